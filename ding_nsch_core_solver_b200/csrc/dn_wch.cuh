// dn_wch.cuh -- the Cahn-Hilliard PCG (solve_preconditioned_cg, ch_sparse_krylov.hpp:515-660) with its 13-point
// ILDLT(0) preconditioner (apply_preconditioner, ch_sparse_krylov.hpp:444-513) swept by many CTAs: the layout and
// the division of labour of dn_wpcg.cuh for the wider stencil.  y is not periodic here (with periodic y the
// 13-point factor is one chain over all rows: apply_seq13).
//
// What bounds it.  A row needs its line's two values before it, the line below up to the next column and the line
// two below at its own column: nx + ny dependent cells a sweep.  In pairs of columns a line may follow the line
// below it two pairs behind, so lane t of a block of 32 lines works on pair c = s - 2t in step s, and the vectors
// lie as [block][step][lane] pairs in that order.
//
// Sweeps.  With D the factor's diagonal, the forward sweep computes y / D directly,
//   w = r / D - sum (L D_col / D) w,     backward  z = w - sum L^T z,
// so that each is a right-hand side and six coefficients per row from a shared ring.  The line below's pair arrives
// by shuffle from the neighbouring lane; a lane keeps the last three it received and passes the oldest on, which is
// the line two below's pair for the next lane.  Coefficients of rows outside the lines are zero.
//
// One block per CTA: warp 0 sweeps, warp 1 (the helper) adds the values of the lines of other blocks -- the two edge
// lines of the block before, with periodic x the two lines across the wrap -- to the right-hand side in the ring and
// clears steps in order, warp 2 (the stager) fills the ring.  The edge lines go through global memory, entries empty
// (NaN sentinel) until their pair arrives and again after their last use.  Entries are numbered in the order in which
// the sweep makes them, so that both sweeps share their code with "first" and "second" column of a pair exchanged.
//
// Measured on B200, one solve: 192 x 384 (4 iterations) 5.8 -> 0.89 ms, 512 x 1024 (17) 207 -> 13.3 ms, against one CTA
// that walked the 2 nx + ny levels with the last eight in a shared ring; 128 x 128 periodic x (4) 15.1 -> 0.56 ms,
// against the same levels on global memory.
//
// The SpMV and update phases run on compact rows as in k_pcg; the update phase stores r / D in sweep order as well,
// and a pass after the sweeps brings z back and takes r.z.
#pragma once

#include "dn_krylov.cuh"
#include "dn_wpcg.cuh"

namespace dn {

constexpr int kCRingGroups = 4;  // groups of kWGroup steps in the shared ring
constexpr int kCRing = kWGroup * kCRingGroups;
constexpr int kCArrays = 7;      // right-hand side and six coefficients
constexpr int kCLag = 2 * (kWLines - 1);

__host__ __device__ inline int c_steps(int ny) { return (w_pairs(ny) + kCLag + kWGroup - 1) / kWGroup * kWGroup; }
__host__ __device__ inline size_t c_vec_pairs(int nx, int ny) { return (size_t)w_blocks(nx) * c_steps(ny) * kWLines; }
// A line of entries: one per step and more in front and behind (the edge lanes write one in every step).
constexpr int kCLinePad = kCLag + 2 * kWGroup;
__host__ __device__ inline int c_line(int ny) { return 2 * kCLinePad + c_steps(ny); }
__host__ __device__ constexpr size_t c_smem() {
  return (size_t)kCArrays * kCRing * kWLines * 16 + 8 * kCRingGroups + 4 * kWCtr;
}
// The wrap's two lines must lie in the last block, and the way round it must be longer than a group.
__host__ __device__ inline bool c_fits(int nx, bool px, bool py) {
  return !py && (!px || (nx > 2 * kWGroup && (nx & (kWLines - 1)) != 1));
}

struct CArgs {
  PcgArgs P;  // operator, vectors on compact rows, stopping rule, record
  int np, S, nblk;
  const double *dinv;      // 1 / D, compact rows
  Pair<double> *v;         // r / D, then w and z, in sweep order
  Pair<double> *f[6], *u[6];  // coefficients in sweep order, forward and backward: own line's last and last but one
                              // value, line below's previous, same and next column, line two below's same column
  Pair<double> *wf[5], *wu[5];  // [np] the wrapped rows' coefficients in entry order: previous, same, next column and
                                // second line of line nx-1 (backward: line 0), first line of line nx-2 (line 1)
  Pair<double> *line[2];   // [nblk][2][c_line] edge lines, forward and backward: next to the edge, one further in
  Pair<double> *wrap[2];   // [2][c_line]
  double *slots;
};

// pair c of line l of block k
__host__ __device__ __forceinline__ size_t c_at(int S, int k, int l, int c) {
  return ((size_t)k * S + c + 2 * l) * kWLines + l;
}

// The coefficients in sweep order, from the factor on compact rows (slots as in Stencil<13>; a slot holds L where its
// column is smaller than the row, and the transposed entry is the mirrored slot of the column's row).
__global__ void k_wch_setup(SpOp A, Factor F, CArgs C) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (size_t)C.nblk * C.S * kWLines) return;
  const int l = (int)(e % kWLines), row = (int)(e / kWLines), k = row / C.S, c = row - k * C.S - 2 * l, i = k * kWLines + l;
  const int n = A.n, ny = A.ny;
  auto coef = [&](int j, int s, bool lower) -> double {  // of slot s in row (i, j): lower (scaled) or upper entry
    const long long r = (long long)i * ny + j, q = slot_col<13>(i, j, s, A.nx, ny, A.px, 0);
    if (q < 0 || (lower ? q >= r : q <= r)) return 0.0;
    if (lower) return F.l[(size_t)s * n + r] * F.d[q] * F.dinv[r];
    return F.l[(size_t)(12 - s) * n + q];
  };
  const bool v0 = i < A.nx && c >= 0 && c < C.np, v1 = v0 && 2 * c + 1 < ny;
  const int fs[6] = {5, 4, 1, 2, 3, 0}, us[6] = {7, 8, 11, 10, 9, 12};
  const int wfs[4] = {9, 10, 11, 12}, wus[4] = {3, 2, 1, 0};
  for (int t = 0; t < 6; ++t) {
    C.f[t][e] = Pair<double>{v0 ? coef(2 * c, fs[t], true) : 0.0, v1 ? coef(2 * c + 1, fs[t], true) : 0.0};
    C.u[t][e] = Pair<double>{v0 ? coef(2 * c, us[t], false) : 0.0, v1 ? coef(2 * c + 1, us[t], false) : 0.0};
  }
  if (!A.px || !v0) return;
  for (int t = 0; t < 4; ++t) {
    if (i == A.nx - 1) C.wf[t][c] = Pair<double>{coef(2 * c, wfs[t], true), v1 ? coef(2 * c + 1, wfs[t], true) : 0.0};
    if (i == 0) C.wu[t][C.np - 1 - c] = Pair<double>{coef(2 * c, wus[t], false), v1 ? coef(2 * c + 1, wus[t], false) : 0.0};
  }
  if (i == A.nx - 2) C.wf[4][c] = Pair<double>{coef(2 * c, 12, true), v1 ? coef(2 * c + 1, 12, true) : 0.0};
  if (i == 1) C.wu[4][C.np - 1 - c] = Pair<double>{coef(2 * c, 0, false), v1 ? coef(2 * c + 1, 0, false) : 0.0};
}

struct CWarp {
  int k;
  unsigned ring, bars, ctr;
};

// First and second column of a pair in sweep direction.
template <bool FWD>
__device__ __forceinline__ double c_first(const Pair<double> &p) { return FWD ? p.x : p.y; }
template <bool FWD>
__device__ __forceinline__ double c_second(const Pair<double> &p) { return FWD ? p.y : p.x; }
template <bool FWD>
__device__ __forceinline__ Pair<double> c_pair(double first, double second) {
  return FWD ? Pair<double>{first, second} : Pair<double>{second, first};
}

// Entry 0 of the lines that a block writes (its edge lines) in sweep direction FWD.
template <bool FWD>
__device__ __forceinline__ Pair<double> *c_edge_line(const CArgs &C, int k, int which) {
  return C.line[FWD ? 0 : 1] + ((size_t)k * 2 + which) * c_line(C.P.A.ny) + kCLinePad;
}
template <bool FWD>
__device__ __forceinline__ Pair<double> *c_wrap_line(const CArgs &C, int which) {
  return C.wrap[FWD ? 0 : 1] + (size_t)which * c_line(C.P.A.ny) + kCLinePad;
}

// The sweep warp's part.
template <bool FWD>
__device__ __forceinline__ bool c_sweep(const CArgs &C, const CWarp &W, long long limit) {
  using P2 = Pair<double>;
  constexpr unsigned E = 16, A = kCRing * kWLines * E, D = kWLines * E;
  const int lane = threadIdx.x & 31, S = C.S, G = S / kWGroup, np = C.np, px = C.P.A.px;
  int *const status = C.P.status;
  const int tl = C.P.A.nx - 1 - kWLines * (C.nblk - 1);
  const bool edge = lane == (FWD ? 0 : 31);  // takes no neighbour from inside the block
  P2 *zg = C.v + (size_t)W.k * S * kWLines + lane + (FWD ? 0 : (size_t)(G - 1) * kWGroup * kWLines);
  // the lanes that hand over: the two lines at the far edge to the next block; lines 0 and 1 (forward), nx-1 and nx-2
  // (backward) across the wrap.  The pair of line l in the n-th step is number n - 2l (forward),
  // n - (S - np) + 2l (backward).
  const int which = FWD ? 31 - lane : lane;
  const bool hand = which >= 0 && which < 2 && (FWD ? W.k + 1 < C.nblk : W.k > 0);
  P2 *to = c_edge_line<FWD>(C, W.k, hand ? which : 0) + (FWD ? -2 * lane : np - S + 2 * lane);
  const int xwhich = FWD ? lane : tl - lane;
  const bool xhand = px && xwhich >= 0 && xwhich < 2 && W.k == (FWD ? 0 : C.nblk - 1);
  P2 *tx = px ? c_wrap_line<FWD>(C, xhand ? xwhich : 0) + (FWD ? -2 * lane : np - S + 2 * lane) : to;
  const unsigned ringE = W.ring + E * lane, ready = W.ctr + (FWD ? kCtrReadyF : kCtrReadyB),
                 done = W.ctr + (FWD ? kCtrDoneF : kCtrDoneB);
  auto from_lane = [&](double v) -> double {
    const double s = FWD ? __shfl_up_sync(0xffffffffu, v, 1) : __shfl_down_sync(0xffffffffu, v, 1);
    return edge ? 0.0 : s;
  };
  // the line below's next, same and previous pair, the line two below's same pair, the own line's last pair; all by
  // first / second
  double n1 = 0.0, n2 = 0.0, m1 = 0.0, m2 = 0.0, o1 = 0.0, o2 = 0.0, t1 = 0.0, t2 = 0.0, l1 = 0.0, l2 = 0.0;
  int seen = 0;
  for (int m = 0; m < G; ++m) {
    if (!wait_ready(ready, (m + 1) * kWGroup, seen, status, limit)) return false;
    __syncwarp();
    const unsigned low = ringE + (unsigned)((FWD ? m * kWGroup : S - (m + 1) * kWGroup) & (kCRing - 1)) * D;
    const bool keep = FWD && m >= G - kCRingGroups;
    P2 v[2][kCArrays];
    auto load = [&](int n) {
      const unsigned at = low + (FWD ? n : kWGroup - 1 - n) * D;
#pragma unroll
      for (int a = 0; a < kCArrays; ++a) lds_pair(at + a * A, v[n & 1][a]);
    };
    load(0);
    P2 o{};
    auto put = [&](int n) {
      const int u = FWD ? n : kWGroup - 1 - n;
      stg_pair(zg + u * kWLines, o);
      if constexpr (FWD) sts_pair_if(low + u * D, o, keep);
      st_pair_if(to + n, o, hand);
      st_pair_if(tx + n, o, xhand);
    };
#pragma unroll
    for (int n = 0; n < kWGroup; ++n) {
      if (n + 1 < kWGroup) load(n + 1);
      if (n == kWGroup - 3) seen = ld_ctr(ready);
      if (n == kWGroup - 1) seen = __shfl_sync(0xffffffffu, seen, 0);
      if (n > 0) put(n - 1);
      const P2(&c)[kCArrays] = v[n & 1];
      // (o2, m1, m2, n1): columns previous .. next of the line below around this pair
      double y1 = c_first<FWD>(c[0]), y2 = c_second<FWD>(c[0]);
      y1 = fma(-c_first<FWD>(c[3]), o2, y1);
      y2 = fma(-c_second<FWD>(c[3]), m1, y2);
      y1 = fma(-c_first<FWD>(c[4]), m1, y1);
      y2 = fma(-c_second<FWD>(c[4]), m2, y2);
      y1 = fma(-c_first<FWD>(c[5]), m2, y1);
      y1 = fma(-c_first<FWD>(c[6]), t1, y1);
      y2 = fma(-c_second<FWD>(c[6]), t2, y2);
      y1 = fma(-c_first<FWD>(c[2]), l1, y1);
      y2 = fma(-c_second<FWD>(c[2]), l2, y2);
      y2 = fma(-c_second<FWD>(c[5]), n1, y2);
      const double x1 = fma(-c_first<FWD>(c[1]), l2, y1);
      const double x2 = fma(-c_second<FWD>(c[1]), x1, y2);
      // for the next step: the oldest pair goes on to the next lane, the new one in behind it
      t1 = from_lane(o1);
      t2 = from_lane(o2);
      o1 = m1;
      o2 = m2;
      m1 = n1;
      m2 = n2;
      n1 = from_lane(x1);
      n2 = from_lane(x2);
      l1 = x1;
      l2 = x2;
      o = c_pair<FWD>(x1, x2);
    }
    put(kWGroup - 1);
    __syncwarp();  // every lane is through with the group; published at the next group's start, as in w_sweep, the ring
                   // of four groups was refilled late (0.635 -> 0.68 ms at 192 x 384)
    if (lane == 0) st_ctr(done, m + 1);
    to += kWGroup;
    tx += kWGroup;
    zg += FWD ? kWGroup * kWLines : -kWGroup * kWLines;
  }
  return true;
}

// The stager's part; see w_stage.
template <bool FWD>
__device__ __forceinline__ bool c_stage(const CArgs &C, const CWarp &W, unsigned &phases, long long limit) {
  constexpr unsigned E = 16, A = kCRing * kWLines * E, kBytes = kWGroup * kWLines * E;
  const int lane = threadIdx.x & 31, S = C.S, G = S / kWGroup;
  int *const status = C.P.status;
  const size_t base = (size_t)W.k * S * kWLines;
  const unsigned done_at = W.ctr + (FWD ? kCtrDoneF : kCtrDoneB), landed_at = W.ctr + (FWD ? kCtrLandedF : kCtrLandedB);
  const int kept = FWD ? 0 : min(G, kCRingGroups);
  int issued = 0, landed = 0;
  long long spins = 0;
  while (landed < G) {
    const int done = warp_ctr(done_at), before = landed;
    while (issued < G && issued < done + kCRingGroups) {
      const int g = FWD ? issued : G - 1 - issued;
      const unsigned slot = (unsigned)(g & (kCRingGroups - 1)), at = W.ring + slot * kBytes + 16 * lane;
      const size_t o = base + (size_t)g * kWGroup * kWLines + lane;
#pragma unroll
      for (int b = 0; b < kWGroup; ++b) {
        if (issued >= kept) cp_async16_at(at + b * 512, C.v + o + b * 32);
#pragma unroll
        for (int a = 0; a < 6; ++a) cp_async16_at(at + b * 512 + (a + 1) * A, (FWD ? C.f[a] : C.u[a]) + o + b * 32);
      }
      mbar_arrive_copies(W.bars + 8 * slot);
      ++issued;
    }
    while (landed < issued) {
      const unsigned slot = (unsigned)((FWD ? landed : G - 1 - landed) & (kCRingGroups - 1));
      if (!__all_sync(0xffffffffu, mbar_done(W.bars + 8 * slot, (phases >> slot) & 1u))) break;
      phases ^= 1u << slot;
      ++landed;
    }
    if (landed > before) {
      if (lane == 0) st_ctr(landed_at, landed);
      spins = 0;
    } else if (give_up(++spins, limit, status)) {
      break;
    }
  }
  for (long long w = 0; landed < issued && w < kSpinLimit; ++w) {  // copies in flight after a wait that gave up
    const unsigned slot = (unsigned)((FWD ? landed : G - 1 - landed) & (kCRingGroups - 1));
    if (!__all_sync(0xffffffffu, mbar_done(W.bars + 8 * slot, (phases >> slot) & 1u))) continue;
    phases ^= 1u << slot;
    ++landed;
  }
  return landed >= G;
}

// The helper's part: in each round its lanes look at the next 32 steps, those from the first on whose rows have landed
// and whose entries have arrived are worked on and cleared together.
template <bool FWD>
__device__ __forceinline__ bool c_help(const CArgs &C, const CWarp &W, long long limit) {
  using P2 = Pair<double>;
  constexpr unsigned E = 16, A = kCRing * kWLines * E;
  const int lane = threadIdx.x & 31, S = C.S, np = C.np;
  int *const status = C.P.status;
  const int tl = C.P.A.nx - 1 - kWLines * (C.nblk - 1);
  const unsigned ready = W.ctr + (FWD ? kCtrReadyF : kCtrReadyB), landed_at = W.ctr + (FWD ? kCtrLandedF : kCtrLandedB);
  const bool has_in = FWD ? W.k > 0 : W.k + 1 < C.nblk;
  const bool wraps = C.P.A.px && W.k == (FWD ? C.nblk - 1 : 0);
  P2 *const e0 = has_in ? c_edge_line<FWD>(C, FWD ? W.k - 1 : W.k + 1, 0) : nullptr;
  P2 *const e1 = has_in ? c_edge_line<FWD>(C, FWD ? W.k - 1 : W.k + 1, 1) : nullptr;
  P2 *const x0 = wraps ? c_wrap_line<FWD>(C, 0) : nullptr, *const x1 = wraps ? c_wrap_line<FWD>(C, 1) : nullptr;
  P2 *const *const wc = FWD ? C.wf : C.wu;
  // number of the pair of the block's first line (in sweep direction), and of the wrapped line, in step n
  const int q_shift = FWD ? 0 : S - np - kCLag, x_shift = FWD ? 2 * tl : S - np;
  const int ln0 = FWD ? 0 : kWLines - 1, ln1 = FWD ? 1 : kWLines - 2, lx0 = FWD ? tl : 0, lx1 = FWD ? tl - 1 : 1;
  int told = 0;
  long long spins = 0;
  auto entry = [&](P2 *line, int q, bool &ok) -> P2 {
    if (q < 0 || q >= np) return P2{0.0, 0.0};
    const P2 v = ld_entry(line + q);
    if (pair_empty(v)) ok = false;
    return v;
  };
  while (told < S) {
    const int n = told + lane, landed = ld_ctr(landed_at);
    const int q = n - q_shift, qx = n - x_shift;
    bool ok = n < S && n < landed * kWGroup;
    P2 a[4], b{}, x[4], y{};
    if (ok && has_in) {
#pragma unroll
      for (int t = 0; t < 4; ++t) a[t] = entry(e0, q - 2 + t, ok);
      b = entry(e1, q, ok);
    }
    if (ok && wraps) {
#pragma unroll
      for (int t = 0; t < 4; ++t) x[t] = entry(x0, qx - 1 + t, ok);
      y = entry(x1, qx, ok);
    }
    const unsigned not_ok = ~__ballot_sync(0xffffffffu, ok);
    const int count = not_ok ? __ffs((int)not_ok) - 1 : 32;  // steps from `told` on that can be cleared
    if (lane < count) {
      const int s = FWD ? n : S - 1 - n;
      const unsigned row = W.ring + (unsigned)(s & (kCRing - 1)) * kWLines * E;
      auto add = [&](int line, double first, double second) {  // into the right-hand side of the line's pair
        P2 r;
        lds_pair(row + line * E, r);
        sts_pair(row + line * E, P2{r.x - (FWD ? first : second), r.y - (FWD ? second : first)});
      };
      auto coef = [&](int line, int t) -> P2 {
        P2 c;
        lds_pair(row + line * E + (t + 1) * A, c);
        return c;
      };
      if (has_in) {
        if (q >= 0 && q < np) {
          const P2 c2 = coef(ln0, 2), c3 = coef(ln0, 3), c4 = coef(ln0, 4), c5 = coef(ln0, 5);
          const double f = c_first<FWD>(c2) * c_second<FWD>(a[1]) + c_first<FWD>(c3) * c_first<FWD>(a[2]) +
                           c_first<FWD>(c4) * c_second<FWD>(a[2]) + c_first<FWD>(c5) * c_first<FWD>(b);
          const double g = c_second<FWD>(c2) * c_first<FWD>(a[2]) + c_second<FWD>(c3) * c_second<FWD>(a[2]) +
                           c_second<FWD>(c4) * c_first<FWD>(a[3]) + c_second<FWD>(c5) * c_second<FWD>(b);
          add(ln0, f, g);
        }
        if (q - 2 >= 0 && q - 2 < np) {
          const P2 c5 = coef(ln1, 5);
          add(ln1, c_first<FWD>(c5) * c_first<FWD>(a[0]), c_second<FWD>(c5) * c_second<FWD>(a[0]));
        }
      }
      if (wraps) {
        if (qx >= 0 && qx < np) {
          const P2 c2 = wc[0][qx], c3 = wc[1][qx], c4 = wc[2][qx], c5 = wc[3][qx];
          const double f = c_first<FWD>(c2) * c_second<FWD>(x[0]) + c_first<FWD>(c3) * c_first<FWD>(x[1]) +
                           c_first<FWD>(c4) * c_second<FWD>(x[1]) + c_first<FWD>(c5) * c_first<FWD>(y);
          const double g = c_second<FWD>(c2) * c_first<FWD>(x[1]) + c_second<FWD>(c3) * c_second<FWD>(x[1]) +
                           c_second<FWD>(c4) * c_first<FWD>(x[2]) + c_second<FWD>(c5) * c_second<FWD>(y);
          add(lx0, f, g);
        }
        if (qx + 2 >= 0 && qx + 2 < np) {
          const P2 c5 = wc[4][qx + 2];
          add(lx1, c_first<FWD>(c5) * c_first<FWD>(x[3]), c_second<FWD>(c5) * c_second<FWD>(x[3]));
        }
      }
    }
    __syncwarp();
    if (lane < count) {  // entries used for the last time
      const P2 none = empty_pair<double>();
      if (has_in && q - 2 >= 0 && q - 2 < np) st_pair_if(e0 + q - 2, none, true);
      if (has_in && q >= 0 && q < np) st_pair_if(e1 + q, none, true);
      if (wraps && qx - 1 >= 0 && qx - 1 < np) st_pair_if(x0 + qx - 1, none, true);
      if (wraps && qx >= 0 && qx < np) st_pair_if(x1 + qx, none, true);
      // the last entry is looked at once more by the step after (which may come in a later round), if there is one
      if (wraps && qx == np - 1 && n == S - 1) st_pair_if(x0 + qx, none, true);
    }
    if (count > 0) {
      told = min(told + count, S);
      if (lane == 0) st_ctr(ready, told);
      spins = 0;
    } else if (give_up(++spins, limit, status)) {
      break;
    }
  }
  return told >= S;
}

__global__ void __launch_bounds__(kBlock, 1) k_wch(CArgs C) {
  using P2 = Pair<double>;
  __shared__ double sh[8 * 32 + 8];
  extern __shared__ __align__(16) char dsm[];
  const PcgArgs &P = C.P;
  const SpOp &A = P.A;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, n = A.n, ny = A.ny, grid = (int)gridDim.x;
  const long long per = (n + gridDim.x - 1) / gridDim.x;
  const long long lo = (long long)blockIdx.x * per, hi = min((long long)n, lo + per);
  const long long limit = spin_limit(P.status);
  const bool in_sweep = (int)blockIdx.x < C.nblk;
  CWarp W{};
  unsigned phases = 0;
  W.k = blockIdx.x;
  W.ring = smem_addr(dsm);
  W.bars = W.ring + (unsigned)((size_t)kCArrays * kCRing * kWLines * 16);
  W.ctr = W.bars + 8 * kCRingGroups;
  if (in_sweep && warp == 2) {
    if (lane < kCRingGroups) mbar_init(W.bars + 8 * lane);
    if (lane < kWCtr) st_ctr(W.ctr + 4 * lane, 0);
  }
  {  // the lines start empty, and v zero outside the lines; the first reduction orders this before any sweep
    const size_t t0 = (size_t)blockIdx.x * kBlock + threadIdx.x, ts = (size_t)gridDim.x * kBlock;
    const size_t nl = (size_t)C.nblk * 2 * c_line(ny), nv = (size_t)C.nblk * C.S * kWLines;
    for (size_t t = t0; t < nl; t += ts) C.line[0][t] = C.line[1][t] = empty_pair<double>();
    if (A.px)
      for (size_t t = t0; t < (size_t)2 * c_line(ny); t += ts) C.wrap[0][t] = C.wrap[1][t] = empty_pair<double>();
    for (size_t t = t0; t < nv; t += ts) {
      const int l = (int)(t % kWLines), row = (int)(t / kWLines), k = row / C.S, c = row - k * C.S - 2 * l;
      if (c < 0 || c >= C.np || k * kWLines + l >= A.nx)
        C.v[t] = P2{0.0, 0.0};
      else if (2 * c + 1 >= ny)
        C.v[t].y = 0.0;
    }
  }
  double *const vs = reinterpret_cast<double *>(C.v);
  auto v_at = [&](long long r) -> size_t {  // of row r, in doubles
    const int i = (int)((unsigned)r / (unsigned)ny), j = (int)((unsigned)r - (unsigned)i * (unsigned)ny);
    return 2 * c_at(C.S, i / kWLines, i % kWLines, j >> 1) + (j & 1);
  };
  int full = 0, app = 0, set, next;
  auto reduce_sets = [](int &count, int base, int &s, int &x) {
    s = base + count % 3;
    x = base + (count + 1) % 3;
    ++count;
  };
  double v2[2] = {0.0, 0.0};
  for (long long r = lo + threadIdx.x; r < hi; r += blockDim.x) {  // r = b - A x0
    const int i = (int)((unsigned)r / (unsigned)ny), j = (int)((unsigned)r - (unsigned)i * (unsigned)ny);
    const double rr = P.b[r] - spmv_row<13>(A, P.x, i, j);
    P.r[r] = rr;
    vs[v_at(r)] = rr * C.dinv[r];
    v2[0] += rr * rr;
    v2[1] += P.b[r] * P.b[r];
  }
  reduce_sets(full, 0, set, next);
  if (!w_reduce<2>(v2, C.slots, set, next, grid, sh, P.status, limit)) return;
  const double rhs_norm = sqrt(max_ref(v2[1], 0.0));
  double absr = sqrt(max_ref(v2[0], 0.0)), relr = absr / max_ref(rhs_norm, 1.0e-30), iter_res = 0.0, rz_old = 0.0;
  if (relr < P.tol || absr < P.tol_abs) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      P.out[0] = 0;
      P.out[1] = absr;
      P.out[2] = relr;
      P.out[3] = 0.0;
    }
    return;
  }
  double *p_old = P.p0, *p_new = P.p1;
  const int max_it = P.max_it > 1 ? P.max_it : 1;
  int iterations = 0;
  for (int it = 0;; ++it) {
    // ---- z = M^-1 r, r.z
    if (in_sweep && warp < 3) {
      bool ok;
      if (warp == 0) {
        ok = c_sweep<true>(C, W, limit);
        __threadfence();  // w, before the stager's copies of it for the backward sweep
        __syncwarp();
        if (lane == 0) st_ctr(W.ctr + kCtrReadyF, -1);  // the ring's last groups hold w now
        if (ok) c_sweep<false>(C, W, limit);
      } else {
        ok = warp == 1 ? c_help<true>(C, W, limit) : c_stage<true>(C, W, phases, limit);
        long long spins = 0;
        while (ok && warp_ctr(W.ctr + kCtrReadyF) != -1) ok = !give_up(++spins, limit, P.status);
        if (ok && warp == 1) c_help<false>(C, W, limit);
        if (ok && warp == 2) c_stage<false>(C, W, phases, limit);
      }
    }
    double none[1] = {0.0};
    reduce_sets(app, 3, set, next);
    if (!w_reduce<1>(none, C.slots, set, next, C.nblk, sh, P.status, limit)) return;
    if (in_sweep && warp == 2 && lane < kWCtr) st_ctr(W.ctr + 4 * lane, 0);
    double rz[1] = {0.0};
    for (long long r = lo + threadIdx.x; r < hi; r += blockDim.x) {
      const double z = __ldcg(vs + v_at(r));
      P.z[r] = z;
      rz[0] += P.r[r] * z;
    }
    reduce_sets(full, 0, set, next);
    if (!w_reduce<1>(rz, C.slots, set, next, grid, sh, P.status, limit)) return;
    if (!isfinite(rz[0]) || rz[0] <= 0.0) {
      if (threadIdx.x == 0) atomicCAS(P.status, kDevOk, it == 0 ? kDevPcgBreakdownRz0 : kDevPcgBreakdownRz);
      return;
    }
    const bool first = it == 0;
    const double beta = first ? 0.0 : rz[0] / rz_old;
    rz_old = rz[0];
    // ---- p = z + beta p, Ap, p.Ap
    double v[3] = {0.0, 0.0, 0.0};
    pcg_spmv_rows<13, double>(P, lo, hi, first, 0.0, beta, p_old, p_new, v);
    reduce_sets(full, 0, set, next);
    if (!w_reduce<3>(v, C.slots, set, next, grid, sh, P.status, limit)) return;
    if (!isfinite(v[1]) || fabs(v[1]) < 1.0e-30) {
      if (threadIdx.x == 0) atomicCAS(P.status, kDevOk, kDevPcgBreakdownPap);
      return;
    }
    // ---- x += alpha p, r -= alpha Ap, norms; r / D in sweep order
    double w[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    pcg_update_rows<double>(P, lo, hi, 0.0, rz[0] / v[1], 0.0, 0.0, p_new, w);
    for (long long r = lo + threadIdx.x; r < hi; r += blockDim.x) vs[v_at(r)] = P.r[r] * C.dinv[r];
    reduce_sets(full, 0, set, next);
    if (!w_reduce<5>(w, C.slots, set, next, grid, sh, P.status, limit)) return;
    iterations = it + 1;
    iter_res = sqrt(w[0] / max_ref(w[1], 1.0e-30));
    absr = sqrt(max_ref(w[4], 0.0));
    relr = absr / max_ref(rhs_norm, 1.0e-30);
    if (relr < P.tol || absr < P.tol_abs || iterations >= max_it) break;
    double *t = p_old;
    p_old = p_new;
    p_new = t;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.out[0] = (double)iterations;
    P.out[1] = absr;
    P.out[2] = relr;
    P.out[3] = iter_res;
    P.out[4] = P.out[5] = P.out[6] = 0.0;
  }
}

}  // namespace dn
