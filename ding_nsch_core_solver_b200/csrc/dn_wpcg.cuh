// dn_wpcg.cuh -- the pressure PCG (solve_preconditioned_cg, ch_sparse_krylov.hpp:515-660) with the ICC(0) /
// ILDLT(0) preconditioner (apply_preconditioner, ch_sparse_krylov.hpp:444-513) as one persistent kernel whose
// vectors live in the order in which the triangular sweeps walk them.
//
// What bounds it.  A triangular solve on the 5-point grid is a dependency chain of nx + ny cells; everything
// else of an iteration is a few microseconds.  The design takes all that is not the chain off the warps that
// walk it.
//
// Layout.  The grid's x-lines are cut into blocks of 32, one sweep warp per block, lane t on line 32k + t.  A
// step of a sweep handles a pair of columns (2c, 2c+1) per lane, lane t one pair behind lane t - 1, so step s
// of block k touches the pairs c = s - t.  Every Krylov vector is stored as [block][step][lane] pairs: a step
// reads and writes 32 contiguous pairs (512 bytes in FP64), there is nothing to transpose, no lane stores to
// its own cache line, and the five-point neighbours of a pair sit at fixed offsets (the same lane one step
// earlier / later, the neighbouring lane one step earlier / later), so the other phases run in this order too.
// The slots outside a line (np + 31 steps for np pairs; lines beyond nx) hold zeros: the recurrence carries exact
// zeros through them and the sweep needs no range checks.
//
// Sweeps.  With q = 1/d^2 (ICC) or 1/D (ILDLT) both factorizations read
//   forward   w = q r - q aS w(j-1) - q aW w(i-1)
//   backward  z = w - q aN z(j+1) - q aE z(i+1).
// q r is stored beside r by the update phase, so that a sweep warp's step is: its inputs from a shared ring (loaded
// a group ahead), one fused multiply-add per cell for the neighbouring line's value (a warp shuffle of the step
// before), one for the own line's, the shuffles, and the store of the result: 27 cycles of shuffle and two FP64
// latencies per pair of columns.  r.z and sum z are taken in a pass of their own over the grid.
//
// Beside each sweep warp run two others, on other schedulers.  The stager fills the ring (asynchronous copies
// counted on mbarriers, eight groups of eight steps).  The helper takes the values that come from outside the block
// -- the previous block's edge line, with periodic x line 0's or nx-1's values, with periodic y the line's own
// other end -- and adds them to the right-hand side in the ring, so that the sweep warp has no special cases; it
// then advances the count of steps that the sweep warp may take.  A lane of the helper works on every 32nd step.
//
// Hand-over.  A block's edge line goes pair by pair into a line of shared memory (same CTA) or of global memory,
// whose entries hold a NaN sentinel until their value arrives and again after the helper has taken it.  Every
// wait is bounded and reports kDevTimeout.
//
// Measured on B200 (per iteration, sweeps forward and backward alone): 192 x 384 split 137 -> 59.5 us, variable
// coefficients 171 -> 64.6 us, 512 x 1024 split 343 -> 152 us, against sweep warps that staged rows through shared
// memory themselves and stored each lane's values to its own line.  A step of a sweep warp costs about 43 ns, of
// which the chain (27 cycles of shuffle, two dependent FP64 operations) is 25 ns; a block boundary costs 32 steps
// and about 1.8 us of hand-over through global memory.
//
// Grid reductions.  Each CTA publishes its partial sums in a slot, every CTA polls all the slots for values (one
// store, one poll: no counter, no second round trip) and adds them in the same order; a slot set is used again
// after two others, by when every CTA has read it.
#pragma once

#include <type_traits>

#include "dn_common.cuh"
#include "dn_krylov.cuh"
#include "dn_wavefront.cuh"

namespace dn {

constexpr int kWBlock = 256;           // threads per CTA
constexpr int kWLines = 32;            // lines per block
constexpr int kWGroup = 8;             // steps per group: staged together, one check of the helper's progress
constexpr int kWRingGroups = 8;        // groups in the shared ring
constexpr int kWRing = kWGroup * kWRingGroups;
constexpr int kWCtr = 8;               // progress counters of a sweep warp: ready, done, landed; forward and backward
constexpr int kWSlot = 8;              // doubles per reduction slot
constexpr int kWSlotSets = 6;          // slot sets per CTA: 3 for the grid-wide sums, 3 for the sweeps' sums
constexpr unsigned long long kSlotEmpty = ~0ull;  // a slot before its value arrives (memset 0xff)

template <typename T>
struct Pair;
template <>
struct __align__(16) Pair<double> {
  double x, y;
};
template <>
struct __align__(8) Pair<float> {
  float x, y;
};

__host__ __device__ inline int w_pairs(int ny) { return (ny + 1) / 2; }
// steps of a block, in whole groups
__host__ __device__ inline int w_steps(int ny) {
  return (w_pairs(ny) + kWLines - 1 + kWGroup - 1) / kWGroup * kWGroup;
}
__host__ __device__ inline int w_blocks(int nx) { return (nx + kWLines - 1) / kWLines; }
// pairs of one vector in sweep order
__host__ __device__ inline size_t w_vec_pairs(int nx, int ny) { return (size_t)w_blocks(nx) * w_steps(ny) * kWLines; }
// A hand-over line: entries for the pairs, between kWLines entries in front and the rest of the steps behind (the
// edge line writes one in every step, zeros where its pair lies outside the line).
__host__ __device__ inline int w_line(int ny) { return kWLines + w_steps(ny); }
// vectors of a block in the ring: right-hand side and q, or (variable operator) right-hand side and the two
// coefficients
__host__ __device__ constexpr int w_ring_arrays(bool var) { return var ? 3 : 2; }
// shared memory of one sweep warp: the ring, the hand-over lines (with periodic x the wrap lines too), one pair per
// line for its ends (periodic y), the mbarriers of the ring's slots and the progress counters
__host__ __device__ inline size_t w_warp_smem(bool var, int ny, int esize, bool px) {
  return ((size_t)w_ring_arrays(var) * kWRing * kWLines + (size_t)(px ? 4 : 2) * w_line(ny)) * 2 * esize +
         (size_t)kWLines * 2 * esize + 8 * kWRingGroups + 4 * kWCtr;
}
// A periodic direction feeds values back into the block that made them (periodic y: a line's first pair into its
// last; periodic x with one block: line 0 into line nx-1), and the helper must have cleared a group and two steps
// before the sweep warp starts it: the way round has to be longer than that.
__host__ __device__ inline bool w_fits(int nx, int ny, bool px, bool py) {
  return (!py || w_pairs(ny) > 2 * kWGroup) && (!px || nx > 2 * kWGroup);
}

template <typename T>
struct WArgs {
  int nx, ny, np, S, nblk;
  int px, py, prec, project, max_it;
  double tol, tol_abs;
  T cx, cy;          // off-diagonals of the constant (split) operator
  T kappa, scale;    // cx / cy; the factor |cy| that the sweeps carry (1 for the variable operator)
  const T *b;        // right-hand side, natural order (row i*ny + j); the iteration starts from x = 0
  T *x_out;          // solution, natural order (not written when the initial residual already stops)
  const T *a5;       // operator slots W,S,C,N,E, natural order
  const T *dinv;     // 1 / max(d, floor), natural order
  // sweep order; v = q r.  Variable operator only: aW and aS of the SpMV, and the sweeps' coefficients q aS, q aW
  // (forward), q aN, q aE (backward).
  Pair<T> *r, *v, *z, *p0, *p1, *x, *ap, *q, *dg, *aw, *as, *ga, *ha, *gn, *he;
  Pair<T> *line_f, *line_b;  // [nblk][w_line] edge lines between CTAs
  Pair<T> *wrap_f, *wrap_b;  // [w_line] periodic-x wrap lines
  double *slots;             // [grid][kWSlotSets][kWSlot]
  int *status;
  double *out;
  double *mon;
  int mon_cap;
  int sw, warp_smem;  // sweep warps per CTA, shared bytes of each
  double *prof;
};

template <typename T>
__device__ __forceinline__ Pair<T> ld_cg(const Pair<T> *p);
template <>
__device__ __forceinline__ Pair<double> ld_cg<double>(const Pair<double> *p) {
  Pair<double> v;
  asm volatile("ld.global.cg.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
  return v;
}
template <>
__device__ __forceinline__ Pair<float> ld_cg<float>(const Pair<float> *p) {
  Pair<float> v;
  asm volatile("ld.global.cg.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
  return v;
}
__device__ __forceinline__ Pair<double> ld_relaxed_pair(const Pair<double> *p) {
  Pair<double> v;
  asm volatile("ld.relaxed.gpu.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ Pair<float> ld_relaxed_pair(const Pair<float> *p) {
  Pair<float> v;
  asm volatile("ld.relaxed.gpu.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}
// Shared memory by its 32-bit address.
__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void lds_pair(unsigned a, Pair<double> &v) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
}
__device__ __forceinline__ void lds_pair(unsigned a, Pair<float> &v) {
  asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
}
__device__ __forceinline__ void sts_pair(unsigned a, const Pair<double> &v) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v.x), "d"(v.y));
}
__device__ __forceinline__ void sts_pair(unsigned a, const Pair<float> &v) {
  asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v.x), "f"(v.y));
}
__device__ __forceinline__ void sts_pair_if(unsigned a, const Pair<double> &v, bool pred) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t@q st.shared.v2.f64 [%0], {%1, %2};\n\t}" ::"r"(a), "d"(v.x),
               "d"(v.y), "r"((int)pred));
}
__device__ __forceinline__ void sts_pair_if(unsigned a, const Pair<float> &v, bool pred) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t@q st.shared.v2.f32 [%0], {%1, %2};\n\t}" ::"r"(a), "f"(v.x),
               "f"(v.y), "r"((int)pred));
}
__device__ __forceinline__ void stg_pair(Pair<double> *p, const Pair<double> &v) {
  asm volatile("st.global.v2.f64 [%0], {%1, %2};" ::"l"(p), "d"(v.x), "d"(v.y));
}
__device__ __forceinline__ void stg_pair(Pair<float> *p, const Pair<float> &v) {
  asm volatile("st.global.v2.f32 [%0], {%1, %2};" ::"l"(p), "f"(v.x), "f"(v.y));
}
// A ring slot's mbarrier: 32 arrivals, one per lane when its copies into the slot have landed.
__device__ __forceinline__ void mbar_init(unsigned bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 32;" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_copies(unsigned bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_done(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile("{\n\t.reg .pred q;\n\tmbarrier.test_wait.parity.shared::cta.b64 q, [%1], %2;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(ok)
               : "r"(bar), "r"(parity)
               : "memory");
  return ok != 0;
}
__device__ __forceinline__ void cp_async16_at(unsigned smem, const void *gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
// The counters: written by one lane after a __syncwarp of its warp, read before the data they stand for.  Shared-memory
// accesses of a CTA's warps are performed in the order of issue; as acquire loads and release stores they would put the
// order in the memory model's terms too, at 3.5% of the sweeps (28.4 -> 29.7 ms at 192 x 384).
__device__ __forceinline__ int ld_ctr(unsigned a) {
  int v;
  asm volatile("ld.volatile.shared.b32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_ctr(unsigned a, int v) {
  asm volatile("st.volatile.shared.b32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}
// Stores under a lane predicate without a branch (the warp stays converged for the next shuffle); the generic
// form reaches a shared line of this CTA or a global one.
__device__ __forceinline__ void st_pair_if(Pair<double> *p, Pair<double> v, bool pred) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t@q st.relaxed.gpu.v2.f64 [%0], {%1, %2};\n\t}" ::"l"(p),
               "d"(v.x), "d"(v.y), "r"((int)pred)
               : "memory");
}
__device__ __forceinline__ void st_pair_if(Pair<float> *p, Pair<float> v, bool pred) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %3, 0;\n\t@q st.relaxed.gpu.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p),
               "f"(v.x), "f"(v.y), "r"((int)pred)
               : "memory");
}
// The sentinel is a signalling NaN, which no arithmetic returns, so its high word alone tells it.
__device__ __forceinline__ bool pair_empty(const Pair<double> &v) {
  constexpr int hi = (int)(kHandEmpty >> 32);
  return __double2hiint(v.x) == hi || __double2hiint(v.y) == hi;
}
__device__ __forceinline__ bool pair_empty(const Pair<float> &v) { return hand_empty(v.x) || hand_empty(v.y); }
template <typename T>
__device__ __forceinline__ Pair<T> empty_pair() {
  return Pair<T>{hand_empty_value<T>(), hand_empty_value<T>()};
}

// A hand-over line's entry, shared or global.
__device__ __forceinline__ Pair<double> ld_entry(const Pair<double> *p) {
  Pair<double> v;
  asm volatile("ld.relaxed.gpu.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ Pair<float> ld_entry(const Pair<float> *p) {
  Pair<float> v;
  asm volatile("ld.relaxed.gpu.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p) : "memory");
  return v;
}

// A sweep warp and its helper: their block, ring and lines, and where the block's edge values go.
template <typename T>
struct WWarp {
  int k;
  unsigned ring, ends, bars, ctr;  // [arrays][kWRing][kWLines], line ends [kWLines], mbarriers, counters (shared)
  bool far_f, far_b;               // whether in_f / in_b lie in global memory
  Pair<T> *in_f, *in_b, *in_xf, *in_xb;  // lines read (forward, backward, wrap forward, wrap backward): entry of
                                         // pair 0; null: none
  Pair<T> *to_f, *to_b, *to_xf, *to_xb;  // lines written: entry of step 0; null: none
};
enum { kCtrReadyF = 0, kCtrDoneF = 4, kCtrReadyB = 8, kCtrDoneB = 12, kCtrLandedF = 16, kCtrLandedB = 20 };  // bytes

// One step's inputs of a sweep warp: the right-hand side, and q (constant operator) or the coefficients of the own
// line's and of the neighbouring line's value.
template <typename T, bool VAR>
struct WStep {
  Pair<T> r, a, b;
};
template <typename T, bool VAR>
__device__ __forceinline__ void load_step(unsigned at, WStep<T, VAR> &v) {
  constexpr unsigned E = sizeof(Pair<T>), A = kWRing * kWLines * E;
  lds_pair(at, v.r);
  lds_pair(at + A, v.a);
  if constexpr (VAR) lds_pair(at + 2 * A, v.b);
}
// A counter's value, the same in every lane.
__device__ __forceinline__ int warp_ctr(unsigned a) { return __shfl_sync(0xffffffffu, ld_ctr(a), 0); }
// Whether a wait after `spins` polls without progress must give up; the same answer in every lane.
__device__ __forceinline__ bool give_up(long long spins, long long limit, int *status) {
  bool up = spins > limit;
  if (!up && (spins & 1023) == 0) up = __shfl_sync(0xffffffffu, *(volatile int *)status, 0) != kDevOk;
  if (up && (threadIdx.x & 31) == 0) atomicCAS(status, kDevOk, kDevTimeout);
  return up;
}
// Waits (bounded) until the helper has cleared `need` steps; `seen` is the count read last.
__device__ __forceinline__ bool wait_ready(unsigned ctr, int need, int &seen, int *status, long long limit) {
  long long spins = 0;
  while (seen < need) {
    seen = warp_ctr(ctr);
    if (seen < need && give_up(++spins, limit, status)) return false;
  }
  return true;
}

// One sweep of a block by its sweep warp: forward (FWD) r -> w, or backward w -> z, both in P.z; KEEP stores the
// results of the groups the other end needs into the ring too (the backward sweep starts from the ring, periodic
// y reads line ends there).  Constant operator: everything is scaled by |aS| (q, w and z by it, the couplings to
// kappa = aW / aS and 1), which the iteration does not see: a constant factor of the preconditioner cancels.
template <typename T, bool VAR, bool FWD, bool PX, bool PY>
__device__ __forceinline__ bool w_sweep(const WArgs<T> &P, const WWarp<T> &W, long long limit) {
  using P2 = Pair<T>;
  constexpr unsigned E = sizeof(P2);
  const int lane = threadIdx.x & 31, S = P.S, G = S / kWGroup;
  const int tl = P.nx - 1 - kWLines * (P.nblk - 1);
  // the lane that takes its neighbour from outside the block takes none here (the helper added it)
  const T kap = lane == (FWD ? 0 : 31) ? T(0) : P.kappa;
  P2 *zg = P.z + (size_t)W.k * S * kWLines + lane + (FWD ? 0 : (size_t)(G - 1) * kWGroup * kWLines);
  P2 *const to = FWD ? W.to_f : W.to_b, *const tx = FWD ? W.to_xf : W.to_xb;
  const bool hand = to != nullptr && lane == (FWD ? 31 : 0);
  const bool xhand = PX && tx != nullptr && lane == (FWD ? 0 : tl);
  P2 *tof = to + (FWD ? 0 : (size_t)(G - 1) * kWGroup), *tox = tx + (FWD ? 0 : (size_t)(G - 1) * kWGroup);
  const unsigned ringE = W.ring + E * lane, ready = W.ctr + (FWD ? kCtrReadyF : kCtrReadyB),
                 done = W.ctr + (FWD ? kCtrDoneF : kCtrDoneB);
  T sa = T(0), sb = T(0), own = T(0);  // the neighbouring lane's last pair, the line's own last value
  int seen = 0;
  WStep<T, VAR> v[4];  // the steps' inputs, loaded kPre steps ahead
  constexpr int kPre = 2;
  if (!wait_ready(ready, kPre, seen, P.status, limit)) return false;
  auto ring_step = [&](int n) -> unsigned {  // n-th step in sweep direction
    return ringE + (unsigned)((FWD ? n : S - 1 - n) & (kWRing - 1)) * kWLines * E;
  };
#pragma unroll
  for (int n = 0; n < kPre; ++n) load_step<T, VAR>(ring_step(n), v[n]);
  // group number m in sweep direction
  auto group = [&](int m, auto keep_t) -> bool {
    constexpr bool KEEP = decltype(keep_t)::value;
    if (!wait_ready(ready, min((m + 1) * kWGroup + kPre, S), seen, P.status, limit)) return false;
    __syncwarp();
    // the groups before this one: their inputs are in registers, their results stored, by every lane
    if (!PY && lane == 0) st_ctr(done, m);
    const unsigned here = ring_step(FWD ? m * kWGroup : m * kWGroup + kWGroup - 1);  // the group's lowest step
    const unsigned next = ring_step((m + 1) * kWGroup);
    P2 o{};
    auto put = [&](int u) {  // a finished step's values
      stg_pair(zg + u * kWLines, o);
      st_pair_if(tof + u, o, hand);
      if constexpr (PX) st_pair_if(tox + u, o, xhand);
      if constexpr (KEEP) sts_pair(here + u * kWLines * E, o);
      if constexpr (PY) {  // the line's first pair (forward) / last pair (backward), for the helper
        const int s = (FWD ? m : G - 1 - m) * kWGroup + u;
        sts_pair_if(W.ends + lane * E, o, s - lane == (FWD ? 0 : P.np - 1));
      }
    };
#pragma unroll
    for (int n = 0; n < kWGroup; ++n) {
      const int u = FWD ? n : kWGroup - 1 - n, before = FWD ? u - 1 : u + 1;
      constexpr int D = kWLines * (int)E;
      load_step<T, VAR>(n + kPre < kWGroup ? here + (FWD ? u + kPre : u - kPre) * D
                                           : next + (FWD ? n + kPre - kWGroup : kWGroup - n - kPre) * D,
                        v[(n + kPre) & 3]);
      if (n == kWGroup - 4) seen = ld_ctr(ready);  // for the next group's check
      if (n == kWGroup - 1) seen = __shfl_sync(0xffffffffu, seen, 0);
      if (n > 0) put(before);
      const WStep<T, VAR> &c = v[n & 3];
      T x0, x1;
      if constexpr (VAR) {
        x0 = fma(-c.b.x, sa, c.r.x);
        x1 = fma(-c.b.y, sb, c.r.y);
        if constexpr (FWD) {
          x0 = fma(-c.a.x, own, x0);
          sa = __shfl_up_sync(0xffffffffu, x0, 1);
          x1 = fma(-c.a.y, x0, x1);
          sb = __shfl_up_sync(0xffffffffu, x1, 1);
        } else {
          x1 = fma(-c.a.y, own, x1);
          sb = __shfl_down_sync(0xffffffffu, x1, 1);
          x0 = fma(-c.a.x, x1, x0);
          sa = __shfl_down_sync(0xffffffffu, x0, 1);
        }
      } else {
        x0 = fma(c.a.x * kap, sa, c.r.x);
        x1 = fma(c.a.y * kap, sb, c.r.y);
        if constexpr (FWD) {
          x0 = fma(c.a.x, own, x0);
          sa = __shfl_up_sync(0xffffffffu, x0, 1);
          x1 = fma(c.a.y, x0, x1);
          sb = __shfl_up_sync(0xffffffffu, x1, 1);
        } else {
          x1 = fma(c.a.y, own, x1);
          sb = __shfl_down_sync(0xffffffffu, x1, 1);
          x0 = fma(c.a.x, x1, x0);
          sa = __shfl_down_sync(0xffffffffu, x0, 1);
        }
      }
      o = P2{x0, x1};
      own = FWD ? x1 : x0;
    }
    put(FWD ? kWGroup - 1 : 0);
    if constexpr (PY) {  // at once: the helper clears the steps that take a line's other end (w_fits) after this
      __syncwarp();
      if (lane == 0) st_ctr(done, m + 1);
    }
    tof += FWD ? kWGroup : -kWGroup;
    tox += FWD ? kWGroup : -kWGroup;
    zg += FWD ? kWGroup * kWLines : -kWGroup * kWLines;
    return true;
  };
  // the last groups' results stay in the ring in the forward sweep: the backward one starts from them
  const int plain = FWD ? max(0, G - kWRingGroups) : G;
  int m = 0;
  for (; m < plain; ++m)
    if (!group(m, std::false_type{})) return false;
  if constexpr (FWD)
    for (; m < G; ++m)
      if (!group(m, std::true_type{})) return false;
  return true;
}

// The stager's part of a sweep: fills the ring and counts the groups that have landed; `phases` holds the parity
// that each slot's mbarrier completes next.
template <typename T, bool VAR, bool FWD>
__device__ __forceinline__ bool w_stage(const WArgs<T> &P, const WWarp<T> &W, unsigned &phases, long long limit) {
  using P2 = Pair<T>;
  constexpr unsigned E = sizeof(P2), A = kWRing * kWLines * E, kBytes = kWGroup * kWLines * E;
  const int lane = threadIdx.x & 31, S = P.S, G = S / kWGroup;
  const size_t base = (size_t)W.k * S * kWLines;
  const unsigned done_at = W.ctr + (FWD ? kCtrDoneF : kCtrDoneB), landed_at = W.ctr + (FWD ? kCtrLandedF : kCtrLandedB);
  const char *const src_r = (const char *)((FWD ? P.v : P.z) + base) + 16 * lane;
  const char *const src_a = (const char *)((VAR ? (FWD ? P.ga : P.gn) : P.q) + base) + 16 * lane;
  const char *const src_b = VAR ? (const char *)((FWD ? P.ha : P.he) + base) + 16 * lane : nullptr;
  // groups in sweep direction; the backward sweep finds w of its first groups in the ring, and q if that is all it needs
  const int kept = FWD ? 0 : min(G, kWRingGroups);
  int issued = VAR ? 0 : kept, landed = issued;
  if (lane == 0) st_ctr(landed_at, landed);
  long long spins = 0;
  while (landed < G) {
    const int done = warp_ctr(done_at), before = landed;  // groups the sweep warp is through with
    while (issued < G && issued < done + kWRingGroups) {
      const int g = FWD ? issued : G - 1 - issued;
      const unsigned slot = (unsigned)(g & (kWRingGroups - 1)), at = W.ring + slot * kBytes + 16 * lane;
      const size_t o = (size_t)g * kBytes;
#pragma unroll
      for (unsigned b = 0; b < kBytes; b += 512) {
        if (!VAR || issued >= kept) cp_async16_at(at + b, src_r + o + b);
        cp_async16_at(at + b + A, src_a + o + b);
        if constexpr (VAR) cp_async16_at(at + b + 2 * A, src_b + o + b);
      }
      mbar_arrive_copies(W.bars + 8 * slot);
      ++issued;
    }
    while (landed < issued) {
      const unsigned slot = (unsigned)((FWD ? landed : G - 1 - landed) & (kWRingGroups - 1));
      if (!__all_sync(0xffffffffu, mbar_done(W.bars + 8 * slot, (phases >> slot) & 1u))) break;
      phases ^= 1u << slot;
      ++landed;
    }
    if (landed > before) {
      if (lane == 0) st_ctr(landed_at, landed);
      spins = 0;
    } else if (give_up(++spins, limit, P.status)) {
      break;
    }
  }
  for (long long w = 0; landed < issued && w < kSpinLimit; ++w) {  // copies in flight after a wait that gave up
    const unsigned slot = (unsigned)((FWD ? landed : G - 1 - landed) & (kWRingGroups - 1));
    if (!__all_sync(0xffffffffu, mbar_done(W.bars + 8 * slot, (phases >> slot) & 1u))) continue;
    phases ^= 1u << slot;
    ++landed;
  }
  return landed >= G;
}

// The helper's part of a sweep: adds the values from outside the block to the landed steps and clears them for the
// sweep warp; see the top.  Lane l works on the steps l, l + 32, ... of the sweep.
template <typename T, bool VAR, bool FWD, bool PX, bool PY>
__device__ __forceinline__ bool w_help(const WArgs<T> &P, const WWarp<T> &W, long long limit) {
  using P2 = Pair<T>;
  constexpr unsigned E = sizeof(P2), A = kWRing * kWLines * E;
  const int lane = threadIdx.x & 31, S = P.S, G = S / kWGroup, np = P.np;
  const int tl = P.nx - 1 - kWLines * (P.nblk - 1);
  const size_t base = (size_t)W.k * S * kWLines;
  const unsigned ready = W.ctr + (FWD ? kCtrReadyF : kCtrReadyB), done_at = W.ctr + (FWD ? kCtrDoneF : kCtrDoneB),
                 landed_at = W.ctr + (FWD ? kCtrLandedF : kCtrLandedB);
  // line that takes the previous block's values, and its entries; the wrapped line and its entries
  constexpr int kInLine = FWD ? 0 : kWLines - 1;
  P2 *const lin = FWD ? W.in_f : W.in_b, *const xin = FWD ? W.in_xf : W.in_xb;
  const bool far = FWD ? W.far_f : W.far_b;  // the entries lie in global memory
  const int xline = FWD ? tl : 0;
  const int el = (P.ny - 1) & 1;
  // periodic y: the coefficient of this lane's line's other end (forward: row ny-1 takes w(0); backward: row 0
  // takes z(ny-1)), and that value once the sweep warp has stored it
  T ecoef = T(0), eval = T(0);
  bool have = !PY;
  const int est = FWD ? lane : np - 1 + lane;  // step whose pair holds the value
  if constexpr (PY) {
    const size_t at = base + (size_t)(FWD ? np - 1 + lane : lane) * kWLines + lane;
    const P2 c = VAR ? (FWD ? P.gn[at] : P.ga[at]) : P.q[at];
    ecoef = (FWD && el) ? c.y : c.x;
    if constexpr (VAR) ecoef = -ecoef;
  }
  int n = lane, told = 0, landed = 0;  // this lane's step in sweep direction; steps cleared; groups landed
  // polls of a far line's entry: two in flight, so that a value is seen half a round trip earlier
  P2 h0{}, h1{};
  int c0 = -1, c1 = -1;
  long long spins = 0;
  while (told < S) {
    if (n >= landed * kWGroup && n < S) landed = ld_ctr(landed_at);
    const int s = FWD ? n : S - 1 - n;
    bool ok = n < S && n < landed * kWGroup;
    // entries this step waits for
    const int c = s - kInLine, cx = s - xline;
    const bool nin = n < S && lin != nullptr && c >= 0 && c < np;
    const bool nx_ = PX && ok && xin != nullptr && cx >= 0 && cx < np;
    P2 hv{T(0), T(0)}, xv{T(0), T(0)};
    if (nin) {
      if (far) {
        hv = h0;
        if (c0 != c || pair_empty(hv)) ok = false;
        h0 = h1;
        c0 = c1;
        h1 = ld_entry(lin + c);
        c1 = c;
      } else {
        hv = ld_entry(lin + c);
        if (pair_empty(hv)) ok = false;
      }
    }
    if constexpr (PX) {
      if (nx_) {
        xv = ld_entry(xin + cx);
        if (pair_empty(xv)) ok = false;
      }
    }
    int eline = -1;
    T ev = T(0), ec = T(0);
    if constexpr (PY) {
      if (!have) {
        const int m = FWD ? est / kWGroup : G - 1 - est / kWGroup;
        if (ld_ctr(done_at) > m) {
          P2 v;
          lds_pair(W.ends + lane * (unsigned)sizeof(T) * 2, v);
          eval = (!FWD && el) ? v.y : v.x;
          have = true;
        }
      }
      eline = FWD ? s - (np - 1) : s;  // the line whose end this step reaches
      const bool mine = ok && eline >= 0 && eline < kWLines;
      const int from = mine ? eline : 0;
      ev = __shfl_sync(0xffffffffu, eval, from);
      ec = __shfl_sync(0xffffffffu, ecoef, from);
      const bool got = __shfl_sync(0xffffffffu, (int)have, from) != 0;
      if (mine && !got) ok = false;
      if (!mine) eline = -1;
    }
    if (ok) {
      const unsigned row = W.ring + (unsigned)(s & (kWRing - 1)) * kWLines * E;
      const unsigned at = row + kInLine * E;
      if (VAR || nin) {
        P2 r, a;
        lds_pair(at, r);
        lds_pair(at + (VAR ? 2 * A : A), a);
        if constexpr (VAR) {
          r = P2{fma(-a.x, hv.x, r.x), fma(-a.y, hv.y, r.y)};
          sts_pair(at + 2 * A, P2{T(0), T(0)});  // the sweep warp's own shuffle has no value for this lane
        } else {
          r = P2{fma(a.x * P.kappa, hv.x, r.x), fma(a.y * P.kappa, hv.y, r.y)};
        }
        sts_pair(at, r);
        if (nin) st_pair_if(lin + c, empty_pair<T>(), true);
      }
      if constexpr (PX) {
        if (nx_) {
          const unsigned xat = row + xline * E;
          P2 r, a;
          lds_pair(xat, r);
          if constexpr (VAR) {  // q aE of line nx-1 (forward), q aW of line 0 (backward)
            a = (FWD ? P.he : P.ha)[base + (size_t)s * kWLines + xline];
            r = P2{fma(-a.x, xv.x, r.x), fma(-a.y, xv.y, r.y)};
          } else {
            lds_pair(xat + A, a);
            r = P2{fma(a.x * P.kappa, xv.x, r.x), fma(a.y * P.kappa, xv.y, r.y)};
          }
          sts_pair(xat, r);
          st_pair_if(xin + cx, empty_pair<T>(), true);
        }
      }
      if constexpr (PY) {
        if (eline >= 0) {
          const unsigned eat = row + eline * E;
          P2 r;
          lds_pair(eat, r);
          if (FWD && el)
            r.y = fma(ec, ev, r.y);
          else
            r.x = fma(ec, ev, r.x);
          sts_pair(eat, r);
        }
      }
      n += 32;
    }
    __syncwarp();
    const int clear = min(__reduce_min_sync(0xffffffffu, n), S);  // every step below has been cleared
    if (clear > told) {
      told = clear;
      if (lane == 0) st_ctr(ready, told);
      spins = 0;
    } else if (give_up(++spins, limit, P.status)) {
      break;
    }
  }
  return told >= S;
}

// A sum as a slot holds it: a NaN that carries the empty slot's bits (a state filled with 0xff has it) as another NaN,
// so that the solve breaks down on it, as on any NaN, and does not wait for a value that has come.
__device__ __forceinline__ double slot_value(double v) { return isnan(v) ? __longlong_as_double(0x7ff8000000000000ll) : v; }

// Sum of K values over the CTA, then over the grid: see the reductions' note at the top.  Every CTA of
// [0, writers) publishes its sums in its slot of set `set`, empties set `next` (read two reductions ago), and
// every CTA adds all slots in the same order.  False when a wait gave up (on every thread of the CTA).
template <int K>
__device__ __forceinline__ bool w_reduce(double (&v)[K], double *slots, int set, int next, int writers, double *sh,
                                         int *status, long long limit) {
  static_assert(K <= kWSlot, "values per slot");
  constexpr int KP = (K + 1) / 2;
  const int tid = threadIdx.x;
  if ((int)blockIdx.x < writers) {
    block_sum<K>(v, sh);
    if (tid == 0) {
      double *mine = slots + (size_t)blockIdx.x * kWSlotSets * kWSlot;
      const double empty = __longlong_as_double((long long)kSlotEmpty);
#pragma unroll
      for (int k = 0; k < kWSlot; k += 2) st_pair_if((Pair<double> *)(mine + next * kWSlot + k), Pair<double>{empty, empty}, true);
      __threadfence();
#pragma unroll
      for (int k = 0; k < KP; ++k)
        st_pair_if((Pair<double> *)(mine + set * kWSlot + 2 * k),
                   Pair<double>{slot_value(v[2 * k]), 2 * k + 1 < K ? slot_value(v[2 * k + 1]) : 0.0}, true);
    }
  }
  double u[K];
#pragma unroll
  for (int k = 0; k < K; ++k) u[k] = 0.0;
  bool ok = true;
  for (int b = tid; b < writers; b += blockDim.x) {
    const double *s = slots + (size_t)b * kWSlotSets * kWSlot + set * kWSlot;
    Pair<double> t[KP];
    long long spins = 0;
    bool miss = true;
    while (miss) {
      miss = false;
#pragma unroll
      for (int k = 0; k < KP; ++k) {
        t[k] = ld_relaxed_pair((const Pair<double> *)(s + 2 * k));
        miss |= (unsigned long long)__double_as_longlong(t[k].x) == kSlotEmpty ||
                (unsigned long long)__double_as_longlong(t[k].y) == kSlotEmpty;
      }
      if (!miss) break;
      ++spins;
      if (spins > limit || ((spins & 1023) == 0 && *(volatile int *)status != kDevOk)) {
        atomicCAS(status, kDevOk, kDevTimeout);
        ok = false;
        break;
      }
    }
    if (!ok) break;
#pragma unroll
    for (int k = 0; k < K; ++k) u[k] += (k & 1) ? t[k >> 1].y : t[k >> 1].x;
  }
  __threadfence();
  if (__syncthreads_or(!ok)) return false;
  block_sum<K>(u, sh);
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = u[k];
  return true;
}

// A row of the sweep order: the 32 pairs of one step, one per lane of the warp that works on it.
struct WRow {
  int k, s, l, c, i;  // block, step, line in the block, pair, grid line
  bool v0, v1;        // the pair's first / second column lies in the grid
  size_t e;           // this lane's pair
};
template <typename T>
__device__ __forceinline__ int w_rows(const WArgs<T> &P) { return P.nblk * P.S; }
template <typename T>
__device__ __forceinline__ WRow w_row(const WArgs<T> &P, int row) {
  WRow R;
  R.k = row / P.S;
  R.s = row - R.k * P.S;
  R.l = threadIdx.x & 31;
  R.c = R.s - R.l;
  R.i = kWLines * R.k + R.l;
  R.v0 = R.i < P.nx && R.c >= 0 && R.c < P.np;
  R.v1 = R.v0 && 2 * R.c + 1 < P.ny;
  R.e = (size_t)row * kWLines + R.l;
  return R;
}
// pair c of line l of block k
template <typename T>
__device__ __forceinline__ size_t w_at(const WArgs<T> &P, int k, int l, int c) {
  return ((size_t)k * P.S + c + l) * kWLines + l;
}

// One row of the SpMV phase: p = z - m_z + beta p_old here and at the neighbours, Ap, and the sums (sum p, p.Ap,
// sum Ap).  The rows one step earlier and later hold the S and N neighbours in this lane and the W and E ones in
// the neighbouring lanes; only the block's edge lanes and the periodic wraps load their own.
template <typename T, bool VAR>
__device__ __forceinline__ void w_spmv_row(const WArgs<T> &P, int row, bool first, T m_z, T beta, const Pair<T> *p_old,
                                           Pair<T> *p_new, double (&v)[3]) {
  using P2 = Pair<T>;
  const WRow R = w_row(P, row);
  const int lane = threadIdx.x & 31, S = P.S, np = P.np, nx = P.nx, ny = P.ny;
  auto pval = [&](size_t e) -> P2 {
    const P2 zc = ld_cg(P.z + e);
    P2 o{zc.x - m_z, zc.y - m_z};
    if (!first) {
      const P2 pc = ld_cg(p_old + e);
      o.x += beta * pc.x;
      o.y += beta * pc.y;
    }
    return o;
  };
  const P2 zero{T(0), T(0)};
  const bool lo = R.s > 0, hi = R.s + 1 < S;
  const P2 pc = pval(R.e);
  const P2 ps = lo ? pval(R.e - kWLines) : zero;
  const P2 pn = hi ? pval(R.e + kWLines) : zero;
  const P2 dg = P.dg[R.e];
  P2 aw, as, awn, asn;  // variable operator: own W, S coefficients and those one step later
  if (VAR) {
    aw = P.aw[R.e];
    as = P.as[R.e];
    awn = hi ? P.aw[R.e + kWLines] : zero;
    asn = hi ? P.as[R.e + kWLines] : zero;
  }
  P2 pw{__shfl_up_sync(0xffffffffu, ps.x, 1), __shfl_up_sync(0xffffffffu, ps.y, 1)};
  P2 pe{__shfl_down_sync(0xffffffffu, pn.x, 1), __shfl_down_sync(0xffffffffu, pn.y, 1)};
  P2 ae = zero;
  if (VAR) ae = P2{__shfl_down_sync(0xffffffffu, awn.x, 1), __shfl_down_sync(0xffffffffu, awn.y, 1)};
  if (R.v0) {
    const int tl = nx - 1 - kWLines * (P.nblk - 1);
    if (R.l == 0) {  // line i-1 belongs to the block before (or, periodic, to the last one)
      pw = R.k > 0 ? pval(w_at(P, R.k - 1, kWLines - 1, R.c)) : P.px ? pval(w_at(P, P.nblk - 1, tl, R.c)) : zero;
    }
    if (R.i == nx - 1) {  // line i+1: line 0 when periodic
      const size_t e = w_at(P, 0, 0, R.c);
      pe = P.px ? pval(e) : zero;
      if (VAR) ae = P.px ? P.aw[e] : zero;
    } else if (lane == 31) {
      const size_t e = w_at(P, R.k + 1, 0, R.c);
      pe = pval(e);
      if (VAR) ae = P.aw[e];
    }
    T s0 = ps.y, n1 = pn.x;  // S of the first column, N of the second (or of a last, unpaired column)
    T asn1 = VAR ? asn.x : T(0);
    const bool end = R.c == np - 1;
    if (P.py && R.c == 0) {
      const P2 t = pval(w_at(P, R.k, R.l, np - 1));
      s0 = ((ny - 1) & 1) ? t.y : t.x;
    }
    if (P.py && end) {
      const size_t e = w_at(P, R.k, R.l, 0);
      n1 = pval(e).x;
      if (VAR) asn1 = P.as[e].x;
    }
    T w0, w1, e0, e1, sc0, sc1, nc0, nc1;
    if (VAR) {
      w0 = aw.x;
      w1 = aw.y;
      e0 = ae.x;
      e1 = ae.y;
      sc0 = as.x;
      sc1 = as.y;
      nc0 = R.v1 ? as.y : asn1;
      nc1 = (!end || P.py) ? asn1 : T(0);
      if (!R.v1 && !P.py) nc0 = T(0);
    } else {
      w0 = w1 = (R.i > 0 || P.px) ? P.cx : T(0);
      e0 = e1 = (R.i < nx - 1 || P.px) ? P.cx : T(0);
      sc0 = (R.c > 0 || P.py) ? P.cy : T(0);
      sc1 = P.cy;
      nc0 = (R.v1 || P.py) ? P.cy : T(0);
      nc1 = (!end || P.py) ? P.cy : T(0);
    }
    const T n0 = R.v1 ? pc.y : n1;
    // in the reference's order and, like it, unfused
    const T a0 = w0 * pw.x + sc0 * s0 + dg.x * pc.x + nc0 * n0 + e0 * pe.x;
    const T a1 = R.v1 ? w1 * pw.y + sc1 * pc.x + dg.y * pc.y + nc1 * n1 + e1 * pe.y : T(0);
    const T p1 = R.v1 ? pc.y : T(0);
    p_new[R.e] = P2{pc.x, p1};
    P.ap[R.e] = P2{a0, a1};
    v[0] += (double)pc.x + (double)p1;
    v[1] += (double)pc.x * (double)a0 + (double)p1 * (double)a1;
    v[2] += (double)a0 + (double)a1;
  } else {
    p_new[R.e] = zero;
  }
}

// One row of the update phase: p -= m_p, x += alpha p, r -= alpha Ap, and the sums for the norms and means.
template <typename T>
__device__ __forceinline__ void w_update_row(const WArgs<T> &P, int row, T m_p, T alpha, T m_x, T m_r, Pair<T> *p_new,
                                             double (&w)[5]) {
  using P2 = Pair<T>;
  const WRow R = w_row(P, row);
  if (!R.v0) return;
  const P2 po = p_new[R.e], ao = P.ap[R.e], xo = P.x[R.e], ro = P.r[R.e];
  const P2 pp{po.x - m_p, R.v1 ? po.y - m_p : T(0)};
  const P2 dl{alpha * pp.x, alpha * pp.y};
  const P2 xx{(xo.x - m_x) + dl.x, R.v1 ? (xo.y - m_x) + dl.y : T(0)};
  const P2 rr{(ro.x - m_r) - alpha * ao.x, R.v1 ? (ro.y - m_r) - alpha * ao.y : T(0)};
  const P2 q = P.q[R.e];
  p_new[R.e] = pp;
  P.x[R.e] = xx;
  P.r[R.e] = rr;
  P.v[R.e] = P2{q.x * rr.x, q.y * rr.y};
  w[0] += (double)dl.x * (double)dl.x + (double)dl.y * (double)dl.y;
  w[1] += (double)xx.x * (double)xx.x + (double)xx.y * (double)xx.y;
  w[2] += (double)xx.x + (double)xx.y;
  w[3] += (double)rr.x + (double)rr.y;
  w[4] += (double)rr.x * (double)rr.x + (double)rr.y * (double)rr.y;
}

// The two vector phases over this warp's rows.
template <typename T, bool VAR>
__device__ __forceinline__ void w_spmv(const WArgs<T> &P, bool first, T m_z, T beta, const Pair<T> *p_old, Pair<T> *p_new,
                                    double (&v)[3]) {
  const int nw = kWBlock / 32, nrows = w_rows(P);
  double a[3] = {0.0, 0.0, 0.0};
  for (int row = blockIdx.x * nw + (threadIdx.x >> 5); row < nrows; row += gridDim.x * nw)
    w_spmv_row<T, VAR>(P, row, first, m_z, beta, p_old, p_new, a);
  v[0] = a[0];
  v[1] = a[1];
  v[2] = a[2];
}
template <typename T>
__device__ __forceinline__ void w_update(const WArgs<T> &P, T m_p, T alpha, T m_x, T m_r, Pair<T> *p_new, double (&w)[5]) {
  const int nw = kWBlock / 32, nrows = w_rows(P);
  double a[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
  for (int row = blockIdx.x * nw + (threadIdx.x >> 5); row < nrows; row += gridDim.x * nw)
    w_update_row<T>(P, row, m_p, alpha, m_x, m_r, p_new, a);
#pragma unroll
  for (int k = 0; k < 5; ++k) w[k] = a[k];
}

// The whole solve.  Same iteration, stopping rule, mean projections and breakdown checks as k_pcg: the residual
// is kept unprojected and the mean of its latest update (m_r) is subtracted on the fly; p's and x's means are
// folded in by the next pass over them.
template <typename T, bool VAR, bool PX, bool PY>
__global__ void __launch_bounds__(kWBlock, 1) k_wpcg(WArgs<T> P) {
  using P2 = Pair<T>;
  __shared__ double sh[8 * 32 + 8];
  extern __shared__ __align__(16) char dsm[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = kWBlock / 32;
  const int gw = blockIdx.x * nw + warp, gstep = gridDim.x * nw, nrows = w_rows(P);
  const int n = P.nx * P.ny;
  const double dn_ = (double)n;
  const long long limit = spin_limit(P.status);
  const int sweep_ctas = (P.nblk + P.sw - 1) / P.sw;

  // ---- this warp's part in the sweeps: a sweep warp (the CTA's first ones), the helper or the stager of one
  const int line = w_line(P.ny);
  auto region = [&](int w) { return (P2 *)(dsm + (size_t)w * P.warp_smem); };
  auto line_of = [&](int w, int which) {
    return region(w) + (size_t)w_ring_arrays(VAR) * kWRing * kWLines + (size_t)which * line + kWLines;
  };
  auto gline = [&](P2 *lines, int k) { return lines + (size_t)k * line + kWLines; };
  const int k0 = blockIdx.x * P.sw;                    // first block of this CTA
  const int nmine = max(0, min(P.sw, P.nblk - k0));    // its sweep warps
  const int tl = P.nx - 1 - kWLines * (P.nblk - 1);
  const int role = warp / P.sw, mine = warp - role * P.sw;  // role 0: sweep warp, 1: helper, 2: stager
  const bool sweeps = role == 0 && mine < nmine, helps = role == 1 && mine < nmine, stages = role == 2 && mine < nmine;
  WWarp<T> W{};
  unsigned phases = 0;
  if (sweeps || helps || stages) {
    const int k = k0 + mine;
    W.k = k;
    W.ring = smem_addr(region(mine));
    W.ctr = W.ring + P.warp_smem - 4 * kWCtr;
    W.bars = W.ctr - 8 * kWRingGroups;
    W.ends = W.bars - kWLines * (unsigned)sizeof(P2);
    W.far_f = mine == 0;
    W.far_b = mine + 1 == nmine;
    // lines from another CTA are read where its edge warp writes them, in global memory
    if (k > 0) W.in_f = mine > 0 ? line_of(mine, 0) : gline(P.line_f, k - 1);
    if (k + 1 < P.nblk) W.in_b = mine + 1 < nmine ? line_of(mine, 1) : gline(P.line_b, k + 1);
    // in step s the block's last line works on pair s - (kWLines - 1), its first on pair s, line nx-1 on pair s - tl
    if (k + 1 < P.nblk) W.to_f = (mine + 1 < nmine ? line_of(mine + 1, 0) : gline(P.line_f, k)) - (kWLines - 1);
    if (k > 0) W.to_b = mine > 0 ? line_of(mine - 1, 1) : gline(P.line_b, k);
    if (PX) {  // line 0 hands its forward values to line nx-1, line nx-1 its backward values to line 0
      const bool near = P.nblk <= P.sw;  // the first and the last block in one CTA
      P2 *const xf = near ? line_of(P.nblk - 1, 2) : gline(P.wrap_f, 0);
      P2 *const xb = near ? line_of(0, 3) : gline(P.wrap_b, 0);
      if (k == 0) W.to_xf = xf;
      if (k == P.nblk - 1) W.in_xf = xf;
      if (k == P.nblk - 1) W.to_xb = xb - tl;
      if (k == 0) W.in_xb = xb;
    }
    if (stages) {
      if (lane < kWRingGroups) mbar_init(W.bars + 8 * lane);
      if (lane < kWCtr) st_ctr(W.ctr + 4 * lane, 0);
      for (int l = 0; l < (PX ? 4 : 2); ++l) {
        P2 *const v = line_of(mine, l);
        for (int t = lane - kWLines; t < line - kWLines; t += 32) v[t] = empty_pair<T>();
      }
    }
  }
  {  // the lines between CTAs start empty; the first reduction orders this before any sweep
    const size_t nl = (size_t)P.nblk * line;
    const size_t t0 = (size_t)blockIdx.x * kWBlock + threadIdx.x, ts = (size_t)gridDim.x * kWBlock;
    for (size_t t = t0; t < nl; t += ts) P.line_f[t] = P.line_b[t] = empty_pair<T>();
    if (PX)
      for (size_t t = t0; t < (size_t)line; t += ts) P.wrap_f[t] = P.wrap_b[t] = empty_pair<T>();
  }

  // ---- into sweep order: r = b (x = 0), the factor's q, the operator; |b|
  double v3[3] = {0.0, 0.0, 0.0};
  for (int row = gw; row < nrows; row += gstep) {
    const WRow R = w_row(P, row);
    const size_t g0 = (size_t)(R.v0 ? R.i : 0) * P.ny + (R.v0 ? 2 * R.c : 0);
    auto take = [&](const T *src) -> P2 { return P2{R.v0 ? src[g0] : T(0), R.v1 ? src[g0 + 1] : T(0)}; };
    const P2 b = take(P.b), d = take(P.dinv);
    const P2 q = P.prec == kPrecICC ? P2{d.x * d.x * P.scale, d.y * d.y * P.scale} : P2{d.x * P.scale, d.y * P.scale};
    P.r[R.e] = b;
    P.v[R.e] = P2{q.x * b.x, q.y * b.y};
    P.x[R.e] = P2{T(0), T(0)};
    P.q[R.e] = q;
    P.dg[R.e] = take(P.a5 + 2 * (size_t)n);
    if (VAR) {
      const P2 w = take(P.a5), s = take(P.a5 + (size_t)n), nn = take(P.a5 + 3 * (size_t)n), e = take(P.a5 + 4 * (size_t)n);
      P.aw[R.e] = w;
      P.as[R.e] = s;
      P.ga[R.e] = P2{q.x * s.x, q.y * s.y};
      P.ha[R.e] = P2{q.x * w.x, q.y * w.y};
      P.gn[R.e] = P2{q.x * nn.x, q.y * nn.y};
      P.he[R.e] = P2{q.x * e.x, q.y * e.y};
    }
    const double b0 = b.x, b1 = b.y;
    v3[0] += b0 + b1;
    v3[1] += b0 * b0 + b1 * b1;
  }
  v3[2] = v3[1];
  const int grid = (int)gridDim.x;
  int full = 0, app = 0;  // reductions of each kind so far
  auto reduce_sets = [](int &count, int base, int &set, int &next) {
    set = base + count % 3;
    next = base + (count + 1) % 3;
    ++count;
  };
  int set, next;
  reduce_sets(full, 0, set, next);
  if (!w_reduce<3>(v3, P.slots, set, next, grid, sh, P.status, limit)) return;
  double m_r = P.project ? v3[0] / dn_ : 0.0;
  double r_sum = v3[0];
  double rn2 = P.project ? max_ref(v3[1] - v3[0] * v3[0] / dn_, 0.0) : v3[1];
  const double rhs_norm = sqrt(max_ref(v3[2], 0.0));
  double absr = sqrt(max_ref(rn2, 0.0));
  double relr = absr / max_ref(rhs_norm, 1.0e-30);
  int iterations = 0;
  double iter_res = 0.0;
  if (relr < P.tol || absr < P.tol_abs) {
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      P.out[0] = 0;
      P.out[1] = absr;
      P.out[2] = relr;
      P.out[3] = 0.0;
    }
    return;
  }

  // z = M^-1 r (scaled by P.scale), then acc[0] = sum z, acc[1] = r.z.  The mean of r is the rounding of its last
  // update; z's own projection and the next update take it out
  auto precondition = [&](double (&acc)[2]) -> bool {
    if (sweeps) {
      const unsigned long long t0 = global_ns();
      bool ok = w_sweep<T, VAR, true, PX, PY>(P, W, limit);
      __threadfence();  // w, before the helper's copies of it for the backward sweep
      __syncwarp();
      if (lane == 0) st_ctr(W.ctr + kCtrReadyF, -1);  // the ring's last groups hold w now
      const unsigned long long t1 = global_ns();
      if (ok) w_sweep<T, VAR, false, PX, PY>(P, W, limit);
      if (P.prof && lane == 0 && W.k < 16) {
        P.prof[4 * W.k] = (double)(t1 - t0);
        P.prof[4 * W.k + 3] = (double)(global_ns() - t1);
      }
    } else if (helps || stages) {
      bool ok = helps ? w_help<T, VAR, true, PX, PY>(P, W, limit) : w_stage<T, VAR, true>(P, W, phases, limit);
      long long spins = 0;  // the forward sweep's results are in the ring and in memory
      while (ok && warp_ctr(W.ctr + kCtrReadyF) != -1) ok = !give_up(++spins, limit, P.status);
      if (ok && helps) w_help<T, VAR, false, PX, PY>(P, W, limit);
      if (ok && stages) w_stage<T, VAR, false>(P, W, phases, limit);
    }
    double none[1] = {0.0};
    int ps, pn;
    reduce_sets(app, 3, ps, pn);
    if (!w_reduce<1>(none, P.slots, ps, pn, sweep_ctas, sh, P.status, limit)) return false;
    if (stages && lane < kWCtr) st_ctr(W.ctr + 4 * lane, 0);  // before the next sweeps: two reductions from here
    acc[0] = acc[1] = 0.0;
    for (int row = gw; row < nrows; row += gstep) {  // zeros outside the lines
      const size_t e = (size_t)row * kWLines + lane;
      const P2 z = ld_cg(P.z + e), r = P.r[e];
      acc[0] += (double)z.x + (double)z.y;
      acc[1] += (double)r.x * (double)z.x + (double)r.y * (double)z.y;
    }
    int fs, fn;
    reduce_sets(full, 0, fs, fn);
    return w_reduce<2>(acc, P.slots, fs, fn, grid, sh, P.status, limit);
  };

  unsigned long long t_p1 = 0, t_p2 = 0, t_pc = 0;
  double m_x = 0.0, rz_old = 0.0;
  const double scale = (double)P.scale;  // z and p carry the factor
  const double pap_min = sizeof(T) == sizeof(float) ? pcg_pap_min<T>() : pcg_pap_min<T>() * scale * scale;
  P2 *p_old = P.p0, *p_new = P.p1;
  const int max_it = P.max_it > 1 ? P.max_it : 1;
  for (int it = 0;; ++it) {
    const unsigned long long t0 = global_ns();
    double acc[2];
    if (!precondition(acc)) return;
    const double m_z = P.project ? acc[0] / dn_ : 0.0;
    const double rz = P.project ? acc[1] - m_z * r_sum : acc[1];  // r^T z with z projected
    if (!isfinite(rz) || rz <= 0.0) {
      if (threadIdx.x == 0) atomicCAS(P.status, kDevOk, it == 0 ? kDevPcgBreakdownRz0 : kDevPcgBreakdownRz);
      return;
    }
    const bool first = it == 0;
    const double beta = first ? 0.0 : rz / rz_old;
    rz_old = rz;
    const unsigned long long t1 = global_ns();
    t_pc += t1 - t0;
    double v[3];
    w_spmv<T, VAR>(P, first, (T)m_z, (T)beta, p_old, p_new, v);
    reduce_sets(full, 0, set, next);
    if (!w_reduce<3>(v, P.slots, set, next, grid, sh, P.status, limit)) return;
    const double m_p = P.project ? v[0] / dn_ : 0.0;
    const double pap = P.project ? v[1] - m_p * v[2] : v[1];
    if (!isfinite(pap) || fabs(pap) < pap_min) {
      if (threadIdx.x == 0) atomicCAS(P.status, kDevOk, kDevPcgBreakdownPap);
      return;
    }
    const double alpha = rz / pap;
    const unsigned long long t2 = global_ns();
    t_p1 += t2 - t1;
    double w[5];
    w_update<T>(P, (T)m_p, (T)alpha, (T)m_x, (T)m_r, p_new, w);
    reduce_sets(full, 0, set, next);
    if (!w_reduce<5>(w, P.slots, set, next, grid, sh, P.status, limit)) return;
    t_p2 += global_ns() - t2;
    m_x = P.project ? w[2] / dn_ : 0.0;
    m_r = P.project ? w[3] / dn_ : 0.0;
    r_sum = w[3];
    rn2 = P.project ? max_ref(w[4] - w[3] * w[3] / dn_, 0.0) : w[4];
    iterations = it + 1;
    iter_res = sqrt(w[0] / max_ref(w[1], 1.0e-30));
    absr = sqrt(max_ref(rn2, 0.0));
    relr = absr / max_ref(rhs_norm, 1.0e-30);
    if (P.mon && it < P.mon_cap && blockIdx.x == 0 && threadIdx.x == 0) {  // the CG monitor's record
      P.mon[4 * it + 0] = absr;
      P.mon[4 * it + 1] = relr;
      P.mon[4 * it + 2] = iter_res;
      P.mon[4 * it + 3] = alpha * scale;
    }
    if (relr < P.tol || absr < P.tol_abs) break;
    if (iterations >= max_it) break;
    P2 *t = p_old;
    p_old = p_new;
    p_new = t;
  }
  // the solution in natural order, its pending projection applied
  const T mx = (P.project && m_x != 0.0) ? (T)m_x : T(0);
  for (int row = gw; row < nrows; row += gstep) {
    const WRow R = w_row(P, row);
    if (!R.v0) continue;
    const P2 x = P.x[R.e];
    const size_t g0 = (size_t)R.i * P.ny + 2 * R.c;
    P.x_out[g0] = x.x - mx;
    if (R.v1) P.x_out[g0 + 1] = x.y - mx;
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    P.out[0] = (double)iterations;
    P.out[1] = absr;
    P.out[2] = relr;
    P.out[3] = iter_res;
    P.out[4] = (double)t_p1 * 1e-6;
    P.out[5] = (double)t_p2 * 1e-6;
    P.out[6] = (double)t_pc * 1e-6;
  }
}

}  // namespace dn
