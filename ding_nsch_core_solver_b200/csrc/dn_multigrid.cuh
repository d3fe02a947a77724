// dn_multigrid.cuh -- the FP32 inner solver of the mixed-precision pressure correction: conjugate gradients
// preconditioned by one geometric multigrid V-cycle.
//
// The mixed form wraps FP32 inner solves of A e = r in an FP64 defect-correction loop that stops on the
// reference's own rule (relative or absolute FP64 residual below pressure_tolerance, the test of
// solve_pressure_correction_*, pressure.cpp:302-365).  The inner preconditioner does not have to be the
// reference's IC(0): the outer loop decides the answer.  ICC/ILDLT triangular solves are one long
// dependency chain across the grid (nx + ny anti-diagonals per sweep), while a V-cycle is a handful of
// fully parallel passes per level, and its iteration count does not grow with the grid.
//
// Hierarchy.  Level 0 is the assembled 5-point operator (k_p_assemble's W,S,C,N,E slots) rounded to FP32.
// Level l+1 halves both extents while both are even, >= 4, and the level has more than kMgCoarseMax cells.
// Its operator is the cell-centred rediscretisation: a coarse face weight is the mean of the two fine face
// weights it covers; the diagonal is the sum of the coarse off-diagonal weights plus half the summed
// boundary excess (diagonal minus off-diagonal sum, non-zero only on Dirichlet sides) of the four children.
// On the coarsest level (<= kMgCoarseMax cells) the operator is inverted exactly in FP64 (Gauss-Jordan on
// the SPD matrix; the pure-Neumann / periodic null space is removed by the rank-one shift A + mean(diag) /
// n * 1 1^T, which leaves the solution of a mean-free right-hand side unchanged) and applied in FP32.
//
// Transfer operators: bilinear cell-centred prolongation P (weights 3/4, 1/4 per direction; across a wall
// the ghost parent mirrors the boundary cell with sign +1 for a Neumann side and -1 for a Dirichlet side;
// periodic directions wrap) and restriction R = P^T.  Smoother: red-black Gauss-Seidel, nu sweeps red-then-
// black before the coarse correction and nu sweeps black-then-red after it, so that the V-cycle is a
// symmetric positive definite operator and the outer iteration is plain CG.  Vectors, operators and the
// SpMV accumulate in FP32; the CG dot products and norms accumulate in FP64.
#pragma once

#include <cooperative_groups.h>

#include <type_traits>

#include "dn_common.cuh"
#include "dn_krylov.cuh"

namespace dn {

constexpr int kMgCoarseMax = 128;  // cells of the directly inverted coarsest level (128^2 doubles of shared memory)
constexpr int kMgMaxLevels = 24;
constexpr int kMgParts = 1024;     // CTAs of the CG vector kernels at most (per-CTA partial sums)
constexpr int kMgSweeps = 2;       // red-black sweeps before and after each coarse correction
constexpr int kMgBottomCells = 8192;  // levels this small run on one CTA of the cluster form (k_mgcg_cluster)

// one level of the hierarchy: operator slots [5][n] (W,S,C,N,E), iterate, right-hand side, residual
struct MgLevel {
  const float *a;
  float *x, *b, *r;
  int nx, ny;
};
// wall folding signs of the bilinear transfer (left, right, bottom, top) and the periodicity
struct MgFold {
  float s[4];
  int px, py;
};

// 1D bilinear weight of coarse index I in the interpolation of fine index i (fine extent 2 * nc)
__device__ __forceinline__ float mg_w1(int i, int I, int nc, int per, float s_lo, float s_hi) {
  const int par = i >> 1;
  int nb = (i & 1) ? par + 1 : par - 1;
  float w = (par == I) ? 0.75f : 0.0f;
  if (nb >= 0 && nb < nc) {
    if (nb == I) w += 0.25f;
  } else if (per) {
    nb = nb < 0 ? nb + nc : nb - nc;
    if (nb == I) w += 0.25f;
  } else if (par == I) {
    w += 0.25f * (nb < 0 ? s_lo : s_hi);
  }
  return w;
}

// coarse b = P^T (fine r) at coarse cell t: the 4 x 4 fine cells whose interpolation it enters
__device__ __forceinline__ void mg_restrict_at(const MgLevel &F, const MgLevel &C, const MgFold &fold, unsigned t) {
  const int I = (int)(t / (unsigned)C.ny), J = (int)(t - (unsigned)I * (unsigned)C.ny);
  float sum = 0.0f;
#pragma unroll
  for (int di = -1; di <= 2; ++di) {
    int i = 2 * I + di;
    if (i < 0 || i >= F.nx) {
      if (!fold.px) continue;
      i = i < 0 ? i + F.nx : i - F.nx;
    }
    const float wx = mg_w1(i, I, C.nx, fold.px, fold.s[0], fold.s[1]);
    if (wx == 0.0f) continue;
    float row = 0.0f;
#pragma unroll
    for (int dj = -1; dj <= 2; ++dj) {
      int j = 2 * J + dj;
      if (j < 0 || j >= F.ny) {
        if (!fold.py) continue;
        j = j < 0 ? j + F.ny : j - F.ny;
      }
      const float wy = mg_w1(j, J, C.ny, fold.py, fold.s[2], fold.s[3]);
      if (wy != 0.0f) row += wy * F.r[(long long)i * F.ny + j];
    }
    sum += wx * row;
  }
  C.b[t] = sum;
}

// fine x += P (coarse x) at fine cell t: its parent and the parents' neighbours toward it
__device__ __forceinline__ void mg_prolong_at(const MgLevel &C, const MgLevel &F, const MgFold &fold, unsigned t) {
  const int i = (int)(t / (unsigned)F.ny), j = (int)(t - (unsigned)i * (unsigned)F.ny);
  int I[2], J[2];
  float wx[2], wy[2];
  I[0] = i >> 1;
  I[1] = (i & 1) ? I[0] + 1 : I[0] - 1;
  wx[0] = 0.75f;
  wx[1] = 0.25f;
  if (I[1] < 0 || I[1] >= C.nx) {
    if (fold.px) {
      I[1] = I[1] < 0 ? I[1] + C.nx : I[1] - C.nx;
    } else {
      wx[0] += 0.25f * (I[1] < 0 ? fold.s[0] : fold.s[1]);
      wx[1] = 0.0f;
      I[1] = I[0];
    }
  }
  J[0] = j >> 1;
  J[1] = (j & 1) ? J[0] + 1 : J[0] - 1;
  wy[0] = 0.75f;
  wy[1] = 0.25f;
  if (J[1] < 0 || J[1] >= C.ny) {
    if (fold.py) {
      J[1] = J[1] < 0 ? J[1] + C.ny : J[1] - C.ny;
    } else {
      wy[0] += 0.25f * (J[1] < 0 ? fold.s[2] : fold.s[3]);
      wy[1] = 0.0f;
      J[1] = J[0];
    }
  }
  float v = 0.0f;
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) v += wx[a] * wy[b] * C.x[(long long)I[a] * C.ny + J[b]];
  F.x[t] += v;
}

// ---------------------------------------------------------------------------------------------------
// The V-cycle of the large grids: one launch per level and direction.
//
// A half sweep does two operations per operator value it reads, so a level is bound by reading its operator
// (five values per cell) as often as it is swept: nine times per V-cycle when every phase is a launch, plus
// the launches themselves, which on the coarser levels are all of the time.  Here a CTA owns a tile of the
// level, reads the operator of the tile and of a halo around it once into registers, and runs all of a
// direction's phases on it: k_mg_down the four half sweeps before the coarse correction, the residual and its
// restriction, k_mg_up the prolongation and the four half sweeps after it.  A phase is wrong in one more ring
// of the region's cells than the phase before (they miss a neighbour), so the halo is as wide as the phases
// are many, and what the tile's own cells hold is what phase-by-phase sweeps of the whole level leave there,
// bit for bit: every cell is updated from the same values in the same order.
//
// A region is kMgRegionRows x kMgRegionCols cells: a lane holds a pair of columns (one cell of each colour), a warp
// kMgRows rows.  Which cell of a pair has the phase's colour depends only on the row, so the choice is made
// at compile time; a row's left and right neighbours come by shuffle, the rows above and below from the same
// thread's registers or, at a warp's edge, through shared memory (one barrier per phase).  Cells outside a
// walled grid get a zero row and stay zero; across a periodic side the region holds copies of the cells of
// the other side.  The swept iterate goes to the level's residual buffer on the way down (no residual is
// stored) and to x on the way up, so no CTA overwrites what another still reads as its halo.
//
// The operator is loaded before griddepcontrol.wait: no kernel of a V-cycle, nor the one launched before it,
// writes an operator.
//
// 32 x 64 regions with three CTAs of eight warps per SM cover 1.9 (down) and 1.5 (up) times the cells, but where
// 64 x 64 ones (1.5 and 1.3 times; one CTA of 16 warps by their registers) load, wait and sweep in turn, they
// overlap.  Measured, us per launch in a chain of launches, 32 x 64 / 64 x 64: level of 2M cells down 29.5 / 34.7,
// up 26.3 / 31.7; of 512K cells 11.2 / 11.8 and 7.8 / 12.3; of at most 100K cells, where a launch is latency,
// 4.8 / 5.8 and 5.1 / 6.1.  A V-cycle of 11 launches per level and a bottom of 8192 cells in global memory took 373 us
// at 1024 x 2048 and 139 us at 192 x 384 cells; this form takes 129 and 41.
// ---------------------------------------------------------------------------------------------------
constexpr int kMgRegionRows = 32, kMgRegionCols = 64;
constexpr int kMgRows = 4;                        // rows of the region per warp (even)
constexpr int kMgWarps = kMgRegionRows / kMgRows;
constexpr int kMgTileThreads = 32 * kMgWarps;
// halo before the tile's first row / column: one ring per phase (half sweeps, residual, restriction), and the
// region's first column is even, so that pairs are aligned; the tile is even in both directions
constexpr int kMgDownRow = 2 * kMgSweeps + 1, kMgDownCol = (kMgDownRow + 1) & ~1;
constexpr int kMgDownRows = kMgRegionRows - 2 * kMgDownRow, kMgDownCols = (kMgRegionCols - kMgDownCol - kMgDownRow) & ~1;
constexpr int kMgUp = 2 * kMgSweeps, kMgUpCols = kMgRegionCols - 2 * kMgUp, kMgUpRows = kMgRegionRows - 2 * kMgUp;
static_assert(kMgRows % 2 == 0 && kMgDownRows % 2 == 0 && kMgUp % 2 == 0, "coarse cells and pairs are not cut");

// The weights of fine cells 2 I - 1 .. 2 I + 2 in coarse cell I of nc >= 2: mg_w1's values, without its branches
__device__ __forceinline__ void mg_w4(int I, int nc, int per, float s_lo, float s_hi, float (&w)[4]) {
  const bool lo = !per && I == 0, hi = !per && I == nc - 1;
  w[0] = lo ? 0.0f : 0.25f;
  w[1] = lo ? 0.75f + 0.25f * s_lo : 0.75f;
  w[2] = hi ? 0.75f + 0.25f * s_hi : 0.75f;
  w[3] = hi ? 0.0f : 0.25f;
}
// sum of w_i w_j r(i, j) over the 4 x 4 fine cells of a coarse cell, a row at a time (a cell outside has weight
// zero and r = 0 or a cell's value)
template <class R>
__device__ __forceinline__ float mg_restrict_sum(const float (&wx)[4], const float (&wy)[4], R &&r) {
  float sum = 0.0f;
#pragma unroll
  for (int a = 0; a < 4; ++a) {
    float row = 0.0f;
#pragma unroll
    for (int b = 0; b < 4; ++b) row += wy[b] * r(a, b);
    sum += wx[a] * row;
  }
  return sum;
}
// index k of an extent of n cells, which may lie outside it: wrapped when periodic, else -1
__device__ __forceinline__ int mg_wrap(int k, int n, int per) {
  if (k >= 0 && k < n) return k;
  if (!per) return -1;
  k %= n;
  return k < 0 ? k + n : k;
}

// A thread's part of a region: kMgRows rows of a pair of columns
struct MgTile {
  float a[kMgRows][4][2], d[kMgRows][2], b[kMgRows][2], x[kMgRows][2];  // a: W, S, N, E
  int row[kMgRows];  // the level's row, -1 outside
  int col;           // the pair's first column, -1 outside
  unsigned lane, warp;
};

// the rows and columns of the region whose first cell is (i0, j0), and its operator
__device__ __forceinline__ void mg_tile_operator(MgTile &T, const MgLevel &L, int i0, int j0, int px, int py) {
  T.lane = threadIdx.x & 31u;
  T.warp = threadIdx.x >> 5;
  T.col = mg_wrap(j0 + 2 * (int)T.lane, L.ny, py);
  const size_t n = (size_t)L.nx * L.ny;
#pragma unroll
  for (int q = 0; q < kMgRows; ++q) {
    T.row[q] = mg_wrap(i0 + (int)T.warp * kMgRows + q, L.nx, px);
    const bool in = T.row[q] >= 0 && T.col >= 0;
    const size_t r = in ? (size_t)T.row[q] * L.ny + T.col : 0;
    constexpr int ks[4] = {0, 1, 3, 4};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const float2 v = in ? __ldg((const float2 *)(L.a + ks[k] * n + r)) : make_float2(0.0f, 0.0f);
      T.a[q][k][0] = v.x;
      T.a[q][k][1] = v.y;
    }
    const float2 v = in ? __ldg((const float2 *)(L.a + 2 * n + r)) : make_float2(1.0f, 1.0f);
    T.d[q][0] = v.x;
    T.d[q][1] = v.y;
  }
}
__device__ __forceinline__ void mg_tile_load(const MgTile &T, const float *g, int ny, float (&v)[kMgRows][2]) {
#pragma unroll
  for (int q = 0; q < kMgRows; ++q) {
    float2 w = make_float2(0.0f, 0.0f);
    if (T.row[q] >= 0 && T.col >= 0) w = *(const float2 *)(g + (size_t)T.row[q] * ny + T.col);
    v[q][0] = w.x;
    v[q][1] = w.y;
  }
}

// the rows a warp's neighbours read: its first and last rows' cells of either colour, as last updated
struct MgEdges {
  float lo[2][kMgWarps + 2][32], hi[2][kMgWarps + 2][32];  // warp w is entry w + 1
};
// a_W x_W + a_S x_S + a_N x_N + a_E x_E of cell s of the pair in row q, summed in that order from zero (a
// coefficient without a neighbour is zero); up, dn: the cells before the first and after the last row
template <int Q, int S>
__device__ __forceinline__ float mg_tile_sum(const MgTile &T, float up, float dn) {
  const float w = Q == 0 ? up : T.x[Q > 0 ? Q - 1 : 0][S];
  const float e = Q == kMgRows - 1 ? dn : T.x[Q < kMgRows - 1 ? Q + 1 : Q][S];
  const float side = S == 0 ? __shfl_up_sync(0xffffffffu, T.x[Q][1], 1) : __shfl_down_sync(0xffffffffu, T.x[Q][0], 1);
  const float so = S == 0 ? side : T.x[Q][0], no = S == 0 ? T.x[Q][1] : side;
  float s = 0.0f;
  s += T.a[Q][0][S] * w;
  s += T.a[Q][1][S] * so;
  s += T.a[Q][2][S] * no;
  s += T.a[Q][3][S] * e;
  return s;
}
// f(row index as a constant) for each of a thread's rows
template <class F>
__device__ __forceinline__ void mg_rows(F &&f) {
  f(std::integral_constant<int, 0>{});
  f(std::integral_constant<int, 1>{});
  f(std::integral_constant<int, 2>{});
  f(std::integral_constant<int, 3>{});
}
static_assert(kMgRows == 4, "mg_rows");
// the rows outside the region (its first and last warps' missing neighbours)
__device__ __forceinline__ void mg_edges_clear(MgEdges &E) {
  if (threadIdx.x < 64) {
    const unsigned c = threadIdx.x >> 5, l = threadIdx.x & 31u;
    E.hi[c][0][l] = 0.0f;
    E.lo[c][kMgWarps + 1][l] = 0.0f;
  }
}
// One half sweep: the cells of colour COLOR, (row + column) & 1, where the region's first row is PAR (mod 2).
// FIRST: the iterate is zero on entry, so the cells take b / diag.
template <int COLOR, int PAR, bool FIRST>
__device__ __forceinline__ void mg_tile_smooth(MgTile &T, MgEdges &E) {
  float up = 0.0f, dn = 0.0f;
  if (!FIRST) {
    up = E.hi[COLOR ^ 1][T.warp][T.lane];
    dn = E.lo[COLOR ^ 1][T.warp + 2][T.lane];
  }
  float v[kMgRows];
  auto cell = [&](auto qc) {
    constexpr int Q = decltype(qc)::value, S = (Q + PAR + COLOR) & 1;
    float s = T.b[Q][S];
    if (!FIRST) s -= mg_tile_sum<Q, S>(T, up, dn);
    v[Q] = s / T.d[Q][S];
  };
  mg_rows(cell);
#pragma unroll
  for (int q = 0; q < kMgRows; ++q) T.x[q][(q + PAR + COLOR) & 1] = v[q];
  E.lo[COLOR][T.warp + 1][T.lane] = v[0];
  E.hi[COLOR][T.warp + 1][T.lane] = v[kMgRows - 1];
  __syncthreads();
}

// Pre-smoothing of level F from a zero iterate, the residual and its restriction into C.b; the iterate goes
// to F.r.  One CTA per tile of kMgDownRows x kMgDownCols cells.
__global__ void __launch_bounds__(kMgTileThreads, 3) k_mg_down(MgLevel F, MgLevel C, MgFold fold) {
  __shared__ MgEdges E;
  __shared__ float rs[kMgRegionRows][kMgRegionCols];
  const int ti = (int)blockIdx.y * kMgDownRows, tj = (int)blockIdx.x * kMgDownCols;  // the tile's first cell
  const int i0 = ti - kMgDownRow, j0 = tj - kMgDownCol;
  constexpr int kPar = kMgDownRow & 1;
  MgTile T;
  mg_tile_operator(T, F, i0, j0, fold.px, fold.py);
  pdl_entry();
  mg_tile_load(T, F.b, F.ny, T.b);
#pragma unroll
  for (int q = 0; q < kMgRows; ++q) T.x[q][0] = T.x[q][1] = 0.0f;
  mg_edges_clear(E);
  mg_tile_smooth<0, kPar, true>(T, E);
  mg_tile_smooth<1, kPar, false>(T, E);
#pragma unroll
  for (int k = 1; k < kMgSweeps; ++k) {
    mg_tile_smooth<0, kPar, false>(T, E);
    mg_tile_smooth<1, kPar, false>(T, E);
  }
  auto residual = [&](auto qc) {
    constexpr int Q = decltype(qc)::value;
    float r[2];
    {
      constexpr int kC = (Q + kPar) & 1;  // colour of cell 0; the rows above and below hold the other one there
      const float up = Q == 0 ? E.hi[kC ^ 1][T.warp][T.lane] : 0.0f;
      const float dn = Q == kMgRows - 1 ? E.lo[kC ^ 1][T.warp + 2][T.lane] : 0.0f;
      r[0] = T.b[Q][0] - (T.d[Q][0] * T.x[Q][0] + mg_tile_sum<Q, 0>(T, up, dn));
    }
    {
      constexpr int kC = (Q + kPar + 1) & 1;
      const float up = Q == 0 ? E.hi[kC ^ 1][T.warp][T.lane] : 0.0f;
      const float dn = Q == kMgRows - 1 ? E.lo[kC ^ 1][T.warp + 2][T.lane] : 0.0f;
      r[1] = T.b[Q][1] - (T.d[Q][1] * T.x[Q][1] + mg_tile_sum<Q, 1>(T, up, dn));
    }
    const int row = (int)T.warp * kMgRows + Q;
    *(float2 *)&rs[row][2 * T.lane] = make_float2(r[0], r[1]);
    const int i = i0 + row, j = j0 + 2 * (int)T.lane;  // the tile's own cells are inside the level as they stand
    if (row >= kMgDownRow && row < kMgDownRow + kMgDownRows && i < F.nx && j >= tj && j < tj + kMgDownCols && j < F.ny)
      *(float2 *)(F.r + (size_t)i * F.ny + j) = make_float2(T.x[Q][0], T.x[Q][1]);
  };
  mg_rows(residual);
  __syncthreads();
  // coarse cells: a warp a row, a lane a column
  const int cj = (int)T.lane, J = tj / 2 + cj;
  if (cj >= kMgDownCols / 2 || J >= C.ny) return;
  float wx[4], wy[4];
  mg_w4(J, C.ny, fold.py, fold.s[2], fold.s[3], wy);
  for (int ci = (int)T.warp; ci < kMgDownRows / 2; ci += kMgWarps) {
    const int I = ti / 2 + ci;
    if (I >= C.nx) break;
    mg_w4(I, C.nx, fold.px, fold.s[0], fold.s[1], wx);
    const float *f = &rs[kMgDownRow + 2 * ci - 1][kMgDownCol + 2 * cj - 1];
    C.b[(size_t)I * C.ny + J] = mg_restrict_sum(wx, wy, [&](int p, int q) { return f[p * kMgRegionCols + q]; });
  }
}

// x = F.r + P (C.x), post-smoothing of level F; the iterate goes to F.x.  One CTA per tile of kMgUpRows x kMgUpCols
// cells.
__global__ void __launch_bounds__(kMgTileThreads, 3) k_mg_up(MgLevel C, MgLevel F, MgFold fold) {
  constexpr int kCo = kMgRegionCols / 2 + 2, kCr = kMgRegionRows / 2 + 2;  // the coarse cells of the region and one ring
  __shared__ MgEdges E;
  __shared__ float cs[kCr][kCo];
  const int ti = (int)blockIdx.y * kMgUpRows, tj = (int)blockIdx.x * kMgUpCols;
  const int i0 = ti - kMgUp, j0 = tj - kMgUp;
  MgTile T;
  mg_tile_operator(T, F, i0, j0, fold.px, fold.py);
  pdl_entry();
  mg_tile_load(T, F.b, F.ny, T.b);
  mg_tile_load(T, F.r, F.ny, T.x);
  for (int t = (int)threadIdx.x; t < kCr * kCo; t += kMgTileThreads) {
    const int ci = t / kCo, cj = t - ci * kCo;
    int I = i0 / 2 - 1 + ci, J = j0 / 2 - 1 + cj;
    // a missing parent at a wall is the boundary cell itself, with weight zero
    I = fold.px ? mg_wrap(I, C.nx, 1) : min(max(I, 0), C.nx - 1);
    J = fold.py ? mg_wrap(J, C.ny, 1) : min(max(J, 0), C.ny - 1);
    cs[ci][cj] = C.x[(size_t)I * C.ny + J];
  }
  mg_edges_clear(E);
  __syncthreads();
  {
    float wy[2][2];
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      wy[s][0] = 0.75f;
      wy[s][1] = 0.25f;
      if (!fold.py && T.col + s == (s == 0 ? 0 : F.ny - 1)) {
        wy[s][0] += 0.25f * (s == 0 ? fold.s[2] : fold.s[3]);
        wy[s][1] = 0.0f;
      }
    }
#pragma unroll
    for (int q = 0; q < kMgRows; ++q) {
      const bool in = T.row[q] >= 0 && T.col >= 0;
      const int o = q & 1;  // the region's first row and a warp's rows are even
      float wx[2] = {0.75f, 0.25f};
      if (!fold.px && T.row[q] == (o == 0 ? 0 : F.nx - 1)) {
        wx[0] += 0.25f * (o == 0 ? fold.s[0] : fold.s[1]);
        wx[1] = 0.0f;
      }
      const int I[2] = {((int)T.warp * kMgRows + q) / 2 + 1, ((int)T.warp * kMgRows + q) / 2 + (o ? 2 : 0)};
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        const int J[2] = {(int)T.lane + 1, (int)T.lane + (s ? 2 : 0)};
        float v = 0.0f;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b) v += wx[a] * wy[s][b] * cs[I[a]][J[b]];
        T.x[q][s] = in ? T.x[q][s] + v : 0.0f;
      }
    }
  }
  // the red cells of the edge rows, which the first half sweep (black) reads
  E.lo[0][T.warp + 1][T.lane] = T.x[0][0];
  E.hi[0][T.warp + 1][T.lane] = T.x[kMgRows - 1][(kMgRows - 1) & 1];
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kMgSweeps; ++k) {
    mg_tile_smooth<1, 0, false>(T, E);
    mg_tile_smooth<0, 0, false>(T, E);
  }
#pragma unroll
  for (int q = 0; q < kMgRows; ++q) {
    const int row = (int)T.warp * kMgRows + q, i = i0 + row, j = j0 + 2 * (int)T.lane;
    if (row >= kMgUp && row < kMgUp + kMgUpRows && i < F.nx && j >= tj && j < tj + kMgUpCols && j < F.ny)
      *(float2 *)(F.x + (size_t)i * F.ny + j) = make_float2(T.x[q][0], T.x[q][1]);
  }
}

// The bottom of the V-cycle in one CTA: levels first .. last-1 (the first at most kMgSmemCells cells, so at
// most kMgBottomLevels levels above the coarsest) smoothed, restricted, the coarsest (last) solved with its
// inverse, then prolonged and smoothed back up to `first`.  One such launch takes the place of two per level,
// which at these sizes cost their latency and nothing else.  A thread holds the operator rows of one pair of
// cells per level in registers, the vectors and the coarsest inverse are in shared memory, and every load of
// operators is issued before the first phase; the phases then cost a barrier and shared-memory latency each.
struct MgChain {
  MgLevel lv[kMgMaxLevels];
  int first, last;
  MgFold fold;
  const float *inv;
};
constexpr int kMgSmemCells = 2048;  // a pair per thread
constexpr int kMgBottomLevels = 2;
constexpr int kMgBottomThreads = kMgSmemCells / 2;
static_assert(kMgSmemCells <= kMgCoarseMax << (2 * kMgBottomLevels), "smoothed levels of the bottom");
// dynamic shared memory: the coarsest inverse, then x, b, r of every level
constexpr size_t kMgBottomSmem = sizeof(float) * ((size_t)kMgCoarseMax * kMgCoarseMax + 3 * 2 * (size_t)kMgSmemCells);

// One pair of cells of a bottom level, by colour: operator rows and where the neighbours' values are
struct MgPair {
  float a[2][4], d[2];
  int c[2][4];  // the W, S, N, E neighbours' cells (a missing one: the cell itself, coefficient zero)
  int cell[2];
  int r, i, j;  // the pair's first cell, its row and column; r < 0: no pair
};
__device__ __forceinline__ void mg_pair_load(MgPair &P, const MgLevel &L, int px, int py) {
  const int n = L.nx * L.ny, half = L.ny >> 1, t = (int)threadIdx.x;
  P.r = -1;
  if (2 * t >= n) return;
  P.i = t / half;
  P.j = 2 * (t - P.i * half);
  P.r = P.i * L.ny + P.j;
  constexpr int ks[4] = {0, 1, 3, 4};
  float2 v[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) v[k] = __ldg((const float2 *)(L.a + (size_t)k * n + P.r));
#pragma unroll
  for (int col = 0; col < 2; ++col) {
    const int s = (P.i + col) & 1;
    P.cell[col] = P.r + s;
    P.d[col] = s ? v[2].y : v[2].x;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const long long c = slot_col<5>(P.i, P.j + s, ks[k], L.nx, L.ny, px, py);
      P.c[col][k] = c >= 0 ? (int)c : P.cell[col];
      P.a[col][k] = c >= 0 ? (s ? v[ks[k]].y : v[ks[k]].x) : 0.0f;
    }
  }
}
__device__ __forceinline__ float mg_pair_sum(const MgPair &P, const float *x, int col) {
  float v = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) v += P.a[col][k] * x[P.c[col][k]];
  return v;
}
template <int COLOR>
__device__ __forceinline__ void mg_pair_smooth(const MgPair &P, const MgLevel &L) {
  if (P.r >= 0) L.x[P.cell[COLOR]] = (L.b[P.cell[COLOR]] - mg_pair_sum(P, L.x, COLOR)) / P.d[COLOR];
  __syncthreads();
}
// the parents of fine index i on one side: its own and the neighbour toward it, with their weights
__device__ __forceinline__ void mg_parents(int i, int nc, int per, float s_lo, float s_hi, int (&I)[2], float (&w)[2]) {
  I[0] = i >> 1;
  I[1] = (i & 1) ? I[0] + 1 : I[0] - 1;
  w[0] = 0.75f;
  w[1] = 0.25f;
  const bool lo = I[1] < 0, hi = I[1] >= nc;
  if (lo || hi) {
    I[1] = per ? (lo ? nc - 1 : 0) : I[0];
    if (!per) {
      w[0] += 0.25f * (lo ? s_lo : s_hi);
      w[1] = 0.0f;
    }
  }
}

__global__ void __launch_bounds__(kMgBottomThreads, 1) k_mg_bottom(const __grid_constant__ MgChain Ch) {
  extern __shared__ float mg_smem[];
  const int tid = (int)threadIdx.x, px = Ch.fold.px, py = Ch.fold.py, ns = Ch.last - Ch.first;
  MgLevel S[kMgBottomLevels + 1];  // the levels with their vectors in shared memory
  MgPair P[kMgBottomLevels];
  float *inv = mg_smem, *q = mg_smem + kMgCoarseMax * kMgCoarseMax;
#pragma unroll
  for (int k = 0; k <= kMgBottomLevels; ++k) {
    if (k > ns) continue;
    S[k] = Ch.lv[Ch.first + k];
    const int n = S[k].nx * S[k].ny;
    S[k].x = q;
    S[k].b = q + n;
    S[k].r = q + 2 * n;
    q += 3 * n;
    if (k < kMgBottomLevels && k < ns) mg_pair_load(P[k], S[k], px, py);
  }
  const int nc = Ch.lv[Ch.last].nx * Ch.lv[Ch.last].ny;
#pragma unroll
  for (int u = 0; u < kMgCoarseMax * kMgCoarseMax / 4 / kMgBottomThreads; ++u) {  // up to 3 floats past nc^2, inside both
    const int k = 4 * (tid + u * kMgBottomThreads);
    if (k < nc * nc) *(float4 *)(inv + k) = __ldg((const float4 *)(Ch.inv + k));
  }
  pdl_entry();
  {
    const MgLevel &G = Ch.lv[Ch.first];
    const int n = G.nx * G.ny;
#pragma unroll
    for (int u = 0; u < kMgSmemCells / kMgBottomThreads; ++u)
      if (tid + u * kMgBottomThreads < n) S[0].b[tid + u * kMgBottomThreads] = G.b[tid + u * kMgBottomThreads];
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kMgBottomLevels; ++k) {
    if (k >= ns) continue;
    const MgLevel &F = S[k], &C = S[k + 1];
    const MgPair &p = P[k];
    if (p.r >= 0) {  // red from a zero iterate
      F.x[p.cell[0]] = F.b[p.cell[0]] / p.d[0];
      F.x[p.cell[1]] = 0.0f;
    }
    __syncthreads();
    mg_pair_smooth<1>(p, F);
    for (int m = 1; m < kMgSweeps; ++m) {
      mg_pair_smooth<0>(p, F);
      mg_pair_smooth<1>(p, F);
    }
    if (p.r >= 0) {
#pragma unroll
      for (int c = 0; c < 2; ++c)
        F.r[p.cell[c]] = F.b[p.cell[c]] - (p.d[c] * F.x[p.cell[c]] + mg_pair_sum(p, F.x, c));
    }
    __syncthreads();
    if (tid < C.nx * C.ny) {  // a quarter of a level of kMgSmemCells: fewer cells than threads
      const int I = tid / C.ny, J = tid - I * C.ny;
      float wx[4], wy[4];
      mg_w4(I, C.nx, px, Ch.fold.s[0], Ch.fold.s[1], wx);
      mg_w4(J, C.ny, py, Ch.fold.s[2], Ch.fold.s[3], wy);
      int row[4], col[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // a cell across a wall has weight zero: any cell's value serves
        const int i = 2 * I + u - 1, j = 2 * J + u - 1;
        row[u] = (px ? (i < 0 ? i + F.nx : (i >= F.nx ? i - F.nx : i)) : min(max(i, 0), F.nx - 1)) * F.ny;
        col[u] = py ? (j < 0 ? j + F.ny : (j >= F.ny ? j - F.ny : j)) : min(max(j, 0), F.ny - 1);
      }
      C.b[tid] = mg_restrict_sum(wx, wy, [&](int u, int w) { return F.r[row[u] + col[w]]; });
    }
    __syncthreads();
  }
#pragma unroll
  for (int k = 0; k <= kMgBottomLevels; ++k) {  // the coarsest level: inv is symmetric, thread i reads column i
    if (k != ns || tid >= nc) continue;
    float s = 0.0f;
    const float *col = inv + tid, *b = S[k].b;
#pragma unroll 16
    for (int m = 0; m < nc; ++m) s += col[m * nc] * b[m];
    S[k].x[tid] = s;
  }
  __syncthreads();
#pragma unroll
  for (int k = kMgBottomLevels - 1; k >= 0; --k) {
    if (k >= ns) continue;
    const MgLevel &F = S[k], &C = S[k + 1];
    const MgPair &p = P[k];
    if (p.r >= 0) {
      int I[2], J[2];
      float wx[2], wy[2];
      mg_parents(p.i, C.nx, px, Ch.fold.s[0], Ch.fold.s[1], I, wx);
#pragma unroll
      for (int s = 0; s < 2; ++s) {
        mg_parents(p.j + s, C.ny, py, Ch.fold.s[2], Ch.fold.s[3], J, wy);
        float v = 0.0f;
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int b = 0; b < 2; ++b) v += wx[a] * wy[b] * C.x[I[a] * C.ny + J[b]];
        F.x[p.r + s] += v;
      }
    }
    __syncthreads();
    for (int m = 0; m < kMgSweeps; ++m) {
      mg_pair_smooth<1>(p, F);
      mg_pair_smooth<0>(p, F);
    }
  }
  float *out = Ch.lv[Ch.first].x;
  const int n = Ch.lv[Ch.first].nx * Ch.lv[Ch.first].ny;
#pragma unroll
  for (int u = 0; u < kMgSmemCells / kMgBottomThreads; ++u)
    if (tid + u * kMgBottomThreads < n) out[tid + u * kMgBottomThreads] = S[0].x[tid + u * kMgBottomThreads];
}

// Coarse operator of level l+1 from the FP64 slots of level l (see the file header), in FP64 with an FP32 copy.
// mass: a uniform diagonal term of level l's operator (the shift of a shifted Laplacian K + m I), kept apart
// from the boundary excess: under R = P^T it aggregates over the four children (4 m on level l+1), while the
// boundary excess, like the face weights, is rediscretised (half the children's sum).
__global__ void k_mg_coarsen(const double *af, int nxf, int nyf, double mass, double *ac, float *acf, int nxc,
                             int nyc) {
  const unsigned nc = (unsigned)nxc * (unsigned)nyc;
  const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nc) return;
  const int I = (int)(t / (unsigned)nyc), J = (int)(t - (unsigned)I * (unsigned)nyc);
  const long long nf = (long long)nxf * nyf;
  auto at = [&](int s, int i, int j) { return af[(size_t)s * nf + (long long)i * nyf + j]; };
  double exc = 0.0;
  for (int a = 0; a < 2; ++a)
    for (int b = 0; b < 2; ++b) {
      const int i = 2 * I + a, j = 2 * J + b;
      const double d = at(2, i, j);
      double e = d + at(0, i, j) + at(1, i, j) + at(3, i, j) + at(4, i, j) - mass;
      if (fabs(e) <= 1.0e-12 * fabs(d)) e = 0.0;  // interior and Neumann rows: round-off of an exact zero
      exc += e;
    }
  const double w = 0.5 * (at(0, 2 * I, 2 * J) + at(0, 2 * I, 2 * J + 1));
  const double s = 0.5 * (at(1, 2 * I, 2 * J) + at(1, 2 * I + 1, 2 * J));
  const double nn = 0.5 * (at(3, 2 * I, 2 * J + 1) + at(3, 2 * I + 1, 2 * J + 1));
  const double e = 0.5 * (at(4, 2 * I + 1, 2 * J) + at(4, 2 * I + 1, 2 * J + 1));
  const double c = -(w + s + nn + e) + 0.5 * exc + 4.0 * mass;
  const double v[5] = {w, s, c, nn, e};
  for (int k = 0; k < 5; ++k) {
    ac[(size_t)k * nc + t] = v[k];
    acf[(size_t)k * nc + t] = (float)v[k];
  }
}

// Level 0 of the CH preconditioner's hierarchy: K + m I with K = -L, L the 5-point Laplacian with reflecting
// rows at walls (build_laplacian_matrix, ch_sparse_krylov.hpp:135-177: a row counts only the neighbours that
// exist), in the W,S,C,N,E slots.
__global__ void k_shifted_laplacian(Grid G, double m, double *a, float *af) {
  const long long n = (long long)G.nx * G.ny;
  const long long r = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= n) return;
  const int i = (int)(r / G.ny), j = (int)(r % G.ny);
  const double cx = 1.0 / (G.dx * G.dx), cy = 1.0 / (G.dy * G.dy);
  const double w = (G.px || i > 0) ? cx : 0.0, e = (G.px || i < G.nx - 1) ? cx : 0.0;
  const double s = (G.py || j > 0) ? cy : 0.0, nn = (G.py || j < G.ny - 1) ? cy : 0.0;
  const double v[5] = {-w, -s, w + e + s + nn + m, -nn, -e};
  for (int k = 0; k < 5; ++k) {
    a[(size_t)k * n + r] = v[k];
    af[(size_t)k * n + r] = (float)v[k];
  }
}

// Inverse of the coarsest operator (n <= kMgCoarseMax cells), dense, by Gauss-Jordan elimination without
// pivoting (the matrix is SPD, shifted by mean(diag) / n on every entry when singular), in FP64 shared
// memory; the FP32 result is stored column-major (= row-major, it is symmetric).  *flag = 1 when a pivot is
// not positive and finite, and the caller then does not use the hierarchy.
__global__ void k_mg_coarse_inverse(const double *a, int nx, int ny, int px, int py, int singular, float *inv,
                                    int *flag) {
  extern __shared__ double M[];
  __shared__ double f[kMgCoarseMax];
  __shared__ double shift, piv;
  const int n = nx * ny, tid = threadIdx.x, nt = blockDim.x;
  for (int k = tid; k < n * n; k += nt) M[k] = 0.0;
  __syncthreads();
  if (tid == 0) {
    double dsum = 0.0;
    for (int r = 0; r < n; ++r) dsum += a[2 * (size_t)n + r];
    shift = singular ? dsum / ((double)n * (double)n) : 0.0;
    *flag = 0;
  }
  __syncthreads();
  for (int r = tid; r < n; r += nt) {
    const int i = r / ny, j = r % ny;
    for (int s = 0; s < 5; ++s) {
      const double v = a[(size_t)s * n + r];
      if (v == 0.0) continue;
      const long long c = slot_col<5>(i, j, s, nx, ny, px, py);
      if (c >= 0) M[r * n + (int)c] += v;  // a row owns its entries: no other thread writes row r
    }
    for (int c = 0; c < n; ++c) M[r * n + c] += shift;
  }
  __syncthreads();
  for (int k = 0; k < n; ++k) {
    if (tid == 0) {
      piv = M[k * n + k];
      if (!(piv > 0.0) || !isfinite(piv)) *flag = 1;
    }
    __syncthreads();
    const double p = piv;
    if (!(p > 0.0) || !isfinite(p)) return;  // uniform across the block
    for (int j = tid; j < n; j += nt) M[k * n + j] = (j == k) ? 1.0 / p : M[k * n + j] / p;
    for (int i = tid; i < n; i += nt) f[i] = (i == k) ? 0.0 : M[i * n + k];
    __syncthreads();
    for (int e = tid; e < n * n; e += nt) {
      const int i = e / n, j = e - (e / n) * n;
      if (i == k) continue;
      M[e] = ((j == k) ? 0.0 : M[e]) - f[i] * M[k * n + j];
    }
    __syncthreads();
  }
  for (int e = tid; e < n * n; e += nt) inv[e] = (float)M[e];
}

// ---------------------------------------------------------------------------------------------------
// CG on the FP32 operator of level 0.  Scalars and the loop control live on the device (slots below): the
// iterations run inside a CUDA graph's conditional while node whose condition k_mgcg_ctrl sets, so the host
// reads nothing until the whole solve has ended.
// ---------------------------------------------------------------------------------------------------
enum MgScal {
  kMgRz = 0, kMgPq = 1, kMgRr = 2, kMgAlpha = 3, kMgBeta = 4, kMgMeanZ = 5, kMgBad = 6,
  kMgIt = 7,   // iterations of this inner solve
  kMgCap = 8,  // its iteration limit
  kMgScalCount = 16
};

// The record of one defect-correction solve (FP64 outer loop around FP32 inner solves), kDcSize doubles on
// the device: what the host reads once the solve's graph has run, and the outer loop's own state.
enum DcSlot {
  kDcTotal = 0,    // inner iterations, all cycles
  kDcCycles = 1,   // outer cycles
  kDcAbs = 2,      // FP64 residual |b - A x| (projected when singular) of the last check
  kDcRel = 3,      // the same relative to |b|
  kDcPrev = 4,     // the residual of the previous cycle (a cycle that does not reduce it ends the multigrid)
  kDcUseMg = 5,    // the next inner solve is the multigrid CG (else the IC/ILDLT persistent PCG)
  kDcIres = 6,     // CH: the last correction's size relative to the iterate
  kDcMean = 7,     // mean of the residual removed before the inner solve (singular systems)
  kDcErr = 8,      // device status of a failed inner solve or factor (0: none)
  kDcIcZero = 9,   // the IC inner solve returned without an iteration
  kDcIcReady = 10, // the FP32 IC/ILDLT factor has been made in this solve
  kDcStarted = 11, // the first check has run
  kDcUsedMg0 = 12, // the solve started with the multigrid inner solver
  kDcIcCycles = 13,// cycles run by the IC inner solver
  kDcMgIts = 14,   // iterations run by the multigrid inner solver
  kDcSize = 16
};

struct MgVec {
  SpOpT<float> A;
  float *x, *r, *z, *p, *q;
  double *part;  // [gridDim.x][3] per-CTA partial sums
  double *scal;
};

// q = A p (the 5-point pressure or the 13-point CH operator), partial sums of p.q
template <int S>
__global__ void k_mgp_apply(MgVec V) {
  pdl_entry();
  __shared__ double sh[32];
  double v[1] = {0.0};
  const unsigned n = (unsigned)V.A.n, ny = (unsigned)V.A.ny;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const int i = (int)(t / ny), j = (int)(t - (unsigned)i * ny);
    const float s = spmv_row<S>(V.A, V.p, i, j);
    V.q[t] = s;
    v[0] += (double)V.p[t] * (double)s;
  }
  block_sum<1>(v, sh);
  if (threadIdx.x == 0) V.part[3 * blockIdx.x] = v[0];
}
// x += alpha p, r -= alpha q, partial sums of r.r
__global__ void k_mgp_update(MgVec V) {
  pdl_entry();
  __shared__ double sh[32];
  double v[1] = {0.0};
  const float alpha = (float)V.scal[kMgAlpha];
  const unsigned n = (unsigned)V.A.n;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    V.x[t] += alpha * V.p[t];
    const float r = V.r[t] - alpha * V.q[t];
    V.r[t] = r;
    v[0] += (double)r * (double)r;
  }
  block_sum<1>(v, sh);
  if (threadIdx.x == 0) V.part[3 * blockIdx.x] = v[0];
}
// partial sums of r.z, z and r (the projected r.z of a singular system needs the last two)
__global__ void k_mgp_rz(MgVec V) {
  pdl_entry();
  __shared__ double sh[3 * 32];
  double v[3] = {0.0, 0.0, 0.0};
  const unsigned n = (unsigned)V.A.n;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const double z = V.z[t], r = V.r[t];
    v[0] += r * z;
    v[1] += z;
    v[2] += r;
  }
  block_sum<3>(v, sh);
  if (threadIdx.x == 0) {
    V.part[3 * blockIdx.x] = v[0];
    V.part[3 * blockIdx.x + 1] = v[1];
    V.part[3 * blockIdx.x + 2] = v[2];
  }
}
// p = (z - mean z) + beta p (first: p = z - mean z; first < 0: the first iteration of the solve)
__global__ void k_mgp_direction(MgVec V, int first) {
  pdl_entry();
  const float beta = (float)V.scal[kMgBeta], mz = (float)V.scal[kMgMeanZ];
  if (first < 0) first = V.scal[kMgIt] == 0.0 ? 1 : 0;
  const unsigned n = (unsigned)V.A.n;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x)
    V.p[t] = first ? V.z[t] - mz : (V.z[t] - mz) + beta * V.p[t];
}
// The scalar step after each reduction, by one warp in a fixed order.
//   mode 0 (after k_mgp_apply):  pq, alpha = rz / pq
//   mode 1 (after k_mgp_update): rr
//   mode 2 (after k_mgp_rz):     mean z, rz' (projected when singular), beta = rz' / rz (0 when first), rz = rz'
// A non-positive or non-finite pq or rz' sets kMgBad (k_mgcg_ctrl then ends the inner solve).  first < 0:
// the first iteration of the solve.
__global__ void k_mgp_scalars(const double *part, int nparts, double *scal, int mode, int first, int project,
                              double n) {
  pdl_entry();
  const int lane = threadIdx.x;
  if (first < 0) first = scal[kMgIt] == 0.0 ? 1 : 0;
  double s0 = 0.0, s1 = 0.0, s2 = 0.0;
  for (int p = lane; p < nparts; p += 32) {
    s0 += part[3 * p];
    if (mode == 2) {
      s1 += part[3 * p + 1];
      s2 += part[3 * p + 2];
    }
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
  s2 = warp_sum(s2);
  if (lane != 0) return;
  if (mode == 0) {
    scal[kMgPq] = s0;
    if (!(s0 > 0.0) || !isfinite(s0)) scal[kMgBad] = 1.0;
    scal[kMgAlpha] = scal[kMgRz] / s0;
  } else if (mode == 1) {
    scal[kMgRr] = s0;
  } else {
    const double mz = project ? s1 / n : 0.0;
    const double rz = project ? s0 - mz * s2 : s0;
    if (!(rz > 0.0) || !isfinite(rz)) scal[kMgBad] = 1.0;
    scal[kMgMeanZ] = mz;
    scal[kMgBeta] = first ? 0.0 : rz / scal[kMgRz];
    scal[kMgRz] = rz;
  }
}

// Start of an inner solve: its scalars cleared and its iteration limit, the outer loop's budget left
// (max(1, max_it - inner iterations so far)).  Sets the while node's condition.
__global__ void k_mgcg_init(double *scal, const double *rec, int max_it, cudaGraphConditionalHandle loop) {
  pdl_entry();
  if (threadIdx.x != 0) return;
  for (int k = 0; k < kMgScalCount; ++k) scal[k] = 0.0;
  scal[kMgCap] = (double)max(1, max_it - (int)rec[kDcTotal]);
  cudaGraphSetConditional(loop, 1u);
}

// End of one inner iteration (after the r.r reduction): counts it, and continues while no breakdown was
// flagged, |r| / |b| >= tol (|b| = the outer residual the inner right-hand side was made from; a NaN ends
// it) and the iteration limit is not reached.
__global__ void k_mgcg_ctrl(double *scal, double *rec, double tol, cudaGraphConditionalHandle loop) {
  pdl_entry();
  if (threadIdx.x != 0) return;
  const double it = scal[kMgIt] + 1.0;
  scal[kMgIt] = it;
  rec[kDcTotal] += 1.0;
  rec[kDcMgIts] += 1.0;
  bool more = it < scal[kMgCap];
  if (scal[kMgBad] != 0.0) {
    more = false;
  } else {
    const double rr = scal[kMgRr], b = rec[kDcAbs];  // std::max semantics: a NaN stays a NaN
    const double rel = sqrt(rr < 0.0 ? 0.0 : rr) / (b < 1.0e-300 ? 1.0e-300 : b);
    if (!(rel >= tol)) more = false;
  }
  cudaGraphSetConditional(loop, more ? 1u : 0u);
}

// ---------------------------------------------------------------------------------------------------
// The inner CG as one thread-block cluster (level-0 grids up to mg_cluster_cells cells).  Small grids leave
// every launch of a V-cycle latency-bound, a few microseconds for a few thousand cells.  Here 1-8 CTAs of 1024 threads, which the hardware schedules
// together, run every iteration of the solve: V-cycles, r.z, direction, A p, p.q and the update as phases
// separated by cluster barriers (barrier.cluster with release / acquire, which orders the global memory the
// phases exchange), dot products reduced through distributed shared memory in rank order, so every CTA holds
// the same scalars and takes the same stopping decision.  One launch per inner solve; nothing waits on
// another launch or spins.  Every cell sees the operations of k_mg_down, k_mg_bottom and k_mg_up, phase for phase.
// ---------------------------------------------------------------------------------------------------
constexpr int kMgClusterThreads = 1024;
constexpr int kMgClusterMax = 8;              // CTAs per cluster at most (the portable cluster size)
constexpr long long kMgClusterCells = 0;  // default: off (set from measurements)
constexpr int kMgClusterSmemMax = 160 * 1024;  // dynamic shared memory of the bottom levels at most

struct MgClusterArgs {
  const MgChain *ch;     // levels 0 .. last of the preconditioner's hierarchy, in device memory (lv[0].b / .x
                         // are replaced per V-cycle)
  SpOpT<float> A;        // the CG operator on level 0 (the 5-point pressure or the 13-point CH operator)
  float *x, *r, *z, *p, *q, *tmp;
  const float *b;        // the inner right-hand side (x is zero on entry)
  int vcycles, project, max_it;
  int bottom;            // the first level of at most kMgBottomCells cells: it and the coarser ones run on CTA 0
                         // in shared memory (3 floats per cell of those levels, dynamic)
  double tol;            // relative to |b| = R[kDcAbs]
  double *R;             // the defect-correction record: iterations added to kDcTotal and kDcMgIts
};

__device__ __forceinline__ void mgc_sync() { cooperative_groups::this_cluster().sync(); }

// K sums over the cluster: the CTA's sums, then every CTA adds the CTAs' sums in rank order (warp 0 reads
// them from distributed shared memory), so all threads of all CTAs hold the same bits.  `slot` alternates
// by `par` so that a CTA writing the next reduction never overwrites sums another CTA is still reading.
template <int K>
__device__ __forceinline__ void mgc_sum(double (&v)[K], double *sh, double (*slot)[4], double *bc, int &par) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  block_sum<K>(v, sh);
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < K; ++k) slot[par][k] = v[k];
  }
  cl.sync();
  if (threadIdx.x == 0) {
    const unsigned cs = cl.num_blocks();
#pragma unroll
    for (int k = 0; k < K; ++k) bc[k] = 0.0;
    for (unsigned j = 0; j < cs; ++j) {
      const double *o = cl.map_shared_rank(&slot[par][0], j);
#pragma unroll
      for (int k = 0; k < K; ++k) bc[k] += o[k];
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < K; ++k) v[k] = bc[k];
  __syncthreads();
  par ^= 1;
}

// The off-diagonal sums a_s x_nb of up to kMgBatch cells at once: every load of the batch is issued
// before any sum is formed (the neighbours' x values do not wait for the coefficients), then each cell's sum
// is taken in slot order over its non-zero coefficients.
constexpr int kMgBatch = 4;
__device__ __forceinline__ void mg_row_sums(const MgLevel &L, const float *x, const int (&ci)[kMgBatch],
                                            const int (&cj)[kMgBatch], const bool (&on)[kMgBatch], long long n,
                                            int px, int py, float (&out)[kMgBatch]) {
  constexpr int ks[4] = {0, 1, 3, 4};
  float av[kMgBatch][4], xv[kMgBatch][4];
#pragma unroll
  for (int u = 0; u < kMgBatch; ++u) {
    const long long r = (long long)ci[u] * L.ny + cj[u];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      av[u][q] = 0.0f;
      xv[u][q] = 0.0f;
      if (on[u]) {
        const long long c = slot_col<5>(ci[u], cj[u], ks[q], L.nx, L.ny, px, py);
        av[u][q] = __ldg(&L.a[(size_t)ks[q] * n + r]);
        if (c >= 0) xv[u][q] = x[c];
        else av[u][q] = 0.0f;  // a missing neighbour is skipped
      }
    }
  }
#pragma unroll
  for (int u = 0; u < kMgBatch; ++u) {
    float s = 0.0f;
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (av[u][q] != 0.0f) s += av[u][q] * xv[u][q];
    out[u] = s;
  }
}

// Red-black Gauss-Seidel half sweep at the colour's cells t0, t0 + st, ... (kMgBatch of them, those below lim;
// (i + j) & 1 == color, ny is even on every smoothed level, so each row holds ny / 2 cells of each colour): no
// cell of the batch reads another's x, and all loads go before the stores.  first: the iterate is zero on entry,
// so the colour's cells take b / diag and the other colour's cells are set to zero.
__device__ __forceinline__ void mg_smooth_batch(const MgLevel &L, int color, int first, int px, int py, unsigned t0,
                                                unsigned st, unsigned lim) {
  const int half = L.ny >> 1;
  const long long n = (long long)L.nx * L.ny;
  int ci[kMgBatch], cj[kMgBatch];
  bool on[kMgBatch];
  float bv[kMgBatch], dv[kMgBatch], rs[kMgBatch];
#pragma unroll
  for (int u = 0; u < kMgBatch; ++u) {
    const unsigned t = t0 + (unsigned)u * st;
    on[u] = t < lim;
    const unsigned tt = on[u] ? t : 0u;
    ci[u] = (int)(tt / (unsigned)half);
    cj[u] = 2 * (int)(tt - (unsigned)ci[u] * (unsigned)half) + ((ci[u] + color) & 1);
    const long long r = (long long)ci[u] * L.ny + cj[u];
    bv[u] = on[u] ? L.b[r] : 0.0f;
    dv[u] = on[u] ? __ldg(&L.a[2 * n + r]) : 1.0f;
  }
  if (!first) mg_row_sums(L, L.x, ci, cj, on, n, px, py, rs);
#pragma unroll
  for (int u = 0; u < kMgBatch; ++u) {
    if (!on[u]) continue;
    const long long r = (long long)ci[u] * L.ny + cj[u];
    float s = bv[u];
    if (!first) s -= rs[u];
    L.x[r] = s / dv[u];
    if (first) L.x[(long long)ci[u] * L.ny + (cj[u] ^ 1)] = 0.0f;
  }
}

// r = b - A x for a batch of cells, loads before stores (r is written, x only read)
__device__ __forceinline__ void mg_residual_batch(const MgLevel &L, int px, int py, unsigned t0, unsigned st,
                                                  unsigned lim) {
  const long long n = (long long)L.nx * L.ny;
  int ci[kMgBatch], cj[kMgBatch];
  bool on[kMgBatch];
  float bv[kMgBatch], dv[kMgBatch], xc[kMgBatch], rs[kMgBatch];
#pragma unroll
  for (int u = 0; u < kMgBatch; ++u) {
    const unsigned t = t0 + (unsigned)u * st;
    on[u] = t < lim;
    const unsigned tt = on[u] ? t : 0u;
    ci[u] = (int)(tt / (unsigned)L.ny);
    cj[u] = (int)(tt - (unsigned)ci[u] * (unsigned)L.ny);
    bv[u] = on[u] ? L.b[tt] : 0.0f;
    dv[u] = on[u] ? __ldg(&L.a[2 * n + tt]) : 0.0f;
    xc[u] = on[u] ? L.x[tt] : 0.0f;
  }
  mg_row_sums(L, L.x, ci, cj, on, n, px, py, rs);
#pragma unroll
  for (int u = 0; u < kMgBatch; ++u)
    if (on[u]) L.r[t0 + (unsigned)u * st] = bv[u] - (dv[u] * xc[u] + rs[u]);
}

// Levels `first` .. last of C in one CTA with __syncthreads between phases (k_mg_bottom's order of phases);
// lv: the levels with their x, b, r (in shared memory for the cluster form).
__device__ void mg_bottom_cta(const MgChain &C, const MgLevel *lv, int first) {
  const unsigned tid = threadIdx.x, nt = blockDim.x;
  const int px = C.fold.px, py = C.fold.py, last = C.last;
  for (int l = first; l < last; ++l) {
    const MgLevel &F = lv[l], &Cl = lv[l + 1];
    const unsigned nf = (unsigned)F.nx * (unsigned)F.ny, nh = nf >> 1, nc = (unsigned)Cl.nx * (unsigned)Cl.ny;
    for (int k = 0; k < kMgSweeps; ++k) {
      for (unsigned t = tid; t < nh; t += kMgBatch * nt) mg_smooth_batch(F, 0, k == 0, px, py, t, nt, nh);
      __syncthreads();
      for (unsigned t = tid; t < nh; t += kMgBatch * nt) mg_smooth_batch(F, 1, 0, px, py, t, nt, nh);
      __syncthreads();
    }
    for (unsigned t = tid; t < nf; t += kMgBatch * nt) mg_residual_batch(F, px, py, t, nt, nf);
    __syncthreads();
    for (unsigned t = tid; t < nc; t += nt) mg_restrict_at(F, Cl, C.fold, t);
    __syncthreads();
  }
  {
    const MgLevel &L = lv[last];
    const int n = L.nx * L.ny;
    for (int i = (int)tid; i < n; i += (int)nt) {  // inv is symmetric: thread i reads column i
      float s = 0.0f;
      for (int k = 0; k < n; ++k) s += __ldg(&C.inv[(size_t)k * n + i]) * L.b[k];
      L.x[i] = s;
    }
    __syncthreads();
  }
  for (int l = last - 1; l >= first; --l) {
    const MgLevel &F = lv[l], &Cl = lv[l + 1];
    const unsigned nf = (unsigned)F.nx * (unsigned)F.ny, nh = nf >> 1;
    for (unsigned t = tid; t < nf; t += nt) mg_prolong_at(Cl, F, C.fold, t);
    __syncthreads();
    for (int k = 0; k < kMgSweeps; ++k) {
      for (unsigned t = tid; t < nh; t += kMgBatch * nt) mg_smooth_batch(F, 1, 0, px, py, t, nt, nh);
      __syncthreads();
      for (unsigned t = tid; t < nh; t += kMgBatch * nt) mg_smooth_batch(F, 0, 0, px, py, t, nt, nh);
      __syncthreads();
    }
  }
}

// One V-cycle x0 = B b0 over every level of `C`.  The levels above `bf` (the first of at most kMgBottomCells
// cells) run on the whole cluster, its threads striding over each phase's cells in batches, with a cluster
// barrier between phases.  The levels from bf down run on CTA 0 alone with their x, b, r in shared memory
// (`smem`, 3 x their cells floats), entered with level bf's b and left with its x through global memory.
__device__ void mgc_vcycle(const MgChain &C, int bf, float *smem, MgLevel *s_lv, float *b0, float *x0, unsigned gt,
                           unsigned GT) {
  const int px = C.fold.px, py = C.fold.py, last = C.last;
  auto level = [&](int l) {
    MgLevel L = C.lv[l];
    if (l == 0) {
      L.b = b0;
      L.x = x0;
    }
    return L;
  };
  for (int l = 0; l < bf; ++l) {
    const MgLevel F = level(l), Cl = level(l + 1);
    const unsigned nf = (unsigned)F.nx * (unsigned)F.ny, nh = nf >> 1, nc = (unsigned)Cl.nx * (unsigned)Cl.ny;
    for (int k = 0; k < kMgSweeps; ++k) {
      for (unsigned t = gt; t < nh; t += kMgBatch * GT) mg_smooth_batch(F, 0, k == 0, px, py, t, GT, nh);
      mgc_sync();
      for (unsigned t = gt; t < nh; t += kMgBatch * GT) mg_smooth_batch(F, 1, 0, px, py, t, GT, nh);
      mgc_sync();
    }
    for (unsigned t = gt; t < nf; t += kMgBatch * GT) mg_residual_batch(F, px, py, t, GT, nf);
    mgc_sync();
    for (unsigned t = gt; t < nc; t += GT) mg_restrict_at(F, Cl, C.fold, t);
    mgc_sync();
  }
  if (cooperative_groups::this_cluster().block_rank() == 0) {
    if (threadIdx.x == 0) {  // the bottom levels' table, their vectors in shared memory
      float *q = smem;
      for (int l = bf; l <= last; ++l) {
        MgLevel L = C.lv[l];
        const unsigned nl = (unsigned)L.nx * (unsigned)L.ny;
        L.x = q;
        L.b = q + nl;
        L.r = q + 2 * nl;
        q += 3 * nl;
        s_lv[l] = L;
      }
    }
    __syncthreads();
    const MgLevel E = level(bf);  // the entry level's global b and x
    const unsigned ne = (unsigned)E.nx * (unsigned)E.ny;
    float *eb = s_lv[bf].b;
    for (unsigned t = threadIdx.x; t < ne; t += blockDim.x) eb[t] = E.b[t];
    __syncthreads();
    mg_bottom_cta(C, s_lv, bf);
    const float *ex = s_lv[bf].x;
    for (unsigned t = threadIdx.x; t < ne; t += blockDim.x) E.x[t] = ex[t];
  }
  mgc_sync();
  for (int l = bf - 1; l >= 0; --l) {
    const MgLevel F = level(l), Cl = level(l + 1);
    const unsigned nf = (unsigned)F.nx * (unsigned)F.ny, nh = nf >> 1;
    for (unsigned t = gt; t < nf; t += GT) mg_prolong_at(Cl, F, C.fold, t);
    mgc_sync();
    for (int k = 0; k < kMgSweeps; ++k) {
      for (unsigned t = gt; t < nh; t += kMgBatch * GT) mg_smooth_batch(F, 1, 0, px, py, t, GT, nh);
      mgc_sync();
      for (unsigned t = gt; t < nh; t += kMgBatch * GT) mg_smooth_batch(F, 0, 0, px, py, t, GT, nh);
      mgc_sync();
    }
  }
}

// The whole inner solve: r = b; per iteration z = M r (vcycles V-cycles, through tmp when two), r.z (the
// mean of z removed when the system is singular), p = (z - mean z) + beta p, q = A p, alpha = r.z / p.q,
// x += alpha p, r -= alpha q; it ends as k_mgcg_ctrl ends the per-phase form: a non-positive or non-finite
// r.z or p.q, |r| < tol |b|, or the iteration budget left in R (at least one iteration).
template <int S>
__global__ void __launch_bounds__(kMgClusterThreads, 1) k_mgcg_cluster(const MgClusterArgs P) {
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const unsigned gt = cl.block_rank() * blockDim.x + threadIdx.x, GT = cl.num_blocks() * blockDim.x;
  __shared__ double sh[3 * 32];
  __shared__ double slot[2][4];
  __shared__ double bc[4];
  __shared__ MgLevel s_lv[kMgMaxLevels];
  extern __shared__ float mgc_smem[];
  int par = 0;
  const unsigned n = (unsigned)P.A.n, ny = (unsigned)P.A.ny;
  const double bnorm = P.R[kDcAbs];
  const int cap = max(1, P.max_it - (int)P.R[kDcTotal]);
  for (unsigned t = gt; t < n; t += GT) P.r[t] = P.b[t];
  mgc_sync();
  double rz_old = 0.0;
  int it = 0;
  for (;;) {
    if (P.vcycles == 2) {
      mgc_vcycle(*P.ch, P.bottom, mgc_smem, s_lv, P.r, P.tmp, gt, GT);
      mgc_vcycle(*P.ch, P.bottom, mgc_smem, s_lv, P.tmp, P.z, gt, GT);
    } else {
      mgc_vcycle(*P.ch, P.bottom, mgc_smem, s_lv, P.r, P.z, gt, GT);
    }
    double v3[3] = {0.0, 0.0, 0.0};
    for (unsigned t = gt; t < n; t += GT) {
      const double z = P.z[t], r = P.r[t];
      v3[0] += r * z;
      v3[1] += z;
      v3[2] += r;
    }
    mgc_sum<3>(v3, sh, slot, bc, par);
    const double mz = P.project ? v3[1] / (double)n : 0.0;
    const double rz = P.project ? v3[0] - mz * v3[2] : v3[0];
    bool bad = !(rz > 0.0) || !isfinite(rz);
    const float beta = it == 0 ? 0.0f : (float)(rz / rz_old), fmz = (float)mz;
    rz_old = rz;
    for (unsigned t = gt; t < n; t += GT) P.p[t] = it == 0 ? P.z[t] - fmz : (P.z[t] - fmz) + beta * P.p[t];
    mgc_sync();
    double v1[1] = {0.0};
    for (unsigned t = gt; t < n; t += GT) {
      const int i = (int)(t / ny), j = (int)(t - (unsigned)i * ny);
      const float s = spmv_row<S>(P.A, P.p, i, j);
      P.q[t] = s;
      v1[0] += (double)P.p[t] * (double)s;
    }
    mgc_sum<1>(v1, sh, slot, bc, par);
    if (!(v1[0] > 0.0) || !isfinite(v1[0])) bad = true;
    const float alpha = (float)(rz / v1[0]);
    double v2[1] = {0.0};
    for (unsigned t = gt; t < n; t += GT) {
      P.x[t] += alpha * P.p[t];
      const float r = P.r[t] - alpha * P.q[t];
      P.r[t] = r;
      v2[0] += (double)r * (double)r;
    }
    mgc_sum<1>(v2, sh, slot, bc, par);
    ++it;
    // std::max semantics, as k_mgcg_ctrl: a NaN ends the solve
    const double rr = v2[0], rel = sqrt(rr < 0.0 ? 0.0 : rr) / (bnorm < 1.0e-300 ? 1.0e-300 : bnorm);
    if (bad || !(rel >= P.tol) || it >= cap) break;
  }
  if (gt == 0) {
    P.R[kDcTotal] += (double)it;
    P.R[kDcMgIts] += (double)it;
  }
  mgc_sync();  // no CTA leaves while another may still read its shared memory
}

}  // namespace dn
