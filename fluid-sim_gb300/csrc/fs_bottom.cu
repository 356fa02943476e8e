// fs_bottom.cu -- the bottom of the multigrid V-cycle: every level of at most
// 64 cells a side in one CTA, in shared memory, the coarse sweeps included
// (src/gpu/multigrid.js:277-330, RBGS(40) on the coarsest level).
//
// What bounds it is the chain of dependent phases: a half-sweep cannot start
// before the one ahead of it has handed on its cells, and one V(2,2) cycle has
// 24 half-sweeps on the levels above the coarsest (64 -> 8) and 80 on it.  So
// the level with most cells and the one-warp levels keep them in registers
// and hand them on by shuffles; the levels between stay in shared memory.
#include <algorithm>
#include <string>

#include "fs_async.cuh"
#include "fs_df.cuh"
#include "fs_internal.cuh"
#include "fs_stencil.cuh"

namespace fs {

// ---------------------------------------------------------------- bottom
// Levels 0..count-1 of the bottom (each n <= 64), all in shared memory.  Per
// level: x, rhs and, for odd n, a ping-pong partner (red-black on an odd
// periodic grid reads cells of its own colour across the wrap, so the
// reference's ping-pong result is kept).
struct BottomLevels {
  int count;
  int n[8];
  float h2[8];
  int off_x[8], off_x2[8], off_r[8];  // float offsets into dynamic smem (-1: none)
  float w;                            // relaxation factor of every sweep
};

// A thread group: the whole CTA, or warp 0 alone (levels <= 16).
struct Group {
  int tid, nthr;
  bool warp;
  __device__ __forceinline__ void sync() const {
    if (warp) __syncwarp();
    else __syncthreads();
  }
};

__device__ __forceinline__ void bottom_smooth(float* sm, const BottomLevels& L, int l, int sweeps, Group G) {
  const int n = L.n[l];
  const float h2 = L.h2[l];
  float* x = sm + L.off_x[l];
  float* x2 = (n & 1) ? sm + L.off_x2[l] : nullptr;
  const float* r = sm + L.off_r[l];
  for (int s = 0; s < 2 * sweeps; s++) {
    const int c = s & 1;
    if (!(n & 1)) {
      for (int k = G.tid; k < n * n; k += G.nthr) {
        int j = k / n, i = k - j * n;
        if (((i + j) & 1) != c) continue;
        int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
        int jm = j == 0 ? n - 1 : j - 1, jp = j + 1 == n ? 0 : j + 1;
        x[k] = gs_update(x[k], x[j * n + im], x[j * n + ip], x[jm * n + i], x[jp * n + i], r[k], h2, L.w);
      }
    } else {
      for (int k = G.tid; k < n * n; k += G.nthr) {
        int j = k / n, i = k - j * n;
        float cur = x[k];
        if (((i + j) & 1) != c) { x2[k] = cur; continue; }
        int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
        int jm = j == 0 ? n - 1 : j - 1, jp = j + 1 == n ? 0 : j + 1;
        x2[k] = gs_update(cur, x[j * n + im], x[j * n + ip], x[jm * n + i], x[jp * n + i], r[k], h2, L.w);
      }
      G.sync();
      float* t = x; x = x2; x2 = t;  // two swaps per sweep: x is back in off_x at the end
    }
    G.sync();
  }
}

__device__ __forceinline__ void bottom_restrict(float* sm, const BottomLevels& L, int l, Group G) {
  const int n = L.n[l], nc = L.n[l + 1];
  const float ih2 = inv_h2(L.h2[l]);
  const float* x = sm + L.off_x[l];
  const float* r = sm + L.off_r[l];
  float* cr = sm + L.off_r[l + 1];
  float* cx = sm + L.off_x[l + 1];
  for (int k = G.tid; k < nc * nc; k += G.nthr) {
    int cj = k / nc, ci = k - cj * nc;
    float r4[4];
    for (int q = 0; q < 4; q++) {
      int i = 2 * ci + (q & 1), j = 2 * cj + (q >> 1);
      int im = i == 0 ? n - 1 : i - 1, ip = i + 1 == n ? 0 : i + 1;
      int jm = j == 0 ? n - 1 : j - 1, jp = j + 1 == n ? 0 : j + 1;
      r4[q] = residual_at(x[j * n + i], x[j * n + im], x[j * n + ip], x[jm * n + i], x[jp * n + i], r[j * n + i], ih2);
    }
    cr[k] = restrict4(r4[0], r4[1], r4[2], r4[3]);
    cx[k] = 0.f;
  }
  G.sync();
}

__device__ __forceinline__ void bottom_prolong(float* sm, const BottomLevels& L, int l, Group G) {
  const int n = L.n[l], nc = L.n[l + 1];
  float* x = sm + L.off_x[l];
  const float* c = sm + L.off_x[l + 1];
  for (int k = G.tid; k < n * n; k += G.nthr) {
    int j = k / n, i = k - j * n;
    int ci0 = (i & 1) ? (i >> 1) : (i >> 1) - 1;
    int cj0 = (j & 1) ? (j >> 1) : (j >> 1) - 1;
    float fx = (i & 1) ? 0.25f : 0.75f, fy = (j & 1) ? 0.25f : 0.75f;
    int x0 = ci0 < 0 ? ci0 + nc : ci0, x1 = ci0 + 1 >= nc ? ci0 + 1 - nc : ci0 + 1;
    int y0 = cj0 < 0 ? cj0 + nc : cj0, y1 = cj0 + 1 >= nc ? cj0 + 1 - nc : cj0 + 1;
    x[k] = __fadd_rn(x[k], prolong_val(c[y0 * nc + x0], c[y0 * nc + x1], c[y1 * nc + x0], c[y1 * nc + x1], fx, fy));
  }
  G.sync();
}

__device__ __forceinline__ void mg_bottom_body(const float* __restrict__ rhs_top, float* __restrict__ x_top,
                                               int has_x, const BottomLevels& L, int pre, int post, int coarse,
                                               float* __restrict__ acc_h, float* __restrict__ acc_l) {
  extern __shared__ float sm[];
  const int tid = threadIdx.x;
  const Group CTA{tid, (int)blockDim.x, false};
  const Group W0{tid, 32, true};
  {
    // the top level's rhs (and iterate) by asynchronous copies, all in flight at once
    const int n = L.n[0];
    for (int k = tid; k < n * n; k += CTA.nthr) {
      cp_async4(&sm[L.off_r[0] + k], rhs_top + k);
      if (has_x) cp_async4(&sm[L.off_x[0] + k], x_top + k);
      else sm[L.off_x[0] + k] = 0.f;
    }
  }
  cp_async_wait_all();
  __syncthreads();
  // first level handled by warp 0 alone
  int ls = 0;
  while (ls < L.count && L.n[ls] > 16) ls++;
  if (ls >= L.count) {
    // every bottom level is a CTA level
    for (int l = 0; l < L.count - 1; l++) {
      bottom_smooth(sm, L, l, pre, CTA);
      bottom_restrict(sm, L, l, CTA);
    }
    bottom_smooth(sm, L, L.count - 1, coarse, CTA);
    for (int l = L.count - 2; l >= 0; l--) {
      bottom_prolong(sm, L, l, CTA);
      bottom_smooth(sm, L, l, post, CTA);
    }
  } else {
    for (int l = 0; l < ls; l++) {
      bottom_smooth(sm, L, l, pre, CTA);
      bottom_restrict(sm, L, l, CTA);
    }
    if (tid < 32) {
      for (int l = ls; l < L.count - 1; l++) {
        bottom_smooth(sm, L, l, pre, W0);
        bottom_restrict(sm, L, l, W0);
      }
      bottom_smooth(sm, L, L.count - 1, coarse, W0);
      for (int l = L.count - 2; l >= ls; l--) {
        bottom_prolong(sm, L, l, W0);
        bottom_smooth(sm, L, l, post, W0);
      }
    }
    __syncthreads();
    for (int l = ls - 1; l >= 0; l--) {
      bottom_prolong(sm, L, l, CTA);
      bottom_smooth(sm, L, l, post, CTA);
    }
  }
  {
    const int n = L.n[0];
    for (int k = tid; k < n * n; k += CTA.nthr) {
      float e = sm[L.off_x[0] + k];
      if (acc_h) {  // the whole hierarchy fits here: add the correction to the pressure
        df p = df_add_f(df{acc_h[k], acc_l[k]}, e);
        acc_h[k] = p.hi;
        acc_l[k] = p.lo;
      } else {
        x_top[k] = e;
      }
    }
  }
}

__global__ void __launch_bounds__(1024) k_mg_bottom(const float* rhs_top, float* x_top, int has_x,
                                                    BottomLevels L, int pre, int post, int coarse, float* acc_h,
                                                    float* acc_l) {
  pdl_wait();
  mg_bottom_body(rhs_top, x_top, has_x, L, pre, post, coarse, acc_h, acc_l);
}

// ------------------------------------------------ bottom, compile-time chains
// The bottom levels are N0, N0/2, ..., NMIN, every size but the coarsest even
// and N0 <= 64: the power-of-two chains down to 8 and the chains 4 b -> 2 b ->
// b of grids of b 2^k cells, b = 9 .. 15 -- all sizes known at compile time.
// Levels > 16 run on the whole CTA (256 threads), levels <= 16 -- including
// the coarse sweeps -- on warp 0 alone.  Same arithmetic (fs_stencil.cuh) and
// order as the generic kernel above.
struct BottomH2 {
  float h2[4];
  float w;  // relaxation factor of every sweep
};

// levels and floats of the chain N0, N0/2, ..., NMIN
template <int N0, int NMIN>
constexpr int chain_levels() {
  return N0 == NMIN ? 1 : 1 + chain_levels<N0 / 2, NMIN>();
}
template <int N0, int NMIN>
constexpr int chain_floats() {
  return N0 == NMIN ? N0 * N0 : N0 * N0 + chain_floats<N0 / 2, NMIN>();
}

constexpr int kBottomThreads = 256;  // threads of the bottom-chain kernels

template <int N, bool WARP>
__device__ __forceinline__ void p2_sync() {
  if (WARP) __syncwarp();
  else __syncthreads();
}

// The chain's loops run a compile-time number of cells per thread (the CTA
// has kBottomThreads threads, warp 0 has 32), fully unrolled, every result of
// a phase computed before any is stored: the cells a phase writes are not
// read in that phase (a colour's cells read only the other colour; restrict
// and prolong write the other level's array, or the cell itself), so the
// loads of a thread's cells are in flight together instead of waiting on the
// stores of the cells before them.  The levels are latency-bound, one phase
// between two barriers after another.
//
// How a phase's cells fall on the threads: COLS columns of ROWS rows, a thread
// per column and RS rows apart (RS even where a row's parity matters), so a
// thread's cells share their column and the offsets of its neighbours, and
// only the first and last rows of the level wrap.  Threads beyond RS * COLS
// idle; the last row of a thread may lie beyond the level.
template <int COLS, int ROWS, bool WARP, bool EVEN>
struct P2Map {
  static constexpr int NT = WARP ? 32 : kBottomThreads;
  static constexpr int FIT = EVEN ? (NT / COLS) & ~1 : NT / COLS;
  static constexpr int RS = FIT < ROWS ? FIT : ROWS;
  static constexpr int PER = (ROWS + RS - 1) / RS;
  static_assert(RS > 0 && (!EVEN || RS % 2 == 0 || RS == ROWS), "a level too wide for its threads");
  // row u of a thread whose first is j0 may lie beyond the level
  static __device__ __forceinline__ bool in(int j0, int u) {
    return (RS * COLS == NT || j0 < RS) && (ROWS % RS == 0 || j0 + u * RS < ROWS);
  }
};

// one red-black half-sweep of colour C on an even level
template <int N, bool WARP, int C>
__device__ __forceinline__ void p2_half(float* x, const float* r, float h2, float w, int j0, int m) {
  using M = P2Map<N / 2, N, WARP, true>;
  const int i = 2 * m + ((j0 + C) & 1);
  const int dl = i == 0 ? N - 1 : -1, dr = i + 1 == N ? 1 - N : 1;
  float nv[M::PER];
#pragma unroll
  for (int u = 0; u < M::PER; u++) {
    const int j = j0 + u * M::RS, k = j * N + i;
    if (!M::in(j0, u)) continue;
    const int db = j == 0 ? (N - 1) * N : -N, dt = j + 1 == N ? -(N - 1) * N : N;
    nv[u] = gs_update(x[k], x[k + dl], x[k + dr], x[k + db], x[k + dt], r[k], h2, w);
  }
#pragma unroll
  for (int u = 0; u < M::PER; u++)
    if (M::in(j0, u)) x[(j0 + u * M::RS) * N + i] = nv[u];
  p2_sync<N, WARP>();
}

// Sweeps of an odd level (the coarsest, one warp).  On an odd periodic grid
// cells of one colour are neighbours across the wrap and read each other's
// value from before the half-sweep (the reference's ping-pong pass), so every
// load comes before any store.  With N odd, (i + j) and j N + i have the same
// parity: colour c is the cells 2 t + c.  A lane's cells and their neighbours
// are the same in every sweep: its own values, their right-hand sides and the
// neighbours' offsets stay in registers, only the neighbours' values go
// through shared memory.
template <int N>
__device__ __forceinline__ void p2_smooth_odd(float* x, const float* r, float h2, int sweeps, float w) {
  constexpr int PER = ((N * N + 1) / 2 + 31) / 32;
  const int lane = threadIdx.x & 31;
  const float *nl[2][PER], *nr[2][PER], *nb[2][PER], *nt[2][PER];
  float *out[2][PER], v[2][PER], q[2][PER];
#pragma unroll
  for (int c = 0; c < 2; c++)
#pragma unroll
    for (int u = 0; u < PER; u++) {
      const int t = 2 * (lane + 32 * u) + c;
      const int e = t < N * N ? t : 0, j = e / N, i = e - j * N;
      out[c][u] = t < N * N ? x + e : nullptr;
      nl[c][u] = x + j * N + (i == 0 ? N - 1 : i - 1);
      nr[c][u] = x + j * N + (i + 1 == N ? 0 : i + 1);
      nb[c][u] = x + (j == 0 ? N - 1 : j - 1) * N + i;
      nt[c][u] = x + (j + 1 == N ? 0 : j + 1) * N + i;
      v[c][u] = x[e];
      q[c][u] = r[e];
    }
  for (int s = 0; s < sweeps; s++)
#pragma unroll
    for (int c = 0; c < 2; c++) {
#pragma unroll
      for (int u = 0; u < PER; u++)
        v[c][u] = gs_update(v[c][u], *nl[c][u], *nr[c][u], *nb[c][u], *nt[c][u], q[c][u], h2, w);
      __syncwarp();
#pragma unroll
      for (int u = 0; u < PER; u++)
        if (out[c][u]) *out[c][u] = v[c][u];
      __syncwarp();
    }
}

// Sweeps of the 8 x 8 level on one warp, in registers: a lane holds the two
// cells of row lane / 4 and columns 2 (lane % 4), + 1, one of each colour; the
// other colour's neighbours are its own other cell and three lanes' (the lane
// to the left or right, the rows below and above).  A half-sweep is a chain
// of a shuffle and the update instead of a store, a warp barrier and a load.
__device__ __forceinline__ void p2_smooth8(float* x, const float* r, float h2, int sweeps, float w) {
  const int lane = threadIdx.x & 31, j = lane >> 2, m = lane & 3, odd = j & 1;
  float* const cell = x + 2 * lane;  // row j starts at 8 j = 2 (4 j)
  float red = cell[odd], black = cell[1 - odd];
  const float rr = r[2 * lane + odd], rb = r[2 * lane + 1 - odd];
  const int below = (lane + 28) & 31, above = (lane + 4) & 31;
  // an even row's red cell is on the left: its left neighbour is the black
  // cell of the lane to the left, its right one the lane's own; odd rows and
  // black cells the other way round
  const int left = (lane & 28) | ((m + 3) & 3), right = (lane & 28) | ((m + 1) & 3);
  const int side_r = odd ? right : left, side_b = odd ? left : right;
  for (int s = 0; s < sweeps; s++) {
    float n = __shfl_sync(0xffffffffu, black, side_r);
    float b = __shfl_sync(0xffffffffu, black, below), t = __shfl_sync(0xffffffffu, black, above);
    red = gs_update(red, odd ? black : n, odd ? n : black, b, t, rr, h2, w);
    n = __shfl_sync(0xffffffffu, red, side_b);
    b = __shfl_sync(0xffffffffu, red, below);
    t = __shfl_sync(0xffffffffu, red, above);
    black = gs_update(black, odd ? n : red, odd ? red : n, b, t, rb, h2, w);
  }
  cell[odd] = red;
  cell[1 - odd] = black;
  __syncwarp();
}

// The update of one colour of a column held in registers (p2_smooth_cols): a[t]
// at rows 2 t + pr, its vertical neighbours b at rows 2 t + 1 - pr (e: the one
// beyond the lane's rows), its horizontal ones the b[t] of the lanes left and
// right.
template <int T, bool SPLIT>
__device__ __forceinline__ void p2_column_half(float (&a)[T], const float (&b)[T], const float (&q)[T], int pr,
                                               int left, int right, float h2, float w) {
  float e = pr ? b[0] : b[T - 1];
  if (SPLIT) e = __shfl_xor_sync(0xffffffffu, e, 16);
#pragma unroll
  for (int t = 0; t < T; t++) {
    const float l = __shfl_sync(0xffffffffu, b[t], left), r = __shfl_sync(0xffffffffu, b[t], right);
    const float below = pr ? b[t] : (t > 0 ? b[t > 0 ? t - 1 : 0] : e);
    const float above = pr ? (t < T - 1 ? b[t < T - 1 ? t + 1 : 0] : e) : b[t];
    a[t] = gs_update(a[t], l, r, below, above, q[t], h2, w);
  }
}

// Sweeps of an even level of at most 16 cells on one warp, in registers: a
// lane holds a column (N = 10, 14), or half of one (N = 12, 16: lanes 0 .. 15
// the lower rows), each colour in an array of its own.
template <int N>
__device__ __forceinline__ void p2_smooth_cols(float* x, const float* r, float h2, int sweeps, float w) {
  constexpr bool SPLIT = N % 4 == 0;
  constexpr int ROWS = SPLIT ? N / 2 : N, T = ROWS / 2;
  static_assert(N <= 16 && N % 2 == 0 && ROWS % 2 == 0, "an even number of rows per lane");
  const int lane = threadIdx.x & 31, half = SPLIT ? lane >> 4 : 0, lc = SPLIT ? lane & 15 : lane;
  const bool act = lc < N;
  const int col = act ? lc : 0, par = col & 1;  // colour 0 is on rows of the column's parity
  const int left = 16 * half + (col == 0 ? N - 1 : col - 1), right = 16 * half + (col + 1 == N ? 0 : col + 1);
  float* const p = x + half * ROWS * N + col;
  const float* const d = r + half * ROWS * N + col;
  float c0[T], c1[T], q0[T], q1[T];
#pragma unroll
  for (int t = 0; t < T; t++) {
    c0[t] = p[(2 * t + par) * N];
    c1[t] = p[(2 * t + 1 - par) * N];
    q0[t] = d[(2 * t + par) * N];
    q1[t] = d[(2 * t + 1 - par) * N];
  }
  for (int s = 0; s < sweeps; s++) {
    p2_column_half<T, SPLIT>(c0, c1, q0, par, left, right, h2, w);
    p2_column_half<T, SPLIT>(c1, c0, q1, 1 - par, left, right, h2, w);
  }
  __syncwarp();
  if (act) {
#pragma unroll
    for (int t = 0; t < T; t++) {
      p[(2 * t + par) * N] = c0[t];
      p[(2 * t + 1 - par) * N] = c1[t];
    }
  }
  __syncwarp();
}

template <int N, bool WARP>
__device__ __forceinline__ void p2_smooth(float* x, const float* r, float h2, int sweeps, float w) {
  if constexpr (N % 2 == 1) {
    static_assert(WARP, "an odd level is the coarsest, on one warp");
    p2_smooth_odd<N>(x, r, h2, sweeps, w);
  } else if constexpr (N == 8) {
    static_assert(WARP, "8 x 8 on one warp");
    p2_smooth8(x, r, h2, sweeps, w);
  } else if constexpr (WARP) {
    p2_smooth_cols<N>(x, r, h2, sweeps, w);
  } else {
    const int tid = WARP ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
    const int j0 = tid / (N / 2), m = tid - j0 * (N / 2);
    for (int s = 0; s < sweeps; s++) {
      p2_half<N, WARP, 0>(x, r, h2, w, j0, m);
      p2_half<N, WARP, 1>(x, r, h2, w, j0, m);
    }
  }
}

// residual of level N restricted into (cr, cx = 0) of level N/2
template <int N, bool WARP>
__device__ __forceinline__ void p2_restrict(const float* x, const float* r, float h2, float* cr, float* cx) {
  constexpr int NC = N / 2;
  using M = P2Map<NC, NC, WARP, false>;
  const int tid = WARP ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const float ih2 = inv_h2(h2);
  const int cj0 = tid / NC, ci = tid - cj0 * NC;
  const int i0 = 2 * ci;
  const int dl0 = i0 == 0 ? N - 1 : -1, dr1 = i0 + 2 == N ? 1 - N : 1;  // left of column i0, right of i0 + 1
  float rv[M::PER];
#pragma unroll
  for (int u = 0; u < M::PER; u++) {
    if (!M::in(cj0, u)) continue;
    const int j = 2 * (cj0 + u * M::RS), k0 = j * N + i0, k1 = k0 + N;
    const int db = j == 0 ? (N - 1) * N : -N, dt = j + 2 == N ? -(N - 1) * N : N;  // below row j, above row j + 1
    const float r00 = residual_at(x[k0], x[k0 + dl0], x[k0 + 1], x[k0 + db], x[k1], r[k0], ih2);
    const float r10 = residual_at(x[k0 + 1], x[k0], x[k0 + 1 + dr1], x[k0 + 1 + db], x[k1 + 1], r[k0 + 1], ih2);
    const float r01 = residual_at(x[k1], x[k1 + dl0], x[k1 + 1], x[k0], x[k1 + dt], r[k1], ih2);
    const float r11 = residual_at(x[k1 + 1], x[k1], x[k1 + 1 + dr1], x[k0 + 1], x[k1 + 1 + dt], r[k1 + 1], ih2);
    rv[u] = restrict4(r00, r10, r01, r11);
  }
#pragma unroll
  for (int u = 0; u < M::PER; u++) {
    if (!M::in(cj0, u)) continue;
    const int k = (cj0 + u * M::RS) * NC + ci;
    cr[k] = rv[u];
    cx[k] = 0.f;
  }
  p2_sync<N, WARP>();
}

// x (level N) += bilinear prolongation of c (level N/2)
template <int N, bool WARP>
__device__ __forceinline__ void p2_prolong(float* x, const float* c) {
  constexpr int NC = N / 2;
  using M = P2Map<N, N, WARP, true>;  // a thread's rows share their parity: both weights are fixed
  const int tid = WARP ? (int)(threadIdx.x & 31) : (int)threadIdx.x;
  const int j0 = tid / N, i = tid - j0 * N;
  const int ci0 = (i & 1) ? (i >> 1) : (i >> 1) - 1;
  const float fx = (i & 1) ? 0.25f : 0.75f, fy = (j0 & 1) ? 0.25f : 0.75f;
  const int x0 = ci0 < 0 ? ci0 + NC : ci0, x1 = ci0 + 1 >= NC ? ci0 + 1 - NC : ci0 + 1;
  float pv[M::PER];
#pragma unroll
  for (int u = 0; u < M::PER; u++) {
    if (!M::in(j0, u)) continue;
    const int j = j0 + u * M::RS, k = j * N + i;
    const int cj0 = (j & 1) ? (j >> 1) : (j >> 1) - 1;
    const int y0 = (cj0 < 0 ? cj0 + NC : cj0) * NC, y1 = (cj0 + 1 >= NC ? cj0 + 1 - NC : cj0 + 1) * NC;
    pv[u] = __fadd_rn(x[k], prolong_val(c[y0 + x0], c[y0 + x1], c[y1 + x0], c[y1 + x1], fx, fy));
  }
#pragma unroll
  for (int u = 0; u < M::PER; u++)
    if (M::in(j0, u)) x[(j0 + u * M::RS) * N + i] = pv[u];
  p2_sync<N, WARP>();
}

// sub-cycle from level N (chain level LVL, at float offset OFF of the chain's
// x and rhs arrays) down to NMIN and back; levels <= 16 are called by warp 0
// only.  Every level's arrays are the shared arrays plus a compile-time
// offset, so all accesses compile as shared-memory accesses.
template <int N, int NMIN, int LVL, int OFF>
__device__ __forceinline__ void p2_cycle(float* sx, float* sr, const BottomH2& H, int pre, int post, int coarse) {
  constexpr bool W = N <= 16;
  float* const x = sx + OFF;
  float* const r = sr + OFF;
  if constexpr (N == NMIN) {
    p2_smooth<N, W>(x, r, H.h2[LVL], coarse, H.w);
  } else {
    static_assert(N % 2 == 0, "every level above the coarsest is even");
    constexpr int OFFC = OFF + N * N;
    p2_smooth<N, W>(x, r, H.h2[LVL], pre, H.w);
    p2_restrict<N, W>(x, r, H.h2[LVL], sr + OFFC, sx + OFFC);
    if constexpr (!W && N / 2 <= 16) {
      if (threadIdx.x < 32) p2_cycle<N / 2, NMIN, LVL + 1, OFFC>(sx, sr, H, pre, post, coarse);
      __syncthreads();
    } else {
      p2_cycle<N / 2, NMIN, LVL + 1, OFFC>(sx, sr, H, pre, post, coarse);
    }
    p2_prolong<N, W>(x, sx + OFFC);
    p2_smooth<N, W>(x, r, H.h2[LVL], post, H.w);
  }
}

// ------------------------------------------ the chain's top level in registers
// The top level (36 .. 64 cells) holds most of the bottom's cells; in shared
// memory its half-sweeps are bound by bank conflicts (a colour's cells are two
// words apart) and take ~800 cycles each at 64 x 64.  Here a warp owns RPW
// rows, a lane two columns of them: a half-sweep takes one shuffle per row
// and the neighbouring warps' edge rows from shared memory (two buffers, one
// barrier).  One solve with 40 coarse sweeps, timed by an event pair (~4 us of
// which the events take): 64 -> 8 16.2 -> 12.3 us and 48 -> 12 24.2 -> 12.7 us
// with the top level and the one-warp levels in registers; 36 -> 9, which the
// generic kernel ran, 60.4 -> 12.4 us.
template <int N>
struct Top {
  static constexpr int RPW = N > 48 ? 8 : 6;              // rows per warp, even
  static constexpr int NW = (N + RPW - 1) / RPW;          // warps that hold rows
  static constexpr int LAST = N - (NW - 1) * RPW;         // rows of the last of them
  static constexpr int LANES = N / 2;
  static_assert(N % 2 == 0 && LANES <= 32 && LAST % 2 == 0 && LAST > 0 && NW <= kBottomThreads / 32, "top level");
  typedef float2 Edge[2][NW][2][LANES];  // [buffer][warp][first, last row]

  float x[RPW][2], r[RPW][2];
  int lane, warp, left, right;  // lanes of the columns left and right (wrapped)
  bool last, act;
  int buf;

  __device__ __forceinline__ Top() {
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    last = warp == NW - 1;
    act = warp < NW && lane < LANES;
    left = lane == 0 ? LANES - 1 : lane - 1;
    right = lane + 1 >= LANES ? 0 : lane + 1;
    buf = 0;
  }
  // whether row k of this warp is one of the level's
  __device__ __forceinline__ bool row(int k) const { return k < LAST || !last; }

  // the rows below and above this warp's
  __device__ __forceinline__ void exchange(Edge& e, float (&below)[2], float (&above)[2]) {
    if (act) {
      e[buf][warp][0][lane] = make_float2(x[0][0], x[0][1]);
      e[buf][warp][1][lane] =
          last ? make_float2(x[LAST - 1][0], x[LAST - 1][1]) : make_float2(x[RPW - 1][0], x[RPW - 1][1]);
    }
    __syncthreads();
    float2 b = make_float2(0.f, 0.f), a = b;
    if (act) {
      b = e[buf][warp == 0 ? NW - 1 : warp - 1][1][lane];
      a = e[buf][last ? 0 : warp + 1][0][lane];
    }
    below[0] = b.x, below[1] = b.y;
    above[0] = a.x, above[1] = a.y;
    buf ^= 1;
  }
  // the value above row k of column c
  __device__ __forceinline__ float up(int k, int c, const float (&above)[2]) const {
    if (k == RPW - 1) return above[c];
    if (k == LAST - 1) return last ? above[c] : x[k + 1][c];
    return x[k + 1][c];
  }

  // colour C: the cells of row k and column c with (k + c) & 1 == C (every
  // warp's first row and every lane's first column are even)
  template <int C>
  __device__ __forceinline__ void half(Edge& e, float h2, float w) {
    float below[2], above[2];
    exchange(e, below, above);
#pragma unroll
    for (int k = 0; k < RPW; k++) {
      if (!row(k)) break;
      const int c = (k + C) & 1;
      const float side = __shfl_sync(0xffffffffu, x[k][1 - c], c == 0 ? left : right);
      const float l = c == 0 ? side : x[k][0], t = c == 0 ? x[k][1] : side;
      x[k][c] = gs_update(x[k][c], l, t, k > 0 ? x[k > 0 ? k - 1 : 0][c] : below[c], up(k, c, above), r[k][c], h2, w);
    }
  }
  __device__ __forceinline__ void smooth(Edge& e, float h2, int sweeps, float w) {
    for (int s = 0; s < sweeps; s++) {
      half<0>(e, h2, w);
      half<1>(e, h2, w);
    }
  }

  // the residual restricted into (cr, cx = 0) of the next level
  __device__ __forceinline__ void restrict_to(Edge& e, float h2, float* cr, float* cx) {
    float below[2], above[2];
    exchange(e, below, above);
    const float ih2 = inv_h2(h2);
#pragma unroll
    for (int k = 0; k < RPW; k += 2) {
      if (!row(k)) break;
      const float l0 = __shfl_sync(0xffffffffu, x[k][1], left), t0 = __shfl_sync(0xffffffffu, x[k][0], right);
      const float l1 = __shfl_sync(0xffffffffu, x[k + 1][1], left), t1 = __shfl_sync(0xffffffffu, x[k + 1][0], right);
      const float b0 = k > 0 ? x[k > 0 ? k - 1 : 0][0] : below[0], b1 = k > 0 ? x[k > 0 ? k - 1 : 0][1] : below[1];
      const float r00 = residual_at(x[k][0], l0, x[k][1], b0, x[k + 1][0], r[k][0], ih2);
      const float r10 = residual_at(x[k][1], x[k][0], t0, b1, x[k + 1][1], r[k][1], ih2);
      const float r01 = residual_at(x[k + 1][0], l1, x[k + 1][1], x[k][0], up(k + 1, 0, above), r[k + 1][0], ih2);
      const float r11 = residual_at(x[k + 1][1], x[k + 1][0], t1, x[k][1], up(k + 1, 1, above), r[k + 1][1], ih2);
      if (act) {
        const int q = (warp * (RPW / 2) + k / 2) * LANES + lane;
        cr[q] = restrict4(r00, r10, r01, r11);
        cx[q] = 0.f;
      }
    }
    __syncthreads();
  }

  // x += bilinear prolongation of the next level's c
  __device__ __forceinline__ void prolong(const float* c) {
    if (!act) return;
    const int j0 = warp * (RPW / 2);
    float b[3], m[3];  // the coarse rows below and of the current pair of fine rows
    auto load = [&](int j, float (&v)[3]) {
      const float* q = c + (j < 0 ? LANES - 1 : j >= LANES ? 0 : j) * LANES;
      v[0] = q[left], v[1] = q[lane], v[2] = q[right];
    };
    load(j0 - 1, b);
    load(j0, m);
#pragma unroll
    for (int k = 0; k < RPW; k += 2) {
      if (!row(k)) break;
      float t[3];
      load(j0 + k / 2 + 1, t);
      x[k][0] = __fadd_rn(x[k][0], prolong_val(b[0], b[1], m[0], m[1], 0.75f, 0.75f));
      x[k][1] = __fadd_rn(x[k][1], prolong_val(b[1], b[2], m[1], m[2], 0.25f, 0.75f));
      x[k + 1][0] = __fadd_rn(x[k + 1][0], prolong_val(m[0], m[1], t[0], t[1], 0.75f, 0.25f));
      x[k + 1][1] = __fadd_rn(x[k + 1][1], prolong_val(m[1], m[2], t[1], t[2], 0.25f, 0.25f));
#pragma unroll
      for (int q = 0; q < 3; q++) b[q] = m[q], m[q] = t[q];
    }
  }
};

// x_top (the level's iterate, read if has_x) or, with acc_h, the double-float
// pressure takes the result
template <int N0, int NMIN>
__device__ __forceinline__ void mg_bottom_chain_body(const float* __restrict__ rhs_top, float* __restrict__ x_top,
                                                     int has_x, const BottomH2& H, int pre, int post, int coarse,
                                                     float* __restrict__ acc_h, float* __restrict__ acc_l) {
  constexpr int L = chain_levels<N0, NMIN>();
  static_assert(L <= 4, "chains of at most four levels");
  const int tid = threadIdx.x;
  if constexpr (N0 > 32) {
    // the levels below the top, one after another
    constexpr int SZ = chain_floats<N0 / 2, NMIN>();
    __shared__ float sx[SZ];
    __shared__ float sr[SZ];
    __shared__ typename Top<N0>::Edge edge;
    Top<N0> top;
    const int64_t at = (int64_t)top.warp * Top<N0>::RPW * N0 + 2 * top.lane;  // the level arrays are 8-byte aligned
#pragma unroll
    for (int k = 0; k < Top<N0>::RPW; k++) {
      const bool in = top.act && top.row(k);
      const float2 z = make_float2(0.f, 0.f);
      const float2 rv = in ? *reinterpret_cast<const float2*>(rhs_top + at + k * N0) : z;
      const float2 xv = in && has_x ? *reinterpret_cast<const float2*>(x_top + at + k * N0) : z;
      top.r[k][0] = rv.x, top.r[k][1] = rv.y;
      top.x[k][0] = xv.x, top.x[k][1] = xv.y;
    }
    top.smooth(edge, H.h2[0], pre, H.w);
    top.restrict_to(edge, H.h2[0], sr, sx);
    p2_cycle<N0 / 2, NMIN, 1, 0>(sx, sr, H, pre, post, coarse);
    top.prolong(sx);
    top.smooth(edge, H.h2[0], post, H.w);
    float* const out = acc_h ? acc_h : x_top;
#pragma unroll
    for (int k = 0; k < Top<N0>::RPW; k++) {
      if (!top.act || !top.row(k)) continue;
      float2* const o = reinterpret_cast<float2*>(out + at + k * N0);
      if (acc_h) {
        float2* const lo = reinterpret_cast<float2*>(acc_l + at + k * N0);
        const float2 hv = *o, lv = *lo;
        const df p0 = df_add_f(df{hv.x, lv.x}, top.x[k][0]), p1 = df_add_f(df{hv.y, lv.y}, top.x[k][1]);
        *o = make_float2(p0.hi, p1.hi);
        *lo = make_float2(p0.lo, p1.lo);
      } else {
        *o = make_float2(top.x[k][0], top.x[k][1]);
      }
    }
  } else {
    constexpr int SZ = chain_floats<N0, NMIN>();
    __shared__ float sx[SZ];
    __shared__ float sr[SZ];
    for (int k = tid; k < N0 * N0; k += blockDim.x) {
      sr[k] = rhs_top[k];
      sx[k] = has_x ? x_top[k] : 0.f;
    }
    __syncthreads();
    if constexpr (N0 <= 16) {
      if (tid < 32) p2_cycle<N0, NMIN, 0, 0>(sx, sr, H, pre, post, coarse);
      __syncthreads();
    } else {
      p2_cycle<N0, NMIN, 0, 0>(sx, sr, H, pre, post, coarse);
    }
    for (int k = tid; k < N0 * N0; k += blockDim.x) {
      const float e = sx[k];
      if (acc_h) {
        const df p = df_add_f(df{acc_h[k], acc_l[k]}, e);
        acc_h[k] = p.hi;
        acc_l[k] = p.lo;
      } else {
        x_top[k] = e;
      }
    }
  }
}

template <int N0, int NMIN>
__global__ void __launch_bounds__(kBottomThreads)
    k_mg_bottom_chain(const float* rhs_top, float* x_top, int has_x, BottomH2 H, int pre, int post, int coarse,
                      float* acc_h, float* acc_l) {
  pdl_wait();
  mg_bottom_chain_body<N0, NMIN>(rhs_top, x_top, has_x, H, pre, post, coarse, acc_h, acc_l);
}

// ------------------------------------------------- batched (one size class)
// whether a class member still runs cycles (the class-wide loop kernel keeps
// the per-member condition in its DevState)
__device__ __forceinline__ bool member_active(const DevState* st, int max_cycles) {
  return !st->converged && !st->nonfinite && st->cycles < max_cycles;
}

struct BottomTab {
  struct {
    const float* rhs;
    float* x;
    float* acc_h;
    float* acc_l;
    const DevState* st;
  } m[kClassMax];
};

template <int N0, int NMIN>
__global__ void __launch_bounds__(kBottomThreads)
    k_mg_bottom_chain_class(const BottomTab tab, BottomH2 H, int pre, int post, int coarse, int max_cycles) {
  pdl_wait();
  const auto& a = tab.m[blockIdx.z];
  if (!member_active(a.st, max_cycles)) return;
  mg_bottom_chain_body<N0, NMIN>(a.rhs, a.x, 0, H, pre, post, coarse, a.acc_h, a.acc_l);
}

__global__ void __launch_bounds__(1024) k_mg_bottom_class(const BottomTab tab, BottomLevels L, int pre, int post,
                                                          int coarse, int max_cycles) {
  pdl_wait();
  const auto& a = tab.m[blockIdx.z];
  if (!member_active(a.st, max_cycles)) return;
  mg_bottom_body(a.rhs, a.x, 0, L, pre, post, coarse, a.acc_h, a.acc_l);
}

// ------------------------------------------------------------------ host
// first level of the bottom solve: every level from there down is <= 64
int bottom_first_level(const Solver* s) {
  int nl = (int)s->lev.size();
  int lb = nl - 1;
  while (lb > 0 && s->lev[lb - 1].n <= 64 && nl - (lb - 1) <= 8) lb--;
  return lb;
}

static size_t bottom_layout(const Solver* s, BottomLevels* B) {
  int lb = bottom_first_level(s);
  int nl = (int)s->lev.size();
  B->count = nl - lb;
  B->w = (float)s->prm.relax;
  int off = 0;
  for (int k = 0; k < B->count; k++) {
    const Level& L = s->lev[lb + k];
    int m = L.n * L.n;
    B->n[k] = L.n;
    B->h2[k] = L.h2;
    B->off_x[k] = off; off += m;
    B->off_r[k] = off; off += m;
    if (L.n & 1) { B->off_x2[k] = off; off += m; }
    else B->off_x2[k] = -1;
  }
  // levels <= 64 hold at most 2 * (64^2 + 32^2 + ...) + 15^2 floats < 48 KB
  return (size_t)off * sizeof(float);
}

// The compile-time chain kernel for the bottom levels from lb, identified by
// its first size (64, 32, 16, 8 down to 8; 4 b, 2 b, b for b = 9 .. 15; 24, 12
// down to 12), or 0 when the levels form another chain (another coarsest size,
// set by mg_min_size, or a grid below 64 cells a side).
static int bottom_chain(const Solver* s, int lb) {
  const std::vector<Level>& L = s->lev;
  for (size_t k = lb; k + 1 < L.size(); k++)
    if ((L[k].n & 1) || L[k + 1].n * 2 != L[k].n) return 0;
  const int nb = L[lb].n, nmin = L.back().n;
  if (nmin == 8 && (nb == 64 || nb == 32 || nb == 16 || nb == 8)) return nb;
  if (nmin == 12 && (nb == 24 || nb == 12)) return nb;
  if (nmin >= 9 && nmin <= 15 && nb == 4 * nmin) return nb;
  return 0;
}

// the chains bottom_chain can return, as cases of a switch
#define FS_CHAINS(CASE)                                                                        \
  CASE(64, 8) CASE(32, 8) CASE(16, 8) CASE(8, 8) CASE(36, 9) CASE(40, 10) CASE(44, 11)         \
  CASE(48, 12) CASE(24, 12) CASE(12, 12) CASE(52, 13) CASE(56, 14) CASE(60, 15)

static BottomH2 bottom_h2(const Solver* s, int lb) {
  BottomH2 H{};
  for (int k = 0; k < (int)s->lev.size() - lb && k < 4; k++) H.h2[k] = s->lev[lb + k].h2;
  H.w = (float)s->prm.relax;
  return H;
}

void launch_bottom(Solver* s, int lb, bool hx, float* acc_h, float* acc_l) {
  const std::vector<Level>& L = s->lev;
  const fs_params& P = s->prm;
  const int nb = L[lb].n;
  const double bytes = (double)nb * nb * (hx ? 12.0 : 8.0);
  const BottomH2 H = bottom_h2(s, lb);
  switch (bottom_chain(s, lb)) {
#define FS_CASE(N0, NM)                                                                                        \
  case N0:                                                                                                     \
    FS_LAUNCH(s, "mg_bottom", bytes,                                                                           \
              launch_dependent(true, k_mg_bottom_chain<N0, NM>, dim3(1), dim3(kBottomThreads), 0, s->stream,   \
                               L[lb].rhs, L[lb].x, hx ? 1 : 0, H, P.mg_pre_smooth, P.mg_post_smooth,           \
                               P.mg_coarse_sweeps, acc_h, acc_l));                                             \
    return;
    FS_CHAINS(FS_CASE)
#undef FS_CASE
  }
  BottomLevels B;
  const size_t smem = bottom_layout(s, &B);
  const int threads = std::min(1024, std::max(32, ((nb * nb / 4 + 31) / 32) * 32));
  FS_LAUNCH(s, "mg_bottom", bytes,
            launch_dependent(true, k_mg_bottom, dim3(1), dim3(threads), smem, s->stream, L[lb].rhs, L[lb].x,
                             hx ? 1 : 0, B, P.mg_pre_smooth, P.mg_post_smooth, P.mg_coarse_sweeps, acc_h, acc_l));
}

void launch_bottom_class(Solver* const* ms, int count, int lb, cudaStream_t st) {
  const Solver* s0 = ms[0];
  const fs_params& P = s0->prm;
  const int nb = s0->lev[lb].n;
  BottomTab tab{};
  for (int i = 0; i < count; i++) {
    const Solver* s = ms[i];
    tab.m[i] = {s->lev[lb].rhs, s->lev[lb].x, lb == 0 ? s->ph : nullptr, lb == 0 ? s->pl : nullptr, s->dev};
  }
  const BottomH2 H = bottom_h2(s0, lb);
  const dim3 grid(1, 1, count);
  switch (bottom_chain(s0, lb)) {
#define FS_CASE(N0, NM)                                                                                        \
  case N0:                                                                                                     \
    launch_dependent(true, k_mg_bottom_chain_class<N0, NM>, dim3(grid), dim3(kBottomThreads), 0, st, tab, H,   \
                     P.mg_pre_smooth, P.mg_post_smooth, P.mg_coarse_sweeps, P.max_cycles);                     \
    return;
    FS_CHAINS(FS_CASE)
#undef FS_CASE
  }
  BottomLevels B;
  const size_t smem = bottom_layout(s0, &B);
  const int threads = std::min(1024, std::max(32, ((nb * nb / 4 + 31) / 32) * 32));
  launch_dependent(true, k_mg_bottom_class, dim3(grid), dim3(threads), smem, st, tab, B, P.mg_pre_smooth,
                   P.mg_post_smooth, P.mg_coarse_sweeps, P.max_cycles);
}

}  // namespace fs
