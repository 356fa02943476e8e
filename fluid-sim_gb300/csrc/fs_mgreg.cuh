// fs_mgreg.cuh -- the smoothing kernels of a multigrid level with a tile's
// region in registers (GB300, sm_103a).
//
// Reference: src/gpu/multigrid.js:277-330 (RBGS(pre) -> residual ->
// restriction, prolongation -> RBGS(post)).
//
// A CTA holds a region of 32 * CPL columns x NW * RPW rows of a level: warp w
// owns rows w * RPW .. + RPW - 1, a lane CPL consecutive columns of them, the
// iterate and the right-hand side of each cell in registers (the layout and
// the sweeps of the flat solvers, fs_flat.cuh).  Both are loaded straight into
// the registers, a row of a warp at a time; a half-sweep costs a row a warp
// publishes on each side, one barrier and one shuffle per row; the residual's,
// the restriction's and the prolongation's neighbours are registers and
// shuffles too.  The cells still right shrink by one ring per half-sweep; the
// tile that is left lies HX columns and HY rows in from the region's edges.
//
// The per-cell arithmetic is fs_stencil.cuh, so a level's values do not depend
// on the region, and equal the one-pass-per-operation kernels'.
#pragma once

#include "fs_df.cuh"
#include "fs_flat.cuh"
#include "fs_internal.cuh"
#include "fs_stencil.cuh"

namespace fs {

// H rings: 2 pre + 1 (down) or 2 post (up)
template <int CPL_, int RPW_, int NW_, int H>
struct MgRegion {
  static constexpr int CPL = CPL_, RPW = RPW_, NW = NW_;
  static constexpr int HX = (H + CPL - 1) / CPL * CPL, HY = (H + 1) & ~1;
  static constexpr int RW = 32 * CPL, RH = RPW * NW, TW = RW - 2 * HX, TH = RH - 2 * HY, THREADS = 32 * NW;
  // CTAs per SM: 80 registers a thread for 32 cells, 64 for fewer
  static constexpr int CTAS = (CPL * RPW >= 32 ? 768 : 1024) / THREADS;
  static_assert(TW > 0 && TH > 0 && RPW % 2 == 0 && CPL % 2 == 0, "a region of 2 x 2 blocks");
};

template <class R>
struct MgCells {
  typedef typename FlatVec<R::CPL>::T V;
  float p[R::RPW][R::CPL], d[R::RPW][R::CPL];
  int lane, warp, xl, yl, gx;  // first column and row of the thread, the column wrapped
  __device__ __forceinline__ MgCells(int n) {
    lane = threadIdx.x & 31;
    warp = threadIdx.x >> 5;
    xl = blockIdx.x * R::TW - R::HX + lane * R::CPL;
    yl = blockIdx.y * R::TH - R::HY + warp * R::RPW;
    gx = flat_wrap(xl, n);  // n is a multiple of CPL: a lane's columns do not straddle the wrap
  }
  // COMPLETE: the field was written before the launch ahead began (see pdl_wait)
  template <bool COMPLETE>
  __device__ __forceinline__ void load(float (&a)[R::RPW][R::CPL], const float* f, int n) const {
#pragma unroll
    for (int r = 0; r < R::RPW; r++) {
      const V* at = reinterpret_cast<const V*>(f + (int64_t)flat_wrap(yl + r, n) * n + gx);
      *reinterpret_cast<V*>(a[r]) = COMPLETE ? __ldg(at) : *at;
    }
  }
  // the rows above and below the thread's, from the neighbouring warps
  typedef float Edge[R::NW][2][R::RW];
  __device__ __forceinline__ void neighbours(Edge& e, float (&below)[R::CPL], float (&above)[R::CPL]) const {
    *reinterpret_cast<V*>(&e[warp][0][lane * R::CPL]) = *reinterpret_cast<const V*>(p[0]);
    *reinterpret_cast<V*>(&e[warp][1][lane * R::CPL]) = *reinterpret_cast<const V*>(p[R::RPW - 1]);
    __syncthreads();
    // beyond the region's edge: any value, the ring it reaches is not written
    *reinterpret_cast<V*>(below) = *reinterpret_cast<const V*>(&e[warp > 0 ? warp - 1 : 0][1][lane * R::CPL]);
    *reinterpret_cast<V*>(above) =
        *reinterpret_cast<const V*>(&e[warp < R::NW - 1 ? warp + 1 : warp][0][lane * R::CPL]);
  }
  // half-sweep s (colour s & 1; the region's first column and row are even)
  __device__ __forceinline__ void half_sweep(Edge* e, int s, float h2, float w) {
    float below[R::CPL], above[R::CPL];
    neighbours(e[s & 1], below, above);
    if (s & 1) flat_rb_rows<R::CPL, R::RPW, 1>(p, d, below, above, h2, w);
    else flat_rb_rows<R::CPL, R::RPW, 0>(p, d, below, above, h2, w);
  }
  // is row r of this thread in the tile and the grid
  __device__ __forceinline__ bool tile_row(int r, int n) const {
    const int row = warp * R::RPW + r;
    return row >= R::HY && row < R::RH - R::HY && yl + r < n;
  }
  __device__ __forceinline__ bool tile_columns(int n) const {
    return lane * R::CPL >= R::HX && lane * R::CPL < R::RW - R::HX && xl < n;
  }
};

// two fields of the region that the CTA `ahead` launches on will load, into L2: a
// 128-byte line per thread and field
template <class R>
__device__ __forceinline__ void prefetch_region(int n, int ahead, const float* f, const float* g) {
  const int b = blockIdx.y * gridDim.x + blockIdx.x + ahead;
  if (b >= (int)(gridDim.x * gridDim.y)) return;
  constexpr int LINES = R::RW / 32;
  for (int k = threadIdx.x; k < LINES * R::RH; k += R::THREADS) {
    const int x = flat_wrap((b % gridDim.x) * R::TW - R::HX + (k % LINES) * 32, n);
    const int y = flat_wrap((int)(b / gridDim.x) * R::TH - R::HY + k / LINES, n);
    prefetch_l2(f + (int64_t)y * n + x);
    prefetch_l2(g + (int64_t)y * n + x);
  }
}

// xin == nullptr: the level starts from zero.  xout == xin is not allowed (the
// halo of a tile is another tile's interior).
template <class R>
__device__ __forceinline__ void mg_down_reg(const float* __restrict__ rhs, const float* __restrict__ xin,
                                            float* __restrict__ xout, float* __restrict__ crhs, int n, float h2,
                                            int pre, float w) {
  constexpr int CPL = R::CPL, RPW = R::RPW;
  typedef typename MgCells<R>::V V;
  __shared__ __align__(16) typename MgCells<R>::Edge edge[2];
  MgCells<R> t(n);
  t.template load<false>(t.d, rhs, n);
  int s = 0;
  if (xin) {
    t.template load<false>(t.p, xin, n);
  } else {
#pragma unroll
    for (int r = 0; r < RPW; r++)
#pragma unroll
      for (int c = 0; c < CPL; c++)
        // the first half-sweep of an iterate of zeros
        t.p[r][c] = ((r + c) & 1) == 0 && pre > 0 ? gs_update(0.f, 0.f, 0.f, 0.f, 0.f, t.d[r][c], h2, w) : 0.f;
    s = 1;
  }
  for (; s < 2 * pre; s++) t.half_sweep(edge, s, h2, w);
  float below[CPL], above[CPL];
  t.neighbours(edge[(2 * pre) & 1], below, above);
  const bool col = t.tile_columns(n);
  const float ih2 = inv_h2(h2);
  const int nc = n >> 1;
  // residual and its restriction (multigrid.js:48-93), a row pair at a time
#pragma unroll
  for (int r0 = 0; r0 < RPW; r0 += 2) {
    float res[2][CPL];
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const int r = r0 + k;
      const float left = __shfl_up_sync(0xffffffffu, t.p[r][CPL - 1], 1);
      const float right = __shfl_down_sync(0xffffffffu, t.p[r][0], 1);
#pragma unroll
      for (int c = 0; c < CPL; c++)
        res[k][c] = residual_at(t.p[r][c], c > 0 ? t.p[r][c > 0 ? c - 1 : 0] : left,
                                c < CPL - 1 ? t.p[r][c < CPL - 1 ? c + 1 : 0] : right,
                                r > 0 ? t.p[r > 0 ? r - 1 : 0][c] : below[c],
                                r < RPW - 1 ? t.p[r < RPW - 1 ? r + 1 : 0][c] : above[c], t.d[r][c], ih2);
    }
    if (!col || !t.tile_row(r0, n)) continue;
    const int64_t at = (int64_t)(t.yl + r0) * n + t.xl;
    *reinterpret_cast<V*>(xout + at) = *reinterpret_cast<const V*>(t.p[r0]);
    *reinterpret_cast<V*>(xout + at + n) = *reinterpret_cast<const V*>(t.p[r0 + 1]);
    float* co = crhs + (int64_t)((t.yl + r0) >> 1) * nc + (t.xl >> 1);
    float cv[CPL / 2];
#pragma unroll
    for (int q = 0; q < CPL / 2; q++)
      cv[q] = restrict4(res[0][2 * q], res[0][2 * q + 1], res[1][2 * q], res[1][2 * q + 1]);
    if (CPL == 4) *reinterpret_cast<float2*>(co) = make_float2(cv[0], cv[CPL / 2 - 1]);
    else *co = cv[0];  // the coarse level may be odd
  }
}

// the residual is the rhs (no sweeps from a zero iterate that nothing reads
// afterwards): its restriction alone, straight from global memory
template <class R>
__device__ __forceinline__ void mg_restrict_rhs(const float* __restrict__ rhs, float* __restrict__ crhs, int n) {
  const int nc = n >> 1;
  for (int k = threadIdx.x; k < (R::TW / 2) * (R::TH / 2); k += R::THREADS) {
    const int cj = k / (R::TW / 2), ci = k - cj * (R::TW / 2);
    const int gci = blockIdx.x * (R::TW / 2) + ci, gcj = blockIdx.y * (R::TH / 2) + cj;
    if (gci >= nc || gcj >= nc) continue;
    const float* q = rhs + (int64_t)(2 * gcj) * n + 2 * gci;
    const float2 q0 = *reinterpret_cast<const float2*>(q);
    const float2 q1 = *reinterpret_cast<const float2*>(q + n);
    crhs[(int64_t)gcj * nc + gci] = restrict4(q0.x, q0.y, q1.x, q1.y);
  }
}

// x += P(coarse) on the region, then the post sweeps.  zero: no sweeps and an
// iterate of zeros that is not read: the correction is the prolongation alone
// (0 + P = P, and a -0 from P gives the same pressure sum as +0).  With ACC the
// tile's correction is added to the double-float pressure (ph, pl) in place
// instead of being written to xout: a cell is read and written by its own tile.
// AHEAD > 0: the CTA fetches a later one's iterate and rhs into L2.
template <class R, bool ACC, int AHEAD>
__device__ __forceinline__ void mg_up_reg(const float* __restrict__ rhs, const float* __restrict__ xin,
                                          float* __restrict__ xout, const float* xc, int n, float h2,
                                          int post, float w, float* __restrict__ ph, float* __restrict__ pl,
                                          bool zero) {
  constexpr int CPL = R::CPL, RPW = R::RPW, CC = CPL / 2, CR = RPW / 2 + 2;
  typedef typename MgCells<R>::V V;
  __shared__ __align__(16) typename MgCells<R>::Edge edge[2];
  MgCells<R> t(n);
  const bool col = t.tile_columns(n);
  if (ACC && col) {
    // the pressure is read after the sweeps: into L2 meanwhile, a 128-byte line per thread
    if ((t.lane * CPL) % 32 == (R::HX % 32) || t.lane * CPL == R::HX) {
#pragma unroll
      for (int r = 0; r < RPW; r++)
        if (t.tile_row(r, n)) {
          prefetch_l2(ph + (int64_t)(t.yl + r) * n + t.xl);
          prefetch_l2(pl + (int64_t)(t.yl + r) * n + t.xl);
        }
    }
  }
  // The coarse rows yl / 2 - 1 .. yl / 2 + RPW / 2: this lane's CC columns, and
  // on the outer lanes the column beyond them (the others' come by shuffle).
  // Fine column 2 i interpolates coarse columns i - 1, i (weight 3/4 on i),
  // column 2 i + 1 columns i, i + 1 (weight 1/4 on i + 1); likewise the rows
  // (PROLONG, multigrid.js:99-131: sample at ((i+1/2)/2 - 1/2, (j+1/2)/2 - 1/2)).
  const int nc = n >> 1, gc = t.gx >> 1, jc = (t.yl >> 1) - 1;
  // the iterate and the rhs were complete before the launch ahead of this one began
  if (!zero) {
    t.template load<true>(t.p, xin, n);
    t.template load<true>(t.d, rhs, n);
  }
  pdl_wait();
  if (AHEAD > 0 && !zero) prefetch_region<R>(n, AHEAD, xin, rhs);
  float cv[CR][CC], side[CR];
  const int gs = flat_wrap(t.lane == 0 ? gc - 1 : gc + CC, nc);
#pragma unroll
  for (int k = 0; k < CR; k++) {
    const float* row = xc + (int64_t)flat_wrap(jc + k, nc) * nc;
    if (CC == 2) {
      const float2 q = *reinterpret_cast<const float2*>(row + gc);
      cv[k][0] = q.x, cv[k][CC - 1] = q.y;
    } else {
      cv[k][0] = row[gc];
    }
    side[k] = t.lane == 0 || t.lane == 31 ? row[gs] : 0.f;
  }
  float m0[CPL], m1[CPL];  // the two coarse rows before, interpolated to the fine columns
#pragma unroll
  for (int k = 0; k < CR; k++) {
    float left = __shfl_up_sync(0xffffffffu, cv[k][CC - 1], 1), right = __shfl_down_sync(0xffffffffu, cv[k][0], 1);
    if (t.lane == 0) left = side[k];
    if (t.lane == 31) right = side[k];
    float m2[CPL];
#pragma unroll
    for (int c = 0; c < CPL; c++) {
      const int i = c / 2;
      m2[c] = (c & 1) ? mix_rn(cv[k][i], i < CC - 1 ? cv[k][i < CC - 1 ? i + 1 : 0] : right, 0.25f)
                      : mix_rn(i > 0 ? cv[k][i > 0 ? i - 1 : 0] : left, cv[k][i], 0.75f);
    }
    if (k >= 2) {
      const int r = 2 * (k - 2);
#pragma unroll
      for (int c = 0; c < CPL; c++) {
        const float top = mix_rn(m0[c], m1[c], 0.75f), bot = mix_rn(m1[c], m2[c], 0.25f);
        t.p[r][c] = zero ? top : __fadd_rn(t.p[r][c], top);
        t.p[r + 1][c] = zero ? bot : __fadd_rn(t.p[r + 1][c], bot);
      }
    }
#pragma unroll
    for (int c = 0; c < CPL; c++) m0[c] = m1[c], m1[c] = m2[c];
  }
  for (int s = 0; s < 2 * post; s++) t.half_sweep(edge, s, h2, w);
  if (!col) return;
  if constexpr (ACC) {
    constexpr int G = RPW < 4 ? RPW : 4;  // rows whose loads are in flight together
    static_assert(RPW % G == 0, "row groups");
#pragma unroll
    for (int r0 = 0; r0 < RPW; r0 += G) {
      float hv[G][CPL], lv[G][CPL];
#pragma unroll
      for (int k = 0; k < G; k++)
        if (t.tile_row(r0 + k, n)) {
          const int64_t at = (int64_t)(t.yl + r0 + k) * n + t.xl;
          *reinterpret_cast<V*>(hv[k]) = *reinterpret_cast<const V*>(ph + at);
          *reinterpret_cast<V*>(lv[k]) = *reinterpret_cast<const V*>(pl + at);
        }
#pragma unroll
      for (int k = 0; k < G; k++)
        if (t.tile_row(r0 + k, n)) {
          const int64_t at = (int64_t)(t.yl + r0 + k) * n + t.xl;
#pragma unroll
          for (int c = 0; c < CPL; c++) {
            const df q = df_add_f(df{hv[k][c], lv[k][c]}, t.p[r0 + k][c]);
            hv[k][c] = q.hi, lv[k][c] = q.lo;
          }
          *reinterpret_cast<V*>(ph + at) = *reinterpret_cast<const V*>(hv[k]);
          *reinterpret_cast<V*>(pl + at) = *reinterpret_cast<const V*>(lv[k]);
        }
    }
  } else {
#pragma unroll
    for (int r = 0; r < RPW; r++)
      if (t.tile_row(r, n))
        *reinterpret_cast<V*>(xout + (int64_t)(t.yl + r) * n + t.xl) = *reinterpret_cast<const V*>(t.p[r]);
  }
}

}  // namespace fs
