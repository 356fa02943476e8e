// fs_flat.cuh -- several Jacobi sweeps or red-black half-sweeps of the flat
// Poisson solvers in one pass over the grid (GB300, sm_103a).
//
// Reference: JACOBI (src/gpu/shaders.js:302-325) and RED_BLACK_GS (:340-372),
// which dispatch one pass over the grid per sweep / colour.
//
// A CTA holds a region of 32 * CPL columns x NW * RPW rows in registers: warp
// w owns rows w * RPW .. + RPW - 1, a lane CPL consecutive columns of them.
// It runs k sweeps there (the cells still right shrink by one ring per sweep)
// and writes the tile that is left: H columns (fixed, so that tiles start on
// 16-byte boundaries) and k rows in from the region's edges.  A cell's
// vertical neighbours are the thread's own registers, or a row a neighbouring
// warp published in shared memory (one barrier per sweep, two buffers); its
// horizontal neighbours are registers too, or one shuffle.  The per-cell
// arithmetic is gs_update, so the result equals one pass per sweep bit for bit.
#pragma once

#include <stdint.h>

#include "fs_stencil.cuh"

namespace fs {

enum FlatMode {
  kFlatJacobi = 0,
  kFlatRbEven = 1,  // nx and ny even: a cell's neighbours are all of the other colour
  kFlatRbOdd = 2    // colours from the wrapped indices; cells of one colour may be neighbours
                    // across the wrap and read each other's old value (the reference's
                    // ping-pong pass, shaders.js:353-358)
};

template <int CPL, int RPW, int NW, int H>
struct FlatTile {
  static constexpr int RW = 32 * CPL, RH = RPW * NW, TW = RW - 2 * H;
  static_assert(TW > 0 && TW % 4 == 0 && H % 4 == 0 && RPW % 2 == 0 && CPL % 2 == 0, "tile shape");
};

// x modulo n for any x >= -n (regions reach less than one grid below zero
// whenever k <= n; smaller grids wrap more than once)
__device__ __forceinline__ int flat_wrap(int x, int n) {
  if (x < 0) x += n;
  if (x >= n) x -= n;
  if ((unsigned)x >= (unsigned)n) {
    x %= n;
    if (x < 0) x += n;
  }
  return x;
}

template <int CPL>
struct FlatVec;
template <>
struct FlatVec<2> {
  typedef float2 T;
};
template <>
struct FlatVec<4> {
  typedef float4 T;
};

// One red-black half-sweep on even grids: the cells of row r and column c with
// (r + c) & 1 == Q.  Their neighbours are not written here, so the order of
// the updates does not matter.
template <int CPL, int RPW, int Q>
__device__ __forceinline__ void flat_rb_rows(float (&p)[RPW][CPL], const float (&d)[RPW][CPL],
                                             const float (&below)[CPL], const float (&above)[CPL], float h2, float w) {
#pragma unroll
  for (int r = 0; r < RPW; r++) {
    // column 0 is updated when (r + Q) is even, column CPL - 1 when it is odd:
    // one neighbour in another lane per row
    const float side = ((r + Q) & 1) == 0 ? __shfl_up_sync(0xffffffffu, p[r][CPL - 1], 1)
                                          : __shfl_down_sync(0xffffffffu, p[r][0], 1);
#pragma unroll
    for (int c = (r + Q) & 1; c < CPL; c += 2) {
      const float l = c > 0 ? p[r][c > 0 ? c - 1 : 0] : side;
      const float t = c < CPL - 1 ? p[r][c < CPL - 1 ? c + 1 : 0] : side;
      const float b = r > 0 ? p[r > 0 ? r - 1 : 0][c] : below[c];
      const float a = r < RPW - 1 ? p[r < RPW - 1 ? r + 1 : 0][c] : above[c];
      p[r][c] = gs_update(p[r][c], l, t, b, a, d[r][c], h2, w);
    }
  }
}

// every cell (Jacobi), or those whose bit of `mask` is set, from the old values
template <int CPL, int RPW, bool MASK>
__device__ __forceinline__ void flat_all_rows(float (&p)[RPW][CPL], const float (&d)[RPW][CPL],
                                              const float (&below)[CPL], const float (&above)[CPL], float h2, float w,
                                              uint32_t mask) {
  float prev[CPL];
#pragma unroll
  for (int c = 0; c < CPL; c++) prev[c] = below[c];
#pragma unroll
  for (int r = 0; r < RPW; r++) {
    const float l = __shfl_up_sync(0xffffffffu, p[r][CPL - 1], 1);
    const float t = __shfl_down_sync(0xffffffffu, p[r][0], 1);
    float nv[CPL];
#pragma unroll
    for (int c = 0; c < CPL; c++) {
      nv[c] = gs_update(p[r][c], c > 0 ? p[r][c > 0 ? c - 1 : 0] : l, c < CPL - 1 ? p[r][c < CPL - 1 ? c + 1 : 0] : t,
                        prev[c], r < RPW - 1 ? p[r < RPW - 1 ? r + 1 : 0][c] : above[c], d[r][c], h2, w);
      if (MASK && !((mask >> (r * CPL + c)) & 1u)) nv[c] = p[r][c];
    }
#pragma unroll
    for (int c = 0; c < CPL; c++) {
      prev[c] = p[r][c];
      p[r][c] = nv[c];
    }
  }
}

// k <= H sweeps (half-sweeps of colours c0, c0 + 1, ...) of (p, d) into o; zero:
// p is taken as 0 and not read.
//
// The launches are programmatic dependents: a CTA may start while the launch
// before it, which writes p and reads o, still runs, loads d (which no launch of
// the solve writes, except that the one ahead of the first may) and then waits
// for that launch to complete before it lets the next one start.
template <int CPL, int RPW, int NW, int H, int MODE>
__global__ void __launch_bounds__(NW * 32) k_flat(const float* p, const float* d, float* o, int nx, int ny,
                                                  float h2, float w, int k, int c0, int zero, int first) {
  using F = FlatTile<CPL, RPW, NW, H>;
  typedef typename FlatVec<CPL>::T V;
  static_assert(MODE != kFlatRbOdd || RPW * CPL <= 32, "one mask bit per cell");
  __shared__ __align__(16) float edge[2][NW][2][F::RW];  // each warp's first and last row
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x0 = blockIdx.x * F::TW - H, y0 = blockIdx.y * (F::RH - 2 * k) - k;
  const int xl = x0 + lane * CPL, yl = y0 + warp * RPW;
  const bool vec = nx % CPL == 0;  // a lane's columns never straddle the wrap
  float pv[RPW][CPL], dv[RPW][CPL];
  if (first) asm volatile("griddepcontrol.wait;" ::: "memory");
  uint32_t odd = 0;  // bit r * CPL + c: the parity of the cell's wrapped indices
  int gx[CPL];
#pragma unroll
  for (int c = 0; c < CPL; c++) gx[c] = flat_wrap(xl + c, nx);
#pragma unroll
  for (int r = 0; r < RPW; r++) {
    const int gy = flat_wrap(yl + r, ny);
    const float* row = d + (int64_t)gy * nx;
    if (vec) {
      *reinterpret_cast<V*>(dv[r]) = *reinterpret_cast<const V*>(row + gx[0]);
    } else {
#pragma unroll
      for (int c = 0; c < CPL; c++) dv[r][c] = row[gx[c]];
    }
#pragma unroll
    for (int c = 0; c < CPL; c++) {
      pv[r][c] = 0.f;
      if (MODE == kFlatRbOdd) odd |= (uint32_t)((gx[c] + gy) & 1) << (r * CPL + c);
    }
  }
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;");
  if (!zero) {
#pragma unroll
    for (int r = 0; r < RPW; r++) {
      const float* row = p + (int64_t)flat_wrap(yl + r, ny) * nx;
      if (vec) {
        *reinterpret_cast<V*>(pv[r]) = *reinterpret_cast<const V*>(row + gx[0]);
      } else {
#pragma unroll
        for (int c = 0; c < CPL; c++) pv[r][c] = row[gx[c]];
      }
    }
  }
  for (int s = 0; s < k; s++) {
    float(*e)[2][F::RW] = edge[s & 1];
    *reinterpret_cast<V*>(&e[warp][0][lane * CPL]) = *reinterpret_cast<const V*>(pv[0]);
    *reinterpret_cast<V*>(&e[warp][1][lane * CPL]) = *reinterpret_cast<const V*>(pv[RPW - 1]);
    __syncthreads();
    // beyond the region's edge: any value, the ring it reaches is not written
    float below[CPL], above[CPL];
    *reinterpret_cast<V*>(below) = *reinterpret_cast<const V*>(&e[warp > 0 ? warp - 1 : 0][1][lane * CPL]);
    *reinterpret_cast<V*>(above) = *reinterpret_cast<const V*>(&e[warp < NW - 1 ? warp + 1 : warp][0][lane * CPL]);
    if (MODE == kFlatJacobi) {
      flat_all_rows<CPL, RPW, false>(pv, dv, below, above, h2, w, 0u);
    } else if (MODE == kFlatRbOdd) {
      flat_all_rows<CPL, RPW, true>(pv, dv, below, above, h2, w, ((c0 + s) & 1) ? odd : ~odd);
    } else if ((c0 + s + y0) & 1) {  // x0 and the warps' first rows are even
      flat_rb_rows<CPL, RPW, 1>(pv, dv, below, above, h2, w);
    } else {
      flat_rb_rows<CPL, RPW, 0>(pv, dv, below, above, h2, w);
    }
  }
  if (lane * CPL < H || lane * CPL >= F::RW - H) return;
#pragma unroll
  for (int r = 0; r < RPW; r++) {
    const int row = warp * RPW + r, gy = yl + r;
    if (row < k || row >= F::RH - k || gy >= ny) continue;
    float* out = o + (int64_t)gy * nx + xl;
    if (vec) {
      if (xl < nx) *reinterpret_cast<V*>(out) = *reinterpret_cast<const V*>(pv[r]);
    } else {
#pragma unroll
      for (int c = 0; c < CPL; c++)
        if (xl + c < nx) out[c] = pv[r][c];
    }
  }
}

}  // namespace fs
