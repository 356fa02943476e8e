// fs_wgrad.cuh -- weight gradients of the 3x3 periodic convolutions on tcgen05.
//
// dW[co][ci][tap] = sum_p G[p][co] X[p + s_tap][ci] as GEMMs with K = the pixels
// of a row segment, one per horizontal tap dx, over tiles of TY rows:
// D_dx[m][n] += sum_k A[m][k] B[n][k] with rows m = xrow * CIN + ci of the TY + 2
// rows of the shifted input X (A) and n = grow * COUT + co of the TY rows of the
// output gradient G (B).  The blocks with xrow - grow = 0, 1, 2 are the vertical
// taps (the others are not used), so one MMA takes all rows of a tile, and D
// accumulates in TMEM over every tile a CTA visits; at the end the TY blocks of
// each vertical tap are added.
//
// Both operands are NHWC in global memory, channels contiguous: MN-major for
// this GEMM.  They are staged as they are, 16 bytes (8 channels of a pixel) at
// a time, into planes of one image row and one channel chunk, [row][chunk]
// [pixel] -- so a plane's 8 consecutive pixels are one core matrix (LBO = 128
// bytes between the two of a K step), the planes follow one another at one
// stride (SBO), and the horizontal taps' operands are descriptors whose start
// addresses differ by one pixel.  Nothing is transposed: the kernel this
// replaces built each of the nine taps' K-major operand with byte permutes
// (288 8 x 8 blocks per 128 pixels at 16 channels), 478 us for 16 -> 16 channels
// at 1024^2 x 4.  The same layout with one MMA per row and horizontal tap took
// 151 us (a 64 x 16 x 16 MMA takes 32 cycles, a 128 x 64 x 16 one hardly more); this
// one takes 62 us (268 MB read, 40 us of HBM time; L1 and shared memory 74% busy,
// the tensor pipe 37%).
//
// The last M block of a layer may have rows beyond (TY + 2) CIN: its descriptor
// runs on into whatever the stage holds there, and those rows of D are not
// read.  Per-CTA partial sums (and the bias sums of G) go to global memory;
// k_wgrad_reduce adds them in a fixed order, so the gradient is deterministic.
#pragma once

#include <cuda_bf16.h>

#include "fs_tc.cuh"

namespace fs {
namespace guess {

constexpr int kWgThreads = 256;  // staging threads; one more warp issues the MMAs

// bytes of one plane of n pixels, such that the `chunks` planes a pixel's
// 16-byte copies go to fall on different banks
__host__ __device__ constexpr int wg_plane(int n, int chunks) {
  const int want = chunks >= 8 ? 16 : 128 / chunks;  // modulo 128
  int b = n * 16;
  while (b % 128 != want) b += 16;
  return b;
}

// TY rows of PX pixels per tile, NDX of the three horizontal taps per CTA
template <int CIN, int COUT, int TY, int PX, int NDX>
struct WgCfg {
  static constexpr int KC = CIN / 8, OC = COUT / 8, RW = PX + 2;
  static constexpr int XP = wg_plane(RW, KC), GP = wg_plane(PX, OC);
  static constexpr int X_BYTES = (TY + 2) * KC * XP, G_BYTES = TY * OC * GP;
  static constexpr int STAGE = (X_BYTES + G_BYTES + 127) & ~127;
  static constexpr int SMEM = 2 * STAGE + 256;
  static constexpr int GROUPS = (TY + 2) * KC;               // 8-row groups of A
  static constexpr int MB = (GROUPS + 15) / 16;              // M blocks
  static constexpr int LAST_M = GROUPS - 16 * (MB - 1) <= 8 ? 64 : 128;
  static constexpr int NN = TY * COUT;                       // columns of D
  static constexpr int COLS = NDX * MB * NN;
  static constexpr int NCOL = COLS <= 32 ? 32 : COLS <= 64 ? 64 : COLS <= 128 ? 128 : COLS <= 256 ? 256 : 512;
  static constexpr int MROWS = 9 * CIN;
  static constexpr int ACC_BYTES = 3 * NDX * CIN * COUT * 4;  // the taps' sums, in the stages' words
  // the last M block reads groups up to here, inside the stage
  static_assert((16 * (MB - 1) + LAST_M / 8) * XP <= X_BYTES + G_BYTES, "A operand within the stage");
  static_assert(ACC_BYTES + kWgThreads * 32 <= 2 * STAGE, "sums and bias fold in the stages' words");
  static_assert(COLS <= 512 && NN <= 256 && NN % 16 == 0 && COUT % 16 == 0 && CIN % 16 == 0 && PX % 16 == 0, "shape");
  static_assert(SMEM <= 227 * 1024, "shared memory of one CTA");
  static_assert(kWgThreads % OC == 0, "a bias thread keeps its channels");
};

// A 16-byte asynchronous copy, or 16 zero bytes.  Through L1 (.ca): past it
// (.cg), whichever way lanes are dealt to pixels and chunks, these kernels were
// much slower (16 -> 16 channels 100 .. 119 us, 62 us here; 64 -> 32 52, 35 here).
__device__ __forceinline__ void wg_copy(uint32_t dst, const void* src, bool real) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(real ? 16 : 0) : "memory");
}

// i modulo n for i >= -n; a division only where the image is smaller than a tile
__device__ __forceinline__ int wg_wrap(int i, int n) {
  if (i < 0) return i + n;
  if (i >= n) {
    i -= n;
    if (i >= n) i %= n;
  }
  return i;
}

// Warps 0 .. 7 stage tiles (and sum the bias gradient from their own copies),
// warp 8 issues the MMAs; two stages, handed over by barriers: full[s] (the
// staging threads' copies have landed) and done[s] (the MMAs that read them).
template <int CIN, int COUT, int TY, int PX, int NDX>
__global__ void __launch_bounds__(kWgThreads + 32, 1) k_wgrad_tc(const uint4* __restrict__ X,
                                                                 const uint4* __restrict__ G, int B, int H, int W,
                                                                 float* __restrict__ part, float* __restrict__ bpart,
                                                                 int* __restrict__ err) {
  using C = WgCfg<CIN, COUT, TY, PX, NDX>;
  extern __shared__ __align__(128) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + 2 * C::STAGE);
  uint64_t* done = full + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(full + 4);
  volatile int* failed = reinterpret_cast<volatile int*>(full + 5);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int dx0 = NDX == 3 ? 0 : blockIdx.y;
  if (warp == 0) {
    tc::tmem_alloc(tslot, C::NCOL);
    tc::tmem_relinquish();
    tc::fence_before_sync();
  }
  if (tid == 0) {
    for (int k = 0; k < 2; k++) {
      tc::mbar_init(&full[k], kWgThreads);
      tc::mbar_init(&done[k], 1);
    }
    tc::mbar_fence_init();
    *failed = 0;
  }
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot, s0 = tc::smem_u32(smem);
  const int ntx = (W + PX - 1) / PX, nty = (H + TY - 1) / TY, ntiles = B * nty * ntx;
  const int mine = blockIdx.x < ntiles ? (ntiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;  // tiles of this CTA
  float bs[8] = {};  // bias sums of channels 8 (tid % OC) ..

  if (warp < kWgThreads / 32) {
    // the G copies of this thread: channel chunk goc, pixels gpx, gpx + GS, ...
    constexpr int GS = kWgThreads / C::OC;
    const int goc = C::OC == 2 ? tid / GS : tid % C::OC, gpx = C::OC == 2 ? tid % GS : tid / C::OC;
    for (int k = 0; k <= mine; k++) {
      if (k < mine) {
        const int t = blockIdx.x + k * gridDim.x, buf = k & 1;
        const int xt = t % ntx, r = t / ntx, y0 = (r % nty) * TY, x0 = xt * PX;
        const int img = (r / nty) * H;
        const uint32_t sx = s0 + buf * C::STAGE, sg = sx + C::X_BYTES;
        if (k >= 2 && !tc::mbar_wait_idle(&done[buf], ((k - 2) >> 1) & 1)) *failed = 1;
        if (*failed) break;
        // columns x0 - 1 .. x0 + PX of rows y0 - 1 .. y0 + TY, wrapped
        const uint4* rows[TY + 2];
#pragma unroll
        for (int row = 0; row < TY + 2; row++) rows[row] = X + (int64_t)(img + wg_wrap(y0 - 1 + row, H)) * (W * C::KC);
        auto column = [&](int px, int kc) {
          const int col = wg_wrap(x0 - 1 + px, W) * C::KC + kc;
          const uint32_t dst = sx + kc * C::XP + px * 16;
#pragma unroll
          for (int row = 0; row < TY + 2; row++) wg_copy(dst + row * C::KC * C::XP, rows[row] + col, true);
        };
        if constexpr (C::KC == 2) {
          // 16 channels: a chunk of neighbouring pixels on neighbouring threads (80 us with
          // the other order)
          static_assert(kWgThreads == 2 * PX, "one column a thread");
          column(tid % PX, tid / PX);
          if (tid % PX < 2) column(PX + tid % PX, tid / PX);
        } else {
          // a pixel's chunks on neighbouring threads
          for (int q = tid; q < C::RW * C::KC; q += kWgThreads) column(q / C::KC, q % C::KC);
        }
        // and the tile's G, zeros beyond the image
#pragma unroll
        for (int px = gpx; px < PX; px += GS) {
          const bool in = x0 + px < W;
          const uint4* col = G + (in ? x0 + px : 0) * C::OC + goc;
          const uint32_t dst = sg + goc * C::GP + px * 16;
#pragma unroll
          for (int row = 0; row < TY; row++) {
            const int gy = y0 + row;
            wg_copy(dst + row * C::OC * C::GP, col + (int64_t)(img + min(gy, H - 1)) * (W * C::OC), in && gy < H);
          }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
      }
      if (k == 0) continue;
      // the tile before: its copies have landed
      const int buf = (k - 1) & 1;
      if (k < mine) asm volatile("cp.async.wait_group 1;" ::: "memory");
      else asm volatile("cp.async.wait_group 0;" ::: "memory");
      tc::fence_async_smem();
      tc::mbar_arrive(&full[buf]);
      if (blockIdx.y == 0) {
        const unsigned char* g = smem + buf * C::STAGE + C::X_BYTES + goc * C::GP;
#pragma unroll
        for (int px = gpx; px < PX; px += GS)
#pragma unroll
          for (int row = 0; row < TY; row++) {
            const uint4 v = *reinterpret_cast<const uint4*>(g + row * C::OC * C::GP + px * 16);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&v);
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const float2 f = __bfloat1622float2(h[e]);
              bs[2 * e] += f.x;
              bs[2 * e + 1] += f.y;
            }
          }
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
  } else {
    const uint32_t leader = tc::elect_one(), ta = __shfl_sync(0xffffffffu, taddr, 0);
    int k = 0;
    for (; k < mine; k++) {
      const int buf = k & 1;
      const bool ok = tc::mbar_wait_idle(&full[buf], (k >> 1) & 1);
      if (__any_sync(0xffffffffu, !ok || *failed)) {
        *failed = 1;
        break;
      }
      tc::fence_after_sync();
      const uint32_t sx = s0 + buf * C::STAGE, sg = sx + C::X_BYTES;
      // the descriptors' address field counts 16-byte units
      const uint64_t ad0 = tc::sdesc(sx + dx0 * 16, 128, C::XP), bd0 = tc::sdesc(sg, 128, C::GP);
#pragma unroll
      for (int s = 0; s < PX / 16; s++) {
#pragma unroll
        for (int d = 0; d < NDX; d++)
#pragma unroll
          for (int j = 0; j < C::MB; j++)
            tc::mma_bf16_warp(leader, ta + (d * C::MB + j) * C::NN, ad0 + 16 * j * (C::XP / 16) + s * 16 + d,
                              bd0 + s * 16, tc::idesc_bf16_mn(j == C::MB - 1 ? C::LAST_M : 128, C::NN),
                              (k > 0 || s > 0) ? 1u : 0u);
      }
      if (leader) tc::mma_commit(&done[buf]);
      __syncwarp();
    }
    // every MMA issued is done before the accumulators are read or released
    // (a commit covers all before it)
    if (k > 0 && !tc::mbar_wait_idle(&done[(k - 1) & 1], ((k - 1) >> 1) & 1)) *failed = 1;
  }
  __syncthreads();
  if (tid == 0 && *failed) atomicExch(err, 1);
  tc::fence_after_sync();
  // The stages are done with: their words hold the taps' sums [dy][d][ci][co]
  // and, behind them, the bias sums of every staging thread.
  float* acc = reinterpret_cast<float*>(smem);
  float* fold = reinterpret_cast<float*>(smem + C::ACC_BYTES);
  if (blockIdx.y == 0 && tid < kWgThreads) {
#pragma unroll
    for (int e = 0; e < 8; e++) fold[tid * 8 + e] = bs[e];
  }
  // Row by row of G, the three blocks of D that hold its vertical taps.  Warp w
  // reads TMEM lanes 32 (w % 4) ..; the two warp groups share the (horizontal
  // tap, M block, 16 channels) chunks.  Row m of D is lane m for M = 128, lane
  // 32 (m / 16) + m % 16 for M = 64.  One thread adds to a sum at a time, in the
  // order of the rows.
  const int q = warp & 3;
  constexpr int CH = COUT / 16;
#pragma unroll 1
  for (int g = 0; g < TY; g++) {
    if (!*failed && warp < kWgThreads / 32) {
#pragma unroll 1
      for (int k = warp >> 2; k < NDX * C::MB * CH; k += kWgThreads / 128) {
        const int d = k / (C::MB * CH), j = (k / CH) % C::MB, c0 = (k % CH) * 16;
        const bool m64 = j == C::MB - 1 && C::LAST_M == 64;
        const int m = 128 * j + (m64 ? 16 * q + lane : 32 * q + lane);
        const int xrow = m / CIN, ci = m - xrow * CIN, dy = xrow - g;
        float v[16];
        tc::tmem_ld16(taddr + ((uint32_t)(32 * q) << 16) + (d * C::MB + j) * C::NN + g * COUT + c0, v);
        if (dy >= 0 && dy < 3 && !(m64 && lane >= 16)) {
          float* dst = acc + ((dy * NDX + d) * CIN + ci) * COUT + c0;
#pragma unroll
          for (int e = 0; e < 16; e++) dst[e] = g == 0 ? v[e] : dst[e] + v[e];
        }
      }
    }
    __syncthreads();
  }
  if (!*failed) {
    for (int k = tid; k < 3 * NDX * CIN * COUT; k += kWgThreads + 32) {
      const int tap = k / (CIN * COUT), r = k - tap * (CIN * COUT), dy = tap / NDX, d = tap - dy * NDX;
      part[((int64_t)blockIdx.x * 9 + dy * 3 + dx0 + d) * CIN * COUT + r] = mine > 0 ? acc[k] : 0.f;
    }
    if (blockIdx.y == 0 && tid < COUT) {  // the threads that hold these channels, in order
      float s = 0.f;
      if (C::OC == 2) {
        for (int k = 0; k < kWgThreads / 2; k++) s += fold[(tid / 8 * (kWgThreads / 2) + k) * 8 + tid % 8];
      } else {
        for (int k = tid / 8; k < kWgThreads; k += C::OC) s += fold[k * 8 + tid % 8];
      }
      bpart[(int64_t)blockIdx.x * COUT + tid] = s;
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, C::NCOL);
}

// grad[off_w + OIHW] = sum over the P partials of row tap * cin + ci, column
// co; grad[off_b + co] = sum of the bias partials.  A warp's lanes take 32
// consecutive elements, the block's eight warps an eighth of the partials
// each, folded in warp order.
__global__ void __launch_bounds__(256) k_wgrad_reduce(const float* __restrict__ part, const float* __restrict__ bpart,
                                                      int P, int cin, int cout, float* __restrict__ gw,
                                                      float* __restrict__ gb) {
  __shared__ float fold[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nw = 9 * cin * cout, e = blockIdx.x * 32 + lane;
  const float* src = e < nw ? part + e : bpart + (e - nw);
  const int64_t step = e < nw ? nw : cout;
  float s = 0.f;
  if (e < nw + cout) {
#pragma unroll 4
    for (int p = warp; p < P; p += 8) s += src[p * step];
  }
  fold[warp][lane] = s;
  __syncthreads();
  if (warp > 0 || e >= nw + cout) return;
#pragma unroll
  for (int k = 1; k < 8; k++) s += fold[k][lane];
  if (e < nw) {
    const int row = e / cout, co = e - row * cout, tap = row / cin, ci = row - tap * cin;
    gw[((int64_t)co * cin + ci) * 9 + tap] = s;
  } else {
    gb[e - nw] = s;
  }
}

}  // namespace guess
}  // namespace fs
