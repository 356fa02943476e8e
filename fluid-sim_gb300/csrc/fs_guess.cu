// fs_guess.cu -- the learned pressure guess: a small periodic U-Net that maps
// the divergence (and the solid mask) at half the grid resolution to an
// initial pressure for the multigrid projection, with its forward pass,
// backward pass and Adam update on the GPU.  No counterpart in the reference.
//
// Network (channels 16/32/64/128 over four levels, NHWC bf16 activations,
// f32 accumulation, every convolution 3x3 periodic on the tcgen05 tensor
// cores -- fs_conv.cu):
//   x0 -A-> a0 -B-> a0b -pool-> q1 -C-> a1 -pool-> q2 -D-> a2 -pool-> q3 -E-> a3
//   a3 -F-> f3;  s2 = up(f3) + a2 -G-> g2;  s1 = up(g2) + a1 -H-> h1;
//   s0 = up(h1) + a0b -I-> i0 -J-> out (channel 0, f32)
// ReLU after every convolution but J.  Parameters are kept in f32 (master
// copy, flattened layer by layer as w[co][ci][3][3] then b[co]) and repacked
// to bf16 after every update, once in the forward layout and once transposed
// and flipped, so that the gradient with respect to a layer's input is the
// same tensor-core convolution.  Weight gradients are a tcgen05 GEMM too,
// with the pixels as its K dimension (k_wgrad_tc), and deterministic per-CTA
// partial sums.
//
// Normalisation (the guess is linear-equivariant in the divergence): with
// h the net's grid spacing and sigma = RMS(h^2 d), the input is h^2 d / sigma
// and the output is p / sigma, so the pressure guess is sigma * out.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>
#include <stdio.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "../../include/fluid.h"
#include "fs_conv.cuh"
#include "fs_df.cuh"
#include "fs_internal.cuh"
#include "fs_reduce.cuh"
#include "fs_tc.cuh"
#include "fs_wgrad.cuh"

struct fs_guess;

namespace fs {
namespace guess {

typedef __nv_bfloat16 bf;
constexpr int NL = 10;
constexpr int kCI[NL] = {16, 16, 16, 32, 64, 128, 64, 32, 16, 16};
constexpr int kCO[NL] = {16, 16, 32, 64, 128, 64, 32, 16, 16, 16};
constexpr int kRelu[NL] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 0};
enum { LA, LB, LC, LD, LE, LF, LG, LH, LI, LJ };

// activation / gradient buffers: (level, channels)
enum Buf {
  X0, A0, A0B, Q1, A1, Q2, A2, Q3, A3, F3, S2, G2, S1, H1, S0, I0,  // forward
  GJ, DI0, DS0, DH1, DS1, DG2, DS2, DF3, DA3, DA0,  // backward
  NBUF
};
constexpr int kBufLevel[NBUF] = {0, 0, 0, 1, 1, 2, 2, 3, 3, 3, 2, 2, 1, 1, 0, 0,
                                 0, 0, 0, 1, 1, 2, 2, 3, 3, 0};
constexpr int kBufCh[NBUF] = {16, 16, 16, 16, 32, 32, 64, 64, 128, 64, 64, 32, 32, 16, 16, 16,
                              16, 16, 16, 16, 32, 32, 64, 64, 128, 16};


struct Net {
  int device = 0;
  cudaStream_t stream = nullptr;  // own stream for the stand-alone entry points
  int64_t off_w[NL], off_b[NL], off_pk[NL];
  int64_t nparam = 0, npk = 0;
  float *theta = nullptr, *grad = nullptr, *m = nullptr, *v = nullptr;
  bf *wpk = nullptr, *wpkT = nullptr;
  float* zero_bias = nullptr;
  int* err = nullptr;
  double* acc = nullptr;  // loss: per-sample mean error [B], loss [B]; guess: sum of squares
  int64_t adam_t = 0;
  double w_p = 1.0, w_r = 0.0;  // loss weights: pressure error, residual (lap of the error)
  int capB = 0, capH = 0, capW = 0;
  bf* buf[NBUF] = {};
  float* out = nullptr;     // [B][H][W]
  float* gin = nullptr;     // solver path: h^2 d at net resolution
  float* gmask = nullptr;   // solver path: mask at net resolution
  float* res = nullptr;     // loss: lap(out - target), [B][H][W]
  float* corr_part = nullptr;
  int64_t corr_cap = 0;
  int64_t launches = 0;
  std::string err_msg;
};

static int64_t level_pixels(const Net* g, int B, int H, int W, int lev) {
  return (int64_t)B * (H >> lev) * (W >> lev);
}

// ------------------------------------------------------------ small kernels
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 q;
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
#pragma unroll
  for (int k = 0; k < 4; k++) h[k] = __floats2bfloat162_rn(f[2 * k], f[2 * k + 1]);
  return q;
}

#define GRID_STRIDE(k, n) for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < (n); k += (int64_t)gridDim.x * blockDim.x)
// element loops of the network's buffers (all below 2^31 elements, checked on the host)
#define GRID_STRIDE32(k, n) for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < (n); k += gridDim.x * blockDim.x)

// sigma = RMS from a sum of squares (1 when it is 0), computed by one thread
// of the block: FP64 runs at 1/54 of the FP32 rate on this part, so it is not
// evaluated per element
__device__ __forceinline__ float block_sigma(const double* __restrict__ sumsq, int64_t nnorm) {
  __shared__ float sig;
  if (threadIdx.x == 0) {
    double r = sqrt(sumsq[0] / (double)nnorm);
    sig = r > 0.0 ? (float)r : 1.f;
  }
  __syncthreads();
  return sig;
}

// x0[p] = (div / sigma, mask, 0, ..., 0); sigma = 1 without a sum of squares.
// A thread writes one half of a pixel, so that a warp's stores are one
// contiguous run (a pixel per thread, 1024^2 x 4: 43 us; 27 us here, of which
// 25 us for the bytes).
__global__ void k_prep(const float* __restrict__ div, const float* __restrict__ mask, uint4* __restrict__ x0,
                       int npix, const double* __restrict__ sumsq, int64_t nnorm) {
  const float inv = sumsq ? 1.f / block_sigma(sumsq, nnorm) : 1.f;
  GRID_STRIDE32(k, 2 * npix) {
    uint4 v = make_uint4(0, 0, 0, 0);
    if (!(k & 1)) {
      const int p = k >> 1;
      const float f[8] = {div[p] * inv, mask ? mask[p] : 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      v = pack8(f);
    }
    x0[k] = v;
  }
}

// ---- The loss.  FP64 runs at 1/54 of the FP32 rate on this part, conversions
// included, so these passes are bound by the number of FP64 instructions a cell
// takes: the error of a cell is formed once and handed to its neighbours, and
// f32 values are widened with integer instructions.  A warp walks down a strip
// of kLossCols columns (lanes 0 and 31 hold its neighbours' columns) with the
// three rows of the stencil in registers.  1024^2 x 4, mean + residual + seed:
// 39 + 175 + 163 us with a thread per cell that converted every operand, 105 + 68 us
// here (mean and residual in one pass).
constexpr int kLossCols = 30, kLossWarps = 8;

// (double)f by integer instructions where f is a normal number
__device__ __forceinline__ double widen(float f) {
  const uint32_t b = __float_as_uint(f);
  if ((b << 1) - 0x01000000u >= 0xfe000000u) return (double)f;  // 0, subnormal, infinite, NaN
  return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + 0x38000000u)), (int)(b << 29));
}

// the block's sum of s, on thread 0
__device__ __forceinline__ double loss_block_sum(double s) {
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double sm[kLossWarps];
  __syncthreads();
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = s;
  __syncthreads();
  double t = 0.0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kLossWarps; w++) t += sm[w];
  return t;
}

// per-sample sum of e = out - target -> acc[b]
__global__ void __launch_bounds__(32 * kLossWarps)
    k_loss_mean(const float* __restrict__ out, const float* __restrict__ tgt, double* __restrict__ acc, int64_t npix) {
  const int b = blockIdx.y;
  double s = 0.0;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < npix; p += (int64_t)gridDim.x * blockDim.x)
    s += widen(out[b * npix + p]) - widen(tgt[b * npix + p]);
  const double t = loss_block_sum(s);
  if (threadIdx.x == 0) atomicAdd(&acc[b], t);
}

// This warp's strip of image blockIdx.y: columns x0 .. x0 + 29, rows y0 .. y1 - 1;
// x is this lane's column, wrapped.
struct LossStrip {
  int x0, x, y0, y1, lane;
  bool any, store;  // the strip exists; this lane's column is one of its own
};
__device__ __forceinline__ LossStrip loss_strip(int H, int W, int rows) {
  LossStrip t;
  const int nx = (W + kLossCols - 1) / kLossCols, k = blockIdx.x * kLossWarps + (threadIdx.x >> 5);
  t.lane = threadIdx.x & 31;
  t.x0 = (k % nx) * kLossCols;
  t.y0 = (k / nx) * rows;
  t.y1 = min(t.y0 + rows, H);
  t.any = t.y0 < H;
  const int x = t.x0 + t.lane - 1;
  t.store = t.lane >= 1 && t.lane <= kLossCols && x < W;
  t.x = (x + W) % W;  // x <= W + 29: wrapped again where the image is narrower
  return t;
}
// c's neighbours' sum and centre: left + right + above + below - 4 c
__device__ __forceinline__ double lap5(double above, double c, double below) {
  const double left = __shfl_up_sync(0xffffffffu, c, 1), right = __shfl_down_sync(0xffffffffu, c, 1);
  return left + right + above + below - 4.0 * c;
}

// res = lap(out - target) (periodic 5-point, unscaled); sum of out - target into
// acc[b], w_r sum res^2 / (B N) into acc[B]
__global__ void __launch_bounds__(32 * kLossWarps)
    k_loss_res(const float* __restrict__ out, const float* __restrict__ tgt, float* __restrict__ res,
               double* __restrict__ acc, int H, int W, int B, int rows, double w_r) {
  const int b = blockIdx.y;
  const int64_t npix = (int64_t)H * W, base = b * npix;
  const LossStrip t = loss_strip(H, W, rows);
  double s = 0.0, m = 0.0;
  if (t.any) {
    auto e = [&](int y) {
      const int64_t q = base + (int64_t)(y < 0 ? y + H : y >= H ? y - H : y) * W + t.x;
      return widen(out[q]) - widen(tgt[q]);
    };
    double above = e(t.y0 - 1), c = e(t.y0);
#pragma unroll 4
    for (int y = t.y0; y < t.y1; y++) {
      const double below = e(y + 1), r = lap5(above, c, below);
      if (t.store) {
        res[base + (int64_t)y * W + t.x] = (float)r;
        s += r * r;
        m += c;
      }
      above = c;
      c = below;
    }
  }
  const double sum = loss_block_sum(s), err = loss_block_sum(m);
  if (threadIdx.x == 0) {
    atomicAdd(&acc[b], err);
    atomicAdd(&acc[B], w_r * sum / ((double)B * npix));
  }
}

// seed gradient dL/dout = (w_p 2 (e - mean_b e) + w_r 2 lap(res)) / (B N) into
// channel 0 of gJ; w_p sum (e - mean)^2 / (B N) into acc[B].  Both are formed in f64,
// the gradient then rounded to f32 and bf16.  That takes 11 f64 instructions a cell
// (148 us at 1024^2 x 4), 8 of them for the gradient, so a cell's gradient is formed
// in double-float (48 bits) on the FP32 pipe first, with a bound on its distance from
// the f64 value: with u = 2^-24 the sums of f32 values are exact but for 10 u^2 of
// their terms, a product or a sum of two double-floats adds 3 to 7 u^2, the rounding
// of the mean and the weights u^2, and the f64 value itself is within 2^-49 of the
// exact one -- together less than 24 u^2 of the terms, 2^-42 of them (64 u^2) with room
// to spare.  Where every value within that bound rounds to the same f32, that is the
// f64 value's rounding too; where not (next to a rounding boundary, or after heavy
// cancellation), and where values or products leave the range in which those bounds
// hold, the cell is done in f64.  66 us without the bound, 68 us with it.
__global__ void __launch_bounds__(32 * kLossWarps)
    k_loss_seed(const float* __restrict__ out, const float* __restrict__ tgt, const float* res,
                double* acc, uint4* __restrict__ gJ, int H, int W, int B, int rows, double w_p,
                double w_r) {
  pdl_wait();
  const int b = blockIdx.y;
  const int64_t npix = (int64_t)H * W, base = b * npix;
  const double mean = acc[b] / (double)npix, scale = 2.0 / ((double)B * npix);
  const df meanf = df_neg(df_from_d(mean)), wp = df_from_d(scale * w_p), wr = df_from_d(scale * w_r);
  // weights whose double-float halves are normal numbers, and products of f32 range
  auto in_range = [](double k) { return k == 0.0 || (k > 1e-28 && k < 1e6); };
  const bool dfok = fabs(mean) < 1e30 && in_range(scale * w_p) && in_range(scale * w_r);
  const float mabs = fabsf(meanf.hi), bound_p = 0x1p-42f * wp.hi, bound_r = res ? 0x1p-42f * wr.hi : 0.f;
  const LossStrip t = loss_strip(H, W, rows);
  double s = 0.0;
  if (t.any) {
    auto row = [&](int y) {
      return res ? res[base + (int64_t)(y < 0 ? y + H : y >= H ? y - H : y) * W + t.x] : 0.f;
    };
    float above = row(t.y0 - 1), c = row(t.y0);
#pragma unroll 4
    for (int y = t.y0; y < t.y1; y++) {
      const int64_t q = base + (int64_t)y * W + t.x;
      const float o = out[q], g0 = tgt[q], below = row(y + 1);
      const float left = __shfl_up_sync(0xffffffffu, c, 1), right = __shfl_down_sync(0xffffffffu, c, 1);
      const double ec = widen(o) - widen(g0) - mean;
      if (t.store) s += ec * ec;
      float g;
      const float size_e = fabsf(o) + fabsf(g0);
      const float size_l = (fabsf(above) + fabsf(below)) + (fabsf(left) + fabsf(right)) + 4.f * fabsf(c);
      const float bound = bound_p * (size_e + mabs) + bound_r * size_l;
      // (above 1e-36 no product's error term is lost to underflow)
      bool done = dfok && size_e + size_l < 1e30f && bound > 1e-36f;
      if (done) {
        df v = df_mul(df_add(two_sum(o, -g0), meanf), wp);
        if (res) {
          const df a = two_sum(left, right), d = two_sum(a.hi, above), e = two_sum(d.hi, below);
          df l = two_sum(e.hi, -4.f * c);
          l.lo = l.lo + ((a.lo + d.lo) + e.lo);
          v = df_add(v, df_mul(fast_two_sum(l.hi, l.lo), wr));
        }
        g = __fadd_rn(v.hi, __fadd_rn(v.lo, bound));
        done = g == __fadd_rn(v.hi, __fsub_rn(v.lo, bound));
      }
      if (!done) {
        double v = w_p * ec;
        if (res)
          v += w_r * ((double)left + (double)right + (double)above + (double)below - 4.0 * (double)c);
        g = (float)(scale * v);
      }
      above = c;
      c = below;
      // the strip's pixels, 16 bytes a lane: channel 0 and zeros, zeros
      const float f[8] = {g, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      const uint32_t first = pack8(f).x;
#pragma unroll
      for (int half = 0; half < 2; half++) {
        const int k = t.lane + 32 * half, px = k >> 1;
        const uint32_t v = __shfl_sync(0xffffffffu, first, (px + 1) & 31);
        if (px < kLossCols && t.x0 + px < W)
          gJ[2 * (base + (int64_t)y * W + t.x0) + k] = make_uint4(k & 1 ? 0u : v, 0u, 0u, 0u);
      }
    }
  }
  const double sum = loss_block_sum(s);
  if (threadIdx.x == 0) atomicAdd(&acc[B], w_p * sum / ((double)B * npix));
}

// ------------------------------------------------------------ parameters
struct PackTable {
  int64_t off_w[NL], off_pk[NL];
  int ci[NL], co[NL];
};

// f32 master -> bf16 forward pack [t][ci/8][co][ci%8] and the transposed,
// flipped pack [t'][co/8][ci][co%8] with t' = (2-ky)*3 + (2-kx)
__global__ void k_pack(const float* __restrict__ theta, bf* __restrict__ wpk, bf* __restrict__ wpkT, PackTable tab) {
  for (int l = 0; l < NL; l++) {
    const int ci_n = tab.ci[l], co_n = tab.co[l];
    const int64_t n = (int64_t)ci_n * co_n * 9;
    GRID_STRIDE(e, n) {
      int tap = (int)(e % 9);
      int ci = (int)((e / 9) % ci_n), co = (int)(e / (9 * (int64_t)ci_n));
      bf w = __float2bfloat16_rn(theta[tab.off_w[l] + e]);
      int ky = tap / 3, kx = tap % 3;
      wpk[tab.off_pk[l] + (((int64_t)tap * (ci_n / 8) + ci / 8) * co_n + co) * 8 + ci % 8] = w;
      int tt = (2 - ky) * 3 + (2 - kx);
      wpkT[tab.off_pk[l] + (((int64_t)tt * (co_n / 8) + co / 8) * ci_n + ci) * 8 + co % 8] = w;
    }
  }
}

__global__ void k_adam(float* __restrict__ theta, const float* __restrict__ grad, float* __restrict__ m,
                       float* __restrict__ v, int64_t n, float lr, float b1, float b2, float eps, float bc1, float bc2) {
  GRID_STRIDE(k, n) {
    float g = grad[k];
    float mk = b1 * m[k] + (1.f - b1) * g;
    float vk = b2 * v[k] + (1.f - b2) * g * g;
    m[k] = mk;
    v[k] = vk;
    theta[k] -= lr * (mk / bc1) / (sqrtf(vk / bc2) + eps);
  }
}

// ------------------------------------------------------------ host side
static int blocks_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  return (int)(b < 1 ? 1 : (b > 152 * 16 ? 152 * 16 : b));
}

struct Ctx {
  Net* g;
  cudaStream_t st;
  Solver* s;  // when run inside a solver step: launches are counted and profiled there
};

#define GL(C, NAME, BYTES, ...)                          \
  do {                                                   \
    if ((C).s) {                                         \
      FS_LAUNCH((C).s, NAME, BYTES, __VA_ARGS__);        \
    } else {                                             \
      __VA_ARGS__;                                       \
      (C).g->launches++;                                 \
    }                                                    \
  } while (0)

static cudaError_t ensure_capacity(Net* g, int B, int H, int W) {
  if (B <= g->capB && H <= g->capH && W <= g->capW) return cudaSuccess;
  int nB = B > g->capB ? B : g->capB, nH = H > g->capH ? H : g->capH, nW = W > g->capW ? W : g->capW;
  for (int k = 0; k < NBUF; k++) {
    if (g->buf[k]) cudaFree(g->buf[k]);
    g->buf[k] = nullptr;
  }
  if (g->out) cudaFree(g->out);
  if (g->gin) cudaFree(g->gin);
  if (g->gmask) cudaFree(g->gmask);
  if (g->res) cudaFree(g->res);
  g->out = g->gin = g->gmask = g->res = nullptr;
  cudaError_t e;
  for (int k = 0; k < NBUF; k++) {
    size_t bytes = (size_t)level_pixels(g, nB, nH, nW, kBufLevel[k]) * kBufCh[k] * 2;
    if ((e = cudaMalloc(&g->buf[k], bytes))) return e;
  }
  size_t npix = (size_t)nB * nH * nW;
  if ((e = cudaMalloc(&g->out, npix * 4))) return e;
  if ((e = cudaMalloc(&g->gin, npix * 4))) return e;
  if ((e = cudaMalloc(&g->gmask, npix * 4))) return e;
  if ((e = cudaMalloc(&g->res, npix * 4))) return e;
  g->capB = nB;
  g->capH = nH;
  g->capW = nW;
  return cudaSuccess;
}

static cudaError_t conv(const Ctx& c, int l, bool transposed, const bf* in, const conv::ConvOut& o, int flags, int B,
                        int H, int W) {
  Net* g = c.g;
  const int ci = transposed ? kCO[l] : kCI[l], co = transposed ? kCI[l] : kCO[l];
  const bf* w = (transposed ? g->wpkT : g->wpk) + g->off_pk[l];
  const float* bias = transposed ? g->zero_bias : g->theta + g->off_b[l];
  cudaError_t e = cudaSuccess;
  const double bytes = (double)(ci + co) * 2 * B * H * W;
  GL(c, "guess_conv", bytes, e = conv::conv3x3(ci, co, flags, in, w, bias, o, B, H, W, g->err, c.st, true));
  return e;
}

#define CK(expr)                          \
  do {                                    \
    cudaError_t _e = (expr);              \
    if (_e != cudaSuccess) return _e;     \
  } while (0)

using conv::ConvOut;

// a plain layer: out (ReLU'd except the network's last, which is f32 planar)
static ConvOut to(void* out) {
  ConvOut o;
  o.out = out;
  return o;
}
// + the 2 x 2 sums times scale (0 where mask, if given, is not > 0)
static ConvOut to_pool(void* out, void* pool, float scale, const void* mask = nullptr) {
  ConvOut o = to(out);
  o.pool = pool;
  o.pool_scale = scale;
  o.pool_mask = mask;
  return o;
}
// + fine + scale * up(out) into up, on the next finer level (out may be null)
static ConvOut to_up(void* out, void* up, const void* fine, float scale, const void* mask = nullptr) {
  ConvOut o = to(out);
  o.up = up;
  o.fine = fine;
  o.scale = scale;
  o.up_mask = mask;
  return o;
}

// the network on x0 (already in buf[X0]); result in out (f32 [B][H][W]).  Pooling and the
// upsampled skip sums are made by the epilogue of the layer before them.
static cudaError_t forward(const Ctx& c, int B, int H, int W, float* out) {
  using namespace conv;
  Net* g = c.g;
  bf** b = g->buf;
  const int Hl1 = H >> 1, Wl1 = W >> 1, Hl2 = H >> 2, Wl2 = W >> 2, Hl3 = H >> 3, Wl3 = W >> 3;
  constexpr int R = kOutStore | kOutRelu;
  CK(conv(c, LA, false, b[X0], to(b[A0]), R, B, H, W));
  CK(conv(c, LB, false, b[A0], to_pool(b[A0B], b[Q1], 0.25f), R | kOutPool, B, H, W));
  CK(conv(c, LC, false, b[Q1], to_pool(b[A1], b[Q2], 0.25f), R | kOutPool, B, Hl1, Wl1));
  CK(conv(c, LD, false, b[Q2], to_pool(b[A2], b[Q3], 0.25f), R | kOutPool, B, Hl2, Wl2));
  CK(conv(c, LE, false, b[Q3], to(b[A3]), R, B, Hl3, Wl3));
  CK(conv(c, LF, false, b[A3], to_up(b[F3], b[S2], b[A2], 1.f), R | kOutUp, B, Hl3, Wl3));
  CK(conv(c, LG, false, b[S2], to_up(b[G2], b[S1], b[A1], 1.f), R | kOutUp, B, Hl2, Wl2));
  CK(conv(c, LH, false, b[S1], to_up(b[H1], b[S0], b[A0B], 1.f), R | kOutUp, B, Hl1, Wl1));
  CK(conv(c, LI, false, b[S0], to(b[I0]), R, B, H, W));
  CK(conv(c, LJ, false, b[I0], to(out), kOutPlanar, B, H, W));
  return cudaSuccess;
}

static cudaError_t ensure_corr(Net* g, int64_t floats) {
  if (floats <= g->corr_cap) return cudaSuccess;
  if (g->corr_part) cudaFree(g->corr_part);
  g->corr_part = nullptr;
  CK(cudaMalloc(&g->corr_part, floats * 4));
  g->corr_cap = floats;
  return cudaSuccess;
}

template <int CIN, int COUT, int TY, int PX, int NDX>
static cudaError_t wgrad_tc(const Ctx& c, int l, Buf xbuf, Buf gbuf, int B, int H, int W) {
  using C = WgCfg<CIN, COUT, TY, PX, NDX>;
  Net* g = c.g;
  auto* kernel = k_wgrad_tc<CIN, COUT, TY, PX, NDX>;
  static std::atomic<uint64_t> attr{0};
  const uint64_t bit = 1ull << (g->device & 63);
  if (!(attr.load() & bit)) {
    CK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM));
    attr.fetch_or(bit);
  }
  // (ordinary launches: as dependent ones these two made the backward pass 2% slower)
  // one wave: as many CTAs as the shared memory lets an SM hold, over the taps' groups
  constexpr int per_sm = C::SMEM <= 110 * 1024 ? 2 : 1;
  const int64_t ntiles = (int64_t)B * ((H + TY - 1) / TY) * ((W + PX - 1) / PX);
  const int P = (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, per_sm * kSMs * NDX / 3));
  const int64_t nw = (int64_t)C::MROWS * COUT;
  CK(ensure_corr(g, (int64_t)P * (nw + COUT)));
  float* part = g->corr_part;
  float* bpart = part + (int64_t)P * nw;
  GL(c, "guess_wgrad", (double)(CIN + COUT) * 2 * B * H * W,
     (kernel<<<dim3(P, 3 / NDX), kWgThreads + 32, C::SMEM, c.st>>>(
         reinterpret_cast<const uint4*>(g->buf[xbuf]), reinterpret_cast<const uint4*>(g->buf[gbuf]), B, H, W, part,
         bpart, g->err)));
  CK(cudaGetLastError());
  GL(c, "guess_wgrad_reduce", (double)P * (nw + COUT) * 4,
     k_wgrad_reduce<<<(int)((nw + COUT + 31) / 32), 256, 0, c.st>>>(part, bpart, P, CIN, COUT, g->grad + g->off_w[l],
                                                                   g->grad + g->off_b[l]));
  return cudaGetLastError();
}

// the (c_in, c_out) pairs of the network: rows and pixels of a tile (two stages
// in shared memory, two CTAs an SM at the wide levels), horizontal taps per CTA
// (one where three would not fit the 512 TMEM columns)
static cudaError_t wgrad(const Ctx& c, int l, Buf xbuf, Buf gbuf, int B, int H, int W) {
  const int ci = kCI[l], co = kCO[l];
#define FS_WG(a, b, ty, px, ndx) \
  if (ci == a && co == b) return wgrad_tc<a, b, ty, px, ndx>(c, l, xbuf, gbuf, B, H, W);
  FS_WG(16, 16, 4, 128, 3)
  FS_WG(16, 32, 2, 128, 3)
  FS_WG(32, 16, 2, 128, 3)
  FS_WG(32, 64, 1, 128, 3)
  FS_WG(64, 128, 1, 128, 1)
  FS_WG(128, 64, 1, 64, 1)
  FS_WG(64, 32, 1, 128, 3)
#undef FS_WG
  return cudaErrorInvalidValue;
}

// loss against target (f32 [B][H][W]) and the gradient of every parameter into g->grad
static cudaError_t backward(const Ctx& c, const float* target, int B, int H, int W) {
  using namespace conv;
  Net* g = c.g;
  bf** b = g->buf;
  const int64_t npix = (int64_t)H * W;
  const int Hl1 = H >> 1, Wl1 = W >> 1, Hl2 = H >> 2, Wl2 = W >> 2, Hl3 = H >> 3, Wl3 = W >> 3;
  CK(cudaMemsetAsync(g->acc, 0, sizeof(double) * (B + 1), c.st));
  const bool with_res = g->w_r != 0.0;
  // rows of a strip: long ones read their two extra rows less often, short ones
  // give small images more warps
  const int64_t cols = (W + kLossCols - 1) / kLossCols;
  const int rows = B * cols * (H / 32) >= kSMs * 16 ? 32 : 8;
  const dim3 lb((unsigned)((cols * ((H + rows - 1) / rows) + kLossWarps - 1) / kLossWarps), B);
  if (with_res)
    GL(c, "guess_loss", npix * B * 12.0,
       k_loss_res<<<lb, 32 * kLossWarps, 0, c.st>>>(g->out, target, g->res, g->acc, H, W, B, rows, g->w_r));
  else
    GL(c, "guess_loss", npix * B * 8.0,
       k_loss_mean<<<dim3((unsigned)std::min<int64_t>((npix + 255) / 256, 256), B), 32 * kLossWarps, 0, c.st>>>(
           g->out, target, g->acc, npix));
  GL(c, "guess_loss", npix * B * 40.0,
     launch_dependent(true, k_loss_seed, lb, dim3(32 * kLossWarps), 0, c.st, g->out, target,
                      with_res ? g->res : nullptr, g->acc, (uint4*)b[GJ], H, W, B, rows, g->w_p, g->w_r));
  CK(cudaGetLastError());
  // Each layer's weight gradient, then the gradient of its input; the ReLU
  // masks, the gradients of the upsampled skip sums (2 x 2 sums) and of the
  // pooling (a quarter of the coarse gradient, added) are made by the epilogue.
  constexpr int M = kOutStore | kOutMask, P = kOutStore | kOutPool | kOutPoolMask, U = kOutUp | kOutUpMask;
  auto masked = [&](Buf out, Buf act) {
    ConvOut o = to(b[out]);
    o.mask = b[act];
    return o;
  };
  CK(wgrad(c, LJ, I0, GJ, B, H, W));
  CK(conv(c, LJ, true, b[GJ], masked(DI0, I0), M, B, H, W));
  CK(wgrad(c, LI, S0, DI0, B, H, W));
  CK(conv(c, LI, true, b[DI0], to_pool(b[DS0], b[DH1], 1.f, b[H1]), P, B, H, W));
  CK(wgrad(c, LH, S1, DH1, B, Hl1, Wl1));
  CK(conv(c, LH, true, b[DH1], to_pool(b[DS1], b[DG2], 1.f, b[G2]), P, B, Hl1, Wl1));
  CK(wgrad(c, LG, S2, DG2, B, Hl2, Wl2));
  CK(conv(c, LG, true, b[DG2], to_pool(b[DS2], b[DF3], 1.f, b[F3]), P, B, Hl2, Wl2));
  CK(wgrad(c, LF, A3, DF3, B, Hl3, Wl3));
  CK(conv(c, LF, true, b[DF3], masked(DA3, A3), M, B, Hl3, Wl3));
  CK(wgrad(c, LE, Q3, DA3, B, Hl3, Wl3));
  CK(conv(c, LE, true, b[DA3], to_up(nullptr, b[DS2], b[DS2], 0.25f, b[A2]), U, B, Hl3, Wl3));
  CK(wgrad(c, LD, Q2, DS2, B, Hl2, Wl2));
  CK(conv(c, LD, true, b[DS2], to_up(nullptr, b[DS1], b[DS1], 0.25f, b[A1]), U, B, Hl2, Wl2));
  CK(wgrad(c, LC, Q1, DS1, B, Hl1, Wl1));
  CK(conv(c, LC, true, b[DS1], to_up(nullptr, b[DS0], b[DS0], 0.25f, b[A0B]), U, B, Hl1, Wl1));
  CK(wgrad(c, LB, A0, DS0, B, H, W));
  CK(conv(c, LB, true, b[DS0], masked(DA0, A0), M, B, H, W));
  CK(wgrad(c, LA, X0, DA0, B, H, W));
  return cudaSuccess;
}

static cudaError_t repack(Net* g, cudaStream_t st) {
  PackTable tab;
  for (int l = 0; l < NL; l++) {
    tab.off_w[l] = g->off_w[l];
    tab.off_pk[l] = g->off_pk[l];
    tab.ci[l] = kCI[l];
    tab.co[l] = kCO[l];
  }
  k_pack<<<152 * 4, 256, 0, st>>>(g->theta, g->wpk, g->wpkT, tab);
  g->launches++;
  return cudaGetLastError();
}

// He-normal initial weights (ReLU layers; the output layer scaled by 0.1),
// zero biases; the padded input channels of layer A start (and stay) at zero.
// Gaussian draws: SplitMix64 + Box-Muller.
static void init_params(std::vector<float>& th, const Net* g, uint64_t seed) {
  uint64_t st = seed * 0x9E3779B97F4A7C15ull + 0x632BE59BD9B4E5ull;
  auto next = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
  };
  auto unif = [&]() { return ((next() >> 11) + 0.5) * (1.0 / 9007199254740992.0); };
  for (int l = 0; l < NL; l++) {
    const int ci = kCI[l], co = kCO[l];
    const double fan = 9.0 * (l == LA ? 2 : ci);
    const double sd = sqrt(2.0 / fan) * (kRelu[l] ? 1.0 : 0.1);
    for (int o = 0; o < co; o++)
      for (int i = 0; i < ci; i++)
        for (int t = 0; t < 9; t++) {
          double u1 = unif(), u2 = unif();
          double z = sqrt(-2.0 * log(u1)) * cos(6.283185307179586 * u2);
          th[g->off_w[l] + ((int64_t)o * ci + i) * 9 + t] = (l == LA && i >= 2) ? 0.f : (float)(z * sd);
        }
    for (int o = 0; o < co; o++) th[g->off_b[l] + o] = 0.f;
  }
}

}  // namespace guess

// ---------------------------------------------------------- solver hooks
// The network runs at 1/f of the grid resolution (f = 1 or 2).
// h^2 * (d averaged over f x f fine cells) at net resolution, the solid mask
// at the net cell centres, and the sum of squares of the former (for sigma).
__global__ void __launch_bounds__(256)
    k_guess_in(const float* __restrict__ dh, const float* __restrict__ dl, int nx, int ny, int f, float h2,
               float* gin, float* gmask, const float* __restrict__ disks, int ndisk, float dxn, float dyn, float lx,
               float ly, float width, RedCtx ctx) {
  const int Wn = nx / f, Hn = ny / f;
  const int n = Wn * Hn;  // grids are capped at 2^30 cells
  double s2 = 0.0;
  GRID_STRIDE32(k, n) {
    int J = k / Wn, I = k - J * Wn;
    int64_t c = (int64_t)(f * J) * nx + f * I;
    // the divergence is a double-float pair (MIXED) or a plain f32 field (dl == nullptr)
    auto at = [&](int64_t q) { return dl ? __fadd_rn(dh[q], dl[q]) : dh[q]; };
    float d = f == 1 ? at(c) : 0.25f * (at(c) + at(c + 1) + at(c + nx) + at(c + nx + 1));
    float x = h2 * d;
    gin[k] = x;
    s2 += (double)x * x;
    float m = 0.f;
    float px = (I + 0.5f) * dxn, py = (J + 0.5f) * dyn;
    for (int q = 0; q < ndisk; q++) {
      float ax = px - disks[7 * q], ay = py - disks[7 * q + 1];
      ax -= lx * floorf(ax / lx + 0.5f);
      ay -= ly * floorf(ay / ly + 0.5f);
      float chi = 0.5f * (1.f - tanhf(fminf(fmaxf((sqrtf(ax * ax + ay * ay) - disks[7 * q + 2]) / width, -10.f), 10.f)));
      m = fmaxf(m, chi);
    }
    gmask[k] = m;
  }
  block_sum2_finish(s2, 0.0, ctx);
}

// pressure guess = sigma * out at the fine cells: a copy for f = 1, the
// bilinear multigrid prolongation stencil for f = 2; pl = 0
__global__ void __launch_bounds__(256) k_guess_out(const float* __restrict__ out, const double* __restrict__ sumsq,
                                                   int64_t nnorm, float* __restrict__ ph, float* __restrict__ pl,
                                                   int nx, int ny, int f) {
  const int Wn = nx / f, Hn = ny / f;
  const float sig = guess::block_sigma(sumsq, nnorm);
  const int n = nx * ny;  // grids are capped at 2^30 cells
  GRID_STRIDE32(k, n) {
    float v;
    if (f == 1) {
      v = out[k] * sig;
    } else {
      int j = k / nx, i = k - j * nx;
      int ci0 = (i & 1) ? (i >> 1) : (i >> 1) - 1, cj0 = (j & 1) ? (j >> 1) : (j >> 1) - 1;
      float fx = (i & 1) ? 0.25f : 0.75f, fy = (j & 1) ? 0.25f : 0.75f;
      int x0 = ci0 < 0 ? ci0 + Wn : ci0, x1 = ci0 + 1 >= Wn ? ci0 + 1 - Wn : ci0 + 1;
      int y0 = cj0 < 0 ? cj0 + Hn : cj0, y1 = cj0 + 1 >= Hn ? cj0 + 1 - Hn : cj0 + 1;
      float a = out[(int64_t)y0 * Wn + x0], b = out[(int64_t)y0 * Wn + x1];
      float c = out[(int64_t)y1 * Wn + x0], d = out[(int64_t)y1 * Wn + x1];
      v = ((1.f - fy) * ((1.f - fx) * a + fx * b) + fy * ((1.f - fx) * c + fx * d)) * sig;
    }
    ph[k] = v;
    if (pl) pl[k] = 0.f;
  }
}

bool guess_supported(const Solver* s, int f) {
  if (f != 1 && f != 2) return false;
  const int m = 8 * f;
  return s->g.nx % m == 0 && s->g.ny % m == 0;
}

// enqueue the guess into (ph, pl) (MIXED) or p32 (F32) on s->stream
int guess_enqueue(Solver* s, fs_guess* handle, int f) {
  guess::Net* g = reinterpret_cast<guess::Net*>(handle);
  const Grid& gr = s->g;
  const int Wn = gr.nx / f, Hn = gr.ny / f;
  const float h2 = (float)(f * f * gr.dxd * gr.dxd);
  guess::Ctx c{g, s->stream, s};
  double* gsum = g->acc;
  RedCtx ctx = red_ctx(s, gsum);
  const int nd = (int)s->disks.size();
  const float* dsk = static_cast<const float*>(s->d_disks);
  const double width = s->prm.solid_mask_width * gr.dxd;
  int blocks = (int)std::min<int64_t>(((int64_t)Wn * Hn + 255) / 256, 152 * 8);
  if (blocks > s->red_cap) blocks = s->red_cap;
  FS_LAUNCH(s, "guess_in", (double)s->n * 8,
            k_guess_in<<<blocks, 256, 0, s->stream>>>(s->mixed ? s->dh : s->div32, s->mixed ? s->dl : nullptr,
                                                      gr.nx, gr.ny, f, h2, g->gin, g->gmask, dsk, nd,
                                                      (float)(f * gr.dxd), (float)(f * gr.dyd), (float)s->prm.lx,
                                                      (float)s->prm.ly, (float)width, ctx));
  const int64_t npn = (int64_t)Wn * Hn;
  FS_LAUNCH(s, "guess_prep", (double)npn * 40,
            guess::k_prep<<<guess::blocks_for(npn), 256, 0, s->stream>>>(g->gin, g->gmask, (uint4*)g->buf[guess::X0],
                                                                         npn, gsum, npn));
  cudaError_t e = guess::forward(c, 1, Hn, Wn, g->out);
  if (e != cudaSuccess) return fail_status(s, FS_ERR_CUDA, std::string("pressure guess: ") + cudaGetErrorString(e));
  FS_LAUNCH(s, "guess_out", (double)s->n * 8,
            k_guess_out<<<guess::blocks_for(s->n), 256, 0, s->stream>>>(
                g->out, gsum, npn, s->mixed ? s->ph : s->p32, s->mixed ? s->pl : nullptr, gr.nx, gr.ny, f));
  return FS_OK;
}

int guess_prepare(Solver* s, fs_guess* handle, int f) {
  guess::Net* g = reinterpret_cast<guess::Net*>(handle);
  cudaError_t e = guess::ensure_capacity(g, 1, s->g.ny / f, s->g.nx / f);
  if (e != cudaSuccess) return fail_status(s, FS_ERR_OUT_OF_MEMORY, std::string("pressure guess buffers: ") + cudaGetErrorString(e));
  return FS_OK;
}

// the divergence, mask and pressure of the last projection at 1/factor of the
// grid resolution (block averages; the mask at the coarse cell centres)
__global__ void k_pair(const float* __restrict__ dh, const float* __restrict__ dl, const float* __restrict__ ph,
                       const float* __restrict__ pl, int nx, int ny, int f, float* div, float* mask, float* p,
                       const float* __restrict__ disks, int ndisk, float dxc, float dyc, float lx, float ly,
                       float width) {
  const int Wc = nx / f, Hc = ny / f;
  const int64_t n = (int64_t)Wc * Hc;
  GRID_STRIDE(k, n) {
    int I = (int)(k % Wc), J = (int)(k / Wc);
    double sd = 0.0, sp = 0.0;
    for (int a = 0; a < f; a++)
      for (int b = 0; b < f; b++) {
        int64_t c = (int64_t)(f * J + a) * nx + f * I + b;
        sd += (double)dh[c] + (dl ? (double)dl[c] : 0.0);
        sp += (double)ph[c] + (pl ? (double)pl[c] : 0.0);
      }
    div[k] = (float)(sd / (f * f));
    p[k] = (float)(sp / (f * f));
    float m = 0.f;
    float px = (I + 0.5f) * dxc, py = (J + 0.5f) * dyc;
    for (int q = 0; q < ndisk; q++) {
      float ax = px - disks[7 * q], ay = py - disks[7 * q + 1];
      ax -= lx * floorf(ax / lx + 0.5f);
      ay -= ly * floorf(ay / ly + 0.5f);
      float chi = 0.5f * (1.f - tanhf(fminf(fmaxf((sqrtf(ax * ax + ay * ay) - disks[7 * q + 2]) / width, -10.f), 10.f)));
      m = fmaxf(m, chi);
    }
    mask[k] = m;
  }
}

int dump_pair(Solver* s, int f, float* div, float* mask, float* p) {
  const Grid& gr = s->g;
  const double width = s->prm.solid_mask_width * gr.dxd;
  const int nd = (int)s->disks.size();
  const int64_t n = (int64_t)(gr.nx / f) * (gr.ny / f);
  float* tmp = nullptr;
  cudaError_t e = cudaMalloc(&tmp, n * 3 * sizeof(float));
  if (e != cudaSuccess) return fail_status(s, FS_ERR_OUT_OF_MEMORY, "fs_dump_pair: cudaMalloc failed");
  k_pair<<<guess::blocks_for(n), 256, 0, s->stream>>>(
      s->mixed ? s->dh : s->div32, s->mixed ? s->dl : nullptr, s->mixed ? s->ph : s->p32, s->mixed ? s->pl : nullptr,
      gr.nx, gr.ny, f, tmp, tmp + n, tmp + 2 * n, static_cast<const float*>(s->d_disks), nd, (float)(f * gr.dxd),
      (float)(f * gr.dyd), (float)s->prm.lx, (float)s->prm.ly, (float)width);
  s->launches++;
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(div, tmp, n * 4, cudaMemcpyDeviceToHost, s->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(mask, tmp + n, n * 4, cudaMemcpyDeviceToHost, s->stream);
  if (e == cudaSuccess) e = cudaMemcpyAsync(p, tmp + 2 * n, n * 4, cudaMemcpyDeviceToHost, s->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s->stream);
  cudaFree(tmp);
  if (e != cudaSuccess) return fail_status(s, FS_ERR_CUDA, std::string("fs_dump_pair: ") + cudaGetErrorString(e));
  return FS_OK;
}

// the same pair into caller-owned device buffers, enqueued on the solver's
// stream (no allocation, no synchronisation)
int dump_pair_device(Solver* s, int f, float* div, float* mask, float* p) {
  const Grid& gr = s->g;
  const double width = s->prm.solid_mask_width * gr.dxd;
  const int nd = (int)s->disks.size();
  const int64_t n = (int64_t)(gr.nx / f) * (gr.ny / f);
  k_pair<<<guess::blocks_for(n), 256, 0, s->stream>>>(
      s->mixed ? s->dh : s->div32, s->mixed ? s->dl : nullptr, s->mixed ? s->ph : s->p32, s->mixed ? s->pl : nullptr,
      gr.nx, gr.ny, f, div, mask, p, static_cast<const float*>(s->d_disks), nd, (float)(f * gr.dxd),
      (float)(f * gr.dyd), (float)s->prm.lx, (float)s->prm.ly, (float)width);
  s->launches++;
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return fail_status(s, FS_ERR_CUDA, std::string("fs_dump_pair_device: ") + cudaGetErrorString(e));
  return FS_OK;
}

}  // namespace fs

// ====================================================================== C ABI
using namespace fs;
using namespace fs::guess;

static thread_local std::string g_guess_err;

static int gfail(Net* g, int code, const std::string& m) {
  if (g) g->err_msg = m;
  record_error(m);
  return code;
}

static int gcuda(Net* g, cudaError_t e, const char* where) {
  if (e == cudaSuccess) return FS_OK;
  return gfail(g, e == cudaErrorMemoryAllocation ? FS_ERR_OUT_OF_MEMORY : FS_ERR_CUDA,
               std::string(where) + ": " + cudaGetErrorString(e));
}

extern "C" FS_API int fs_guess_create(int32_t device, uint64_t seed, fs_guess** out) {
  if (!out) return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_guess_create: NULL out");
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
    return gfail(nullptr, FS_ERR_NO_DEVICE, "fs_guess_create: no CUDA device");
  if (device < 0 || device >= ndev) return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_guess_create: bad device");
  cudaError_t e = cudaSetDevice(device);
  if (e != cudaSuccess) return gcuda(nullptr, e, "cudaSetDevice");
  Net* g = new Net();
  g->device = device;
  int64_t k = 0, kp = 0;
  for (int l = 0; l < NL; l++) {
    g->off_w[l] = k;
    k += (int64_t)kCI[l] * kCO[l] * 9;
    g->off_b[l] = k;
    k += kCO[l];
    g->off_pk[l] = kp;
    kp += (int64_t)kCI[l] * kCO[l] * 9;
  }
  g->nparam = k;
  g->npk = kp;
  std::vector<float> th(k);
  init_params(th, g, seed);
#define GA(p, bytes)                                   \
  if ((e = cudaMalloc(&(p), (bytes))) != cudaSuccess) { \
    fs_guess_destroy(reinterpret_cast<fs_guess*>(g));  \
    return gcuda(nullptr, e, "fs_guess_create");        \
  }
  GA(g->theta, k * 4);
  GA(g->grad, k * 4);
  GA(g->m, k * 4);
  GA(g->v, k * 4);
  GA(g->wpk, kp * 2);
  GA(g->wpkT, kp * 2);
  GA(g->zero_bias, 256 * 4);
  GA(g->err, 4);
  GA(g->acc, 4096 * 8);
#undef GA
  if ((e = cudaStreamCreateWithFlags(&g->stream, cudaStreamNonBlocking)) != cudaSuccess) {
    fs_guess_destroy(reinterpret_cast<fs_guess*>(g));
    return gcuda(nullptr, e, "cudaStreamCreate");
  }
  cudaMemsetAsync(g->grad, 0, k * 4, g->stream);
  cudaMemsetAsync(g->m, 0, k * 4, g->stream);
  cudaMemsetAsync(g->v, 0, k * 4, g->stream);
  cudaMemsetAsync(g->zero_bias, 0, 256 * 4, g->stream);
  cudaMemsetAsync(g->err, 0, 4, g->stream);
  cudaMemcpyAsync(g->theta, th.data(), k * 4, cudaMemcpyHostToDevice, g->stream);
  repack(g, g->stream);
  e = cudaStreamSynchronize(g->stream);
  if (e != cudaSuccess) {
    fs_guess_destroy(reinterpret_cast<fs_guess*>(g));
    return gcuda(nullptr, e, "fs_guess_create");
  }
  *out = reinterpret_cast<fs_guess*>(g);
  return FS_OK;
}

extern "C" FS_API void fs_guess_destroy(fs_guess* h) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g) return;
  cudaSetDevice(g->device);
  if (g->stream) cudaStreamSynchronize(g->stream);
  for (int k = 0; k < NBUF; k++)
    if (g->buf[k]) cudaFree(g->buf[k]);
  float* fl[] = {g->theta, g->grad, g->m, g->v, g->zero_bias, g->out, g->gin, g->gmask, g->res, g->corr_part};
  for (float* p : fl)
    if (p) cudaFree(p);
  if (g->wpk) cudaFree(g->wpk);
  if (g->wpkT) cudaFree(g->wpkT);
  if (g->err) cudaFree(g->err);
  if (g->acc) cudaFree(g->acc);
  if (g->stream) cudaStreamDestroy(g->stream);
  delete g;
}

extern "C" FS_API int64_t fs_guess_num_params(const fs_guess* h) {
  const Net* g = reinterpret_cast<const Net*>(h);
  return g ? g->nparam : -1;
}

extern "C" FS_API int fs_guess_get_params(fs_guess* h, float* host, int64_t n) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g || !host) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_get_params: NULL argument");
  if (n != g->nparam) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_get_params: wrong parameter count");
  cudaSetDevice(g->device);
  cudaError_t e = cudaMemcpyAsync(host, g->theta, n * 4, cudaMemcpyDeviceToHost, g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  return gcuda(g, e, "fs_guess_get_params");
}

extern "C" FS_API int fs_guess_set_params(fs_guess* h, const float* host, int64_t n) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g || !host) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_set_params: NULL argument");
  if (n != g->nparam) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_set_params: wrong parameter count");
  cudaSetDevice(g->device);
  cudaError_t e = cudaMemcpyAsync(g->theta, host, n * 4, cudaMemcpyHostToDevice, g->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(g->m, 0, n * 4, g->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(g->v, 0, n * 4, g->stream);
  if (e == cudaSuccess) e = repack(g, g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  g->adam_t = 0;
  return gcuda(g, e, "fs_guess_set_params");
}

static int check_shape(Net* g, int B, int H, int W, const char* who) {
  if (B < 1 || H < 8 || W < 8 || H % 8 || W % 8)
    return gfail(g, FS_ERR_INVALID_ARGUMENT, std::string(who) + ": batch >= 1 and H, W multiples of 8 (>= 8)");
  if ((int64_t)B * H * W * 16 >= ((int64_t)1 << 31))
    return gfail(g, FS_ERR_INVALID_ARGUMENT, std::string(who) + ": batch x H x W x 16 must stay below 2^31");
  return FS_OK;
}

static int read_err(Net* g, const char* who) {
  int h = 0;
  cudaError_t e = cudaMemcpyAsync(&h, g->err, 4, cudaMemcpyDeviceToHost, g->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(g->stream);
  if (e != cudaSuccess) return gcuda(g, e, who);
  if (h) {
    cudaMemsetAsync(g->err, 0, 4, g->stream);
    return gfail(g, FS_ERR_CUDA, std::string(who) + ": a tensor-core completion wait timed out");
  }
  return FS_OK;
}

// out = network(div_n, mask): device pointers, f32 [B][H][W]
extern "C" FS_API int fs_guess_predict(fs_guess* h, const float* d_div, const float* d_mask, int32_t B, int32_t H,
                                       int32_t W, float* d_out) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g || !d_div || !d_out) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_predict: NULL argument");
  int rc = check_shape(g, B, H, W, "fs_guess_predict");
  if (rc) return rc;
  cudaSetDevice(g->device);
  cudaError_t e = ensure_capacity(g, B, H, W);
  if (e != cudaSuccess) return gcuda(g, e, "fs_guess_predict");
  Ctx c{g, g->stream, nullptr};
  const int64_t np = (int64_t)B * H * W;
  k_prep<<<blocks_for(np), 256, 0, g->stream>>>(d_div, d_mask, (uint4*)g->buf[X0], np, nullptr, 1);
  g->launches++;
  if ((e = forward(c, B, H, W, d_out)) != cudaSuccess) return gcuda(g, e, "fs_guess_predict");
  return read_err(g, "fs_guess_predict");
}

static int loss_grad_impl(Net* g, const float* d_div, const float* d_mask, const float* d_tgt, int B, int H, int W,
                          double* loss, const char* who) {
  int rc = check_shape(g, B, H, W, who);
  if (rc) return rc;
  if (B > 4000) return gfail(g, FS_ERR_INVALID_ARGUMENT, std::string(who) + ": batch above 4000");
  cudaSetDevice(g->device);
  cudaError_t e = ensure_capacity(g, B, H, W);
  if (e != cudaSuccess) return gcuda(g, e, who);
  Ctx c{g, g->stream, nullptr};
  const int64_t np = (int64_t)B * H * W;
  k_prep<<<blocks_for(np), 256, 0, g->stream>>>(d_div, d_mask, (uint4*)g->buf[X0], np, nullptr, 1);
  g->launches++;
  if ((e = forward(c, B, H, W, g->out)) != cudaSuccess) return gcuda(g, e, who);
  if ((e = backward(c, d_tgt, B, H, W)) != cudaSuccess) return gcuda(g, e, who);
  if (loss) {
    e = cudaMemcpyAsync(loss, g->acc + B, 8, cudaMemcpyDeviceToHost, g->stream);
    if (e != cudaSuccess) return gcuda(g, e, who);
  }
  return FS_OK;
}

extern "C" FS_API int fs_guess_loss_grad(fs_guess* h, const float* d_div, const float* d_mask, const float* d_target,
                                         int32_t B, int32_t H, int32_t W, double* loss, float* d_grad) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g || !d_div || !d_target) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_loss_grad: NULL argument");
  int rc = loss_grad_impl(g, d_div, d_mask, d_target, B, H, W, loss, "fs_guess_loss_grad");
  if (rc) return rc;
  if (d_grad) {
    cudaError_t e = cudaMemcpyAsync(d_grad, g->grad, g->nparam * 4, cudaMemcpyDeviceToDevice, g->stream);
    if (e != cudaSuccess) return gcuda(g, e, "fs_guess_loss_grad");
  }
  return read_err(g, "fs_guess_loss_grad");
}

extern "C" FS_API int fs_guess_train_step(fs_guess* h, const float* d_div, const float* d_mask, const float* d_target,
                                          int32_t B, int32_t H, int32_t W, float lr, double* loss) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g || !d_div || !d_target) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_train_step: NULL argument");
  if (!(lr > 0.f)) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_train_step: lr must be positive");
  int rc = loss_grad_impl(g, d_div, d_mask, d_target, B, H, W, loss, "fs_guess_train_step");
  if (rc) return rc;
  g->adam_t++;
  const float b1 = 0.9f, b2 = 0.999f;
  const float bc1 = (float)(1.0 - pow(0.9, (double)g->adam_t)), bc2 = (float)(1.0 - pow(0.999, (double)g->adam_t));
  k_adam<<<blocks_for(g->nparam), 256, 0, g->stream>>>(g->theta, g->grad, g->m, g->v, g->nparam, lr, b1, b2, 1e-8f,
                                                      bc1, bc2);
  g->launches++;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = repack(g, g->stream);
  if (e != cudaSuccess) return gcuda(g, e, "fs_guess_train_step");
  return loss ? read_err(g, "fs_guess_train_step") : FS_OK;
}

extern "C" FS_API int fs_guess_set_loss(fs_guess* h, double w_pressure, double w_residual) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_set_loss: NULL handle");
  if (!(w_pressure >= 0) || !(w_residual >= 0) || !(w_pressure + w_residual > 0) || !std::isfinite(w_pressure) ||
      !std::isfinite(w_residual))
    return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_set_loss: weights must be finite, >= 0, not both 0");
  g->w_p = w_pressure;
  g->w_r = w_residual;
  return FS_OK;
}

extern "C" FS_API int fs_guess_sync(fs_guess* h) {
  Net* g = reinterpret_cast<Net*>(h);
  if (!g) return gfail(g, FS_ERR_INVALID_ARGUMENT, "fs_guess_sync: NULL handle");
  return read_err(g, "fs_guess_sync");
}

extern "C" FS_API int64_t fs_guess_launch_count(const fs_guess* h) {
  const Net* g = reinterpret_cast<const Net*>(h);
  return g ? g->launches : -1;
}

// ---------------------------------------------------- training-pair files
// "FSPAIR" file: a 40-byte little-endian header then three f32 fields.
//   0  char[8]  magic "FSPAIR\0\1"
//   8  uint32   version (1)
//  12  uint32   nx
//  16  uint32   ny
//  20  uint32   dtype (0 = f32)
//  24  double   dx, the grid spacing of the stored fields
//  32  uint32   nfields (3: div, mask, p)
//  36  uint32   reserved (0)
//  40  div[ny][nx], mask[ny][nx], p[ny][nx]
static const char kPairMagic[8] = {'F', 'S', 'P', 'A', 'I', 'R', 0, 1};

extern "C" FS_API int fs_write_pair_file(const char* path, int32_t nx, int32_t ny, double dx, const float* div,
                                         const float* mask, const float* p) {
  if (!path || !div || !mask || !p || nx < 1 || ny < 1 || !(dx > 0))
    return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_write_pair_file: bad argument");
  FILE* f = fopen(path, "wb");
  if (!f) return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, std::string("fs_write_pair_file: cannot open ") + path);
  unsigned char hdr[40] = {};
  uint32_t u[7] = {1u, (uint32_t)nx, (uint32_t)ny, 0u, 0u, 3u, 0u};
  memcpy(hdr, kPairMagic, 8);
  memcpy(hdr + 8, &u[0], 4);
  memcpy(hdr + 12, &u[1], 4);
  memcpy(hdr + 16, &u[2], 4);
  memcpy(hdr + 20, &u[3], 4);
  memcpy(hdr + 24, &dx, 8);
  memcpy(hdr + 32, &u[5], 4);
  memcpy(hdr + 36, &u[6], 4);
  const size_t n = (size_t)nx * ny;
  bool ok = fwrite(hdr, 1, 40, f) == 40 && fwrite(div, 4, n, f) == n && fwrite(mask, 4, n, f) == n &&
            fwrite(p, 4, n, f) == n;
  ok = (fclose(f) == 0) && ok;
  return ok ? FS_OK : gfail(nullptr, FS_ERR_CUDA, "fs_write_pair_file: write failed");
}

// With div == NULL only the header is read (to size the buffers).
extern "C" FS_API int fs_read_pair_file(const char* path, int32_t* nx, int32_t* ny, double* dx, float* div,
                                        float* mask, float* p) {
  if (!path || !nx || !ny || !dx) return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_read_pair_file: bad argument");
  FILE* f = fopen(path, "rb");
  if (!f) return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, std::string("fs_read_pair_file: cannot open ") + path);
  unsigned char hdr[40];
  uint32_t ver, unx, uny, dtype, nf;
  bool ok = fread(hdr, 1, 40, f) == 40 && memcmp(hdr, kPairMagic, 8) == 0;
  if (ok) {
    memcpy(&ver, hdr + 8, 4);
    memcpy(&unx, hdr + 12, 4);
    memcpy(&uny, hdr + 16, 4);
    memcpy(&dtype, hdr + 20, 4);
    memcpy(dx, hdr + 24, 8);
    memcpy(&nf, hdr + 32, 4);
    ok = ver == 1 && dtype == 0 && nf == 3 && unx > 0 && uny > 0 && unx < (1u << 20) && uny < (1u << 20);
  }
  if (!ok) {
    fclose(f);
    return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_read_pair_file: not a version-1 f32 FSPAIR file");
  }
  *nx = (int32_t)unx;
  *ny = (int32_t)uny;
  if (div) {
    const size_t n = (size_t)unx * uny;
    if (!mask || !p) {
      fclose(f);
      return gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_read_pair_file: NULL field buffer");
    }
    ok = fread(div, 4, n, f) == n && fread(mask, 4, n, f) == n && fread(p, 4, n, f) == n;
  }
  fclose(f);
  return ok ? FS_OK : gfail(nullptr, FS_ERR_INVALID_ARGUMENT, "fs_read_pair_file: truncated file");
}
