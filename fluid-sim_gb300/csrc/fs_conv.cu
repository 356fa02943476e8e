// fs_conv.cu -- 3x3 periodic convolution of NHWC bf16 images on the tcgen05
// tensor cores (implicit GEMM), the building block of the pressure-guess
// network.  No counterpart in the reference.
//
// out[b, y, x, co] = bias[co] + sum_{ky, kx, ci} w[co, ci, ky, kx] * in[b, y + ky - 1, x + kx - 1, ci]
// with periodic wrap in x and y (the flow domain is periodic), optional ReLU.
//
// GEMM view: M = 128 consecutive pixels of one image row, N = C_out (or a part
// of it), K = 9 taps x C_in.  The input rows of a tile are staged as they are in
// memory, in planes of one row and one 8-channel chunk, [row][chunk][130 pixels],
// so that 8 consecutive pixels of a plane form one 128-byte core matrix and
// every tap's A operand is the same tile seen through a descriptor whose start
// address is shifted by (dy, dx) -- no data is rearranged per tap.  Weights are
// packed on the host side of the network as [tap][kc][co][8 ci] (the B operand,
// K-major); a CTA's part of them stays in shared memory for all its tiles.
//
// A CTA walks down strips of the image 128 pixels wide, TY rows a tile, with a
// warp group per role: warps 0 .. 7 read accumulators back (lane = pixel) and do
// the epilogue, half of a tile each, warps 8 .. 11 stage rows with 16-byte
// asynchronous copies, warp 12 issues the MMAs.  The rows go to a ring of planes
// in shared memory, so that a row is read once per strip and not once per tile
// that needs it (1.5 times at TY = 4, three times at TY = 1: an SM gets ~14 bytes
// a clock from L2, which is what bounds this kernel with the wide layers); ring
// and the two accumulator sets in TMEM are handed over by barriers.
//
// The one-tile-per-CTA kernel this replaces spent its time in the chain of
// TMEM allocation, weight and tile staging, MMAs and epilogue (45% warps active,
// tensor core 28% busy): 95 us for 16 -> 16 channels at 1024^2 x 4 against 56 us
// here.  A 128 x 16 x 16 MMA takes 32 cycles however narrow it is, which makes 32 us
// of those 56 (its math is 8 of the 32: the tensor pipe is 16% active, and what is
// busiest is L1 and shared memory, 72%); the 268 MB are 40 us of HBM time.
// One 1024^2 forward pass, with the pooling and skip-sum passes it absorbs:
// 323 -> 212 us.  Two CTAs an SM and eight epilogue warps each: the layers that
// write the skip sum wait for the four finer pixels, which are therefore all
// loaded before the accumulator is waited for (32 -> 16 channels at 512^2: 36 ->
// 27 us); with masks as well that takes 128 registers, and one CTA an SM is
// faster than two that spill (92 against 129 us at 512^2 x 4).
//
// A convolution is a dependent launch (launch_dependent): barriers, TMEM and the
// weights are set up while the layer before it finishes, 1024^2 predict 225 -> 208
// us.
//
// The epilogue also does what the network's next element-wise pass would do
// with the layer's output while it is in registers (ConvOut): the rounding to
// bf16 between the two is kept, so the results are the separate passes'.
//
// Images narrower than 128 pixels are staged wrapped around, so the extra
// lanes compute copies of real pixels and are not stored.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <atomic>
#include <string>
#include <type_traits>

#include "../../include/fluid.h"
#include "fs_conv.cuh"
#include "fs_internal.cuh"
#include "fs_tc.cuh"

namespace fs {
void record_error(const std::string& msg);
}

namespace fs {
namespace conv {

constexpr int kTX = 128;       // pixels per M tile
constexpr int kTW = kTX + 2;   // staged tile width (halo of 1)
constexpr int kEpi = 256;      // threads of the epilogue: two groups of four warps
constexpr int kStage = 128;    // threads that stage
constexpr int kThreads = kEpi + kStage + 32;

__host__ __device__ constexpr int align128(int x) { return (x + 127) & ~127; }

// bytes of a plane of kTW pixels, such that the KC 16-byte copies of a pixel go
// to different banks
__host__ __device__ constexpr int plane_bytes(int kc) {
  const int want = kc >= 8 ? 16 : 128 / kc;  // modulo 128
  int b = kTW * 16;
  while (b % 128 != want) b += 16;
  return b;
}

// TY rows per tile, NS output channels per CTA, D tiles staged ahead
template <int CIN, int COUT, int TY, int NS, int D>
struct Cfg {
  static constexpr int KC = CIN / 8;
  static constexpr int NSPLIT = COUT / NS;                   // CTAs sharing one pixel tile
  static constexpr int PLANE = plane_bytes(KC);
  static constexpr int ROW = KC * PLANE;                     // one image row of the ring
  // rows of the ring: tile k's new rows may overwrite those last used by tile k - D - 1
  static constexpr int NR = TY * (D + 1) + 2;
  static constexpr int RING = align128(NR * ROW);
  static constexpr int WTAP = KC * NS * 16;                  // bytes of one tap of this CTA's weights
  static constexpr int W_BYTES = align128(9 * WTAP);
  static constexpr int NACC = TY * NS;                       // columns of one accumulator set
  static constexpr int NCOL =
      2 * NACC <= 32 ? 32 : 2 * NACC <= 64 ? 64 : 2 * NACC <= 128 ? 128 : 2 * NACC <= 256 ? 256 : 512;
  // + 128 bytes of barriers and the TMEM slot, and this CTA's biases (which the caller
  // aligns to a word only: the epilogue reads them four at a time from here)
  static constexpr int SMEM = RING + W_BYTES + 128 + align128(NS * 4);
  // CTAs of one SM: shared memory, TMEM columns and what is worth having
  static constexpr int BY_SMEM = 226 * 1024 / (SMEM + 1024), BY_TMEM = 512 / NCOL;
  static constexpr int FIT = BY_SMEM < BY_TMEM ? BY_SMEM : BY_TMEM, PER_SM = FIT < 2 ? FIT : 2;
  // the epilogue groups share a tile by 16-channel chunks or, with one chunk, by rows
  static constexpr bool BY_CHUNK = NS >= 32;
  static constexpr int EROWS = BY_CHUNK ? TY : TY / 2;
  static_assert(CIN % 16 == 0 && NS % 16 == 0 && NS <= 256 && COUT % NS == 0, "channel counts");
  static_assert(2 * NACC <= 512 && PER_SM >= 1 && SMEM <= 227 * 1024, "TMEM columns, shared memory");
  static_assert(8 * (2 * (D + 1) + 4) + 12 <= 128, "barriers, TMEM slot and flag");
};

// CTAs per SM: one where the epilogue holds 64 registers of loads in flight
template <int F, typename C>
struct Per {
  static constexpr int SM = (F & kOutUpMask) ? 1 : C::PER_SM;
};

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ float2 unpack_bf16(uint32_t w) {
  return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
}
// w's two values where a's are > 0, else 0
__device__ __forceinline__ uint32_t relu_mask(uint32_t w, uint32_t a) {
  const float2 f = unpack_bf16(a);
  return (f.x > 0.f ? w & 0xffffu : 0u) | (f.y > 0.f ? w & 0xffff0000u : 0u);
}

// 16 channels of one pixel as bf16 pairs
struct Px16 {
  uint32_t w[8];
};
__device__ __forceinline__ Px16 load16(const void* base, int64_t px, int channels, int c0) {
  const uint4* p = reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(base) + px * channels + c0);
  const uint4 a = p[0], b = p[1];
  return Px16{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
}
__device__ __forceinline__ void store16(void* base, int64_t px, int channels, int c0, const Px16& v) {
  uint4* p = reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(base) + px * channels + c0);
  p[0] = make_uint4(v.w[0], v.w[1], v.w[2], v.w[3]);
  p[1] = make_uint4(v.w[4], v.w[5], v.w[6], v.w[7]);
}

// What the epilogue of one pixel's 16 channels reads besides the accumulator:
// loaded before the accumulator is waited for.
template <int F>
struct Extra {
  Px16 mask, fine[(F & kOutUp) ? 4 : 1], up_mask[(F & kOutUpMask) ? 4 : 1];
  // pixel q of the four above (y, x) on the next finer level
  static __device__ __forceinline__ int64_t above(int64_t b, int y, int x, int H, int W, int q) {
    return (b * 2 * H + 2 * y + (q >> 1)) * (2 * (int64_t)W) + 2 * x + (q & 1);
  }
  __device__ __forceinline__ void load(const ConvOut& o, int64_t b, int y, int x, int H, int W, int channels, int c0) {
    if (F & kOutMask) mask = load16(o.mask, (b * H + y) * W + x, channels, c0);
    if (F & kOutUp) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int64_t fp = above(b, y, x, H, W, q);
        // fine and up may be one buffer (a pixel is read and written by one thread): a plain load
        const __nv_bfloat16* px = reinterpret_cast<const __nv_bfloat16*>(o.fine) + fp * channels + c0;
        const uint4* sp = reinterpret_cast<const uint4*>(px);
        const uint4 s0 = sp[0], s1 = sp[1];
        fine[(F & kOutUp) ? q : 0] = Px16{{s0.x, s0.y, s0.z, s0.w, s1.x, s1.y, s1.z, s1.w}};
        if (F & kOutUpMask) up_mask[(F & kOutUpMask) ? q : 0] = load16(o.up_mask, fp, channels, c0);
      }
    }
  }
};

// Epilogue of one pixel's 16 channels v (bf16), except pooling.  F: kOut* flags.
template <int F>
__device__ __forceinline__ void finish16(const ConvOut& o, const Extra<F>& e, Px16 v, int64_t b, int y, int x, int H,
                                         int W, int channels, int c0) {
  if (F & kOutMask) {
#pragma unroll
    for (int k = 0; k < 8; k++) v.w[k] = relu_mask(v.w[k], e.mask.w[k]);
  }
  if (F & kOutStore) store16(o.out, (b * H + y) * W + x, channels, c0, v);
  if (F & kOutUp) {
    // fine + scale * v, and where a mask is given 0 where that is not > 0
#pragma unroll
    for (int q = 0; q < 4; q++) {
      Px16 s;
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const float2 c = unpack_bf16(v.w[k]), f = unpack_bf16(e.fine[(F & kOutUp) ? q : 0].w[k]);
        s.w[k] = pack_bf16(__fmaf_rn(o.scale, c.x, f.x), __fmaf_rn(o.scale, c.y, f.y));
        if (F & kOutUpMask) s.w[k] = relu_mask(s.w[k], e.up_mask[(F & kOutUpMask) ? q : 0].w[k]);
      }
      store16(o.up, Extra<F>::above(b, y, x, H, W, q), channels, c0, s);
    }
  }
}

// The 2 x 2 block of this lane's and its neighbour's pixel in two rows, summed
// (times pool_scale) for 8 of the 16 channels: the even lane makes channels c0
// .. c0 + 7 of the pooled pixel, the odd one the others.  Every lane calls it.
template <int F>
__device__ __forceinline__ void pool16(const ConvOut& o, const Px16& r0, const Px16& r1, bool store, int64_t b, int y,
                                       int x, int H, int W, int channels, int c0) {
  const int odd = threadIdx.x & 1;
  uint32_t out[4];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    // the words of the half this lane does not make go to the neighbour
    const uint32_t g0 = __shfl_xor_sync(0xffffffffu, odd ? r0.w[k] : r0.w[k + 4], 1);
    const uint32_t g1 = __shfl_xor_sync(0xffffffffu, odd ? r1.w[k] : r1.w[k + 4], 1);
    const uint32_t m0 = odd ? r0.w[k + 4] : r0.w[k], m1 = odd ? r1.w[k + 4] : r1.w[k];
    const float2 a = unpack_bf16(odd ? g0 : m0), c = unpack_bf16(odd ? m0 : g0);   // row y: left, right
    const float2 d = unpack_bf16(odd ? g1 : m1), e = unpack_bf16(odd ? m1 : g1);   // row y + 1
    out[k] = pack_bf16((((0.f + a.x) + c.x) + d.x + e.x) * o.pool_scale,
                       (((0.f + a.y) + c.y) + d.y + e.y) * o.pool_scale);
  }
  if (!store) return;
  const int64_t at = ((b * (H >> 1) + (y >> 1)) * (int64_t)(W >> 1) + (x >> 1)) * channels + c0 + 8 * odd;
  if (F & kOutPoolMask) {
    const uint4 a = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(o.pool_mask) + at);
    out[0] = relu_mask(out[0], a.x);
    out[1] = relu_mask(out[1], a.y);
    out[2] = relu_mask(out[2], a.z);
    out[3] = relu_mask(out[3], a.w);
  }
  *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(o.pool) + at) = make_uint4(out[0], out[1], out[2], out[3]);
}

// i modulo n for i >= -n; a division only where the image is smaller than a tile
__device__ __forceinline__ int wrap_near(int i, int n) {
  if (i < 0) return i + n;
  if (i >= n) {
    i -= n;
    if (i >= n) i %= n;
  }
  return i;
}

// through L1: past it (.cg) the wide layers took 5 .. 10% longer
__device__ __forceinline__ void copy16(uint32_t dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

// Strips of rows_per rows, 128 pixels wide, of the images: strip t is image b,
// first row y0, first pixel x0.
struct Strips {
  int nx, nv, count, rows_per, H;
  __host__ __device__ void at(int t, int& b, int& y0, int& x0) const {
    const int r = t / nx;
    x0 = (t - r * nx) * kTX;
    b = r / nv;
    y0 = (r - b * nv) * rows_per;
  }
  // tiles of TY rows of strip t
  __device__ int tiles(int t, int TY) const {
    int b, y0, x0;
    at(t, b, y0, x0);
    return (min(rows_per, H - y0) + TY - 1) / TY;
  }
};
// A CTA's tiles in order: strips blockIdx.x, + gridDim.x, ..., each from its top.
// ring: the ring row of the tile's first row (its image row y - 1).
template <int TY, int NR>
struct Walk {
  const Strips& S;
  int strip, left, k, b, y, x0, ring;
  bool first;  // first tile of a strip
  __device__ __forceinline__ explicit Walk(const Strips& s) : S(s), strip(blockIdx.x), left(0), k(-1), ring(0) {
    if (strip < S.count) start();
  }
  __device__ __forceinline__ void start() {
    S.at(strip, b, y, x0);
    left = S.tiles(strip, TY);
    first = true;
    k++;
  }
  __device__ __forceinline__ bool done() const { return left <= 0; }
  __device__ __forceinline__ void next() {
    if (--left > 0) {
      y += TY;
      ring += TY;
      first = false;
      k++;
    } else {
      ring += TY + 2;  // a new strip shares no rows
      strip += gridDim.x;
      if (strip < S.count) start();
    }
    while (ring >= NR) ring -= NR;
  }
};

template <int CIN, int COUT, int TY, int NS, int D, int F>
__global__ void __launch_bounds__(kThreads, (Per<F, Cfg<CIN, COUT, TY, NS, D>>::SM))
    k_conv3x3(const uint4* in, const uint4* __restrict__ wpk,
                                                         const float* __restrict__ bias, const ConvOut o,
                                                         const Strips strips, int H, int W, int* __restrict__ err) {
  using C = Cfg<CIN, COUT, TY, NS, D>;
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* wbuf = smem + C::RING;
  // barriers of tile k at index k % (D + 1), of accumulator set k % 2
  uint64_t* full = reinterpret_cast<uint64_t*>(wbuf + C::W_BYTES);  // the tile's rows are staged
  uint64_t* empty = full + D + 1;                                   // its MMAs are done
  uint64_t* ready = empty + D + 1;                                  // the set's MMAs are done
  uint64_t* taken = ready + 2;                                      // the set is read back
  uint32_t* tslot = reinterpret_cast<uint32_t*>(taken + 2);
  volatile int* failed = reinterpret_cast<volatile int*>(tslot + 2);
  float* sbias = reinterpret_cast<float*>(wbuf + C::W_BYTES + 128);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n0 = blockIdx.y * NS;  // first output channel
  if (warp == 0) {
    tc::tmem_alloc(tslot, C::NCOL);
    tc::tmem_relinquish();
    tc::fence_before_sync();
  }
  if (tid == 0) {
    for (int k = 0; k < D + 1; k++) {
      tc::mbar_init(&full[k], kStage);
      tc::mbar_init(&empty[k], 1);
    }
    for (int k = 0; k < 2; k++) {
      tc::mbar_init(&ready[k], 1);
      tc::mbar_init(&taken[k], kEpi);
    }
    tc::mbar_fence_init();
    *failed = 0;
  }
  // every tap's weights: global rows [tap][kc][co] of 16 bytes, this CTA's co in
  // [n0, n0 + NS)
  for (int k = tid; k < 9 * C::KC * NS; k += kThreads) {
    const int blk = k / NS, co = k - blk * NS;
    copy16(tc::smem_u32(wbuf) + k * 16, wpk + blk * COUT + n0 + co);
  }
  if (tid < ((F & kOutPlanar) ? 1 : NS)) sbias[tid] = bias[n0 + tid];
  asm volatile("cp.async.wait_all;" ::: "memory");
  tc::fence_async_smem();
  __syncthreads();
  tc::fence_after_sync();
  pdl_wait();  // the weights and biases were written long before the launch ahead
  const uint32_t taddr = *tslot, s0 = tc::smem_u32(smem), w0 = tc::smem_u32(wbuf);
  Walk<TY, C::NR> t(strips);

  if (warp >= kEpi / 32 && warp < (kEpi + kStage) / 32) {
    const int st = tid - kEpi;
    bool ok = true;
    int landed = 0;  // tiles handed over
    // hands the next tile over: its copies have landed
    auto land = [&] {
      tc::fence_async_smem();
      tc::mbar_arrive(&full[landed % (D + 1)]);
      landed++;
    };
    for (; !t.done(); t.next()) {
      const int k = t.k;
      // a new strip begins when all tiles before it are done: hand the last one over
      if (t.first && k > 0) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        land();
      }
      // the rows that go, or all rows before a new strip, are done with
      const int w = t.first ? k - 1 : k - D - 1;
      if (w >= 0) ok = tc::mbar_wait_idle(&empty[w % (D + 1)], (w / (D + 1)) & 1);
      if (!ok || *failed) {
        *failed = 1;
        break;
      }
      // columns x0 - 1 .. x0 + 128 of image rows y - 1 .. y + TY, wrapped; the
      // first two are there already unless the strip begins
      auto rows = [&](auto from) {
        constexpr int R0 = decltype(from)::value;
        const uint4* src[TY + 2 - R0];
        uint32_t dst[TY + 2 - R0];
#pragma unroll
        for (int r = R0; r < TY + 2; r++) {
          int q = t.ring + r;
          if (q >= C::NR) q -= C::NR;
          src[r - R0] = in + ((int64_t)t.b * H + wrap_near(t.y - 1 + r, H)) * W * C::KC;
          dst[r - R0] = s0 + q * C::ROW;
        }
        for (int q = st; q < kTW * C::KC; q += kStage) {
          // 16 channels: a chunk of neighbouring pixels on neighbouring threads; more:
          // a pixel's chunks on neighbouring threads
          const int xx = C::KC == 2 ? q % kTW : q / C::KC, kc = C::KC == 2 ? q / kTW : q % C::KC;
          const int off = kc * C::PLANE + xx * 16;
          const int64_t col = (int64_t)wrap_near(t.x0 - 1 + xx, W) * C::KC + kc;
#pragma unroll
          for (int r = 0; r < TY + 2 - R0; r++) copy16(dst[r] + off, src[r] + col);
        }
      };
      if (t.first) rows(std::integral_constant<int, 0>());
      else rows(std::integral_constant<int, 2>());
      asm volatile("cp.async.commit_group;" ::: "memory");
      // the tile before this one, whose copies are older
      if (landed < k) {
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        land();
      }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (t.k >= 0 && ok) land();
  } else if (warp == (kEpi + kStage) / 32) {
    constexpr uint32_t IDESC = tc::idesc_bf16(128, NS);
    const uint32_t leader = tc::elect_one(), ta = __shfl_sync(0xffffffffu, taddr, 0);
    int issued = 0;
    for (; !t.done(); t.next()) {
      const int k = t.k, set = k & 1;
      bool ok = tc::mbar_wait_idle(&full[k % (D + 1)], (k / (D + 1)) & 1);
      if (k >= 2) ok = tc::mbar_wait_idle(&taken[set], (k / 2 - 1) & 1) && ok;
      if (__any_sync(0xffffffffu, !ok || *failed)) {
        *failed = 1;
        break;
      }
      tc::fence_after_sync();
      // the descriptors' address field counts 16-byte units
      const uint64_t ad = tc::sdesc(s0, C::PLANE, 128), bd = tc::sdesc(w0, NS * 16, 128);
      const uint32_t d0 = ta + set * C::NACC;
      // by vertical tap and row (in the order of the taps for each row)
#pragma unroll 1
      for (int dy = 0; dy < 3; dy++) {
        const uint64_t by = bd + dy * (3 * C::WTAP / 16);
#pragma unroll
        for (int r = 0; r < TY; r++) {
          int q = t.ring + r + dy;
          if (q >= C::NR) q -= C::NR;
          const uint64_t ay = ad + q * (C::ROW / 16);
#pragma unroll
          for (int dx = 0; dx < 3; dx++)
#pragma unroll
            for (int j = 0; j < C::KC / 2; j++)
              tc::mma_bf16_warp(leader, d0 + r * NS, ay + 2 * j * (C::PLANE / 16) + dx,
                                by + (dx * C::WTAP + 2 * j * NS * 16) / 16, IDESC,
                                (dy > 0 || dx > 0 || j > 0) ? 1u : 0u);
        }
      }
      if (leader) {
        tc::mma_commit(&empty[k % (D + 1)]);
        tc::mma_commit(&ready[set]);
      }
      __syncwarp();
      issued = k + 1;
    }
    // every MMA issued is done before the TMEM is released (a commit covers all before it)
    if (issued > 0 && !tc::mbar_wait_idle(&ready[(issued - 1) & 1], ((issued - 1) / 2) & 1)) *failed = 1;
  } else {
    const int quarter = warp & 3, group = warp >> 2, p = 32 * quarter + lane;  // this thread's pixel of the tile
    const int r0 = C::BY_CHUNK ? 0 : group * C::EROWS;
    constexpr int CSTEP = C::BY_CHUNK ? 32 : 16;
    const int cfirst = C::BY_CHUNK ? 16 * group : 0;
    // the biases of a thread's one chunk stay in registers (4 x 1024^2 gradient 1887 us with
    // them read from shared memory for every pixel, 1846 us so); not where two CTAs an SM
    // and the loads of a skip sum leave none for them
    constexpr bool HELD = NS <= CSTEP && !(F & kOutPlanar) && !((F & kOutUp) && Per<F, C>::SM > 1);
    float held[HELD ? 16 : 1];
#pragma unroll
    for (int e = 0; e < (HELD ? 16 : 1); e++) held[e] = sbias[HELD ? cfirst + e : 0];
    for (; !t.done() && !*failed; t.next()) {
      const int set = t.k & 1, x = t.x0 + p;
      const uint32_t d0 = taddr + set * C::NACC + ((uint32_t)(32 * quarter) << 16);
#pragma unroll 1
      for (int c0 = cfirst; c0 < NS && !*failed; c0 += CSTEP) {
        Px16 prev;
#pragma unroll
        for (int rr = 0; rr < C::EROWS; rr++) {
          const int r = r0 + rr, y = t.y + r;
          const bool in_image = x < W && y < H;
          Extra<F> extra;
          if (in_image) extra.load(o, t.b, y, x, H, W, COUT, n0 + c0);
          if (rr == 0 && c0 == cfirst) {
            if (!tc::mbar_wait_idle(&ready[set], (t.k / 2) & 1)) *failed = 1;
            if (__any_sync(0xffffffffu, *failed != 0)) break;
            tc::fence_after_sync();
          }
          float v[16];
          tc::tmem_ld16(d0 + r * NS + c0, v);
          if (rr == C::EROWS - 1 && c0 + CSTEP >= NS) {
            // this thread's last read of the set: it may be written again
            tc::fence_before_sync();
            tc::mbar_arrive(&taken[set]);
          }
          if constexpr ((F & kOutPlanar) != 0) {
            if (in_image) reinterpret_cast<float*>(o.out)[((int64_t)t.b * H + y) * W + x] = v[0] + held[0];
          } else {
            Px16 w;
#pragma unroll
            for (int e = 0; e < 16; e += 4) {
              float4 bv;
              if constexpr (HELD) bv = make_float4(held[e], held[e + 1], held[e + 2], held[e + 3]);
              else bv = *reinterpret_cast<const float4*>(sbias + c0 + e);
              v[e] += bv.x, v[e + 1] += bv.y, v[e + 2] += bv.z, v[e + 3] += bv.w;
            }
#pragma unroll
            for (int e = 0; e < 16; e++)
              if (F & kOutRelu) v[e] = fmaxf(v[e], 0.f);
#pragma unroll
            for (int e = 0; e < 8; e++) w.w[e] = pack_bf16(v[2 * e], v[2 * e + 1]);
            if (in_image) finish16<F>(o, extra, w, t.b, y, x, H, W, COUT, n0 + c0);
            if constexpr ((F & kOutPool) != 0) {
              if (rr % 2 == 0) prev = w;
              else pool16<F>(o, prev, w, in_image, t.b, y - 1, x, H, W, COUT, n0 + c0);
            }
          }
        }
      }
    }
  }
  __syncthreads();
  if (tid == 0 && *failed) atomicExch(err, 1);
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, C::NCOL);
}

// ------------------------------------------------------------ GEMM check
// D[128][N] = A[128][K] B[N][K]^T from row-major bf16 A and B: exercises the
// descriptors, the instruction descriptor and the TMEM read-back on one tile.
// Operands are staged with LBO = 128 and SBO = 256 bytes, so that every
// address either field could produce stays inside the staged block.
template <int N>
__global__ void __launch_bounds__(128) k_gemm_check(const uint16_t* __restrict__ A, const uint16_t* __restrict__ B,
                                                    float* __restrict__ D, int K, int* __restrict__ err) {
  __shared__ __align__(128) uint16_t sa[128 * 64];  // up to K = 64
  __shared__ __align__(128) uint16_t sb[N * 64];
  __shared__ uint64_t bar;
  __shared__ uint32_t tslot;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int NCOL = N < 32 ? 32 : N;
  if (warp == 0) {
    tc::tmem_alloc(&tslot, NCOL);
    tc::tmem_relinquish();
    tc::fence_before_sync();
  }
  if (tid == 0) {
    tc::mbar_init(&bar, 1);
    tc::mbar_fence_init();
  }
  // element (row m, k) -> K step s = k / 16, chunk c = (k / 8) % 2, group g = m / 8:
  // byte offset s * (rows * 32) + g * 256 + c * 128 + (m % 8) * 16 + (k % 8) * 2
  for (int e = tid; e < 128 * K; e += 128) {
    int m = e / K, k = e % K;
    sa[(k / 16) * (128 * 16) + (m / 8) * 128 + ((k / 8) % 2) * 64 + (m % 8) * 8 + (k % 8)] = A[e];
  }
  for (int e = tid; e < N * K; e += 128) {
    int n = e / K, k = e % K;
    sb[(k / 16) * (N * 16) + (n / 8) * 128 + ((k / 8) % 2) * 64 + (n % 8) * 8 + (k % 8)] = B[e];
  }
  tc::fence_async_smem();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = tslot;
  if (tid == 0) {
    for (int s = 0; s < K / 16; s++)
      tc::mma_bf16(taddr, tc::sdesc(tc::smem_u32(sa + s * 128 * 16), 128, 256),
                   tc::sdesc(tc::smem_u32(sb + s * N * 16), 128, 256), tc::idesc_bf16(128, N), s > 0 ? 1u : 0u);
    tc::mma_commit(&bar);
  }
  __syncthreads();
  bool ok = tc::mbar_wait(&bar, 0);
  tc::fence_after_sync();
  if (!ok) {
    if (tid == 0) atomicExch(err, 1);
  } else {
    const int m = 32 * warp + lane;
    for (int c0 = 0; c0 < N; c0 += 16) {
      float v[16];
      tc::tmem_ld16(taddr + ((uint32_t)(32 * warp) << 16) + c0, v);
      for (int k = 0; k < 16; k++) D[m * N + c0 + k] = v[k];
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(taddr, NCOL);
}

// ------------------------------------------------------------------ host
template <int CIN, int COUT, int TY, int NS, int D, int F>
static cudaError_t launch_t(const void* in, const void* w, const float* bias, const ConvOut& o, int B, int H, int W,
                            int* err, cudaStream_t st, bool dependent) {
  using C = Cfg<CIN, COUT, TY, NS, D>;
  static_assert(!(F & kOutPool) || C::EROWS % 2 == 0, "pooled rows in pairs");
  // the dynamic shared-memory limit is an attribute of the function on each device
  static std::atomic<uint64_t> attr_set{0};
  int dev = 0;
  cudaError_t e0 = cudaGetDevice(&dev);
  if (e0 != cudaSuccess) return e0;
  const uint64_t bit = 1ull << (dev & 63);
  if (!(attr_set.load() & bit)) {
    cudaError_t e = cudaFuncSetAttribute(k_conv3x3<CIN, COUT, TY, NS, D, F>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM);
    if (e != cudaSuccess) return e;
    attr_set.fetch_or(bit);
  }
  // one strip per CTA where the images allow: as many vertical parts as there
  // are slots for (whole tiles each)
  const int slots = kSMs * Per<F, C>::SM / C::NSPLIT, nx = (W + kTX - 1) / kTX, rows = (H + TY - 1) / TY;
  const int64_t columns = (int64_t)B * nx;
  const int parts = (int)(columns >= slots ? 1 : slots / columns < rows ? slots / columns : rows);
  const int per = (rows + parts - 1) / parts, nv = (rows + per - 1) / per;
  const int64_t count = columns * nv;
  if (count >= (int64_t)1 << 31) return cudaErrorInvalidValue;
  const Strips strips{nx, nv, (int)count, per * TY, H};
  return launch_dependent(dependent, k_conv3x3<CIN, COUT, TY, NS, D, F>,
                          dim3((unsigned)(count < slots ? count : slots), C::NSPLIT), dim3(kThreads), C::SMEM, st,
                          static_cast<const uint4*>(in), static_cast<const uint4*>(w), bias, o, strips, H, W, err);
}

// (c_in, c_out, rows per tile, output channels per CTA, tiles staged ahead)
#define FS_CONV_PAIRS(CASE) \
  CASE(16, 16, 4, 16, 2) CASE(16, 32, 4, 32, 2) CASE(32, 16, 2, 16, 2) CASE(32, 64, 2, 64, 2) \
  CASE(64, 32, 1, 32, 2) CASE(64, 128, 1, 64, 2) CASE(128, 64, 1, 32, 1)

template <int F>
static cudaError_t dispatch(int cin, int cout, const void* in, const void* w, const float* bias, const ConvOut& o,
                            int B, int H, int W, int* err, cudaStream_t st, bool dependent) {
  // pooled layers widen or keep the channels, upsampled ones narrow them
  constexpr bool pool = (F & kOutPool) != 0, planar = (F & kOutPlanar) != 0, up = (F & kOutUp) != 0;
#define FS_CASE(ci, co, ty, ns, d)                                                      \
  if constexpr ((!pool || (co >= ci && ty > 1)) && (!up || co < ci) && (!planar || co == 16)) { \
    if (cin == ci && cout == co)                                                             \
      return launch_t<ci, co, ty, ns, d, F>(in, w, bias, o, B, H, W, err, st, dependent); \
  }
  FS_CONV_PAIRS(FS_CASE)
#undef FS_CASE
  return cudaErrorInvalidValue;
}

bool supported(int cin, int cout) {
#define FS_CASE(ci, co, ty, ns, d) \
  if (cin == ci && cout == co) return true;
  FS_CONV_PAIRS(FS_CASE)
#undef FS_CASE
  return false;
}

cudaError_t conv3x3(int cin, int cout, int flags, const void* in, const void* w, const float* bias, const ConvOut& o,
                    int B, int H, int W, int* err, cudaStream_t st, bool dependent) {
  switch (flags) {
#define FS_CASE(f) \
  case f: return dispatch<f>(cin, cout, in, w, bias, o, B, H, W, err, st, dependent);
    FS_CASE(kOutStore)                                              // a plain layer
    FS_CASE(kOutStore | kOutRelu)
    FS_CASE(kOutPlanar)                                             // the network's output
    FS_CASE(kOutStore | kOutRelu | kOutPool)                        // forward: + the pooled level below
    FS_CASE(kOutStore | kOutRelu | kOutUp)                          // forward: + the skip sum of the level above
    FS_CASE(kOutStore | kOutMask)                                   // backward: a masked gradient
    FS_CASE(kOutStore | kOutPool | kOutPoolMask)                    // backward: + the gradient of the upsampling
    FS_CASE(kOutUp | kOutUpMask)                                    // backward: the gradient of the pooling
#undef FS_CASE
  }
  return cudaErrorInvalidValue;
}

cudaError_t gemm_check(int n, const void* a, const void* b, float* d, int k, int* err, cudaStream_t st) {
  if (n == 16) k_gemm_check<16><<<1, 128, 0, st>>>((const uint16_t*)a, (const uint16_t*)b, d, k, err);
  else if (n == 64) k_gemm_check<64><<<1, 128, 0, st>>>((const uint16_t*)a, (const uint16_t*)b, d, k, err);
  else return cudaErrorInvalidValue;
  return cudaGetLastError();
}

}  // namespace conv
}  // namespace fs

// ------------------------------------------------------------------ C ABI
using namespace fs;

static int conv_fail(int code, const std::string& m) {
  record_error(m);
  return code;
}

extern "C" FS_API int fs_conv3x3_bf16(const void* d_in, const void* d_wpacked, const float* d_bias, void* d_out,
                                      int32_t batch, int32_t h, int32_t w, int32_t c_in, int32_t c_out,
                                      int32_t epilogue, int32_t* d_err, void* stream) {
  if (!d_in || !d_wpacked || !d_bias || !d_out || !d_err)
    return conv_fail(FS_ERR_INVALID_ARGUMENT, "fs_conv3x3_bf16: NULL pointer");
  if (batch < 1 || batch > 8192 || h < 1 || w < 1 || epilogue < 0 || epilogue > 2)
    return conv_fail(FS_ERR_INVALID_ARGUMENT, "fs_conv3x3_bf16: bad shape or epilogue");
  if (!conv::supported(c_in, c_out) || (epilogue == 2 && c_out != 16))
    return conv_fail(FS_ERR_UNSUPPORTED, "fs_conv3x3_bf16: channel pair " + std::to_string(c_in) + "->" +
                                             std::to_string(c_out) + " not instantiated");
  if (((uintptr_t)d_in | (uintptr_t)d_wpacked | (uintptr_t)d_out) & 15)
    return conv_fail(FS_ERR_INVALID_ARGUMENT, "fs_conv3x3_bf16: buffers must be 16-byte aligned");
  conv::ConvOut o;
  o.out = d_out;
  const int flags = epilogue == 0   ? conv::kOutStore
                    : epilogue == 1 ? conv::kOutStore | conv::kOutRelu
                                    : conv::kOutPlanar;
  cudaError_t e = conv::conv3x3(c_in, c_out, flags, d_in, d_wpacked, d_bias, o, batch, h, w, d_err,
                                static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return conv_fail(FS_ERR_CUDA, std::string("fs_conv3x3_bf16: ") + cudaGetErrorString(e));
  return FS_OK;
}

extern "C" FS_API int fs_tc_gemm_check(const void* d_a, const void* d_b, float* d_d, int32_t n, int32_t k,
                                       int32_t* d_err, void* stream) {
  if (!d_a || !d_b || !d_d || !d_err) return conv_fail(FS_ERR_INVALID_ARGUMENT, "fs_tc_gemm_check: NULL pointer");
  if ((n != 16 && n != 64) || k < 16 || k > 64 || k % 16)
    return conv_fail(FS_ERR_INVALID_ARGUMENT, "fs_tc_gemm_check: n must be 16 or 64, k a multiple of 16 <= 64");
  cudaError_t e = conv::gemm_check(n, d_a, d_b, d_d, k, d_err, static_cast<cudaStream_t>(stream));
  if (e != cudaSuccess) return conv_fail(FS_ERR_CUDA, std::string("fs_tc_gemm_check: ") + cudaGetErrorString(e));
  return FS_OK;
}
