// fs_flat.cu -- the flat Poisson solvers (Jacobi, red-black Gauss-Seidel) with
// several sweeps per launch (k_flat, fs_flat.cuh).
//
// One launch per sweep or colour (k_jacobi, k_rb_half) costs what a launch
// costs, ~4.5 us in a stream and ~2.5 us of it on the GPU, where the sweep
// itself needs well under 1 us: 40 Jacobi sweeps took 170 us at 256^2 and 250
// us at 1280 x 720, 40 red-black sweeps 340 us at 333 x 500.  k_flat runs up
// to 12 sweeps or half-sweeps per launch (20 on small grids) on a region in registers; the cells
// a region shares with its neighbours are computed by each of them (2.6x the
// useful cells for the 64 x 64 region at 12, 1.9x for the 128 x 64 one),
// which the idle issue slots pay for.  The same solves, captured: 18.5 us,
// 43 us and 37 us; with the first launch of a solve a dependent one too, steps of
// these sizes take 32.6 -> 29.8, 84.5 -> 81.6 and 46.6 -> 45.6 us.
#include <algorithm>
#include <atomic>
#include <utility>

#include "fs_flat.cuh"
#include "fs_internal.cuh"

namespace fs {

// Dynamic shared memory that leaves room for one CTA an SM only.  A launch of the
// small region with at most one CTA an SM asks for it: its CTAs are placed while the
// kernel ahead still holds some SMs, and where registers leave room for three an SM
// two of them can share one and take twice the time.  Whether they do depends on
// what else runs: eight steps at 256^2 with the velocity copied in and out 312 us,
// 247 us with the limit (64 KB, two an SM: 318); steps alone at 256^2, red-black, 35.8
// -> 34.1 us; from 16^2 to 446^2 no size is slower.  Launches with more CTAs than SMs
// need the room: 8000 x 24 with 40 sweeps 43.7 -> 48.4 us a step.
constexpr int kFlatAlone = 100 * 1024;

template <int CPL, int RPW, int NW, int H, int MODE>
static int flat_alone_bytes(int device) {
  static std::atomic<uint64_t> set{0};  // the limit is an attribute of the function on each device
  const uint64_t bit = 1ull << (device & 63);
  if (!(set.load() & bit)) {
    if (cudaFuncSetAttribute(k_flat<CPL, RPW, NW, H, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, kFlatAlone) !=
        cudaSuccess) {
      cudaGetLastError();
      return 0;
    }
    set.fetch_or(bit);
  }
  return kFlatAlone;
}

template <int CPL, int RPW, int NW, int H, int MODE>
static void flat_t(Solver* s, float** x, float** y, const float* d, int n, float h2, bool zero) {
  using F = FlatTile<CPL, RPW, NW, H>;
  const Grid& g = s->g;
  const int launches = (n + H - 1) / H, k = (n + launches - 1) / launches;  // as even as they come
  for (int done = 0; done < n; done += k) {
    const int now = std::min(k, n - done);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((g.nx + F::TW - 1) / F::TW, (g.ny + F::RH - 2 * now - 1) / (F::RH - 2 * now));
    cfg.blockDim = dim3(NW * 32);
    cfg.stream = s->stream;
    if (RPW == 4 && (int64_t)cfg.gridDim.x * cfg.gridDim.y <= kSMs)
      cfg.dynamicSmemBytes = flat_alone_bytes<CPL, RPW, NW, H, MODE>(s->device);
    cudaLaunchAttribute pdl = {};
    pdl.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    pdl.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &pdl;
    cfg.numAttrs = 1;
    FS_LAUNCH(s, MODE == kFlatJacobi ? "jacobi" : "red_black", (double)s->n * (zero ? 8 : 12),
              cudaLaunchKernelEx(&cfg, k_flat<CPL, RPW, NW, H, MODE>, (const float*)*x, d, *y, g.nx, g.ny, h2,
                                 (float)s->prm.relax, now, done & 1, zero ? 1 : 0, done == 0 ? 1 : 0));
    zero = false;
    std::swap(*x, *y);
  }
}

// The region: 64 x 64 cells (16 warps of 4 rows) spreads a small grid over
// more CTAs, 128 x 64 (8 warps of 8 rows, 4 columns a lane) spends fewer
// shuffles and less overlap on a large one.  40 Jacobi / red-black sweeps,
// 64 x 64 against 128 x 64: 18.5 / 28.7 against 24.6 / 36.9 us at 256^2, 18.5
// / 31.2 against 24.6 / 36.9 at 384^2, 28.7 / 49.0 against 24.7 / 41.6 at
// 512^2, 53.1 / 90.1 against 38.9 / 55.3 at 1000^2.
constexpr int64_t kFlatLarge = 200000;

// Does a solve of n sweeps have at most one CTA an SM if up to H go into a launch
// of the small region?  Fewer, deeper launches pay while they fit the chip: steps
// with 40 Jacobi / red-black sweeps at H = 12, 16, 20: 256^2 29.6 / 39.9, 27.7 /
// 36.0, 26.1 / 34.5 us (121 CTAs); 384^2 31.7 / 42.0, 29.7 / 38.1, 35.5 / 48.3 (256
// CTAs at 20); 440^2 33.9 / 44.2, 39.9 / 52.3, 46.6 / 65.9 (182 at 16).
static bool flat_fits(const Solver* s, int n, int H) {
  const int launches = (n + H - 1) / H, k = (n + launches - 1) / launches, tw = 64 - 2 * H, th = 64 - 2 * k;
  return (int64_t)((s->g.nx + tw - 1) / tw) * ((s->g.ny + th - 1) / th) <= kSMs;
}

template <int MODE>
static void flat_mode(Solver* s, float** x, float** y, const float* d, int n, float h2, bool zero) {
  if (s->n >= kFlatLarge) flat_t<4, 8, 8, 12, MODE>(s, x, y, d, n, h2, zero);
  else if (flat_fits(s, n, 20)) flat_t<2, 4, 16, 20, MODE>(s, x, y, d, n, h2, zero);
  else if (flat_fits(s, n, 16)) flat_t<2, 4, 16, 16, MODE>(s, x, y, d, n, h2, zero);
  else flat_t<2, 4, 16, 12, MODE>(s, x, y, d, n, h2, zero);
}

// `iterations` sweeps of the flat solver on (*x, d), *y the second buffer (the
// two pointers are swapped so that *x is the result); zero: *x starts from 0,
// whatever it holds.  kernel_variant 1 runs one pass per sweep or colour.
void flat_sweeps(Solver* s, float** x, float** y, const float* d, int iterations, bool zero) {
  const Grid& g = s->g;
  const float h2 = g.dx * g.dx;
  const bool rb = s->prm.pressure_solver == FS_PRESSURE_RED_BLACK;
  if (s->prm.kernel_variant == 0 && iterations > 0) {
    if (!rb) flat_mode<kFlatJacobi>(s, x, y, d, iterations, h2, zero);
    else if (s->odd) flat_mode<kFlatRbOdd>(s, x, y, d, 2 * iterations, h2, zero);
    else flat_mode<kFlatRbEven>(s, x, y, d, 2 * iterations, h2, zero);
    return;
  }
  if (zero) launch_fill(s, *x, 0.f, s->n);
  for (int k = 0; k < iterations; k++) {
    if (!rb) {
      launch_jacobi(s, *x, d, *y, h2, g.nx, g.ny);
      std::swap(*x, *y);
      continue;
    }
    for (int colour = 0; colour < 2; colour++) {
      launch_rb_half(s, *x, d, s->odd ? *y : *x, h2, colour, g.nx, g.ny);
      if (s->odd) std::swap(*x, *y);
    }
  }
}

}  // namespace fs
