// fs_multigrid.cu -- fused multigrid V-cycle for GB300 (sm_103a).
//
// The V-cycle of src/gpu/multigrid.js:277-330 (RBGS(pre) -> residual ->
// restriction -> ... -> coarse RBGS(40) -> prolongation -> RBGS(post)) costs
// the reference 8 + 5 passes per level plus 80 coarse passes (~184 dispatches
// at 2048^2).  Here one V-cycle is:
//
//   k_mg_down   per level n > 64: a tile with a halo of 2 * pre + 1 cells is
//               held in registers, the pre-smoothing red-black sweeps run
//               there (the valid region shrinks one ring per half-sweep), then
//               the residual and its 2x2 restriction are formed; only the
//               tile's x and the coarse right-hand side go back to HBM;
//   k_mg_bottom one CTA runs every level <= 64 (fs_bottom.cu);
//   k_mg_up     per level n > 64: prolongation-add of the coarse correction on
//               the tile plus a halo of 2 * post, then the post-smoothing sweeps.
//
// The tiles are fs_mgreg.cuh's.  With the tile in shared memory instead (64 x 64,
// a TMA copy per field) each update took five shared-memory loads and a store,
// which bound the kernels: level 0 of 4096^2, down 62 us and up into the
// pressure 80 us, against 36 us and 70 us here (22 us and 62 us of HBM time).
// The per-cell arithmetic is fs_stencil.cuh, shared with the one-pass-per-
// operation kernels, so the fused cycle reproduces them bit for bit.
#include <string>
#include <utility>

#include "fs_df.cuh"
#include "fs_internal.cuh"
#include "fs_mgreg.cuh"

namespace fs {

template <class R>
__global__ void __launch_bounds__(R::THREADS, R::CTAS)
    k_mg_down(const float* rhs, const float* xin, float* __restrict__ xout,
                  float* __restrict__ crhs, int n, float h2, int pre, float w, const int* first_cycle, int first_pre,
                  int first_x_unused) {
  pdl_wait();
  // the first cycle of a projection may run fewer sweeps on this level
  // (fs_params mg_first_pre, at most pre): first_pre >= 0 applies it, inside
  // a captured loop only while the loop's cycle count is still 0;
  // first_x_unused: that cycle's up kernel on this level runs no sweeps
  // either and does not read the iterate
  const bool first = first_pre >= 0 && (!first_cycle || *first_cycle == 0);
  if (first) pre = first_pre;
  if (first && pre == 0 && first_x_unused && !xin) mg_restrict_rhs<R>(rhs, crhs, n);
  else mg_down_reg<R>(rhs, xin, xout, crhs, n, h2, pre, w);
}

template <class R, bool ACC, int AHEAD>
__global__ void __launch_bounds__(R::THREADS, R::CTAS)
    k_mg_up(const float* __restrict__ rhs, const float* __restrict__ xin, float* __restrict__ xout,
                const float* xc, int n, float h2, int post, float w, float* __restrict__ ph,
                float* __restrict__ pl, const int* first_cycle, int first_post, int first_x_zero) {
  // as k_mg_down; first_x_zero: that cycle's down kernel on this level ran no
  // sweeps, so the iterate is zero
  const bool first = first_post >= 0 && (!first_cycle || *first_cycle == 0);
  if (first) post = first_post;
  mg_up_reg<R, ACC, AHEAD>(rhs, xin, xout, xc, n, h2, post, w, ph, pl, ACC && first && post == 0 && first_x_zero);
}

// ------------------------------------------------- batched (one size class)
// The members of a batch with the same grid and multigrid settings run each
// kernel of their refinement cycles as one launch, member = blockIdx.z, with
// their pointers in a table passed by value among the kernel parameters.  A
// member whose tolerance loop has ended (the per-member condition the
// class-wide loop kernel keeps in its DevState) leaves the launch at once, so
// every member runs exactly the cycles it would run alone.
__device__ __forceinline__ bool member_active(const DevState* st, int max_cycles) {
  return !st->converged && !st->nonfinite && st->cycles < max_cycles;
}

struct DownTab {
  struct {
    const float* rhs;
    float* xout;
    float* crhs;
    const DevState* st;
  } m[kClassMax];
};
struct UpTab {
  struct {
    const float* rhs;
    const float* xin;
    float* xout;
    const float* xc;
    float* ph;
    float* pl;
    const DevState* st;
  } m[kClassMax];
};
static_assert(sizeof(UpTab) + 64 <= 32764, "kernel parameter limit");

template <class R>
__global__ void __launch_bounds__(R::THREADS, R::CTAS)
    k_mg_down_class(const __grid_constant__ DownTab tab, int n, float h2, int pre, float w, int max_cycles) {
  pdl_wait();
  const auto& a = tab.m[blockIdx.z];
  if (!member_active(a.st, max_cycles)) return;
  mg_down_reg<R>(a.rhs, nullptr, a.xout, a.crhs, n, h2, pre, w);
}

template <class R, bool ACC>
__global__ void __launch_bounds__(R::THREADS, R::CTAS)
    k_mg_up_class(const __grid_constant__ UpTab tab, int n, float h2, int post, float w, int max_cycles) {
  const auto& a = tab.m[blockIdx.z];
  if (!member_active(a.st, max_cycles)) {  // (the loop state was set before the cycle began)
    pdl_wait();
    return;
  }
  mg_up_reg<R, ACC, 0>(a.rhs, a.xin, a.xout, a.xc, n, h2, post, w, a.ph, a.pl, false);
}

// ------------------------------------------------------------------ host
// A tile kernel's region by its side class T (fs_set_mg_tiles): 64 is 128 x 64
// cells (32 a thread, three CTAs an SM: down 40 us at 4096^2, two CTAs 48 us,
// 512 threads of 16 cells 51 us), 32 is 128 x 32, 16 is 64 x 32.  The up kernel
// that adds into the pressure takes the 128 x 32 cells in class 64 too: 74 us
// at 4096^2, with 128 x 64 in 512 threads 78 us, in 256 80 us (two CTAs) and
// 96 us (three, which spill).
template <int T, int H, bool ACC = false>
struct RegionOf {
  typedef MgRegion<4, ACC ? 4 : 8, 8, H> R;
};
template <int H, bool ACC>
struct RegionOf<32, H, ACC> {
  typedef MgRegion<4, 4, 8, H> R;
};
template <int H, bool ACC>
struct RegionOf<16, H, ACC> {
  typedef MgRegion<2, 4, 8, H> R;
};

// side class of a level of n cells (launches timed with an event on each side,
// ~4 us of them that; class 64 / 32 / 16): 2048 cells, down 15 / 19 / 21 us, up 16 /
// 17 / 20; 1024, down 10 / 9.5 / 10, up 10 / 9 / 10; 512, down 9 / 7.6 / 7.6, up 8.2 /
// 8.1 / 8.1; 256, down 9 / 7.4 / 6.9, up 8.2 / 8.1 / 6.3
static int tile_for(int n) {
  const int c64 = (n + 63) / 64, c32 = (n + 31) / 32;
  if (c64 * c64 >= 1024) return 64;
  if (c32 * c32 >= 256) return 32;
  return 16;
}

// A side T serves a level of n cells only if T <= n / 2 and its regions' four columns
// a lane divide the level; side 16, with two columns a lane, serves every tile level (n
// > 64 and even; n = 2 mod 4 only as the last above an odd bottom level, so n <= 126).
static bool tile_fits(int t, int n) { return t == 16 || (n % 4 == 0 && 2 * t <= n); }

int mg_tile(const Solver* s, int l) {
  const int n = s->lev[l].n;
  if (l >= 0 && l < 16 && s->tile_level[l] && tile_fits(s->tile_level[l], n)) return s->tile_level[l];
  return tile_for(n);
}

// profile name of a tile kernel: one entry per level ("mg_down_l0", ...)
static std::string level_name(const Solver* s, const Level& L, const char* base) {
  return std::string(base) + "_l" + std::to_string(&L - s->lev.data());
}

// CTAs between the one whose region an up kernel's CTA fetches into L2 and itself:
// two an SM ahead, on levels whose fields L2 does not hold (4096^2: 71 us with it, 75
// without, the pressure fetched as well 77; the down kernel is not bound by its
// loads).  Steps with it and without: 2048^2 560 / 558 us, 2304^2 658 / 658, 2560^2 773 /
// 774, 2816^2 894 / 905, 3072^2 1010 / 1025, 3584^2 1297 / 1324, 4096^2 1559 / 1587.
constexpr int kAheadFrom = 2896, kAhead = 2 * kSMs;

template <class R>
static dim3 region_grid(int n, int members = 1) {
  return dim3((n + R::TW - 1) / R::TW, (n + R::TH - 1) / R::TH, members);
}

// first >= 0: the sweeps of this level in the first cycle of a projection;
// cyc: the loop's cycle count on the device that decides (nullptr: the host
// knows this is the first cycle)
template <int T, int H>
static void down_t(Solver* s, Level& L, const Level& C, bool has_x, bool zero, int first, const int* cyc,
                   bool x_unused) {
  typedef typename RegionOf<T, H>::R R;
  double bytes = (double)L.n * L.n * (has_x && !zero ? 12.0 : 8.0) + (double)C.n * C.n * 4.0;
  // a first cycle the host knows is profiled under its own name
  const std::string name = level_name(s, L, "mg_down") + (first >= 0 && !cyc ? "_first" : "");
  FS_LAUNCH(s, name.c_str(), bytes,
            launch_dependent(true, k_mg_down<R>, region_grid<R>(L.n), dim3(R::THREADS), 0, s->stream, L.rhs,
                             has_x && !zero ? L.x : nullptr, has_x ? L.x2 : L.x, C.rhs, L.n, L.h2,
                             s->prm.mg_pre_smooth, (float)s->prm.relax, cyc,
                             first < s->prm.mg_pre_smooth ? first : s->prm.mg_pre_smooth, x_unused ? 1 : 0));
  if (has_x) std::swap(L.x, L.x2);
}

template <int H>
static void down(Solver* s, Level& L, const Level& C, bool has_x, bool zero, int first, const int* cyc, bool x_unused) {
  switch (mg_tile(s, (int)(&L - s->lev.data()))) {
    case 64: down_t<64, H>(s, L, C, has_x, zero, first, cyc, x_unused); break;
    case 32: down_t<32, H>(s, L, C, has_x, zero, first, cyc, x_unused); break;
    default: down_t<16, H>(s, L, C, has_x, zero, first, cyc, x_unused); break;
  }
}

template <int T, int H>
static void up_t(Solver* s, Level& L, const Level& C, float* acc_h, float* acc_l, int first, const int* cyc,
                 bool x_zero) {
  const int fp = first < s->prm.mg_post_smooth ? first : s->prm.mg_post_smooth;
  double bytes = (double)L.n * L.n * (acc_h ? 24.0 : 12.0) + (double)C.n * C.n * 4.0;
  const bool ahead = L.n >= kAheadFrom && T == 64;
  constexpr int AHEAD = T == 64 ? kAhead : 0;
  if (acc_h) {
    typedef typename RegionOf<T, H, true>::R R;
    auto* kernel = ahead ? k_mg_up<R, true, AHEAD> : k_mg_up<R, true, 0>;
    FS_LAUNCH(s, first >= 0 && !cyc ? "mg_up_acc_first" : "mg_up_acc", bytes,
              launch_dependent(true, kernel, region_grid<R>(L.n), dim3(R::THREADS), 0, s->stream, L.rhs, L.x, nullptr,
                               C.x, L.n, L.h2, s->prm.mg_post_smooth, (float)s->prm.relax, acc_h, acc_l, cyc, fp,
                               x_zero ? 1 : 0));
    return;
  }
  typedef typename RegionOf<T, H>::R R;
  auto* kernel = ahead ? k_mg_up<R, false, AHEAD> : k_mg_up<R, false, 0>;
  FS_LAUNCH(s, level_name(s, L, "mg_up").c_str(), bytes,
            launch_dependent(true, kernel, region_grid<R>(L.n), dim3(R::THREADS), 0, s->stream, L.rhs, L.x, L.x2, C.x,
                             L.n, L.h2, s->prm.mg_post_smooth, (float)s->prm.relax, nullptr, nullptr, cyc, fp,
                             x_zero ? 1 : 0));
  std::swap(L.x, L.x2);
}

template <int H>
static void up(Solver* s, Level& L, const Level& C, float* acc_h, float* acc_l, int first, const int* cyc,
               bool x_zero) {
  switch (mg_tile(s, (int)(&L - s->lev.data()))) {
    case 64: up_t<64, H>(s, L, C, acc_h, acc_l, first, cyc, x_zero); break;
    case 32: up_t<32, H>(s, L, C, acc_h, acc_l, first, cyc, x_zero); break;
    default: up_t<16, H>(s, L, C, acc_h, acc_l, first, cyc, x_zero); break;
  }
}

// the fused cycle needs even tile levels, a bottom of <= 8 levels each <= 64,
// and 1 <= pre, post <= 3
bool mg_fused_supported(const Solver* s) {
  const fs_params& P = s->prm;
  if (P.mg_pre_smooth < 1 || P.mg_pre_smooth > 3 || P.mg_post_smooth < 1 || P.mg_post_smooth > 3) return false;
  int lb = bottom_first_level(s);
  for (int l = 0; l < lb; l++)
    if (s->lev[l].n & 1) return false;
  if ((int)s->lev.size() - lb > 8) return false;
  for (size_t l = lb; l < s->lev.size(); l++)
    if (s->lev[l].n > 64) return false;
  return true;
}

void mg_vcycle_fused(Solver* s, bool first_has_x, float* acc_h, float* acc_l, bool zero) {
  std::vector<Level>& L = s->lev;
  const int lb = bottom_first_level(s);
  const fs_params& P = s->prm;
  // the finest level of a MIXED refinement cycle (acc_h: the correction goes
  // into the double-float pressure) may run fewer sweeps in the first cycle of
  // a projection: the host knows which cycle it enqueues (mg_cycle_index >= 0)
  // except inside a captured tolerance loop, where the kernels read the loop's
  // cycle count on the device
  int fpre = -1, fpost = -1;
  const int* cyc = nullptr;
  if (acc_h && s->mg_cycle_index <= 0) {
    fpre = P.mg_first_pre;
    fpost = P.mg_first_post;
    if (s->mg_cycle_index < 0 && (fpre >= 0 || fpost >= 0)) cyc = &s->dev->cycles;
  }
  for (int l = 0; l < lb; l++) {
    bool hx = l == 0 && first_has_x;
    const int f = l == 0 ? fpre : -1;
    const bool xu = l == 0 && fpost == 0;  // the first cycle's up kernel reads no iterate here
    switch (P.mg_pre_smooth) {
      case 1: down<3>(s, L[l], L[l + 1], hx, zero && l == 0, f, cyc, xu); break;
      case 2: down<5>(s, L[l], L[l + 1], hx, zero && l == 0, f, cyc, xu); break;
      default: down<7>(s, L[l], L[l + 1], hx, zero && l == 0, f, cyc, xu); break;
    }
  }
  const bool hx = lb == 0 && first_has_x && !zero;
  float* bah = lb == 0 ? acc_h : nullptr;
  float* bal = lb == 0 ? acc_l : nullptr;
  launch_bottom(s, lb, hx, bah, bal);
  for (int l = lb - 1; l >= 0; l--) {
    float* ah = l == 0 ? acc_h : nullptr;
    float* al = l == 0 ? acc_l : nullptr;
    const int f = l == 0 ? fpost : -1;
    const bool xz = l == 0 && fpre == 0;  // the first cycle's down kernel left a zero iterate here
    switch (P.mg_post_smooth) {
      case 1: up<2>(s, L[l], L[l + 1], ah, al, f, cyc, xz); break;
      case 2: up<4>(s, L[l], L[l + 1], ah, al, f, cyc, xz); break;
      default: up<6>(s, L[l], L[l + 1], ah, al, f, cyc, xz); break;
    }
  }
}


// ------------------------------------------------------- batched V-cycle
// mg_vcycle_fused(s, false, ph, pl) of a MIXED refinement cycle for every
// member of one size class (same grid and multigrid settings), one launch per
// level and phase; the level pointers of each member move exactly as in the
// single-solver cycle.  Returns the number of launches it recorded.
template <int T, int H>
static void down_class_t(Solver* const* ms, int count, int l, cudaStream_t st) {
  typedef typename RegionOf<T, H>::R R;
  const Level& L0 = ms[0]->lev[l];
  DownTab tab{};
  for (int i = 0; i < count; i++) {
    Level& L = ms[i]->lev[l];
    tab.m[i] = {L.rhs, L.x, ms[i]->lev[l + 1].rhs, ms[i]->dev};
  }
  launch_dependent(true, k_mg_down_class<R>, region_grid<R>(L0.n, count), dim3(R::THREADS), 0, st, tab, L0.n, L0.h2,
                   ms[0]->prm.mg_pre_smooth, (float)ms[0]->prm.relax, ms[0]->prm.max_cycles);
}

// tile side for a level of a class: an override of the class's members, else
// like tile_for counting the CTAs of all members (the tiles give the same
// values whatever their size)
static int tile_for_class(const Solver* s0, int l, int count) {
  const int n = s0->lev[l].n;
  if (l < 16 && s0->tile_level[l] && tile_fits(s0->tile_level[l], n)) return s0->tile_level[l];
  for (int t : {64, 32}) {
    int c = (n + t - 1) / t;
    if (tile_fits(t, n) && c * c * count >= 256) return t;
  }
  return 16;
}

int mg_tile_class(const Solver* s0, int l, int count) { return tile_for_class(s0, l, count); }

template <int H>
static void down_class(Solver* const* ms, int count, int l, cudaStream_t st) {
  switch (tile_for_class(ms[0], l, count)) {
    case 64: down_class_t<64, H>(ms, count, l, st); break;
    case 32: down_class_t<32, H>(ms, count, l, st); break;
    default: down_class_t<16, H>(ms, count, l, st); break;
  }
}

template <int T, int H, bool ACC>
static void up_class_t(Solver* const* ms, int count, int l, cudaStream_t st) {
  typedef typename RegionOf<T, H, ACC>::R R;
  const Level& L0 = ms[0]->lev[l];
  UpTab tab{};
  for (int i = 0; i < count; i++) {
    Solver* s = ms[i];
    Level& L = s->lev[l];
    tab.m[i] = {L.rhs, L.x, ACC ? nullptr : L.x2, s->lev[l + 1].x, ACC ? s->ph : nullptr, ACC ? s->pl : nullptr,
                s->dev};
    if (!ACC) std::swap(L.x, L.x2);
  }
  launch_dependent(true, k_mg_up_class<R, ACC>, region_grid<R>(L0.n, count), dim3(R::THREADS), 0, st, tab, L0.n,
                   L0.h2, ms[0]->prm.mg_post_smooth, (float)ms[0]->prm.relax, ms[0]->prm.max_cycles);
}

template <int H>
static void up_class(Solver* const* ms, int count, int l, cudaStream_t st) {
  const bool acc = l == 0;
  switch (tile_for_class(ms[0], l, count)) {
    case 64: acc ? up_class_t<64, H, true>(ms, count, l, st) : up_class_t<64, H, false>(ms, count, l, st); break;
    case 32: acc ? up_class_t<32, H, true>(ms, count, l, st) : up_class_t<32, H, false>(ms, count, l, st); break;
    default: acc ? up_class_t<16, H, true>(ms, count, l, st) : up_class_t<16, H, false>(ms, count, l, st); break;
  }
}

int mg_vcycle_class(Solver* const* ms, int count, cudaStream_t st) {
  Solver* s0 = ms[0];
  for (int i = 0; i < count; i++) {  // level 0 is the correction of the refinement cycle
    ms[i]->lev[0].x = ms[i]->e32;
    ms[i]->lev[0].x2 = ms[i]->e32b;
  }
  const int lb = bottom_first_level(s0);
  const fs_params& P = s0->prm;
  int launches = 0;
  for (int l = 0; l < lb; l++, launches++) {
    switch (P.mg_pre_smooth) {
      case 1: down_class<3>(ms, count, l, st); break;
      case 2: down_class<5>(ms, count, l, st); break;
      default: down_class<7>(ms, count, l, st); break;
    }
  }
  launch_bottom_class(ms, count, lb, st);
  launches++;
  for (int l = lb - 1; l >= 0; l--, launches++) {
    switch (P.mg_post_smooth) {
      case 1: up_class<2>(ms, count, l, st); break;
      case 2: up_class<4>(ms, count, l, st); break;
      default: up_class<6>(ms, count, l, st); break;
    }
  }
  return launches;
}
}  // namespace fs
