// One warp on 32 host threads, for the warp-level code of csrc/fk_group.cuh.
// __syncwarp(mask) is a barrier that orders memory between its lanes; a vote is
// exchanged by relaxed atomics and orders nothing, as on the GPU.  Built with
// ThreadSanitizer, a shared-memory access of one lane that nothing orders with
// another lane's is reported.
//   group_step_host race      every system, steps that reach the seventh attempt
//   group_step_host compare   step sizes over many decades: group form = thread form, bit for bit
//   group_step_host status    statuses of a set of sources after its adjoint phase
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <thread>
#include <type_traits>
#include <vector>

using std::max;
using std::min;
#define __device__
#define __host__
#define __global__
#define __constant__
#define __shared__
#define __grid_constant__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)
#define __align__(n)
#define asm(...) r = 1.0 / x   // the approximate reciprocal of rinv
struct alignas(16) double2 { double x, y; };
struct int2 { int x, y; };
inline double2 make_double2(double x, double y) { return {x, y}; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __dsub_rn(double a, double b) { return a - b; }
inline double __drcp_rn(double a) { return 1.0 / a; }
inline double __longlong_as_double(long long v) { double d; memcpy(&d, &v, 8); return d; }
template <class T> inline T __ldg(const T* p) { return *p; }
inline int __popc(unsigned v) { return __builtin_popcount(v); }
inline int __ffs(unsigned v) { return __builtin_ffs(v); }
inline unsigned long long clock64() { return 0; }
struct { unsigned x; } threadIdx, blockIdx, blockDim, gridDim;
inline void __syncthreads() {}
template <class T> T atomicAdd(T* p, T v);     // of the kernels, which are not instantiated here
template <class T, class U> T atomicCAS(T* p, U a, U b);
template <class T, class U> T atomicExch(T* p, U a);
void __threadfence_block();
void __nanosleep(unsigned);
template <class T> T __shfl_sync(unsigned, T, int);
template <class T> T __shfl_down_sync(unsigned, T, int);
unsigned __reduce_or_sync(unsigned, unsigned);
bool __all_sync(unsigned, bool);
using cudaError_t = int;
using cudaStream_t = void*;

static thread_local int LANE;
static void wait_change(const std::atomic<int>& g, int old, std::memory_order o) {
  while (g.load(o) == old) std::this_thread::yield();
}
static void __syncwarp(unsigned mask = 0xffffffffu) {
  struct Bar { std::atomic<unsigned> mask{0}; std::atomic<int> count{0}, gen{0}; };
  static Bar bars[64];
  Bar* b = bars;
  for (;; ++b) {   // the barrier of this set of lanes
    unsigned m = 0;
    if (b->mask.compare_exchange_strong(m, mask, std::memory_order_relaxed) || m == mask) break;
  }
  const int g = b->gen.load(std::memory_order_relaxed);
  if (b->count.fetch_add(1, std::memory_order_acq_rel) == __builtin_popcount(mask) - 1) {
    b->count.store(0, std::memory_order_relaxed);
    b->gen.store(g + 1, std::memory_order_release);
  } else {
    wait_change(b->gen, g, std::memory_order_acquire);
  }
}
static unsigned __ballot_sync(unsigned, bool p) {
  static std::atomic<unsigned> bits[3];
  static std::atomic<int> count{0}, gen{0};
  const int g = gen.load(std::memory_order_relaxed);
  if (p) bits[g % 3].fetch_or(1u << LANE, std::memory_order_relaxed);
  if (count.fetch_add(1, std::memory_order_relaxed) == 31) {
    bits[(g + 1) % 3].store(0, std::memory_order_relaxed);
    count.store(0, std::memory_order_relaxed);
    gen.store(g + 1, std::memory_order_relaxed);
  } else {
    wait_change(gen, g, std::memory_order_relaxed);
  }
  return bits[g % 3].load(std::memory_order_relaxed);
}
static bool __any_sync(unsigned m, bool p) { return __ballot_sync(m, p) != 0; }

#define GEM_NS gem_fast
#define GEM_FAST 1
#include "fk_group.cuh"

using namespace gem;
using namespace gem_fast;

template <class F> void warp(F f) {
  std::vector<std::thread> t;
  for (int l = 0; l < 32; ++l) t.emplace_back([=, &f] { LANE = l; f(l); });
  for (auto& x : t) x.join();
}

static FKStatic P;
static Tab tab;
static GroupTab T;
static std::vector<double> poly(4 * POLY_STRIDE);

// one layer of three knot intervals, every constant a cubic that varies by some per cent
static void setup() {
  P.nlay = 2; P.nk = 4; P.equidis = 0;
  tab.iktop[1] = 0; tab.iktop[2] = 4;
  for (int i = 0; i < 5; ++i) tab.rk[i] = tab.kb[i] = 1000.0 + 300.0 * i;
  for (int j = 0; j < 4; ++j)
    for (int v = 0; v < 16; ++v) {
      double* q = &poly[j * POLY_STRIDE + 4 * v];
      q[0] = 1e-10 * (v + 1); q[1] = -2e-8 * (v + 2); q[2] = 1e-5 * (v - 7); q[3] = v == 0 ? 3.0 : (v & 1 ? 60.0 + 10.0 * v : 0.5 + 0.1 * v);
    }
  group_tab(T);
}

static void env(Env& e, int nr) {
  e.tab = &tab; e.spl = nullptr; e.poly = poly.data(); e.nl = 2;
  e.omre = 0.05 + 0.01 * nr; e.omim = -1e-3; e.dll1 = 30.0 * (30.0 + nr);
}

template <int PH> void lane_state(Lane& L, double x, double h, double y, int nr) {
  memset((void*)&L, 0, sizeof L);
  env(L.e, nr);
  L.x = x; L.h = h; L.jknot = 1;
  for (int v = 0; v < 5; ++v) L.y[v] = dz{y * (1.0 - 0.3 * v + 0.1 * nr), y * 0.2 * (v - nr)};
}

// one step of the groups; returns the attempts, the groups' items in G
template <int PH, int SYS, bool ISO>
std::vector<int> groups(std::vector<GroupItem<PH>>& G, unsigned active) {
  constexpr int GL = GroupShape<PH>::GL;
  std::vector<int> res(32 / GL);
  warp([&](int l) {
    const int r = group_step<PH, SYS, ISO>(P, G[l / GL], T, active >> (l / GL) & 1, l);
    if (l % GL == 0) res[l / GL] = r;
  });
  return res;
}

template <int PH, int SYS, bool ISO> void race() {
  std::vector<GroupItem<PH>> G(32 / GroupShape<PH>::GL);
  for (double eps : {1e-30, 1e-4}) {
    P.eps = eps;
    for (unsigned active : {0xfu, 0x2u}) {
      for (size_t g = 0; g < G.size(); ++g) lane_state<PH>(G[g].L, 1250.0, 100.0, 1.0, (int)g);
      groups<PH, SYS, ISO>(G, active);
    }
  }
}

static int seen[8], beyond;   // steps by their result; accepted ones beside an attempt that overflowed

template <int PH, int SYS, bool ISO> int compare() {
  constexpr int NG = 32 / GroupShape<PH>::GL, NV = SysNV<SYS>::NV, NVD = PhaseNV<PH>::NV;
  std::vector<GroupItem<PH>> G(NG);
  std::vector<double2> D(4 * NVD * 32), scratch(32 * FK_LANE_STEP_SLOTS);
  int bad = 0;
  for (double eps : {1e-6, 1e-2, 1e3})
    for (int k = -6; k <= 64; ++k) {
      P.eps = eps;
      const double h = 500.0 * pow(10.0, k < 8 ? k / 4.0 : k - 6.0), y = k < 8 ? 1.0 : 1e-100;
      std::vector<Lane> L(32);
      for (int l = 0; l < 32; ++l) lane_state<PH>(L[l], 1010.0, h, y, l % NG);
      for (int g = 0; g < NG; ++g) G[g].L = L[g];
      const std::vector<int> rg = groups<PH, SYS, ISO>(G, 0xffu);
      std::vector<int> rt(32);
      warp([&](int l) {
        dz ye[5];
        Counters cnt{};
        Lane& q = L[l];
        bs_step<SYS, NVD, 4, ISO>(P, q.e, l < NG, q.h, q.x, q.y, ye, rt[l], D.data(), l, Slot{&scratch[l * FK_LANE_STEP_SLOTS], 1}, cnt, q.jknot);
        if (rt[l])
          for (int v = 0; v < NV; ++v) q.y[v] = ye[v];
      });
      for (int g = 0; g < NG; ++g) {
        bool over = false;
        for (int i = 0; i < 6 * NV; ++i) over |= !std::isfinite(G[g].Y[i].x);
        ++seen[rt[g]];
        beyond += rt[g] && over;
        if (rg[g] == rt[g] && !memcmp(G[g].L.y, L[g].y, NV * sizeof(dz))) continue;
        if (++bad < 4) printf("phase %d system %d eps %g h %g: group form %d, thread form %d\n", PH, SYS, eps, h, rg[g], rt[g]);
      }
    }
  return bad;
}

// item k of nkf, sources: two of moments, the force.  Failures: item 0 none, item 1 the toroidal or
// spheroidal phase, item 2 the second source, item 3 the first and the force, item 4 the force
static int set_status() {
  constexpr int NKF = 5, NN = 3, BLK = NKF * 20 * NN, FBLK = NKF * 10 * NN;
  int status[NKF] = {0, 7, 0, 0, 0}, src[3 * NKF] = {0, 0, 0, 2, 0, 0, 0, 1, 0, 0, 0, 0, 0, 3, 1};
  const int want[NKF] = {0, 7, 1, 2, 1}, from[NKF] = {3, 3, 2, 1, 3};   // first source whose block is cleared
  std::vector<double2> g64(2 * BLK + FBLK, double2{1.0, 1.0});
  std::vector<float> re(g64.size(), 1.0f), im(re);
  FKLaunch L{};
  L.nkf = NKF; L.nsrc = 3; L.src_blk = BLK; L.status = status; L.status_src = src;
  L.gf64 = g64.data(); L.gfre = re.data(); L.gfim = im.data();
  L.src_type[0] = L.src_type[1] = 1;
  blockDim.x = 128;
  for (threadIdx.x = 0; threadIdx.x < 128; ++threadIdx.x) fk_set_status_kernel(L, NN);
  int bad = memcmp(status, want, sizeof want) != 0;
  for (int b = 0; b < 3; ++b) {
    const int nsp = b < 2 ? 20 : 10, nsph = b < 2 ? 16 : 8;   // the toroidal spectra, the last ones of a node, stay
    for (int o = 0; o < NKF * nsp * NN; ++o) {
      const int k = o % NKF, q = o / NKF % nsp, at = b * BLK + o;
      const double v = b >= from[k] && q < nsph ? 0.0 : 1.0;
      bad += g64[at].x != v || g64[at].y != v || re[at] != v || im[at] != v;
    }
  }
  return bad;
}

int main(int argc, char** argv) {
  setup();
  if (argc > 1 && !strcmp(argv[1], "race")) {
    race<PH_TOR, SYS_TOROIDAL, true>();
    race<PH_SPH, SYS_MINORS, true>();
    race<PH_SPH, SYS_MINORS, false>();
    race<PH_SPH, SYS_FLUID, true>();
    race<PH_SPH, SYS_RADIAL, false>();
    race<PH_ADJ, SYS_SOLIDT, true>();
    return 0;
  }
  if (argc > 1 && !strcmp(argv[1], "status")) return set_status();
  const int bad = compare<PH_TOR, SYS_TOROIDAL, true>() + compare<PH_SPH, SYS_MINORS, false>() +
                  compare<PH_SPH, SYS_RADIAL, true>() + compare<PH_ADJ, SYS_SOLIDT, true>();
  printf("steps by attempts:");
  for (int v : seen) printf(" %d", v);
  printf("; accepted beside an overflow: %d; different: %d\n", beyond, bad);
  return bad || !beyond || !seen[3] || !seen[4] || !seen[5] || !seen[6] || !seen[7] || !seen[0];
}
