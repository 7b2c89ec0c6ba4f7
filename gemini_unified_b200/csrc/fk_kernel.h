// Launch-level structures of the FK kernels (device pointers only).
#pragma once
#include <cstdint>

#include "gem_device.cuh"

namespace gem {

// Schedules of a solver phase kernel: threads per block (one block per SM) of
// the plain and of the fast build.  The autotuner picks one per phase.  Batched
// configuration, fast build, toroidal / spheroidal / adjoint phase in ms: 256
// threads 65.6 / 203 / 107, 384 threads 56.2 / 210 / 99.8, 512 threads 55.3 /
// 210 / 108; the defaults are the fastest but for the toroidal phase, where 512
// threads are 0.9 ms faster.  The plain build tries 0..2 only.
constexpr int FK_NSCHED = 6;
constexpr int FK_SCHED_BLOCK[2][FK_NSCHED] = {{384, 512, 256, 384, 512, 256}, {256, 384, 512, 320, 448, 192}};
constexpr int FK_SCHED_DEFAULT[3] = {1, 0, 1};   // toroidal, spheroidal, adjoint
// Largest number of solves a phase of the fast build runs in the group form, 16
// or 8 lanes per solve.  The thread form takes the time of the longest solve
// whatever the number below its 37,888 lanes, the group form's grows with the
// solves once its 3,552 groups are busy, so the two break even at the number
// that the groups do in the time of the longest solve's chain.  Both forms were timed
// on slabs of 2,000 to 65,000 solves at the top and at the middle of a band, PREM to
// 0.02 .. 0.2 Hz and a crust to 0.4 .. 2 Hz, isotropic or not; per model the break-even lies at
//   with a core     toroidal 36,700 .. 48,000   spheroidal 25,500 .. 49,700
//   without         toroidal 18,100 .. 24,400   spheroidal  9,900 .. 15,500
// and the line at or below the least of them (ms, thread and group form: PREM to 0.2 Hz, 22,278
// solves, toroidal 11.1 and 6.1, spheroidal 55.7 and 30.1; PREM to 0.02 Hz, 26,500,
// spheroidal break-even 25,500; crust to 1 Hz, 9,331, spheroidal 2.84 and 2.18).
// An adjoint solve stops at every node, so the thread form's chain grows with the
// nodes and the break-even with it: 4 nodes 7,400 .. 7,900, 11 nodes 8,300 ..
// 10,400 (crust 11,400), 32 nodes 15,200 .. 19,800, 37 nodes 16,800 .. 21,700.  With 4 nodes
// the group form is behind as soon as a third solve per group begins, at 7,104 (0.40 and
// 0.35 ms); a set of sources on 11 nodes gains up to the line (7,635 positions: 7.3 and 8.6 ms for the call).
constexpr int FK_GROUP_MAX[2][3] = {{18000, 9500, 8000}, {36000, 25000, 8000}};   // without and with a core
constexpr int FK_GROUP_NODES = 30, FK_GROUP_MAX_ADJ = 13500;                       // adjoint phase of many nodes
constexpr int fk_group_max(bool core, int phase, int nnod) {
  return phase == 2 && nnod >= FK_GROUP_NODES ? FK_GROUP_MAX_ADJ : FK_GROUP_MAX[core][phase];
}
// candidate deferrals of the bookkeeping passes (lanes waiting, trips waited);
// the last waits for the whole warp: its lanes, on adjacent degrees of one
// frequency, reach their sub-interval ends within a few steps of each other
constexpr int FK_NDEFER = 6;
constexpr int FK_DEFER_MIN[FK_NDEFER] = {1, 8, 16, 32, 32, 32};
constexpr int FK_DEFER_WAIT[FK_NDEFER] = {0, 6, 10, 24, 48, 1000000};
constexpr int FK_DEFER_DEFAULT = 4;
// queue granularity: consecutive queue positions a lane reserves per fetch (it
// takes the next of its run without the queue until the run is used up), or,
// with FK_QCHUNK > 0, runs of that many positions the warps of a block share
constexpr int FK_NGRAN = 4;
constexpr int FK_GRAN[FK_NGRAN] = {1, 2, 4, 1};
constexpr int FK_QCHUNK[FK_NGRAN] = {0, 0, 0, 1024};
constexpr int FK_GRAN_DEFAULT = 0;
constexpr int MAX_LAYER_KNOTS = 64;    // knots per layer handled by the spline kernel
// per-lane scratch elements (double2) of one Bulirsch-Stoer step, after the
// lane's node storage: A(x0) y0 and the results of the sixth and fourth attempt
constexpr int FK_LANE_STEP_SLOTS = 15;

// radii of the turning-radius search per frequency and motion type: 400 steps of
// (R - r0) / 400 reach the top within rounding, in whole warps
constexpr int START_ENTRIES = 416;

struct PrepArgs {
  int nslot, nk, nlay, attmode;
  double df, fref;
  const int* jf;        // [nslot] frequency index of each slot
  const double* ro;     // 1-based knot arrays [nk+1]
  const double* vpv;
  const double* vph;
  const double* vsv;
  const double* vsh;
  const double* eta;
  const double* qkinv;
  const double* qminv;
  const double* rk;
  const int* iktop;     // 1-based [nlay+1]
  const int* ikbot;
  double* spl;          // [nslot][nk+1][SPL_STRIDE]
};

struct FKLaunch {
  const double* spl;    // spline tables [nslot][nk+1][SPL_STRIDE]
  const double* poly;   // cubic coefficients per knot interval [nslot][nk+1][POLY_STRIDE] (fast variant)
  const int* jf;        // [nslot]
  const int* koff;      // [nslot] output index of (slot, iwn = 1)
  const int2* items;    // (slot, iwn) of each output index k
  const int* order;     // queue position -> k, most expensive first
  int nitems;
  unsigned nqueue;      // queue positions: nitems, or nsrc * nitems in the adjoint phase of a set of sources
  long long nkf;        // extent of the wavenumber-frequency index in the outputs
  double2* gf64;        // optional FP64 output (nkf, nsp, nnod)
  float* gfre;          // optional FP32 real part
  float* gfim;          // optional FP32 imaginary part
  int* status;          // optional per-k status
  double2* scratch;     // per-thread node storage, element-major
  long long nthreads;   // scratch stride
  unsigned int* queue;  // work-queue counters, one per phase (zeroed before launch)
  double2* start_tab;   // [nslot][2][START_ENTRIES] (radius, velocity) of the turning-radius search
  int nslot;
  double* rstart;       // [2][nkf] start radius, toroidal then spheroidal
  double2* um;          // [jre*6][nkf] upward minors at nodes 1..jre
  double2* dm;          // [(nnod-jre+1)*6][nkf] downward minors at nodes jre..nnod
  double2* dets;        // [nkf] spheroidal determinant at the receiver
  unsigned long long* stats;   // 6 counters
  unsigned long long* prof;    // optional lockstep counters [8]
  unsigned long long* warp_ns; // optional per-warp (start, end) globaltimer stamps
  const signed char* prop_kopt;   // optional proposed order target per (phase, k): [3][nkf]
  const float* prop_hs;           // optional proposed multiplier of the initial step per (phase, k): [3][nkf]
  struct StepRec* steplog;     // optional record of every step attempt
  unsigned long long steplog_cap;
  unsigned long long* steplog_n;
  // deferral of the bookkeeping between integrations: a pass runs when
  // adv_min lanes wait, one has waited adv_wait trips, or none integrates
  int adv_min, adv_wait;
  int qgran;            // queue positions reserved per fetch (FK_GRAN)
  int qchunk;           // > 0: runs of queue positions shared by the warps of a block (FK_QCHUNK)
  // toroidal and adjoint phase of a set of source nodes (nsrc > 0): per source b
  // its node and type (0 force, 1 moment), passed by value; its output block
  // starts at element b * src_blk; status_src [nsrc][nkf]: adjoint status per source
  int nsrc;
  int* status_src;
  long long src_blk;
  unsigned char src_node[MAXNOD + 2];
  unsigned char src_type[MAXNOD + 2];
};
static_assert(MAXNOD + 1 <= 255, "source-node table entries are bytes");

// One Bulirsch-Stoer step attempt as the step log records it (32 bytes).
struct StepRec {
  double x;             // radius at the start of the step
  double h;             // step tried (signed)
  int k;                // item (wavenumber-frequency index of the run)
  float lgy;            // log10 of the mean |y| of the solution, including the renormalisation
  short nl;             // layer
  signed char sys;      // system (toroidal, minors, fluid, radial, adjoint)
  signed char result;   // attempt at which the step converged (3..7); 0: rejected
  short phase;          // phase kernel (0 toroidal, 1 spheroidal, 2 adjoint)
  short nstep;          // step number within the sub-interval
};

struct FKStatic;
}  // namespace gem

#include <cuda_runtime.h>
namespace gem {
cudaError_t launch_prep(const PrepArgs& A, int* d_err, cudaStream_t st);
cudaError_t launch_poly(const PrepArgs& A, double* poly, cudaStream_t st);
}  // namespace gem

// Two builds of the solver: gem_plain (parity path, no FMA contraction) and
// gem_fast (FMA, division-free spline, reciprocal complex inverses).
#define GEM_DECLARE_SOLVER(NS)                                                                          \
  namespace NS {                                                                                     \
  /* phase < 0: start radii; 0 toroidal, 1 spheroidal minors, 2 adjoint + spheroidal spectra;     */ \
  /* 3: status of a set of sources after its adjoint phase;                                       */ \
  /* sched: index into FK_SCHED_BLOCK[build]                                                     */ \
  cudaError_t launch_fk_phase(int phase, int sched, const gem::FKStatic& P, const gem::FKLaunch& L, int grid,  \
                              cudaStream_t st);                                                      \
  int fk_phase_blocks_per_sm(int phase, int sched);                                                  \
  int fk_lane_slot_per_node();                                                                       \
  }
GEM_DECLARE_SOLVER(gem_plain)
GEM_DECLARE_SOLVER(gem_fast)
namespace gem_fast {
// group form of a phase (fk_group.cuh): 16 or 8 lanes per solve, one block per SM
cudaError_t launch_fk_group(int phase, const gem::FKStatic& P, const gem::FKLaunch& L, int grid, cudaStream_t st);
}
namespace gem_ray {
// travel-time table by ray tracing (raytable.cu): one thread per turning radius
cudaError_t launch_ray_table(const gem::FKStatic& P, const double* spl, int ntp, int stype, double eps, double drtp,
                             double a0, double* rtp, double* slowness, float* table, int* status, cudaStream_t st);
}
namespace gem {
}  // namespace gem
