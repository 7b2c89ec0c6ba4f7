// One build of the FK solver kernels: the including file defines GEM_NS and
// GEM_FAST (gem_plain / 0 and gem_fast / 1) and GEM_PHASE (0 toroidal, 1
// spheroidal, 2 adjoint phase, start radii and the dispatch).
#include <cuda_runtime.h>

#include <type_traits>

#include "fk_kernel.h"
#include "fk_solver.cuh"
#include "fk_phases.cuh"
#if GEM_FAST
#include "fk_group.cuh"
#endif

namespace GEM_NS {
namespace {

template <int PH, int BLK>
size_t phase_smem() {
  return (size_t)(BLK / 32) * PhaseDiag<PH, BLK>::L * PhaseNV<PH>::NV * 32 * sizeof(double2);
}

template <int PH, int BLK>
cudaError_t phase_attr() {
  static bool done = false;
  if (done) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(fk_phase_kernel<PH, BLK>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)phase_smem<PH, BLK>());
  if (e == cudaSuccess) done = true;
  return e;
}

template <int PH, int BLK>
cudaError_t launch_ph(const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  cudaError_t e = phase_attr<PH, BLK>();
  if (e != cudaSuccess) return e;
  fk_phase_kernel<PH, BLK><<<grid, BLK, phase_smem<PH, BLK>(), st>>>(P, L);
  return cudaGetLastError();
}

template <int PH, int BLK>
int bps() {
  if (phase_attr<PH, BLK>() != cudaSuccess) return 1;
  int nb = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, fk_phase_kernel<PH, BLK>, BLK, phase_smem<PH, BLK>()) !=
      cudaSuccess)
    return 1;
  return nb < 1 ? 1 : nb;
}

// calls f with the schedule's block size as a compile-time constant
template <class F>
auto with_block(int sched, F f) {
  if (sched < 0 || sched >= FK_NSCHED) sched = 0;
  constexpr const int(&B)[FK_NSCHED] = FK_SCHED_BLOCK[GEM_FAST];
  switch (sched) {
    case 1: return f(std::integral_constant<int, B[1]>());
    case 2: return f(std::integral_constant<int, B[2]>());
    case 3: return f(std::integral_constant<int, B[3]>());
    case 4: return f(std::integral_constant<int, B[4]>());
    case 5: return f(std::integral_constant<int, B[5]>());
    default: return f(std::integral_constant<int, B[0]>());
  }
}

template <int PH>
cudaError_t launch_sched(int sched, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  return with_block(sched, [&](auto b) { return launch_ph<PH, b.value>(P, L, grid, st); });
}

template <int PH>
int bps_sched(int sched) {
  return with_block(sched, [&](auto b) { return bps<PH, b.value>(); });
}

#if GEM_FAST
template <int PH>
cudaError_t launch_grp(const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  static_assert(group_smem<PH>() + sizeof(Tab) + sizeof(GroupTab) + 1024 <= 227 * 1024, "one block per SM");
  cudaError_t e = cudaFuncSetAttribute(fk_group_kernel<PH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)group_smem<PH>());
  if (e != cudaSuccess) return e;
  fk_group_kernel<PH><<<grid, GP_WARPS * 32, group_smem<PH>(), st>>>(P, L);
  return cudaGetLastError();
}
#endif

}  // namespace

// one translation unit per phase (GEM_PHASE): they compile side by side
#if GEM_PHASE == 0
cudaError_t launch_fk_tor(int sched, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  return launch_sched<PH_TOR>(sched, P, L, grid, st);
}
int bps_fk_tor(int sched) { return bps_sched<PH_TOR>(sched); }
#if GEM_FAST
cudaError_t launch_grp_tor(const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  return launch_grp<PH_TOR>(P, L, grid, st);
}
#endif
#elif GEM_PHASE == 1
cudaError_t launch_fk_sph(int sched, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  return launch_sched<PH_SPH>(sched, P, L, grid, st);
}
int bps_fk_sph(int sched) { return bps_sched<PH_SPH>(sched); }
#if GEM_FAST
cudaError_t launch_grp_sph(const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  return launch_grp<PH_SPH>(P, L, grid, st);
}
#endif
#else
cudaError_t launch_fk_tor(int sched, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st);
cudaError_t launch_fk_sph(int sched, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st);
int bps_fk_tor(int sched);
int bps_fk_sph(int sched);

cudaError_t launch_fk_phase(int phase, int sched, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  switch (phase) {
    case PH_TOR: return launch_fk_tor(sched, P, L, grid, st);
    case PH_SPH: return launch_fk_sph(sched, P, L, grid, st);
    case PH_ADJ: return launch_sched<PH_ADJ>(sched, P, L, grid, st);
    case 3:
      fk_set_status_kernel<<<(unsigned)((L.nkf + 127) / 128), 128, 0, st>>>(L, P.nnod);
      return cudaGetLastError();
    default:
      start_table_kernel<<<2 * L.nslot, START_ENTRIES, 0, st>>>(P, L);
      fk_setup_kernel<<<grid, 128, 0, st>>>(P, L);
      return cudaGetLastError();
  }
}

int fk_phase_blocks_per_sm(int phase, int sched) {
  switch (phase) {
    case PH_TOR: return bps_fk_tor(sched);
    case PH_SPH: return bps_fk_sph(sched);
    case PH_ADJ: return bps_sched<PH_ADJ>(sched);
    default: return 8;
  }
}

int fk_lane_slot_per_node() { return LaneLayout::PER_NODE; }

#if GEM_FAST
cudaError_t launch_grp_tor(const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st);
cudaError_t launch_grp_sph(const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st);
cudaError_t launch_fk_group(int phase, const FKStatic& P, const FKLaunch& L, int grid, cudaStream_t st) {
  switch (phase) {
    case PH_TOR: return launch_grp_tor(P, L, grid, st);
    case PH_SPH: return launch_grp_sph(P, L, grid, st);
    default: return launch_grp<PH_ADJ>(P, L, grid, st);
  }
}
#endif
#endif

}  // namespace GEM_NS
