// vlct_kern_impl.cuh -- explicit instantiation and runtime dispatch of the
// kernel templates for one precision R.  Included once per precision TU.
#pragma once
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "vlct_aux.cuh"
#include "vlct_launch.h"
#include "vlct_passive.cuh"
#include "vlct_split.cuh"
#include "vlct_stage.cuh"

namespace vlct {

namespace {
// Device ordinals a per-device cache covers.
constexpr int kMaxDevices = 64;

// CTAs of a kernel that the current device holds at once, asked for once per
// device (the query costs as much as a launch) and kept in `cache`.
inline cudaError_t resident_ctas(const void* k, int threads, size_t smem,
                                 std::atomic<int>* cache, int& out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  out = dev < kMaxDevices ? cache[dev].load(std::memory_order_acquire) : 0;
  if (out > 0) return cudaSuccess;
  int nsm = 1, per_sm = 1;
  e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, smem);
  if (e != cudaSuccess) return e;
  out = std::max(1, per_sm) * std::max(1, nsm);
  if (dev < kMaxDevices) cache[dev].store(out, std::memory_order_release);
  return cudaSuccess;
}

template <class R, bool MHD, bool DE>
cudaError_t timestep_one(const AuxBlock<R>* b, int nb, int cpb, size_t cells,
                         const PhysParams& phys, typename SpeedBits<R>::T* smax,
                         cudaStream_t st) {
  auto* k = timestep_kernel<R, MHD, DE>;
  if (cpb <= 0) {
    static std::atomic<int> cache[kMaxDevices];
    int resident = 1;
    const cudaError_t e = resident_ctas((const void*)k, 256, 0, cache, resident);
    if (e != cudaSuccess) return e;
    // at least a pass of an FP64 CTA, two of an FP32 one: one FP64 block of 16^3 in
    // 41 CTAs 19 us, in 10 33 us
    cpb = wave_chunks(nb, resident, cells, sizeof(R) == 8 ? 256 : 512);
  }
  k<<<nb * cpb, 256, 0, st>>>(b, nb, cpb, phys, smax);
  return cudaGetLastError();
}

// One stage as the kernels of vlct_split.cuh, group after group of jobs.
template <class R, int SOLVER, int RECON, bool DE>
cudaError_t stage_split(const StageBlock<R>* b, const SplitLaunch& sp, const StageInfo& info,
                        const PhysParams& phys, cudaStream_t st) {
  constexpr bool MHD = SOLVER != SOLVER_HLLC;
  R* ws = static_cast<R*>(sp.ws);
  static const int nsm = [] {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
      n = 1;
    return n;
  }();
  for (int k = 0; k < sp.ngroups; k++) {
    const SplitGroup& G = sp.groups[k];
    const SplitJob* jobs = sp.jobs + G.first;
    const unsigned gx = (unsigned)((G.cells + kSplitThreads - 1) / kSplitThreads);
    const dim3 cells(gx, G.count);
    // faces a thread takes: as many as leave 256 threads to every SM
    int kmax = 1;
    if (RECON != RECON_NN)
      kmax = (int)std::max<size_t>(1, std::min<size_t>(12, 3 * G.total / ((size_t)nsm * 256)));
    const int kmin = (kmax + 1) / 2;
    const dim3 faces((gx + kmin - 1) / kmin, G.count, 3);
    split_prim_kernel<R, SOLVER, RECON == RECON_NN, DE><<<cells, kSplitThreads, 0, st>>>(b, jobs, ws, info, phys);
    split_flux_kernel<R, SOLVER, RECON, DE><<<faces, kSplitThreads, 0, st>>>(b, jobs, ws, info, phys, kmax);
    if constexpr (MHD) split_emf_kernel<R, DE><<<cells, kSplitThreads, 0, st>>>(b, jobs, ws, info);
    split_update_kernel<R, MHD, DE><<<cells, kSplitThreads, 0, st>>>(b, jobs, ws, info, phys);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// One stage as the fused kernel, on a persistent grid: as many CTAs as fit on
// the GPU at once (asked for once per device: the query costs as much as a
// launch).
template <class R, int SOLVER, int RECON, bool DE, int EXTRA>
cudaError_t stage_fused(const StageBlock<R>* b, const StageTile* t, int nt,
                        const StageInfo& info, const PhysParams& phys, int grid,
                        cudaStream_t st) {
  auto* k = stage_kernel<R, SOLVER, RECON, DE, EXTRA>;
  constexpr size_t smem = stage_smem_bytes<R, SOLVER, RECON, DE>();
  constexpr int threads = StageBounds<R, SOLVER, RECON>::threads;
  static std::atomic<int> resident[kMaxDevices], ready[kMaxDevices];
  int dev = 0, fit = 1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= kMaxDevices || !ready[dev].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (dev < kMaxDevices) ready[dev].store(1, std::memory_order_release);
  }
  e = resident_ctas((const void*)k, threads, smem, resident, fit);
  if (e != cudaSuccess) return e;
  if (nt <= 0) return cudaSuccess;
  if (grid <= 0) grid = fit;
  k<<<std::min(grid, nt), threads, smem, st>>>(b, t, nt, info, phys);
  return cudaGetLastError();
}

template <class R, int SOLVER, int RECON, bool DE>
cudaError_t stage_one(const StageBlock<R>* b, const StageTile* t, int nt,
                      const StageInfo& info, const PhysParams& phys, int grid,
                      cudaStream_t st, const SplitLaunch& split) {
  if constexpr (std::is_same<R, double>::value) {
    if (split.ngroups > 0) {
      cudaError_t e = stage_split<R, SOLVER, RECON, DE>(b, split, info, phys, st);
      if (e == cudaSuccess && info.npass > 0 && nt > 0) {
        passive_kernel<R, RECON><<<nt, 256, 0, st>>>(b, t, info, phys);
        e = cudaGetLastError();
      }
      return e;
    }
  }
  const bool all = info.gravity != 0 || info.npass > 0;
  const bool fc = info.fc != nullptr || info.block_fc != 0;
  // the flux-storing-only variant exists for the hydro solver (flux
  // correction is hydro only); the others take the full variant
  cudaError_t e;
  if (all || (fc && SOLVER != SOLVER_HLLC))
    e = stage_fused<R, SOLVER, RECON, DE, EXTRA_ALL>(b, t, nt, info, phys, grid, st);
  else if (fc)
    e = stage_fused<R, SOLVER, RECON, DE, SOLVER == SOLVER_HLLC ? EXTRA_FC : EXTRA_ALL>(
        b, t, nt, info, phys, grid, st);
  else
    e = stage_fused<R, SOLVER, RECON, DE, EXTRA_NONE>(b, t, nt, info, phys, grid, st);
  if (e == cudaSuccess && SOLVER != SOLVER_HLLC && info.final_stage && nt > 0) {
    ring_bfield_kernel<R><<<nt, 128, 0, st>>>(b, t, info);
    e = cudaGetLastError();
  }
  // the passive scalars, on the same tiles, with the density fluxes the
  // stage kernel wrote
  if (e == cudaSuccess && info.npass > 0 && nt > 0) {
    passive_kernel<R, RECON><<<nt, 256, 0, st>>>(b, t, info, phys);
    e = cudaGetLastError();
  }
  return e;
}

template <class R, int SOLVER, bool DE>
cudaError_t stage_recon(int recon, const StageBlock<R>* b, const StageTile* t,
                        int nt, const StageInfo& info, const PhysParams& phys,
                        int grid, cudaStream_t st, const SplitLaunch& split) {
  switch (recon) {
    case RECON_NN: return stage_one<R, SOLVER, RECON_NN, DE>(b, t, nt, info, phys, grid, st, split);
    case RECON_PLM: return stage_one<R, SOLVER, RECON_PLM, DE>(b, t, nt, info, phys, grid, st, split);
    case RECON_PLM_ATHENA:
      return stage_one<R, SOLVER, RECON_PLM_ATHENA, DE>(b, t, nt, info, phys, grid, st, split);
  }
  return cudaErrorInvalidValue;
}

template <class R, int SOLVER>
cudaError_t stage_de(int recon, bool de, const StageBlock<R>* b,
                     const StageTile* t, int nt, const StageInfo& info,
                     const PhysParams& phys, int grid, cudaStream_t st,
                     const SplitLaunch& split) {
  return de ? stage_recon<R, SOLVER, true>(recon, b, t, nt, info, phys, grid, st, split)
            : stage_recon<R, SOLVER, false>(recon, b, t, nt, info, phys, grid, st, split);
}

}  // namespace

template <>
cudaError_t launch_stage<VLCT_REAL>(int solver, int recon, bool de,
                                    const StageBlock<VLCT_REAL>* b,
                                    const StageTile* t, int nt,
                                    const StageInfo& info,
                                    const PhysParams& phys, int grid,
                                    cudaStream_t st, const SplitLaunch& split) {
  switch (solver) {
    case SOLVER_HLLE: return stage_de<VLCT_REAL, SOLVER_HLLE>(recon, de, b, t, nt, info, phys, grid, st, split);
    case SOLVER_HLLC: return stage_de<VLCT_REAL, SOLVER_HLLC>(recon, de, b, t, nt, info, phys, grid, st, split);
    case SOLVER_HLLD: return stage_de<VLCT_REAL, SOLVER_HLLD>(recon, de, b, t, nt, info, phys, grid, st, split);
  }
  return cudaErrorInvalidValue;
}

template <>
cudaError_t launch_timestep<VLCT_REAL>(bool mhd, bool de,
                                       const AuxBlock<VLCT_REAL>* b, int nb,
                                       int cpb, size_t cells, const PhysParams& phys,
                                       void* d_smax, double courant,
                                       int global_min, double* d_dt,
                                       double* d_dt_min, cudaStream_t st) {
  typedef typename SpeedBits<VLCT_REAL>::T T;
  T* smax = (T*)d_smax;
  cudaError_t e = cudaMemsetAsync(smax, 0, sizeof(T) * 3 * (size_t)nb, st);
  if (e != cudaSuccess) return e;
  if (mhd)
    e = de ? timestep_one<VLCT_REAL, true, true>(b, nb, cpb, cells, phys, smax, st)
           : timestep_one<VLCT_REAL, true, false>(b, nb, cpb, cells, phys, smax, st);
  else
    e = de ? timestep_one<VLCT_REAL, false, true>(b, nb, cpb, cells, phys, smax, st)
           : timestep_one<VLCT_REAL, false, false>(b, nb, cpb, cells, phys, smax, st);
  if (e != cudaSuccess) return e;
  timestep_finish_kernel<VLCT_REAL><<<1, 256, 0, st>>>(b, nb, smax, courant, global_min,
                                                       d_dt, d_dt_min);
  return cudaGetLastError();
}

template <>
cudaError_t launch_refresh<VLCT_REAL>(const AuxBlock<VLCT_REAL>* b, const int* nbr,
                                      int nb, int g, int cpb, size_t shell, bool mhd, int max_m,
                                      cudaStream_t st) {
  // the decode of refresh_shell_kernel is exact while (shell elements of a
  // field) x (largest divisor) < 2^32; bound the shell by the whole field
  const unsigned long long mm = (unsigned long long)max_m + 1;
  const bool quick = mm * mm * mm * mm < (1ull << 32);
  if (cpb <= 0) {
    // One wave of CTAs, of a pass each at least, where that leaves none more than
    // 6000 ghost cells, with B, twice the arrays, 2000 (4000 in small blocks: FP32, 200
    // of 16^3, 400 CTAs 33 us, 1000 37; FP64 hydro, one block of 64^3:
    // 304 CTAs 9.9 us, 456 12.1; FP32, eight of 128^3: 456 CTAs 55.5 us, 4864 61.7).  More
    // work in chunks of 1700, with B 1100: a CTA's pointer tables cost it two memory
    // round trips (FP32, 512 blocks of 32^3: 6656 CTAs 193 us, 2048 206, 9728 197; MHD, 30
    // of 56^3: 1740 CTAs 74 us, 450 82).
    static std::atomic<int> cache[2][kMaxDevices];
    int resident = 1;
    const cudaError_t e =
        resident_ctas(quick ? (const void*)refresh_shell_kernel<VLCT_REAL>
                            : (const void*)refresh_kernel<VLCT_REAL>,
                      256, 0, cache[quick], resident);
    if (e != cudaSuccess) return e;
    const size_t one = (size_t)resident / nb;
    const size_t most = !mhd ? 6000 : one <= 2 ? 4000 : 2000;
    const bool wave = 4 * one * nb >= 3 * (size_t)resident && shell <= most * one;
    cpb = (int)std::max<size_t>(1, wave ? std::min(one, shell / 256) : shell / (mhd ? 1100 : 1700));
  }
  if (quick)
    refresh_shell_kernel<VLCT_REAL><<<nb * cpb, 256, 0, st>>>(b, nbr, nb, g, cpb);
  else
    refresh_kernel<VLCT_REAL><<<nb * cpb, 256, 0, st>>>(b, nbr, nb, g, NCELL + 11, cpb);
  return cudaGetLastError();
}

template <>
cudaError_t launch_copy_faces<VLCT_REAL>(int m0, int m1, int m2, int S1,
                                         const VLCT_REAL* fx, const VLCT_REAL* fy,
                                         const VLCT_REAL* fz, VLCT_REAL* ox,
                                         VLCT_REAL* oy, VLCT_REAL* oz,
                                         cudaStream_t st) {
  copy_faces_kernel<VLCT_REAL><<<256, 256, 0, st>>>(m0, m1, m2, S1, S1, fx, fy, fz,
                                                    ox, oy, oz);
  return cudaGetLastError();
}

template <>
cudaError_t launch_diag<VLCT_REAL>(const AuxBlock<VLCT_REAL>* b, int nb, int g, int cpb,
                                   bool mhd, bool de, double* partial, double* out,
                                   cudaStream_t st) {
  diag_kernel<VLCT_REAL><<<nb * cpb, 256, 0, st>>>(b, nb, g, cpb, mhd ? 1 : 0, de ? 1 : 0,
                                                   partial);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  diag_finish_kernel<<<1, 256, 0, st>>>(partial, nb * cpb, out);
  return cudaGetLastError();
}

template <>
cudaError_t launch_bfield_from_potential<VLCT_REAL>(
    int m0, int m1, int m2, const double* ax, const double* ay, const double* az,
    double dx, double dy, double dz, VLCT_REAL* bfx, VLCT_REAL* bfy, VLCT_REAL* bfz,
    VLCT_REAL* bx, VLCT_REAL* by, VLCT_REAL* bz, cudaStream_t st) {
  bfield_from_potential_kernel<VLCT_REAL><<<1024, 256, 0, st>>>(m0, m1, m2, ax, ay, az, dx, dy,
                                                               dz, bfx, bfy, bfz);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  center_bfield_kernel<VLCT_REAL><<<1024, 256, 0, st>>>(m0, m1, m2, bfx, bfy, bfz, bx, by, bz);
  return cudaGetLastError();
}

}  // namespace vlct
