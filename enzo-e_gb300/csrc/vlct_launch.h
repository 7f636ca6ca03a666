// vlct_launch.h -- typed launch entry points of the kernels (one set per
// precision; FP64 lives in kern_f64.cu compiled with --fmad=false, FP32 in
// kern_f32.cu).
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <stddef.h>

#include "vlct_types.h"

namespace vlct {

template <class R> struct AuxBlock;

// Largest tile extent that can be asked for, per precision.
template <class R> struct TileLimits;
template <> struct TileLimits<double> { static constexpr int TMAX = 16; };
template <> struct TileLimits<float> { static constexpr int TMAX = 40; };

// The kind of a fused stage kernel, and what a CTA of it holds of a tile of
// tx x ty columns: its columns with their halo, one a thread, and the ring of
// cells around them that PLM's stencil reaches.  nn: nearest-neighbour
// reconstruction.
//
// Threads and CTAs per SM: FP32 MHD stages want up to 166 registers a thread
// and run at 128 (two CTAs of 256); more, smaller-register CTAs spill (256^3
// HLLD + PLM box, cycle: 256 x 2 5.65 ms; NN at 224 x 3 and PLM at 224 x 2 6.05;
// both at 288 x 2 7.07).  Hydro stages are lighter: NN four CTAs of 256, PLM two
// of 320 (960-leaf HLLC mesh with flux correction, cycle: 6.00 ms; 3 x 256 and
// 2 x 288 5.98; 2 x 288 and 2 x 384 6.11; 3 x 256 both, slower while the tiles
// covered the layer around the updated cells too, 5.80: not taken up yet).
struct StageKind {
  bool f64, nn, mhd;
  constexpr int threads() const { return !f64 && !mhd && !nn ? 320 : 256; }
  // CTAs an SM holds at once
  constexpr int ctas() const { return f64 ? 1 : (mhd || !nn ? 2 : 4); }
  static constexpr int ring = 96;
  bool fits(int tx, int ty) const {
    return (tx + 2) * (ty + 2) <= threads() && 2 * (tx + ty + 4) <= ring;
  }
};

template <class R>
cudaError_t launch_stage(int solver, int recon, bool de,
                         const StageBlock<R>* d_blocks, const StageTile* d_tiles,
                         int ntiles, const StageInfo& info,
                         const PhysParams& phys, int grid, cudaStream_t st,
                         const SplitLaunch& split = SplitLaunch());

// Chunks a block is cut into by a kernel that takes nb x chunks CTAs of which the GPU
// holds `resident` at once, for blocks of `work` items, at least `least` of them a
// chunk.  A grid of exactly the CTAs held is best, as a few more make the whole GPU
// wait for them (FP32 hydro timestep, 16 blocks of 64^3: 608 CTAs, four on each SM,
// 44 us; 656 54 us; 304 56 us; 4864 47 us); where nb divides that badly, the fewest
// waves that are nine tenths full.
inline int wave_chunks(long nb, long resident, size_t work, size_t least) {
  const long most = std::max<long>(1, (long)(work / least));
  long best = 1;
  double full = 0.0;
  for (long w = 1; w <= 8 && full < 0.9; w++) {
    const long c = w * resident / nb;
    if (c >= most) return (int)most;
    const double f = (double)(c * nb) / (double)(w * resident);
    if (f > full + 1e-9) {
      full = f;
      best = c;
    }
  }
  return (int)best;
}

// chunks_per_block 0: as fills the GPU best, blocks having `cells` cells on average
template <class R>
cudaError_t launch_timestep(bool mhd, bool de, const AuxBlock<R>* d_blocks,
                            int nblocks, int chunks_per_block, size_t cells,
                            const PhysParams& phys, void* d_smax,
                            double courant, int global_min, double* d_dt,
                            double* d_dt_min, cudaStream_t st);

// max_m: the largest ghosted extent of any block (selects the multiply-high
// shell decode when it is exact for every block); chunks_per_block 0: as fills the
// GPU best, blocks having `shell` ghost cells on average
template <class R>
cudaError_t launch_refresh(const AuxBlock<R>* d_blocks, const int* d_nbr,
                           int nblocks, int g, int chunks_per_block, size_t shell, bool mhd, int max_m,
                           cudaStream_t st);

template <class R>
cudaError_t launch_copy_faces(int m0, int m1, int m2, int S1, const R* fx,
                              const R* fy, const R* fz, R* ox, R* oy, R* oz,
                              cudaStream_t st);

// FP64 conserved totals / div B of every block's active zones into out[8];
// partial: nb * cpb * 8 doubles of scratch.
template <class R>
cudaError_t launch_diag(const AuxBlock<R>* d_blocks, int nblocks, int g, int cpb,
                        bool mhd, bool de, double* partial, double* out,
                        cudaStream_t st);

// face B from an edge vector potential (double), then the centred B
template <class R>
cudaError_t launch_bfield_from_potential(int m0, int m1, int m2, const double* ax,
                                         const double* ay, const double* az, double dx,
                                         double dy, double dz, R* bfx, R* bfy, R* bfz,
                                         R* bx, R* by, R* bz, cudaStream_t st);

cudaError_t launch_set_scalar(double* p, double v, cudaStream_t st);

}  // namespace vlct
