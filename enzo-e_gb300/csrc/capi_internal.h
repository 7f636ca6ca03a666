// capi_internal.h -- host-side internals shared by the C ABI translation units.
#pragma once
#include <cuda_runtime.h>

#include <string>
#include <vector>

#include "../../include/mhdvlct_gb300.h"
#include "vlct_launch.h"
#include "vlct_types.h"

namespace mhdint {
// Tiles and z-chunks of the per-block path's stages.
struct PlainDecomp {
  int tx[2] = {8, 8}, ty[2] = {8, 8};
  int zchunk[2] = {0, 0};
};
}  // namespace mhdint

struct mhdvlct_handle {
  MhdVlctParams params;
  int solver = 2;        // vlct::Solver
  int recon = 1;         // reconstruction of the last stage
  int mhd = 1;
  int de = 0;
  int euler = 0;
  vlct::PhysParams phys;
  std::string err;
  // plain-path scratch, reused while the block geometry and dtype repeat
  int cache_dtype = -1;
  int cache_m[3] = {0, 0, 0};
  int cache_np = 0;            // passive-scalar scratch fields in the cache
  // the per-block path's decomposition of the last extents and dtype
  mhdint::PlainDecomp dc;
  int dc_dtype = -1;
  int dc_m[3] = {0, 0, 0};
  void* scratch = nullptr;     // one device allocation
  size_t scratch_bytes = 0;
  // the split stages' jobs of that geometry (FP64): per stage, and the
  // elements of workspace they share; split: the scratch holds them
  std::vector<vlct::SplitJob> sp_jobs[2];
  std::vector<vlct::SplitGroup> sp_groups[2];
  size_t sp_ws = 0;
  bool split = false;
  bool use_split = true;       // false: the fused kernels, as without room (tests)
  // mesh-refresh tables (pointer table, regions, chunks), reused across calls
  void* rf_dev = nullptr;
  size_t rf_bytes = 0;
  cudaEvent_t rf_done = nullptr;  // recorded after the last refresh launch
  std::vector<char> rf_host;
};

// Whether FP64 steps on this handle, and batches created on it from now on, run
// the split stages where their workspace can be had (the default) or the fused
// kernels, which otherwise run only where it cannot.  For tests.
extern "C" int mhdvlct_internal_use_split(mhdvlct_handle* h, int on);

namespace mhdint {

// Set the handle's error text and return the code.
int fail(mhdvlct_handle* h, int code, const std::string& msg);

// Stage geometry of the VL scheme: stale depth at entry and after the
// immediate staling of the reconstruction (EnzoReconstructorNN.hpp:31-35,
// EnzoReconstructorPLM.hpp:153-157).
struct StagePlan {
  int nstages;
  int recon[2];
  int s[2];
  int S[2];
  double dt_factor[2];
};
StagePlan stage_plan(const mhdvlct_handle* h);

// The kind of stage i (vlct_launch.h) on fields of a dtype.
vlct::StageKind stage_kind(const mhdvlct_handle* h, int dtype, int i);

// The cells that a stage updates, which its tiles cover.  m: ghosted extents of
// the block, S: stale depth after reconstruction.
struct Window {
  int lo, len[3];
};
Window stage_window(const int m[3], int S);

// A work decomposition of a stage: tile extents and z-chunk length (0: the
// whole window).
struct Decomp {
  int tx = 0, ty = 0, zchunk = 0;
};
// The tile of at most tx x ty columns (0: any) that the fused kernel holds and
// that covers an lx x ly window with the least work.
void fit_tile(const vlct::StageKind& k, int lx, int ly, int& tx, int& ty);
// Columns that fit_tile cuts an lx x ly window into.
long tile_columns(const vlct::StageKind& k, int lx, int ly, int tx, int ty);
// Tile and z-chunk for `nblocks` windows alone on a GPU of nsm SMs.
Decomp decompose(const vlct::StageKind& k, const Window& w, long nblocks, int nsm);

// Split a stage's window into tiles of at most tile_x x tile_y columns (as
// fit_tile gives them).
void make_tiles(int block, const int m[3], int S, int tile_x, int tile_y, int zchunk,
                std::vector<vlct::StageTile>& out);

// The jobs of a split stage over blocks of ghosted extents m (3 per block),
// blocks `ids` of them (all when empty), in groups whose workspace is bounded
// (by max_elems too, when given); ws_elems is raised to the elements the
// largest group needs.  No jobs when a block's planes are so wide that the fused
// kernel is the faster form.
void split_plan(const std::vector<int>& m, const std::vector<int>& ids, int S, bool final,
                bool mhd, bool de, std::vector<vlct::SplitJob>& jobs,
                std::vector<vlct::SplitGroup>& groups, size_t& ws_elems, size_t max_elems = 0);

// Device field pointers of a block view.
template <class R>
vlct::FieldSet<R> fieldset_of(const MhdBlockView* b);

// SM count of the current device (asked for once).
int sm_count();

// The batched form (batch.cu).  batch_create is mhdvlct_batch_create_ex with,
// when ordered_stream is not null, every device allocation, free and set-up
// copy of the batch ordered on that stream (cudaMallocFromPoolAsync from
// `pool`, or cudaMallocAsync when pool is null; cudaFreeAsync), so that
// creating or destroying it never waits for other streams' work.
int batch_create(mhdvlct_handle* h, const int* dims, const double* widths, int nblocks,
                 int ghost, int dtype, int npassive, int gravity,
                 cudaStream_t ordered_stream, cudaMemPool_t pool, mhdvlct_batch** out);
// Device address of the batch's simulated-time accumulator: the sum of dt
// over the cycles of the last mhdvlct_batch_run call.
const double* batch_time_device(const mhdvlct_batch* b);

// Mesh ghost refresh (refresh.cu): a validated plan of refresh faces over a
// set of block views -- the per-block field pointer table and the device
// records of the regions and their CTA chunks.
struct RefreshPlan {
  std::vector<void*> ptrs;  // MHD_NFIELD_SLOTS pointers per block
  std::vector<char> items;  // region records
  std::vector<char> chunks; // CTA chunk records
  int nchunks = 0;
  int dtype = MHD_DTYPE_F64;
};
int plan_refresh(mhdvlct_handle* h, const MhdBlockView* blocks, int nblocks,
                 const MhdRefreshFace* faces, int nfaces, unsigned conservative,
                 RefreshPlan& plan);
cudaError_t launch_refresh_faces(int dtype, const void* d_items, const void* d_chunks,
                                 int nchunks, void* const* d_ptrs, cudaStream_t st);

// Flux correction (fluxcorrect.cu): a validated plan -- the corrected faces,
// their CTA chunks and the blocks' field and flux pointers in one blob to
// upload once -- and its launch.
struct FluxCorrectPlan {
  std::vector<char> blob;
  size_t o_chunks = 0, o_blocks = 0;
  int nchunks = 0;
  int dtype = MHD_DTYPE_F64;
  int params[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};  // kernel parameters
};
int plan_flux_correct(mhdvlct_handle* h, const MhdBlockView* blocks, int nblocks,
                      const MhdFluxCorrection* fluxes, const MhdRefreshFace* faces,
                      int nfaces, unsigned conservative, FluxCorrectPlan& plan);
cudaError_t launch_flux_correct(const FluxCorrectPlan& plan, const void* d_blob,
                                cudaStream_t st);

}  // namespace mhdint
