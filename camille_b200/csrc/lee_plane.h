// Stage and filter kernels of 2-D blocks (lee_plane.cu): declarations shared with the host.
#pragma once

#include <cuda.h>

#include "lee_internal.h"

namespace lee {

constexpr int kPlaneFdHalf = 2;    // the 4th-order difference
constexpr int kPlaneFilterNb = 5;  // closure rows per line end, at most
constexpr int kPlaneCols = 64;     // columns of a warp (two per thread)
constexpr int kPlaneRows = 4;      // rows of a stage CTA (one per warp)
constexpr int kPlaneMaxRows = 65535 * kPlaneRows;  // of a block: a grid's second dimension counts row groups
constexpr int kPlaneBatchTall = 8; // rows of a batched stage tile
constexpr int kPlaneSlots = 3;     // tiles whose boxes a batched filter CTA holds (the next ones in flight)
constexpr int kPlaneWarps = 8;     // warps of a filter CTA
constexpr int kPlaneBatchRows = 2; // rows a warp of the batched filter finishes

// The TMA box of a batched filter tile (halo of 4): rows start on 16 bytes.
template <typename T>
struct PlaneFilterBox {
  static constexpr int HX = 4;
  static constexpr int BX = kPlaneCols + 2 * HX, BY = kPlaneWarps * kPlaneBatchRows + 8;
  static constexpr int FB = BX * BY;
};
void plane_filter_box(int* bx, int* by);

// Difference weights by closure class (TmaStageParams::w).
template <typename T>
struct PlaneWeights {
  T w[6][5];
};

template <typename T>
struct PlaneStage {
  StageParams<T> s;
  T w[6][5];
  int overlap;  // launch while the stream's previous kernel still runs (the kernel waits for its end)
};

// One field of a filter launch: the pre-filter values, their rounding error (compensated), the
// outputs.
template <typename T>
struct PlaneFilterField {
  const T* x;
  const T* err;
  T* y;
  T* comp;
};

template <typename T>
struct PlaneFilter {
  int nx, ny, px;
  int rows;  // rows a warp finishes, 1 or 2
  int nb;    // closure rows per line end
  T w[1 + 2 * kPlaneFilterNb + 1][11];  // by class, offsets -hf..hf (TmaFilterParams::w)
  const int8_t* code[2];  // a block with holes: closure codes along xi and eta, and the mask
  const int* iblank;
  T blend;
  PlaneFilterField<T> f[kMaxVars];
  int overlap;  // as in PlaneStage
};

// traits: the block's layout traits and the stage's kind (not the increment kind)
template <typename T>
cudaError_t launch_plane_stage(const PlaneStage<T>& p, int traits, cudaStream_t s);
template <typename T>
cudaError_t launch_plane_filter(const PlaneFilter<T>& p, int hf, int V, cudaStream_t s);
// One launch over tiles (block, x0, y0, -) of kPlaneCols x kPlaneBatchTall points of many blocks.
template <typename T>
cudaError_t launch_plane_stage_batch(const StageParams<T>* prm, const int4* tiles, int n, const PlaneWeights<T>& w,
                                     int kind, bool jm_fields, cudaStream_t s);
// ... of kPlaneCols x kPlaneWarps * kPlaneBatchRows points; p gives nb, w and blend; maps: the four
// input fields' tensor maps of each block. A wait on a copy gives up after wait_ns and sets err.
template <typename T>
cudaError_t launch_plane_filter_batch(const BatchFilterInst<T>* inst, const CUtensorMap* maps, const int4* tiles, int n,
                                      const PlaneFilter<T>& p, int* err, unsigned long long wait_ns, cudaStream_t s);

}  // namespace lee
