// The row-grid kernels of the triangle form factor: FP32C on the tensor cores (ff_tri_mma.cu) and
// FP64 (ff_tri_f64.cu).
#pragma once

#include "ff_tri.cuh"

namespace hgx {

// Floats per tile of the in-plane array: (dx0, dx1, dy0, dy1) per pair of triangles, then the
// tile's largest in-plane offset and three unused.
constexpr int MMA_XY = TILE * 2 + 4;

// Triangle tiles of one call (ff_tri.cu prepares them): the FP32 tiles in the scalar layout,
// their anchors, the in-plane offsets alone (MMA_XY floats per tile), and per tile (largest |n~| component, smallest dz, largest dz, 0).
struct MmaTiles {
  const float* tiles;
  const double4* anchors;
  const float* xy;
  const float4* info;
  int ntiles, ntri;
};

// Enqueues the form factor of a row grid (g->mode 1 or 2).
int ff_rows_mma(hgx_ctx c, hgx_qgrid g, const MmaTiles& t, const Rot9& R, void* out, int ff_type);

// The same in FP64.  HGX_ERR_NO_MEMORY: nothing was enqueued, the plain kernel takes the call (no room for the
// split sums, or a grid on which it is the faster one).
int ff_rows_f64(hgx_ctx c, hgx_qgrid g, const double* sd, int ntri, const Rot9& R, void* out, int ff_type);

}  // namespace hgx
