// The tensor-core backward pass of the mesh adjoint (mesh_adjoint_mma.cu).
#pragma once

#include "hgx_internal.cuh"

namespace hgx {

struct BwmArgs {
  const float* tiles;        // the forward's FP32 tiles, anchors and slot -> triangle map
  const double4* anchors;
  const int* perm;
  int ntri, ntiles;
  const float4* seeds;       // 2 per pixel: (P03, M03), (P21, M21)
  const double* qx;
  const double* qy;
  const double2* rowqz;      // nrow x 4
  int nrow, ncol;
  double* partial;           // [splits][ntri][6], the slabs' sums added in order
  // set by bwm_run: items per row, 32-pixel chunks per item, and the slab's arrays
  int nch, nck;
  unsigned char* b;
  uint32_t* rec;
  float* xy;
  float* colmax;
  unsigned* err;
};

// How the pass is cut: slabs of `rows` rows, each in `splits` row ranges per group of 128
// triangles.  slabs == 0: the grid is too narrow for it.
struct BwmPlan {
  int nch, nck, rows, slabs, splits;
};
BwmPlan bwm_plan(hgx_ctx c, hgx_qgrid g, int ntiles, int ntri);
int bwm_run(hgx_ctx c, const BwmPlan& p, BwmArgs a);

}  // namespace hgx
