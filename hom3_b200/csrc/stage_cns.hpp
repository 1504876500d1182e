// stage_cns.hpp -- what the host side of the CNS tile stage shares with its
// kernels (stage_cns.cuh): the shared-memory layout and the launches.
#pragma once
#include <cuda_runtime.h>

#include "stage_halo.hpp"

namespace h3c {

// The slopes a face reads: the transverse slopes of momentum and density
// (cns/physics.hpp:305-338 reads no energy slope), [sd][v] for v <= nd.
template <int ND> constexpr int kCnsSlopeVars = ND + 1;

// Whether the tables are a "brick" grid's: every tile a whole Morton brick, or
// at least with no more layer-1 cells than one (H1 of them: 256 around 8x8x4
// cells, 64 around 16x16) and no more faces whose minus side lies outside the
// tile than fit its border list (kCnsBorder: 32 + 32 + 64 of an 8x8x4 brick,
// 16 + 16 of a 16x16 one, each direction's padded to whole warps).  Bricks
// take the kernel variant with constant row strides and the border list.
template <int ND> constexpr int kCnsBrickH1 = ND == 3 ? 256 : 64;
template <int ND> constexpr int kCnsBorder = ND == 3 ? 128 : 64;

// Shared memory of one block.  In FP64 the copies land in the primitive
// rows themselves (the tile and first-layer cells' states are the first nv
// rows of the primitives) and only the second layer has a landing area of
// its own; in FP32 (R = float) the FP64 states land in a separate area.
//   mbarrier (16) | plus fluxes [nv][256] f64 | primitives [nv + nd + 2][S1] R | slopes [nd (nd + 1)][S1] R |
//   bricks: border fluxes [nv][kCnsBorder] R | landing: FP32 [nv][S] f64, FP64 the second layer's [nv][S - S1] |
//   neighbour slots [FP32: 2][2nd][256] u16
template <class R, int ND>
__host__ __device__ constexpr bool cns_land_in_prims() {
  return sizeof(R) == sizeof(double);
}
template <class R, int ND>
__host__ __device__ constexpr size_t cns_layout_bytes(int hmax, int h1max, bool brick) {
  const size_t rows = 2 * ND + 4 + ND * kCnsSlopeVars<ND>;
  return 16 + 8 * (size_t)(ND + 2) * kHaloTile + sizeof(R) * rows * (kHaloTile + h1max) +
         (brick ? sizeof(R) * (size_t)(ND + 2) * kCnsBorder<ND> : 0) +
         (cns_land_in_prims<R, ND>() ? 8 * (size_t)(ND + 2) * (hmax - h1max) : 8 * (size_t)(ND + 2) * (kHaloTile + hmax)) +
         (cns_land_in_prims<R, ND>() ? 1 : 2) * 2 * (size_t)(2 * ND) * kHaloTile;
}

struct CnsLaunch {
  const double* qin;
  double* out;
  const Geometry& g;
  const CnsHaloGeom& h;
  const PhysConst& pc;
  const Scalars* sc;
  long long* dtmin;
  int* status;
  int grid;
  size_t smem;
  cudaStream_t st;
};

// Opt-in and resident blocks per SM of the variants with these modes, and a
// stage with its ghost-slope pass; instantiated per dimension and precision.
template <int ND, class R>
int cns_prepare_v(unsigned modes, size_t smem, bool brick);
template <int ND, class R>
void cns_stage_v(int mode, bool fuse, const GhostTables& gt, double* gsl, const CnsLaunch& a);

}  // namespace h3c
