// stage_split.hpp -- host interface of the Euler/AUSM tile stage with
// precomputed flux splits (h3c_stage_split.cu), shared with h3c_solver.cu.
#pragma once
#include "stage_halo.hpp"

namespace h3c {

// Device tables: the halo lists of stage_halo.hpp, and per cell its face
// neighbours' slots packed for one load (split_pack).
struct SplitGeom {
  const uint4* __restrict__ pack3;  // 3D: u16 slots of positions 0..5, level, 0
  const uint2* __restrict__ pack2;  // 2D: u16 slots of positions 0..3
  HaloGeom h;                       // halo ids, offsets, groups
};

// Packs lnb [2nd][ld] (and in 3D the level bytes) into pack [n] (16 bytes per cell in 3D, 8 in 2D).
size_t split_pack_bytes(int nd, long long n);
void split_pack(int nd, const unsigned short* lnb, const unsigned char* lvl, long long ld, long long n, void* pack,
                cudaStream_t st);

// Halo entries a block keeps in shared memory, and its dynamic shared memory.
int split_halo_slots(int nd);
size_t split_smem_bytes(int nd, bool mixed);
// Opts the instantiations a solver launches (stage_modes, with or without
// coarse/fine faces) into their dynamic shared memory where that needs an
// opt-in (outside capture); false when the kernel cannot be launched.
bool split_prepare(int nd, bool mixed, unsigned modes, bool hang, size_t smem);

// One stage: out = rk_combine<mode>(g.q0, qin, dt/dx R(qin)), with the fused
// next-step CFL minimum into dtmin when fuse; grid blocks take the tiles round-robin.
void split_stage(int nd, bool mixed, int mode, bool hang, bool fuse, const double* qin, double* out,
                 const Geometry& g, const SplitGeom& h, const PhysConst& pc, const Scalars* sc, long long* dtmin,
                 unsigned grid, size_t smem, cudaStream_t st);

}  // namespace h3c
