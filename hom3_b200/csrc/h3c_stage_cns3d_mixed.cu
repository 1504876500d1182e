// h3c_stage_cns3d_mixed.cu -- the 3D variants with FP32 fluxes of the CNS tile stage.
// A device module is loaded whole by the first call
// that touches it, so these lie in modules of their own: a process's first CNS
// grid took 18 ms to load all of them, 4 to 6 for its own.
#include "stage_cns.cuh"

namespace h3c {

template int cns_prepare_v<3, float>(unsigned, size_t, bool);
template void cns_stage_v<3, float>(int, bool, const GhostTables&, double*, const CnsLaunch&);

}  // namespace h3c
