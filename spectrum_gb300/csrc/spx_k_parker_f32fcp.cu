// spx_k_parker_f32fcp.cu -- the parker stepping kernels in float arithmetic with analytic field
// derivatives, specialised for DiffusionFullConstant and the boundary layout of one time boundary,
// two planes and one momentum boundary (diffusive shock acceleration).
#include "spx_k_family.cuh"

SPX_FAMILY_TU_DK(parker, f32fcp, kParker, kDfFull, kLayoutPlanes)
