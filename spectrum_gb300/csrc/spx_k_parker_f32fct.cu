// spx_k_parker_f32fct.cu -- the parker stepping kernels in float arithmetic with analytic field
// derivatives, specialised for DiffusionFullConstant and the boundary layout of one time boundary
// and no other (pure diffusion).
#include "spx_k_family.cuh"

SPX_FAMILY_TU_DK(parker, f32fct, kParker, kDfFull, kLayoutTime)
