// Instantiations of the fused streaming kernel for H_FIRST=true, float sums.
#include "fused_inst.cuh"

ZG_FUSED_INSTANCE(h_f32, true, false)
