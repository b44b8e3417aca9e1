// Instantiations of the fused streaming kernel for H_FIRST=false, float sums.
#include "fused_inst.cuh"

ZG_FUSED_INSTANCE(v_f32, false, false)
