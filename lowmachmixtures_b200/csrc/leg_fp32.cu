// leg_fp32.cu - the cluster legs of the V-cycle (leg.cuh), FP32 preconditioner.
#include "leg.cuh"

namespace lmm {
LMM_INSTANTIATE_LEG(float)
}  // namespace lmm

// the bounds-check table and record of this translation unit (empty
// unless built with -DLMM_BOUNDS_CHECK)
LMM_BC_UNIT(leg_fp32)
