// leg_fp64.cu - the cluster legs of the V-cycle (leg.cuh), FP64, built without FMA contraction.
#include "leg.cuh"

namespace lmm {
LMM_INSTANTIATE_LEG(double)
}  // namespace lmm

// the bounds-check table and record of this translation unit (empty
// unless built with -DLMM_BOUNDS_CHECK)
LMM_BC_UNIT(leg_fp64)
