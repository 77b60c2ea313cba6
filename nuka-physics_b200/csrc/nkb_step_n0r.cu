// step_kernel<0, true>: free rigid bodies, no articulation.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBodies, 0, true, false, false, kPartWhole)
}  // namespace nkb
