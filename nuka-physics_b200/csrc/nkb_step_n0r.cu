// step_kernel<0, true>: free rigid bodies, no articulation.
#define NKB_TEAM_BUILD
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBodies, 0, true, false, false, kPartWhole)
}  // namespace nkb
