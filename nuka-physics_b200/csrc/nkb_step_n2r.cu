// step_kernel<2, true>: two coordinates per lane, with free rigid bodies.
#define NKB_TEAM_BUILD
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepWideRigid, 2, true, false, false, kPartWhole)
}  // namespace nkb
