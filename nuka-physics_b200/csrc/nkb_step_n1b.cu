// step_kernel, one coordinate per lane, no contacts.  Without the contact stages (7-link arms, 150 envs, 41 steps) 1.55 ms against
// 1.69.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBare, 1, false, false, false, kPartBare)
}  // namespace nkb
