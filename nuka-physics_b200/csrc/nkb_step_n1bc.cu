// step_kernel, one coordinate per lane, no contacts, with the controllers of modes 3 and 4 (operational space, 4 steps: 1024 arms 251
// us against 258 with the contact stages, 4096 arms 1030 and 1058).
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBareControl, 1, false, false, true, kPartBare)
}  // namespace nkb
