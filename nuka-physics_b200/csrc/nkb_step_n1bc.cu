// step_kernel, one coordinate per lane, no contacts, with the controllers of modes 3 and 4.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBareControl, 1, false, false, true, kPartBare)
}  // namespace nkb
