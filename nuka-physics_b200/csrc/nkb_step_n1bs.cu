// step_kernel, one coordinate per lane, no contacts, 128 registers: four warps per scheduler (4096 arms, 32 steps: 3.18 ms; 4.01 with
// three, 3.39 with the 128-register build that has the contact stages).
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBareSlim, 1, false, true, false, kPartBare)
}  // namespace nkb
