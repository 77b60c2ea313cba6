// step_kernel, one coordinate per lane, no contacts, 128 registers: four warps per scheduler (4096 arms, 32 steps: 3.1 ms, 3.9 with
// three).
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStepBareSlim, 1, false, true, false, kPartBare)
}  // namespace nkb
