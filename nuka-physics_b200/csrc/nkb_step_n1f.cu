// step_kernel, straight-line stages of a split step: one coordinate per lane, without free rigid bodies, 128 registers.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStagesNarrow, 1, false, true, false, kPartStages)
}  // namespace nkb
