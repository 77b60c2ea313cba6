// step_kernel, straight-line stages of a split step: two coordinates per lane, without free rigid bodies.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStagesWide, 2, false, false, false, kPartStages)
}  // namespace nkb
