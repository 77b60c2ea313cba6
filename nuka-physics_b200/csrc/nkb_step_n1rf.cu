// step_kernel, straight-line stages of a split step: one coordinate per lane, with free rigid bodies.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kStagesNarrowRigid, 1, true, false, false, kPartStages)
}  // namespace nkb
