// step_kernel, constraint solve of a split step: two coordinates per lane, without free rigid bodies.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kSolveWide, 2, false, false, false, kPartSolve)
}  // namespace nkb
