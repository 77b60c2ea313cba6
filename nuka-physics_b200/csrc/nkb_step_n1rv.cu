// step_kernel, constraint solve of a split step: one coordinate per lane, with free rigid bodies.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kSolveNarrowRigid, 1, true, false, false, kPartSolve)
}  // namespace nkb
