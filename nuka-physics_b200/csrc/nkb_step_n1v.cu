// step_kernel, constraint solve of a split step: one coordinate per lane, without free rigid bodies, 128 registers.
#include "nkb_step.cuh"

namespace nkb {
NKB_STEP_VARIANT(kSolveNarrow, 1, false, true, false, kPartSolve)
}  // namespace nkb
