// stage_strip_d3.cu -- the strip form of the stage kernel for MCV3, split
// precision.  Compiled without FMA contraction: its fused operations are
// written out, so that one grid and several grids in a launch give the same bits.
#include "mcv_strip.cuh"

namespace mcv {

StageLauncher strip_launcher_d3() { return StripConfig<3>::make(); }

}  // namespace mcv
