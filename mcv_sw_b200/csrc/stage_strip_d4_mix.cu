// stage_strip_d4_mix.cu -- the strip form of the stage kernel for MCV4, split precision.
// Compiled without FMA contraction: its fused operations are written out, so
// that one grid and several grids in a launch give the same bits.
#include "mcv_strip_table.cuh"

namespace mcv {

StageLauncher strip_launcher_d4_mix() { return StripConfig<4, true>::make(); }

}  // namespace mcv
