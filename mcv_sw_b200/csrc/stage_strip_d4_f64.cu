// stage_strip_d4_f64.cu -- the strip form of the stage kernel for MCV4, FP64.
// Compiled without FMA contraction: its fused operations are written out, so
// that one grid and several grids in a launch give the same bits.
#include "mcv_strip_table.cuh"

namespace mcv {

StageLauncher strip_launcher_d4_f64() { return StripConfig<4, false>::make(); }

}  // namespace mcv
