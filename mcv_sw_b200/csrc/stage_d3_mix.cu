// stage_d3_mix.cu -- stage-kernel instantiations for MCV3, split precision:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from; split-precision sweeps run on packed FP32
// pairs.
// the TMA walk entries form each loaded column's linear references once per
// work item (OPT bit 2); the walks of 3 cells also balance the sweep walks (bit 1).
// which of them wins where (RK4 step, us; the 12x12 tiles these replaced in
// brackets): 4x4 up to Nc=26, 6x6 to 37 (35.0 at 32 [39.0]), 8x8 per-cell items to 45
// (38.4 at 40, 8x8 TMA 39.1), 8x8 TMA to 90 (42.7 at 64 [45.9]), the 12x12 walks from
// there to 165 (55.4 at 96 [55.0]; strips 58.3), strips beyond (119 at 181, 12x12 132).
// tried(): the cells of a launch between which the autotuner times them; 8x8 TMA also
// where a direct tile wins, for groups, which run persistent forms.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d3_mix();  // stage_strip_d3_mix.cu

const StageLauncher *stage_launchers_d3_mix(int *count) {
  static const StageLauncher table[] = {
    StageConfig<3, 16, 12, 448, 2, true, 0>::make().never_tried(),
    StageConfig<3, 8, 8, 448, 2, true, 0>::make().tried(1200, 2100),
    StageConfig<3, 6, 6, 320, 2, true, 0>::make().tried(500, 1400),
    StageConfig<3, 4, 4, 224, 3, true, 0>::make().tried(0, 700),
    StageConfig<3, 8, 8, 224, 3, true, 2, true, 2>::make().tried(0, 12000),
    StageConfig<3, 12, 12, 320, 2, true, 2, true, 2>::make().tried(3500, 45000),
    StageConfig<3, 12, 12, 320, 2, true, 3, true, 3>::make().tried(3500, 45000),
    strip_launcher_d3_mix().tried(12000)};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
