// stage_d3_f64.cu -- stage-kernel instantiations for MCV3, FP64:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from.
// which of them wins where (RK4 step, us; the 12x12 and 8x8 per-cell items these
// replaced in brackets): 4x4 up to Nc=38 (28.8 at 32 [30.9], 6x4 30.8), 6x4 to 48,
// 8x8 walked by 448 threads at 40..64 (45.8 at 64 [47.1]), by 224 from 45 to 128 (62.6
// at 96 [67.8]; strips 68.2), 12x12 at 80 (53.5, 8x8 55.0), strips beyond (88.3 at 128,
// 8x8 89.0).  tried(): the cells of a launch between which the autotuner times them.
// The TMA tiles are for groups, which run persistent forms.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d3_f64();  // stage_strip_d3_f64.cu

const StageLauncher *stage_launchers_d3_f64(int *count) {
  static const StageLauncher table[] = {
    StageConfig<3, 12, 12, 320, 2, false, 2>::make().tried(6000, 7500),
    StageConfig<3, 8, 8, 224, 4, false, 2>::make().tried(2000, 65536),
    StageConfig<3, 8, 8, 448, 2, false, 2>::make().tried(1500, 5000),
    StageConfig<3, 4, 4, 224, 3, false, 0>::make().tried(0, 1500),
    StageConfig<3, 6, 4, 224, 3, false, 0>::make().tried(1400, 3072),
    StageConfig<3, 8, 8, 224, 2, false, 0, true>::make().never_tried(),
    strip_launcher_d3_f64().tried(9000)};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
