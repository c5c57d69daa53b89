// stage_d3_f64.cu -- stage-kernel instantiations for MCV3, FP64:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from.
// which of them wins where (RK4 step, us; the 12x12 and 8x8 per-cell items these
// replaced in brackets): 4x4 and 6x4 up to Nc=32 (28.8 at 32 [30.9]), 8x8 walked by
// 448 threads at 48..64 (34.9 at 48 [38.9]), by 224 from there to 128 (62.8 at 96
// [67.8]), strips beyond.  The TMA tiles are for groups, which run persistent forms.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d3_f64();  // stage_strip_d3_f64.cu

const StageLauncher *stage_launchers_d3_f64(int *count) {
  static const StageLauncher table[] = {
    StageConfig<3, 12, 12, 320, 2, false, 2>::make(),
    StageConfig<3, 8, 8, 224, 4, false, 2>::make(),
    StageConfig<3, 8, 8, 448, 2, false, 2>::make(),
    StageConfig<3, 4, 4, 224, 3, false, 0>::make(),
    StageConfig<3, 6, 4, 224, 3, false, 0>::make(),
    StageConfig<3, 8, 8, 224, 2, false, 0, true>::make(),
    strip_launcher_d3_f64()};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
