// stage_d4_f64.cu -- stage-kernel instantiations for MCV4, FP64:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from.
// which of them wins where (RK4 step, us; the per-cell items these replaced in
// brackets): 4x4 by 384 threads up to Nc=26 (28.8 at 16 [32.9], 26.7 at 8 [32.9]), by 256
// to 34 (32.9 at 28; 8x8 39.0), 6x4 at 24, the walked tiles from 36 to 96 (104 at 90
// [115]; strips 110), strips beyond (109 at 96, 8x8 111; 127 at 112, 153).  tried(): the
// cells of a launch between which the autotuner times them.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d4_f64();  // stage_strip_d4_f64.cu

const StageLauncher *stage_launchers_d4_f64(int *count) {
  static const StageLauncher table[] = {
    StageConfig<4, 8, 8, 320, 2, false, 2>::make().tried(900, 40000),
    StageConfig<4, 6, 6, 256, 3, false, 3>::make().tried(1100, 14000),
    StageConfig<4, 4, 4, 384, 2, false, 0>::make().tried(0, 700),
    StageConfig<4, 4, 4, 256, 3, false, 0>::make().tried(250, 1200),
    StageConfig<4, 6, 4, 384, 2, false, 0>::make().tried(350, 700),
    StageConfig<4, 6, 6, 256, 2, false, 0, true>::make().never_tried(),
    StageConfig<4, 8, 8, 640, 1, false, 2, true>::make().tried(2000, 14000),
    strip_launcher_d4_f64().tried(8500)};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
