// stage_d4_f64.cu -- stage-kernel instantiations for MCV4, FP64:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from.
// which of them wins where (RK4 step, us; the per-cell items these replaced in
// brackets): 4x4 and 6x4 up to Nc=32 (28.8 at 16 [32.9], 26.7 at 8 [32.9]), the walked
// tiles from 48 to 96 (104 at 90 [115]), strips beyond.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d4_f64();  // stage_strip_d4_f64.cu

const StageLauncher *stage_launchers_d4_f64(int *count) {
  static const StageLauncher table[] = {
    StageConfig<4, 8, 8, 320, 2, false, 2>::make(),
    StageConfig<4, 6, 6, 256, 3, false, 3>::make(),
    StageConfig<4, 4, 4, 384, 2, false, 0>::make(),
    StageConfig<4, 4, 4, 256, 3, false, 0>::make(),
    StageConfig<4, 6, 4, 384, 2, false, 0>::make(),
    StageConfig<4, 6, 6, 256, 2, false, 0, true>::make(),
    StageConfig<4, 8, 8, 640, 1, false, 2, true>::make(),
    strip_launcher_d4_f64()};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
