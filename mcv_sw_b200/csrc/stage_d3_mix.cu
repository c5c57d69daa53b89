// stage_d3_mix.cu -- stage-kernel instantiations for MCV3, split precision:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from; split-precision sweeps run on packed FP32
// pairs.
// the TMA walk entries form each loaded column's linear references once per
// work item (OPT bit 2); the walks of 3 cells also balance the sweep walks (bit 1).
// which of them wins where (RK4 step, us; the 12x12 tiles these replaced in
// brackets): 8x8 and smaller up to Nc=64 (34.9 at 32 [39.0], 42.3 at 64 [45.8]), the
// 12x12 walks from there to 150 (55.0 at 96 [55.0]), strips beyond.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d3_mix();  // stage_strip_d3_mix.cu

const StageLauncher *stage_launchers_d3_mix(int *count) {
  static const StageLauncher table[] = {
    StageConfig<3, 16, 12, 448, 2, true, 0>::make(),
    StageConfig<3, 8, 8, 448, 2, true, 0>::make(),
    StageConfig<3, 6, 6, 320, 2, true, 0>::make(),
    StageConfig<3, 4, 4, 224, 3, true, 0>::make(),
    StageConfig<3, 8, 8, 224, 3, true, 2, true, 2>::make(),
    StageConfig<3, 12, 12, 320, 2, true, 2, true, 2>::make(),
    StageConfig<3, 12, 12, 320, 2, true, 3, true, 3>::make(),
    strip_launcher_d3_mix()};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
