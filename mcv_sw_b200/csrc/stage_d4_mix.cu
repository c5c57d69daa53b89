// stage_d4_mix.cu -- stage-kernel instantiations for MCV4, split precision:
// the tile shapes (cells x cells, threads, CTAs per SM the registers must allow,
// sweep style (0: per-cell items, n: walks of n cells), TMA-staged persistent
// form) the autotuner chooses from; split-precision sweeps run on packed FP32
// pairs.
// the last entry's option bits (OPT 3) balance the sweep walks and form
// each loaded column's linear references once per work item.
// which of them wins where (RK4 step, us; the 8x8 per-cell items these replaced in
// brackets): 4x4 up to Nc=33 (34.9 at 16 [39.1]), 6x6 at 36..40 (43.3 at 36; 8x8 walked
// 45.2), 8x8 TMA walks from 41 to 124 (46.8 at 48 [48.1]; 122 at 120, strips 128), strips
// beyond (130 at 128, walks 138).  The strips' first two stages, which are timed, are
// 5% ahead of the walks' where the steps are even, so they are not tried below 124.
// tried(): the cells of a launch between which the autotuner times them; 640 threads
// also where a direct tile wins, for groups, which run persistent forms.
#include "mcv_stage.cuh"

namespace mcv {

StageLauncher strip_launcher_d4_mix();  // stage_strip_d4_mix.cu

const StageLauncher *stage_launchers_d4_mix(int *count) {
  static const StageLauncher table[] = {
    StageConfig<4, 8, 8, 320, 2, true, 2>::make().tried(800, 2100),
    StageConfig<4, 4, 4, 256, 3, true, 0>::make().tried(0, 1100),
    StageConfig<4, 6, 6, 256, 3, true, 0>::make().tried(1150, 1700),
    StageConfig<4, 8, 8, 640, 1, true, 2, true, 3>::make().tried(0, 1800),
    StageConfig<4, 8, 8, 320, 2, true, 0, true>::make().tried(2000, 3072),
    StageConfig<4, 8, 8, 320, 2, true, 2, true, 3>::make().tried(1700, 30000),
    strip_launcher_d4_mix().tried(15500)};
  *count = (int)(sizeof(table) / sizeof(table[0]));
  return table;
}

}  // namespace mcv
