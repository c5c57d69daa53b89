// mcv_strip_table.cuh -- launch table of the strip kernels.
#pragma once
#include "mcv_strip.cuh"
#include "mcv_strip64.cuh"

namespace mcv {

// Launch table of the strip form (split precision, or FP64).
template <int D, bool MIXED>
struct StripConfig {
  template <int KIND>
  using S = std::conditional_t<MIXED, StripSmem<D, KIND>, Strip64Smem<D, KIND>>;
  template <int KIND, int NB, bool IDENT>
  static constexpr auto kernel() {
    if constexpr (MIXED) return &strip_kernel<D, KIND, NB, IDENT>;
    else return &strip64_kernel<D, KIND, NB, IDENT>;
  }
  template <int KIND, int NB, bool IDENT>
  static void launch_nb(dim3 grid, cudaStream_t s, const StageBatch<NB> &b) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(32 * S<KIND>::WPB);
    cfg.dynamicSmemBytes = (size_t)S<KIND>::WPB * S<KIND>::BYTES;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel<KIND, NB, IDENT>(), b);
  }
  template <int KIND>
  static void launch(dim3 grid, cudaStream_t s, const StageBatch<1> &b) {
    launch_nb<KIND, 1, false>(grid, s, b);
  }
  template <int KIND>
  static void launch_ident(dim3 grid, cudaStream_t s, const StageBatch<1> &b) {
    launch_nb<KIND, 1, true>(grid, s, b);
  }
  template <int KIND>
  static void launch_batch(dim3 grid, cudaStream_t s, const StageBatch<kMaxGrids> &b) {
    launch_nb<KIND, kMaxGrids, false>(grid, s, b);
  }
  template <int KIND>
  static cudaError_t attr() {
    const int bytes = S<KIND>::WPB * S<KIND>::BYTES;
    cudaError_t e = cudaFuncSetAttribute(kernel<KIND, 1, false>(), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel<KIND, 1, true>(), cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(kernel<KIND, kMaxGrids, false>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                               bytes);
    return e;
  }
  static cudaError_t prepare() {
    cudaError_t e;
    if ((e = attr<0>()) || (e = attr<1>()) || (e = attr<2>()) || (e = attr<3>()) || (e = attr<4>()) ||
        (e = attr<5>()) || (e = attr<6>()))
      return e;
    return cudaSuccess;
  }
  static int blocks_per_sm() { return 1; }
  static StageLauncher make() {
    return StageLauncher{kStripCells, 1, 32 * S<1>::WPB, 1, 0, true, (size_t)S<1>::WPB * S<1>::BYTES, S<1>::RE, S<1>::H,
                    {&launch<0>, &launch<1>, &launch<2>, &launch<3>, &launch<4>, &launch<5>, &launch<6>},
                    {&launch_ident<0>, &launch_ident<1>, &launch_ident<2>, &launch_ident<3>, &launch_ident<4>,
                     &launch_ident<5>, &launch_ident<6>},
                    {&launch_batch<0>, &launch_batch<1>, &launch_batch<2>, &launch_batch<3>, &launch_batch<4>,
                     &launch_batch<5>, &launch_batch<6>}, &prepare, &blocks_per_sm,
                    {S<0>::WPB, S<1>::WPB, S<2>::WPB, S<3>::WPB, S<4>::WPB, S<5>::WPB, S<6>::WPB}};
  }
};

}  // namespace mcv
