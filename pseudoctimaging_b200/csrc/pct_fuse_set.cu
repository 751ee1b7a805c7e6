// The plain kernel for one register tile set (PCT_TILE_SET, given by the build), every half window. See
// pct_fuse_tma.cuh.
#include "pct_fuse_tma.cuh"

namespace pct {
namespace fuse {
namespace {

// One subject, persistent over its work items. MB = CTAs per SM the register budget is sized for.
template <int HW, int RX, int TZ, int LY, int MB>
__global__ void __launch_bounds__(kThreads, MB)
    fuse_tma_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmL,
                    TmaParams p) {
  extern __shared__ unsigned char smem_raw[];
  Pipe pp = pipe_init(smem_raw);
  p.sv.tmA = &tmA;
  p.sv.tmL = &tmL;
  for (int item = p.item_begin + blockIdx.x; item < p.item_end; item += gridDim.x) {
    if (!run_item<HW, RX, TZ, LY>(p.sv, item, pp, p.err, p.timeout_ns, p.withhold_cta)) {
      pipe_drain(pp, p.timeout_ns);
      return;
    }
  }
}

template <int SET, int HW>
cudaError_t launch_tiles_hw(int blocks, const CUtensorMap &tmA, const CUtensorMap &tmL,
                            const TmaParams &p, const LaunchHooks &wt, cudaStream_t stream) {
  using T = TileOf<SET, HW>;
  using C = Cfg<HW, T::RX, T::TZ>;
  auto kern = fuse_tma_kernel<HW, T::RX, T::TZ, T::LY, T::MB>;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM)) !=
      cudaSuccess)
    return e;
  if (wt.start && (e = cudaEventRecord(wt.start, stream)) != cudaSuccess) return e;
  kern<<<blocks, kThreads, C::SMEM, stream>>>(tmA, tmL, p);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  return wt.stop ? cudaEventRecord(wt.stop, stream) : cudaSuccess;
}

}  // namespace

template <>
cudaError_t launch_tiles<PCT_TILE_SET>(int hw, int blocks, const CUtensorMap &tmA,
                                       const CUtensorMap &tmL, const TmaParams &p,
                                       const LaunchHooks &wt, cudaStream_t stream) {
  switch (hw) {
    case 1: return launch_tiles_hw<PCT_TILE_SET, 1>(blocks, tmA, tmL, p, wt, stream);
    case 2: return launch_tiles_hw<PCT_TILE_SET, 2>(blocks, tmA, tmL, p, wt, stream);
    case 3: return launch_tiles_hw<PCT_TILE_SET, 3>(blocks, tmA, tmL, p, wt, stream);
    case 4: return launch_tiles_hw<PCT_TILE_SET, 4>(blocks, tmA, tmL, p, wt, stream);
    case 5: return launch_tiles_hw<PCT_TILE_SET, 5>(blocks, tmA, tmL, p, wt, stream);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace fuse
}  // namespace pct
