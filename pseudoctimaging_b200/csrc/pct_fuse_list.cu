// The plain kernel's tiles over an offset list (the centre prior) and over a list of masked items (the
// learned form's fallback). See pct_fuse_tma.cuh.
#include "pct_fuse_tma.cuh"

namespace pct {
namespace fuse {
namespace {

// An offset list (the centre prior) over the tiles of one subject. Counts its own evaluations
// where pct_learned_stats reads them. Issue-bound like the full search, plus the first planes of each
// run (a run of k = 81 has 3.9 offsets on average). y-pairs (2,6), 192x208x96, 8 atlases: k = 7
// 0.25 ms (0.58 by the rescoring's items), k = 81 1.34 ms (2.56), k = 123 2.03 ms (3.78); (2,4) 0.30 /
// 1.40 / 2.08, (3,4) 0.32 / 1.33 / 2.01 (without the sums kept per 64 offsets, which cost 1.5 % and
// halve the error against FP64: 8.1e-8 instead of 1.5e-7).
template <int HW, int RX, int TZ>
__global__ void __launch_bounds__(kThreads, 1)
    fuse_runs_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmL,
                     TmaParams p, const __grid_constant__ OffsetRuns runs,
                     unsigned long long *__restrict__ stats, unsigned long long evaluated) {
  extern __shared__ unsigned char smem_raw[];
  Pipe pp = pipe_init(smem_raw);
  p.sv.tmA = &tmA;
  p.sv.tmL = &tmL;
  if (blockIdx.x == 0 && threadIdx.x < 2) stats[threadIdx.x] = threadIdx.x ? evaluated : 0;
  for (int item = p.item_begin + blockIdx.x; item < p.item_end; item += gridDim.x) {
    if (!run_item<HW, RX, TZ, 1, false, true>(p.sv, item, pp, p.err, p.timeout_ns, -1, &runs)) {
      pipe_drain(pp, p.timeout_ns);
      return;
    }
  }
}

// The full search over a device-side list of masked items (count on the device, so the launch
// needs no host round trip): each item is up to two flagged atlases of one tile, its sums written
// to the partial slot of its pair.
template <int HW, int RX, int TZ, int LY, int MB>
__global__ void __launch_bounds__(kThreads, MB)
    fuse_list_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmL,
                     TmaParams p, const int *__restrict__ items, const int *__restrict__ count) {
  extern __shared__ unsigned char smem_raw[];
  Pipe pp = pipe_init(smem_raw);
  p.sv.tmA = &tmA;
  p.sv.tmL = &tmL;
  const int n = *count;
  for (int i = blockIdx.x; i < n; i += gridDim.x) {
    if (!run_item<HW, RX, TZ, LY, true>(p.sv, items[i], pp, p.err, p.timeout_ns, -1)) {
      pipe_drain(pp, p.timeout_ns);
      return;
    }
  }
}

template <int HW>
cudaError_t launch_runs_hw(const OffsetRuns &runs, int blocks, const CUtensorMap &tmA,
                           const CUtensorMap &tmL, const TmaParams &p, unsigned long long *stats,
                           unsigned long long evaluated, cudaStream_t stream) {
  using T = TileOf<6, HW>;
  using C = Cfg<HW, T::RX, T::TZ, true>;
  auto kern = fuse_runs_kernel<HW, T::RX, T::TZ>;
  constexpr int smem = C::SMEM + C::SUMS;
  static_assert(2 * (smem + 1024) <= 228 * 1024, "2 CTAs per SM");
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  kern<<<blocks, kThreads, smem, stream>>>(tmA, tmL, p, runs, stats, evaluated);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_runs(const OffsetRuns &runs, int blocks, const CUtensorMap &tmA,
                        const CUtensorMap &tmL, const TmaParams &p, unsigned long long *stats,
                        unsigned long long evaluated, cudaStream_t stream) {
  switch (runs.reach) {
    case 1: return launch_runs_hw<1>(runs, blocks, tmA, tmL, p, stats, evaluated, stream);
    case 2: return launch_runs_hw<2>(runs, blocks, tmA, tmL, p, stats, evaluated, stream);
    case 3: return launch_runs_hw<3>(runs, blocks, tmA, tmL, p, stats, evaluated, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_list(int sms, const CUtensorMap &tmA, const CUtensorMap &tmL, const TmaParams &p,
                        const int *items, const int *count, cudaStream_t stream) {
  using T = TileOf<0, 5>;
  using C = Cfg<5, T::RX, T::TZ>;
  auto kern = fuse_list_kernel<5, T::RX, T::TZ, T::LY, T::MB>;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM)) !=
      cudaSuccess)
    return e;
  int per_sm = 1;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, C::SMEM)) !=
      cudaSuccess)
    return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  kern<<<sms * per_sm, kThreads, C::SMEM, stream>>>(tmA, tmL, p, items, count);
  return cudaGetLastError();
}

}  // namespace fuse
}  // namespace pct
