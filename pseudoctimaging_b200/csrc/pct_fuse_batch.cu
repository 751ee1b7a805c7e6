// The batched kernel for one register tile set (PCT_TILE_SET, given by the build). See pct_fuse_tma.cuh.
#include "pct_fuse_tma.cuh"

namespace pct {
namespace fuse {
namespace {

// Many subjects (uneven sizes, atlas counts and NH in {7, 9, 11}), one persistent launch: work
// items of all subjects are numbered consecutively, the longest windows and items first; a CTA takes
// the next one whenever it is done (a counter, read while the item before it runs) and dispatches
// it to the tile code of its subject's window.
template <int SET>
__global__ void __launch_bounds__(kThreads, BatchTileOf<SET, 5>::MB) fuse_batch_kernel(const BatchParams bp) {
  extern __shared__ unsigned char smem_raw[];
  // The current subject's view, copied into shared memory when the subject changes: the tile
  // code then reads its fields from there as it needs them instead of keeping the values it
  // loaded from global memory in registers (the single-subject kernel reads them from its
  // parameters).
  __shared__ __align__(16) SubjectView s_sv;
  static_assert(sizeof(SubjectView) % 4 == 0 && sizeof(SubjectView) <= 4 * kThreads, "copy");
  Pipe pp = pipe_init(smem_raw);
  int s = 0, cur = -1;
  __shared__ int s_next;
  int item = blockIdx.x;
  while (item < bp.total_items) {
    int next = 0;
    if (threadIdx.x == 0) next = (int)gridDim.x + atomicAdd(bp.next, 1);
    while (s + 1 < bp.nsub && bp.subjects[s + 1].item_begin <= item) ++s;
    if (s != cur) {  // uniform over the CTA
      __syncthreads();  // every thread is done with the previous subject's view
      if (threadIdx.x < sizeof(SubjectView) / 4)
        reinterpret_cast<int *>(&s_sv)[threadIdx.x] =
            reinterpret_cast<const int *>(bp.subjects + s)[threadIdx.x];
      __syncthreads();
      cur = s;
    }
    const SubjectView &sv = s_sv;
    const int local = item - sv.item_begin;
    bool ok = true;
    switch (sv.hw) {
      case 5: ok = run_item<5, BatchTileOf<SET, 5>::RX, BatchTileOf<SET, 5>::TZ, BatchTileOf<SET, 5>::LY>(sv, local, pp, bp.err, bp.timeout_ns, -1); break;
      case 4: ok = run_item<4, BatchTileOf<SET, 4>::RX, BatchTileOf<SET, 4>::TZ, BatchTileOf<SET, 4>::LY>(sv, local, pp, bp.err, bp.timeout_ns, -1); break;
      default: ok = run_item<3, BatchTileOf<SET, 3>::RX, BatchTileOf<SET, 3>::TZ, BatchTileOf<SET, 3>::LY>(sv, local, pp, bp.err, bp.timeout_ns, -1); break;
    }
    if (!ok) {
      pipe_drain(pp, bp.timeout_ns);
      return;
    }
    if (threadIdx.x == 0) s_next = next;
    __syncthreads();
    item = s_next;
  }
}

}  // namespace

template <>
cudaError_t batch_ctas_per_sm<PCT_TILE_SET>(int *per_sm) {
  constexpr int smem = batch_smem<PCT_TILE_SET>();
  auto kern = fuse_batch_kernel<PCT_TILE_SET>;
  const cudaError_t e =
      cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, kern, kThreads, smem);
}

template <>
cudaError_t launch_batch_items<PCT_TILE_SET>(const BatchParams &bp, int blocks, cudaStream_t stream) {
  fuse_batch_kernel<PCT_TILE_SET><<<blocks, kThreads, batch_smem<PCT_TILE_SET>(), stream>>>(bp);
  return cudaGetLastError();
}

}  // namespace fuse
}  // namespace pct
