// NaN median fill after the path (RegularizationStep + Median,
// NewPatchedBrainPureC.cpp:1024-1047,1059-1106; PatchBasedPseudoCT.cu:1501-1595).
//
// The reference sweeps the interior in z, x, y order and replaces each NaN, in place, by the
// median of the non-NaN values of its 3x3x3 neighbourhood, so a voxel sees the fills of voxels
// before it in the sweep and the NaNs of voxels after it. That order is reproduced exactly,
// in parallel and without rounds: a NaN voxel is filled once none of its NaN neighbours that come
// EARLIER in the sweep is still NaN. Its earlier neighbours then hold their final fills (a value
// never changes again) and its later NaN neighbours are still NaN (each of them waits for it), so
// the median sees exactly what the sequential sweep would, whenever it looks.
//
// So one launch does a whole volume: the NaN voxels are listed, one warp takes each (27 lanes load
// the neighbourhood, the median comes from the values' ranks), and a warp whose voxel is not ready
// looks again; where warps have many voxels, lanes first test theirs for readiness. Looks are
// bounded; the host launches again while a launch still filled something, which also ends it where
// NaN in the border leaves voxels that nothing can fill. What bounds it is the chain of dependent
// fills, one L2 round trip each, and the host's one wait. 222x222x112 with a thousand NaN voxels,
// a copy before and the rounding and HU map after it: 77 us, 546 us with a launch per round, a host
// read every 4 to 64 rounds and one thread sorting each neighbourhood; the fill alone with 5 %, 30 %
// and all of the interior NaN: 0.27, 23 and 153 ms (0.86, 54 and 271).
#include <cuda_runtime.h>
#include <math.h>
#include <stddef.h>
#include <stdint.h>

#include "pct_internal.h"

namespace pct {
namespace {

// Lists the interior's NaN voxels: one warp per row along y, four loads in flight per lane.
__global__ void collect_nan_kernel(const float *__restrict__ vol, int nx, int ny, int nz, int lo,
                                   int *__restrict__ list, int *__restrict__ count) {
  const int ix = nx - 2 * lo, iy = ny - 2 * lo, rows = ix * (nz - 2 * lo);
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < rows; r += nwarps) {
    const int z = r / ix + lo, x = r % ix + lo;
    const int k0 = (z * nx + x) * ny + lo;
    for (int c = 0; c < iy; c += 128) {
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int y = c + 32 * j + lane;
        v[j] = y < iy ? vol[k0 + y] : 0.f;
      }
      if (!__any_sync(0xffffffffu, isnan(v[0]) || isnan(v[1]) || isnan(v[2]) || isnan(v[3]))) continue;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned m = __ballot_sync(0xffffffffu, isnan(v[j]));
        if (!m) continue;
        int at = 0;
        if (lane == 0) at = atomicAdd(count, __popc(m));
        at = __shfl_sync(0xffffffffu, at, 0);
        if ((m >> lane) & 1) list[at + __popc(m & ((1u << lane) - 1))] = k0 + c + 32 * j + lane;
      }
    }
  }
}

// One look at NaN voxel k by a whole warp: fills it if it is ready. Median() of the reference:
// stable order of the non-NaN values among the 27 in (z, x, y) order, the middle one or the double
// average of the two middle ones. Here each value's place in that order is counted.
enum Look { kWaits, kFilled, kNanMedian };  // kNanMedian: ready, but the average of both infinities
__device__ __forceinline__ Look try_fill(float *vol, int nx, int ny, int nz, int lo, int k, int lane) {
  const int nxy = nx * ny;
  const int z = k / nxy, x = k % nxy / ny, y = k % ny;
  const int dz = lane / 9 - 1, dx = lane / 3 % 3 - 1, dy = lane % 3 - 1;
  const bool on = lane < 27;
  const float v = on ? *((volatile const float *)vol + k + dz * nxy + dx * ny + dy) : 0.f;
  const bool nan = on && isnan(v);
  // An earlier interior NaN neighbour is still pending. (NaNs outside the interior are never
  // filled by the reference; they only drop out of the median.)
  const bool pending = nan && lane < 13 && z + dz >= lo && z + dz < nz - lo && x + dx >= lo &&
                       x + dx < nx - lo && y + dy >= lo && y + dy < ny - lo;
  if (__any_sync(0xffffffffu, pending)) return kWaits;
  const unsigned have = __ballot_sync(0xffffffffu, on && !nan);
  const int cnt = __popc(have);
  if (cnt == 0) return kWaits;
  int rank = 0;
#pragma unroll
  for (int j = 0; j < 27; ++j) {
    const float u = __shfl_sync(0xffffffffu, v, j);
    rank += (((have >> j) & 1) && (u < v || (u == v && j < lane))) ? 1 : 0;
  }
  const bool mine = (have >> lane) & 1;
  const unsigned hi = __ballot_sync(0xffffffffu, mine && rank == cnt / 2);
  const unsigned low = __ballot_sync(0xffffffffu, mine && rank == cnt / 2 - 1);
  const float b = __shfl_sync(0xffffffffu, v, __ffs(hi) - 1);
  const float a = __shfl_sync(0xffffffffu, v, low ? __ffs(low) - 1 : 0);
  const float m = (cnt & 1) == 0 ? (float)(((double)a + (double)b) / 2.0) : b;
  if (isnan(m)) return kNanMedian;
  if (lane == 0) *((volatile float *)vol + k) = m;
  return kFilled;
}

// Whether none of NaN voxel k's earlier interior neighbours is NaN (one thread).
__device__ __forceinline__ bool ready(const float *vol, int nx, int ny, int nz, int lo, int k) {
  const int nxy = nx * ny;
  const int z = k / nxy, x = k % nxy / ny, y = k % ny;
  bool pending = false;
#pragma unroll
  for (int j = 0; j < 13; ++j) {
    const int dz = j / 9 - 1, dx = j / 3 % 3 - 1, dy = j % 3 - 1;
    const float v = *((volatile const float *)vol + k + dz * nxy + dx * ny + dy);
    pending |= isnan(v) && z + dz >= lo && z + dz < nz - lo && x + dx >= lo && x + dx < nx - lo &&
               y + dy >= lo && y + dy < ny - lo;
  }
  return !pending;
}

constexpr int kLooks = 256;  // passes over a warp's pending voxels per launch

// The looks of one warp with many voxels. It also ends them when no warp fills anything any more: it reads the fill
// counter before every PER-th look and ends where two reads are equal and it filled nothing between
// them (too early an end costs one more launch, about 15 us). Without the reads a volume that nothing
// can fill went through all looks: 222x222x112, all NaN, 76 ms; 0.77 now, 0.88 with a launch per round.
template <int PER>
__device__ __forceinline__ void fill_looks(float *vol, int nx, int ny, int nz, int lo,
                                           const int *__restrict__ list, int n, int w, int nwarps,
                                           int lane, unsigned long long *fills,
                                           unsigned long long *nan_medians) {
  unsigned nans = 0;
  unsigned long long seen = ~0ull;  // the counter as last read
  for (int first = 0; first < kLooks; first += PER) {
    const unsigned long long now = *(volatile unsigned long long *)fills;
    bool left = false, any = false;
    for (int look = first; look < first + PER; ++look) {
      unsigned filled = 0;
      left = false;
      // the warp's voxels are w, w + nwarps, ...: 32 of them are tested at once, the pending taken
      // one by one
      for (int base = w; base < n; base += 32 * nwarps) {
        const long long i = base + (long long)lane * nwarps;
        const int k = i < n ? list[i] : -1;
        unsigned todo = __ballot_sync(0xffffffffu, k >= 0 && isnan(*((volatile const float *)vol + max(k, 0))));
        if (__popc(todo) > 2) {  // only the ready ones cost a warp's look
          const bool go = ((todo >> lane) & 1) && ready(vol, nx, ny, nz, lo, k);
          const unsigned to = __ballot_sync(0xffffffffu, go);
          left |= to != todo;
          todo = to;
        }
        while (todo) {
          const int j = __ffs(todo) - 1;
          todo &= todo - 1;
          const Look r = try_fill(vol, nx, ny, nz, lo, __shfl_sync(0xffffffffu, k, j), lane);
          filled += r == kFilled;
          nans += r == kNanMedian && look == 0;
          left |= r == kWaits;
        }
        if (PER == 1 && filled) {  // (a long look: the others read it sooner)
          any = true;
          if (lane == 0) atomicAdd(fills, (unsigned long long)filled);
          filled = 0;
        }
        if (base > n - 1 - 32 * nwarps) break;  // (the next base could overflow)
      }
      if (PER > 1 && filled) {
        any = true;
        if (lane == 0) atomicAdd(fills, (unsigned long long)filled);
      }
      if (!left) break;
    }
    if (!left || (!any && __all_sync(0xffffffffu, now == seen))) break;
    seen = any ? ~0ull : now;
  }
  if (lane == 0 && nans) atomicAdd(nan_medians, (unsigned long long)nans);
}

// The same for at most 32 voxels per warp, which stay in its lanes' registers: a look is one round trip
// to L2, and the counter is read after every sixteenth.
__device__ __forceinline__ void fill_few(float *vol, int nx, int ny, int nz, int lo,
                                         const int *__restrict__ list, int n, int w, int nwarps,
                                         int lane, unsigned long long *fills,
                                         unsigned long long *nan_medians) {
  const long long i = w + (long long)lane * nwarps;
  const int k = i < n ? list[i] : -1;
  // (a launch after the first one finds some filled)
  unsigned todo = __ballot_sync(0xffffffffu, k >= 0 && isnan(*((volatile const float *)vol + max(k, 0))));
  unsigned long long seen = ~0ull;
  for (int look = 0; todo && look < kLooks; ++look) {
    unsigned filled = 0, nans = 0;
    for (unsigned left = todo; left; left &= left - 1) {
      const int j = __ffs(left) - 1;
      const Look r = try_fill(vol, nx, ny, nz, lo, __shfl_sync(0xffffffffu, k, j), lane);
      if (r == kWaits) continue;
      todo &= ~(1u << j);
      filled += r == kFilled;
      nans += r == kNanMedian;
    }
    if (lane == 0 && filled) atomicAdd(fills, (unsigned long long)filled);
    if (lane == 0 && nans) atomicAdd(nan_medians, (unsigned long long)nans);
    if ((look & 15) != 15) continue;
    const unsigned long long now = *(volatile unsigned long long *)fills;
    if (__all_sync(0xffffffffu, now == seen)) break;
    seen = now;
  }
}

// A look takes 1 us with a voxel or two per warp and 300 us with a thousand, so the fewer there are,
// the more looks lie between two reads of the counter (64x64x32, all NaN: 0.09 ms as with a launch per
// round; 0.15 with eight looks between reads in the middle form, 1.8 without reads).
__global__ void __launch_bounds__(256) fill_kernel(float *vol, int nx, int ny, int nz, int lo,
                                                   const int *__restrict__ list,
                                                   const int *__restrict__ count,
                                                   unsigned long long *fills,
                                                   unsigned long long *nan_medians) {
  const int n = *count;
  const int lane = threadIdx.x & 31;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (n <= 2 * nwarps)
    fill_few(vol, nx, ny, nz, lo, list, n, w, nwarps, lane, fills, nan_medians);
  else if (n <= 64 * nwarps)
    fill_looks<4>(vol, nx, ny, nz, lo, list, n, w, nwarps, lane, fills, nan_medians);
  else
    fill_looks<1>(vol, nx, ny, nz, lo, list, n, w, nwarps, lane, fills, nan_medians);
}

}  // namespace

size_t regularize_scratch_bytes(long long nvox) {
  // An index list of at most nvox entries, its length and two counters.
  return (size_t)nvox * sizeof(int) + 64;
}

cudaError_t launch_regularize(float *vol, int nx, int ny, int nz, int nh, void *scratch,
                              cudaStream_t stream, long long *fills_out, int *rounds_out) {
  const int lo = (nh - 1) / 2 + 1;
  if (fills_out) *fills_out = 0;
  if (rounds_out) *rounds_out = 0;
  if (nx <= 2 * lo || ny <= 2 * lo || nz <= 2 * lo) return cudaSuccess;
  char *base = static_cast<char *>(scratch);
  struct Counters {
    unsigned long long fills, nan_medians;
    int listed;
  } host{};
  int *count = reinterpret_cast<int *>(base + offsetof(Counters, listed));
  int *list = reinterpret_cast<int *>(base + 64);
  cudaError_t e = cudaMemsetAsync(base, 0, 64, stream);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  collect_nan_kernel<<<sms * 8, 256, 0, stream>>>(vol, nx, ny, nz, lo, list, count);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  unsigned long long *fills = reinterpret_cast<unsigned long long *>(base);
  long long filled = 0;
  int launches = 0;
  for (;;) {
    const Counters before = host;
    // (every CTA resident: a warp may wait for a fill of another)
    fill_kernel<<<sms * 4, 256, 0, stream>>>(vol, nx, ny, nz, lo, list, count,
                                             fills, fills + 1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = cudaMemcpyAsync(&host, base, sizeof(host), cudaMemcpyDeviceToHost, stream)) !=
        cudaSuccess)
      return e;
    if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    ++launches;
    // A launch that filled nothing means that only voxels with no non-NaN neighbour remain (possible
    // only with NaN in the border) and those whose median is NaN, with what waits for either, and no
    // later one could fill them. A NaN median counts as a fill, as the voxel's one visit in a sweep
    // does; the volume stood still in this launch, so its first look met each of them once.
    filled = (long long)host.fills;
    if (host.fills >= (unsigned long long)host.listed) break;
    if (host.fills == before.fills) {
      filled += (long long)(host.nan_medians - before.nan_medians);
      break;
    }
  }
  if (fills_out) *fills_out = filled;
  if (rounds_out) *rounds_out = launches;
  return cudaSuccess;
}

}  // namespace pct
