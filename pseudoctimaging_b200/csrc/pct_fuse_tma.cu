// Planning and launches of the plain kernel and its batched, list and masked forms (pct_fuse_tma.cuh), the
// combine of partial sums and the repack of stacks for TMA.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "pct_fuse_tma.cuh"

namespace pct {
namespace {

using namespace fuse;

PFN_cuTensorMapEncodeTiled_v12000 encode_fn() {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  if (!fn) {
    void *ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(ptr);
  }
  return fn;
}

}  // namespace

void *tensor_map_encoder() { return reinterpret_cast<void *>(encode_fn()); }

namespace {

// 4-D map over a pitched volume stack [num][nz][nx][pitch], box = one x-row slab of
// `box_z` planes x `box_y` columns. Out-of-volume elements read as zero.
cudaError_t make_slab_map(CUtensorMap *map, const float *base, int nx, int ny, int nz, int num,
                          int pitch, int box_y, int box_z) {
  auto fn = encode_fn();
  if (!fn) return cudaErrorNotSupported;
  const cuuint64_t dims[4] = {(cuuint64_t)ny, (cuuint64_t)nx, (cuuint64_t)nz, (cuuint64_t)num};
  const cuuint64_t strides[3] = {(cuuint64_t)pitch * 4, (cuuint64_t)pitch * 4 * nx,
                                 (cuuint64_t)pitch * 4 * nx * nz};
  const cuuint32_t box[4] = {(cuuint32_t)box_y, 1u, (cuuint32_t)box_z, 1u};
  const cuuint32_t estr[4] = {1u, 1u, 1u, 1u};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, const_cast<float *>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// Sums the per-group partial (product, sum_weight) of every interior voxel of planes [z0, z1) in
// group order and applies the output rule, so the result does not depend on which CTA ran which
// group.
__global__ void combine_groups_kernel(const float *__restrict__ partial, int groups, int nx, int ny,
                                      int z0, int z1, int lo, long long nvox,
                                      float *__restrict__ out) {
  const int ix = nx - 2 * lo, iy = ny - 2 * lo;
  const long long total = (long long)ix * iy * (z1 - z0);
  asm volatile("griddepcontrol.wait;" ::: "memory");  // the sums are complete
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int y = (int)(i % iy) + lo;
    const long long r = i / iy;
    const int x = (int)(r % ix) + lo;
    const int z = (int)(r / ix) + z0;
    const long long v = (long long)z * nx * ny + (long long)x * ny + y;
    float pr = 0.f, sw = 0.f;
    for (int g = 0; g < groups; ++g) {
      pr += partial[(2LL * g) * nvox + v];
      sw += partial[(2LL * g + 1) * nvox + v];
    }
    out[v] = fuse_result(pr, sw);
  }
}

// The same for every subject of a batch that runs in groups.
__global__ void combine_batch_kernel(const SubjectView *__restrict__ subjects, int nsub) {
  for (int s = blockIdx.y; s < nsub; s += gridDim.y) {
    const SubjectView &sv = subjects[s];
    const int groups = sv.groups, lo = sv.lo;
    if (groups < 2) continue;
    const int ix = sv.nx - 2 * lo, iy = sv.ny - 2 * lo;
    const long long total = (long long)ix * iy * (sv.nz - 2 * lo);
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
      const int y = (int)(i % iy) + lo;
      const long long r = i / iy;
      const int x = (int)(r % ix) + lo;
      const int z = (int)(r / ix) + lo;
      const long long v = (long long)z * sv.nxy + (long long)x * sv.ny + y;
      float pr = 0.f, sw = 0.f;
      for (int g = 0; g < groups; ++g) {
        pr += sv.partial[(2LL * g) * sv.nvox + v];
        sw += sv.partial[(2LL * g + 1) * sv.nvox + v];
      }
      sv.out[v] = fuse_result(pr, sw);
    }
  }
}

// The combine over the interior planes [z0, z1) (clipped to the interior).
cudaError_t launch_combine_groups(const Geometry &g, const float *partial, int groups, float *out,
                                  int z0, int z1, cudaStream_t stream) {
  z0 = std::max(z0, g.lo);
  z1 = std::min(z1, g.nz - g.lo);
  if (z1 <= z0 || g.ix <= 0 || g.iy <= 0) return cudaSuccess;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // Launched while the fusion drains (it waits for it on the device): 1 us less between the two.
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(sms * 8);
  cfg.blockDim = dim3(256);
  cfg.stream = stream;
  cudaLaunchAttribute attr{};
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, combine_groups_kernel, partial, groups, g.nx, g.ny, z0, z1, g.lo,
                            g.nvox(), out);
}

cudaError_t launch_combine_groups(const Geometry &g, const float *partial, int groups, float *out,
                                  cudaStream_t stream) {
  return launch_combine_groups(g, partial, groups, out, 0, g.nz, stream);
}

int sm_count() {
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms;
}

template <class T, int HW>
void tile_counts(const Geometry &g, FusePlan *pl) {
  constexpr int XC = Cfg<HW, T::RX, T::TZ>::XC;
  pl->rx = T::RX;
  pl->tz = T::TZ;
  pl->tiles_y = (g.iy + kOutY - 1) / kOutY;
  pl->tiles_x = (g.ix + XC - 1) / XC;
  pl->tiles_z = (g.iz + 2 * T::TZ - 1) / (2 * T::TZ);
  pl->tiles = pl->tiles_y * pl->tiles_x * pl->tiles_z;
}

// Measured cost of one output voxel of a tile, padding included, for all NH^3 offsets of one atlas
// (ns of the whole chip; 222x222x112, 10 atlases, two CTAs per SM), by half window and tile: (3,4) (NH 9: (3,3)
// with the label ring, NH 5: (3,3), NH 3: (4,2)), (2,5), (2,6), (2,4). Within a few per cent of
// each other, so that what decides is how much of the volume's last tiles is padding (NH 11 at
// 222x222x112: (2,5) tiles the 210 x 210 x 100 interior with 4 % less of it than (3,4)).
constexpr int kTileChoices[4] = {0, 5, 6, 7};
constexpr float kTileCost[5][4] = {{0.0185f, 0.0162f, 0.0146f, 0.0195f},
                                   {0.0635f, 0.0642f, 0.0643f, 0.0629f},
                                   {0.1708f, 0.1625f, 0.1575f, 0.1685f},
                                   {0.3510f, 0.3376f, 0.3356f, 0.3344f},
                                   {0.6020f, 0.5990f, 0.5970f, 0.6080f}};

// Expected time (us) of the volume's work items, `natl` atlases and 1 / splits of the window each:
// rounds of the persistent grid, the last one cheaper when it leaves SMs with one CTA (one warp per
// scheduler takes 0.61 of the time of two sharing it; 0.85 behind several full rounds), plus what each
// item spends on its windows, taps and stores and, with partial sums, the combine. Behind one full round
// the remainder takes 0.44 of a round up to 110 of 296 slots (37 %) and a whole one from 112 on, and the
// CTAs that take a second item pay its windows again: 7,000 plans of 380 shapes, where the rule for more
// rounds put 1.08 rounds of 8 groups (40x23x93, 8 atlases, NH 3: 47 us) before half a round of 4 (39).
// Of those shapes' best plans the chosen one is 1.2 % behind on average, 5 % or more on 36 of 380, 22 %
// at worst (2.0 %, 54 and 40 % with that rule for one round too).
double expected_us(const Geometry &g, const FusePlan &pl, int slots, double voxel_ns, int natl,
                   int splits, int groups) {
  const double rounds = (double)pl.tiles * groups / slots;
  const double full = std::floor(rounds), rem = rounds - full;
  const double voxels = (double)kOutY * kWarps * pl.rx * 2 * pl.tz;
  const double round = 1e-3 * slots * voxels * voxel_ns * natl / splits;  // items of average length
  const double longest = round * splits * ((g.nh + splits - 1) / splits) / g.nh;
  double t = 0.0, items = std::max(1.0, rounds);  // items: of a CTA that takes the most of them
  if (full < 1.0) {
    t = (rem <= 0.5 ? 0.61 : 1.0) * longest;
  } else if (full == 1.0 && rem > 0.0) {
    t = (rem < 0.365 ? 1.44 : 2.0) * round + longest - round;
    items = 1.85;
  } else if (rem > 0.0) {
    t = std::min((full + (rem <= 0.5 ? 0.85 : 1.0)) * round, (rounds + 0.4) * round) + longest - round;
  } else {
    t = full * round + longest - round;
  }
  t += items * (6.0 + 1.0 * natl);
  if (groups > 1) t += 2.5 + (double)g.ix * g.iy * g.iz * 16.0 * groups / 5e6;
  return t;
}

// Chooses the atlas groups and, once every atlas is a group of its own, the ranges of the window's
// rows that the items of a tile are split into, for one tile shape: fills *pl and returns its
// expected time. Small volumes have fewer tiles than the chip has room for (64x64x32, one atlas:
// 42 tiles on 148 SMs, 81 us for one CTA's 343 offsets), so their windows are split over CTAs.
// Three groups or more are taken over fewer when they cost at most 3 % more: the host-pointer path
// overlaps its uploads with the fusion group by group, and the FP32 sums are shorter.
double choose_groups(const Geometry &g, int slots, double voxel_ns, size_t partial_limit,
                     bool may_split, FusePlan *pl) {
  const int ns = g.nh;
  auto bytes_of = [&](int groups) {
    return groups > 1 ? (size_t)groups * 2 * (size_t)g.nvox() * sizeof(float) : 0;
  };
  auto time_of = [&](int agroups, int splits) {
    const int groups = agroups * splits;
    if (bytes_of(groups) > partial_limit || (long long)pl->tiles * groups >= (1LL << 31)) return -1.0;
    return expected_us(g, *pl, slots, voxel_ns, g.num / agroups, splits, groups);
  };
  int agroups = 1, splits = 1;
  double best = time_of(1, 1);
  auto consider = [&](int a, int sp) {
    const double t = time_of(a, sp);
    if (t < 0.0 || t >= best) return;
    best = t;
    agroups = a;
    splits = sp;
  };
  for (int a = 2; a <= g.num; ++a)
    if (g.num % a == 0) consider(a, 1);
  for (int sp = 2; may_split && sp <= ns; ++sp) consider(g.num, sp);
  if (splits == 1 && agroups < 3)
    for (int a = 3; a <= g.num; ++a) {
      if (g.num % a) continue;
      const double t = time_of(a, 1);
      if (t < 0.0 || t > 1.03 * best) continue;
      best = t;
      agroups = a;
      break;
    }
  pl->atlas_groups = agroups;
  pl->splits = splits;
  pl->groups = agroups * splits;
  pl->partial_bytes = bytes_of(pl->groups);
  return best;
}

template <int SET, int HW>
double plan_hw(const Geometry &g, int sms, double voxel_ns, size_t partial_limit, FusePlan *pl,
               bool may_split = true) {
  using T = TileOf<SET, HW>;
  // two CTAs share an SM's shared memory (228 KB, 1 KB reserved per CTA) and registers
  static_assert(T::MB > 1 || 2 * (Cfg<HW, T::RX, T::TZ>::SMEM + 1024) <= 228 * 1024, "2 CTAs per SM");
  tile_counts<T, HW>(g, pl);
  pl->set = SET;
  const int slots = sms * (T::MB > 1 ? T::MB : 2);
  const double t = choose_groups(g, slots, voxel_ns, partial_limit, may_split, pl);
  const long long items = (long long)pl->tiles * pl->groups;
  pl->ctas = (int)(items < slots ? items : slots);
  return t;
}

SubjectView subject_view(const Geometry &g, const SlabInputs &in, float *out, double div,
                         float *partial, const FusePlan &pl) {
  SubjectView sv{};
  sv.img = in.img;
  sv.out = out;
  sv.partial = partial;
  sv.nx = g.nx;
  sv.ny = g.ny;
  sv.nz = g.nz;
  sv.nxy = g.nx * g.ny;
  sv.nvox = g.nvox();
  sv.scale = (float)sqrt(1.4426950408889634 / div);
  sv.tiles_y = pl.tiles_y;
  sv.tiles_x = pl.tiles_x;
  sv.ntiles = pl.tiles;
  sv.groups = pl.groups;
  sv.splits = pl.splits;
  sv.atlases_per_group = g.num / pl.atlas_groups;
  sv.hw = g.hw;
  sv.lo = g.lo;
  return sv;
}

template <int SET, int HW>
cudaError_t launch_hw(const Geometry &g, const SlabInputs &in, float *out, double div,
                      float *partial, int *err, const LaunchHooks &wt, const FusePlan &pl,
                      int item_begin, int item_end, cudaStream_t stream) {
  using T = TileOf<SET, HW>;
  using C = Cfg<HW, T::RX, T::TZ>;
  if (pl.groups > 1 && !partial) return cudaErrorInvalidValue;
  const bool whole = item_begin < 0;  // every item, then the combine
  if (whole) {
    item_begin = 0;
    item_end = pl.groups * pl.tiles;
  } else if ((pl.groups < 2 && !out) || item_begin >= item_end || item_end > pl.groups * pl.tiles) {
    return cudaErrorInvalidValue;
  }
  cudaError_t e;
  CUtensorMap tmA, tmL;
  if ((e = make_slab_map(&tmA, in.atlas, g.nx, g.ny, g.nz, g.num, in.pitch, C::YB, C::ZA)) !=
      cudaSuccess)
    return e;
  if ((e = make_slab_map(&tmL, in.label, g.nx, g.ny, g.nz, g.num, in.pitch, C::YB, C::ZL)) !=
      cudaSuccess)
    return e;
  TmaParams p{};
  p.sv = subject_view(g, in, out, div, partial, pl);
  p.err = err;
  p.timeout_ns = 2000000000ull;  // 2 s per wait; a step's copies land in microseconds
  p.withhold_cta = -1;
  if (wt.timeout_ns) {
    p.timeout_ns = wt.timeout_ns;
    p.withhold_cta = 0;
  }
  p.item_begin = item_begin;
  p.item_end = item_end;
  const int blocks = std::min(pl.ctas, p.item_end - p.item_begin);
  if ((e = launch_tiles<SET>(HW, blocks, tmA, tmL, p, wt, stream)) != cudaSuccess) return e;
  if (whole && pl.groups > 1) return launch_combine_groups(g, partial, pl.groups, out, stream);
  return cudaSuccess;
}

template <int SET>
double plan_set(const Geometry &g, int sms, double voxel_ns, size_t limit, FusePlan *pl) {
  switch (g.hw) {
    case 1: return plan_hw<SET, 1>(g, sms, voxel_ns, limit, pl);
    case 2: return plan_hw<SET, 2>(g, sms, voxel_ns, limit, pl);
    case 3: return plan_hw<SET, 3>(g, sms, voxel_ns, limit, pl);
    case 4: return plan_hw<SET, 4>(g, sms, voxel_ns, limit, pl);
    default: return plan_hw<SET, 5>(g, sms, voxel_ns, limit, pl);
  }
}

double plan_internal(const Geometry &g, int set, int sms, double voxel_ns, size_t limit,
                     FusePlan *pl) {
  switch (set) {
    case 1: return plan_set<1>(g, sms, voxel_ns, limit, pl);
    case 2: return plan_set<2>(g, sms, voxel_ns, limit, pl);
    case 3: return plan_set<3>(g, sms, voxel_ns, limit, pl);
    case 4: return plan_set<4>(g, sms, voxel_ns, limit, pl);
    case 5: return plan_set<5>(g, sms, voxel_ns, limit, pl);
    case 6: return plan_set<6>(g, sms, voxel_ns, limit, pl);
    case 7: return plan_set<7>(g, sms, voxel_ns, limit, pl);
    default: return plan_set<0>(g, sms, voxel_ns, limit, pl);
  }
}

template <int SET>
cudaError_t launch_set(const Geometry &g, const SlabInputs &in, float *out, double div,
                       float *partial, int *err, const LaunchHooks &wt, const FusePlan &pl, int ib,
                       int ie, cudaStream_t stream) {
  switch (g.hw) {
    case 1: return launch_hw<SET, 1>(g, in, out, div, partial, err, wt, pl, ib, ie, stream);
    case 2: return launch_hw<SET, 2>(g, in, out, div, partial, err, wt, pl, ib, ie, stream);
    case 3: return launch_hw<SET, 3>(g, in, out, div, partial, err, wt, pl, ib, ie, stream);
    case 4: return launch_hw<SET, 4>(g, in, out, div, partial, err, wt, pl, ib, ie, stream);
    case 5: return launch_hw<SET, 5>(g, in, out, div, partial, err, wt, pl, ib, ie, stream);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_any(const Geometry &g, const SlabInputs &in, float *out, double div,
                       float *partial, int *err, const LaunchHooks &wt, const FusePlan &pl, int ib,
                       int ie, cudaStream_t s) {
  switch (pl.set) {
    case 0: return launch_set<0>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 1: return launch_set<1>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 2: return launch_set<2>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 3: return launch_set<3>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 4: return launch_set<4>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 5: return launch_set<5>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 6: return launch_set<6>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    case 7: return launch_set<7>(g, in, out, div, partial, err, wt, pl, ib, ie, s);
    default: return cudaErrorInvalidValue;
  }
}

// Tiles and slab box sizes of one subject in the batched kernel.
template <int SET, int HW>
void batch_plan_hw(const Geometry &g, FusePlan *pl, int *yb, int *za, int *zl) {
  using T = BatchTileOf<SET, HW>;
  using C = Cfg<HW, T::RX, T::TZ>;
  tile_counts<T, HW>(g, pl);
  *yb = C::YB;
  *za = C::ZA;
  *zl = C::ZL;
}

template <int SET>
cudaError_t batch_plan(int hw, const Geometry &g, FusePlan *pl, int *yb, int *za, int *zl) {
  *pl = FusePlan{};
  pl->groups = pl->atlas_groups = pl->splits = 1;  // (the batch's plan says how many: plan_batch)
  switch (hw) {
    case 5: batch_plan_hw<SET, 5>(g, pl, yb, za, zl); return cudaSuccess;
    case 4: batch_plan_hw<SET, 4>(g, pl, yb, za, zl); return cudaSuccess;
    case 3: batch_plan_hw<SET, 3>(g, pl, yb, za, zl); return cudaSuccess;
    default: return cudaErrorInvalidValue;
  }
}

// Atlas groups of a batch's subjects: items no longer than a twelfth of the whole batch's time (a last
// item then keeps the other SMs waiting for about a twenty-fourth of it), not below 80 us. Six
// subjects with 2..8 atlases, items of up to 1.5 ms: 7.18 ms against 7.75 with one group each and a
// fixed stride over the items; a sixth and a twenty-fourth of the time: 7.25 and 7.27. Without the room
// for the partial sums every subject is one group.
BatchPlan plan_batch_groups(const Geometry *geoms, const int *tiles, const double *atlas_us, int n,
                            int slots, size_t partial_limit) {
  BatchPlan plan;
  plan.groups.assign(n, 1);
  double total = 0.0;
  for (int i = 0; i < n; ++i) total += atlas_us[i] * geoms[i].num * tiles[i] / slots;
  const double target = std::max(80.0, total / 12);
  for (int i = 0; i < n; ++i) {
    int g = 1;
    while (g < geoms[i].num && (geoms[i].num % g || atlas_us[i] * geoms[i].num / g > target)) ++g;
    if (tiles[i] == 0 || (long long)tiles[i] * g >= (1LL << 31)) g = 1;
    plan.groups[i] = g;
    if (g > 1) plan.partial_bytes += (size_t)g * 2 * (size_t)geoms[i].nvox() * sizeof(float);
  }
  if (plan.partial_bytes > partial_limit) {
    plan.groups.assign(n, 1);
    plan.partial_bytes = 0;
  }
  return plan;
}

template <int SET>
cudaError_t plan_batch_set(const Geometry *geoms, int n, size_t partial_limit, BatchPlan *plan) {
  std::vector<int> tiles(n);
  std::vector<double> us(n);
  const int slots = 2 * sm_count();
  for (int i = 0; i < n; ++i) {
    FusePlan pl;
    int yb, za, zl;
    const cudaError_t e = batch_plan<SET>(geoms[i].hw, geoms[i], &pl, &yb, &za, &zl);
    if (e != cudaSuccess) return e;
    const bool work = geoms[i].ix > 0 && geoms[i].iy > 0 && geoms[i].iz > 0;
    tiles[i] = work ? pl.tiles : 0;
    us[i] = 1e-3 * slots * kOutY * kWarps * pl.rx * 2 * pl.tz * kTileCost[geoms[i].hw - 1][3];
    if (n == 1 && work) {  // alone: by its rounds of the grid, as the single-subject kernel
      choose_groups(geoms[0], slots, kTileCost[geoms[0].hw - 1][3], partial_limit, false, &pl);
      plan->groups.assign(1, pl.groups);
      plan->partial_bytes = pl.partial_bytes;
      return cudaSuccess;
    }
  }
  *plan = plan_batch_groups(geoms, tiles.data(), us.data(), n, slots, partial_limit);
  return cudaSuccess;
}

template <int SET>
cudaError_t launch_batch_set(const BatchSubjectIn *subs, int n, const BatchPlan &plan, float *partial,
                             void *dev_scratch, int *err, cudaStream_t stream, BatchSetup *setup) {
  // Order subjects by window (largest first), so CTAs working at the same time mostly run the
  // same tile code, and within a window by the length of their items.
  if ((int)plan.groups.size() != n || (plan.partial_bytes && !partial)) return cudaErrorInvalidValue;
  std::vector<int> order(n);
  for (int i = 0; i < n; ++i) order[i] = i;
  auto length = [&](int i) { return subs[i].geom.num / plan.groups[i]; };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
    return subs[a].geom.hw != subs[b].geom.hw ? subs[a].geom.hw > subs[b].geom.hw
                                              : length(a) > length(b);
  });
  std::vector<SubjectView> views(n);
  std::vector<CUtensorMap> maps(2 * (size_t)n);
  int total = 0;
  cudaError_t e;
  for (int k = 0; k < n; ++k) {
    const BatchSubjectIn &b = subs[order[k]];
    FusePlan pl;
    int yb, za, zl;
    if ((e = batch_plan<SET>(b.geom.hw, b.geom, &pl, &yb, &za, &zl)) != cudaSuccess) return e;
    if ((e = make_slab_map(&maps[2 * k], b.in.atlas, b.geom.nx, b.geom.ny, b.geom.nz, b.geom.num,
                           b.in.pitch, yb, za)) != cudaSuccess)
      return e;
    if ((e = make_slab_map(&maps[2 * k + 1], b.in.label, b.geom.nx, b.geom.ny, b.geom.nz,
                           b.geom.num, b.in.pitch, yb, zl)) != cudaSuccess)
      return e;
    pl.groups = pl.atlas_groups = plan.groups[order[k]];
    SubjectView sv = subject_view(b.geom, b.in, b.out, b.div, partial, pl);
    if (pl.groups > 1) partial += (size_t)pl.groups * 2 * (size_t)b.geom.nvox();
    if (b.geom.ix <= 0 || b.geom.iy <= 0 || b.geom.iz <= 0) pl.tiles = 0;
    if ((long long)total + (long long)pl.tiles * pl.groups >= (1LL << 31)) return cudaErrorInvalidValue;
    sv.item_begin = total;
    total += pl.tiles * pl.groups;
    views[k] = sv;
  }
  // Device copies: maps first (64-byte aligned), then the subject views pointing at them.
  unsigned char *base = static_cast<unsigned char *>(dev_scratch);
  CUtensorMap *d_maps = reinterpret_cast<CUtensorMap *>(base);
  SubjectView *d_views = reinterpret_cast<SubjectView *>(base + maps.size() * sizeof(CUtensorMap));
  for (int k = 0; k < n; ++k) {
    views[k].tmA = d_maps + 2 * k;
    views[k].tmL = d_maps + 2 * k + 1;
  }
  if ((e = cudaMemcpyAsync(d_maps, maps.data(), maps.size() * sizeof(CUtensorMap),
                           cudaMemcpyHostToDevice, stream)) != cudaSuccess)
    return e;
  if ((e = cudaMemcpyAsync(d_views, views.data(), views.size() * sizeof(SubjectView),
                           cudaMemcpyHostToDevice, stream)) != cudaSuccess)
    return e;
  // Host copies must outlive the asynchronous transfers.
  if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;

  int per_sm = 1;
  if ((e = batch_ctas_per_sm<SET>(&per_sm)) != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const int slots = sm_count() * per_sm;
  setup->params_ready = true;
  setup->items = total;
  setup->blocks = total < slots ? total : slots;
  setup->set = SET;
  setup->bp_subjects = d_views;
  setup->bp_nsub = n;
  setup->bp_err = err;
  setup->combine = plan.partial_bytes > 0;
  return cudaSuccess;
}

}  // namespace

size_t batch_scratch_bytes(int n) {
  return 2 * (size_t)n * sizeof(CUtensorMap) + (size_t)n * sizeof(SubjectView) + 256;
}

cudaError_t plan_batch(const Geometry *geoms, int n, int set, size_t partial_limit, BatchPlan *plan) {
  switch (set) {
    case 0: return plan_batch_set<0>(geoms, n, partial_limit, plan);
    case 1: return plan_batch_set<1>(geoms, n, partial_limit, plan);
    case 2: return plan_batch_set<2>(geoms, n, partial_limit, plan);
    case 3: return plan_batch_set<3>(geoms, n, partial_limit, plan);
    case 4: return plan_batch_set<4>(geoms, n, partial_limit, plan);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t prepare_batch(const BatchSubjectIn *subs, int n, int set, const BatchPlan &plan,
                          float *partial, void *dev_scratch, int *err, cudaStream_t stream,
                          BatchSetup *setup) {
  for (int i = 0; i < n; ++i)
    if (subs[i].geom.hw < 3 || subs[i].geom.hw > 5) return cudaErrorInvalidValue;
  switch (set) {
    case 0: return launch_batch_set<0>(subs, n, plan, partial, dev_scratch, err, stream, setup);
    case 1: return launch_batch_set<1>(subs, n, plan, partial, dev_scratch, err, stream, setup);
    case 2: return launch_batch_set<2>(subs, n, plan, partial, dev_scratch, err, stream, setup);
    case 3: return launch_batch_set<3>(subs, n, plan, partial, dev_scratch, err, stream, setup);
    case 4: return launch_batch_set<4>(subs, n, plan, partial, dev_scratch, err, stream, setup);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_prepared_batch(const BatchSetup &setup, cudaStream_t stream) {
  if (!setup.params_ready) return cudaErrorInvalidValue;
  if (setup.items == 0) return cudaSuccess;
  BatchParams bp{static_cast<const SubjectView *>(setup.bp_subjects), setup.bp_nsub, setup.items,
                 setup.bp_err, setup.bp_err + 1, 2000000000ull};
  cudaError_t e;
  switch (setup.set) {
    case 0: e = launch_batch_items<0>(bp, setup.blocks, stream); break;
    case 1: e = launch_batch_items<1>(bp, setup.blocks, stream); break;
    case 2: e = launch_batch_items<2>(bp, setup.blocks, stream); break;
    case 3: e = launch_batch_items<3>(bp, setup.blocks, stream); break;
    case 4: e = launch_batch_items<4>(bp, setup.blocks, stream); break;
    default: return cudaErrorInvalidValue;
  }
  if (e != cudaSuccess || !setup.combine) return e;
  combine_batch_kernel<<<dim3(sm_count() * 2, std::min(setup.bp_nsub, 65535)), 256, 0, stream>>>(
      bp.subjects, setup.bp_nsub);
  return cudaGetLastError();
}

bool make_offset_runs(const std::vector<std::array<int, 3>> &offsets, OffsetRuns *runs) {
  int reach = 0;
  for (const auto &o : offsets)
    reach = std::max(reach, std::max(std::abs(o[0]), std::max(std::abs(o[1]), std::abs(o[2]))));
  if (reach < 1 || reach > kMaxRunReach) return false;
  *runs = OffsetRuns{};
  runs->reach = reach;
  runs->count = (int)offsets.size();
  const int ns = 2 * reach + 1;
  std::vector<char> has((size_t)ns * ns * ns, 0);
  for (const auto &o : offsets) {
    char &h = has[((size_t)(o[1] + reach) * ns + o[2] + reach) * ns + o[0] + reach];
    if (h) return false;
    h = 1;
  }
  for (int u = 0; u < ns; ++u)
    for (int v = 0; v < ns; ++v) {
      const char *h = &has[((size_t)u * ns + v) * ns];
      int first = ns, last = -1, n = 0;
      for (int w = 0; w < ns; ++w)
        if (h[w]) {
          first = std::min(first, w);
          last = w;
          ++n;
        }
      if (n && last - first + 1 != n) return false;  // not one run of dw
      runs->w0[u][v] = (unsigned char)(n ? first : 0);
      runs->len[u][v] = (unsigned char)n;
    }
  return true;
}

namespace {
template <int SET, int HW>
cudaError_t launch_runs_hw(const Geometry &g, const SlabInputs &in, float *out, double div,
                           float *partial, int *err, const FusePlan &pl, const OffsetRuns &runs,
                           unsigned long long *stats, unsigned long long evaluated,
                           cudaStream_t stream) {
  using T = TileOf<SET, HW>;
  using C = Cfg<HW, T::RX, T::TZ, true>;
  if (pl.groups > 1 && !partial) return cudaErrorInvalidValue;
  cudaError_t e;
  CUtensorMap tmA, tmL;
  if ((e = make_slab_map(&tmA, in.atlas, g.nx, g.ny, g.nz, g.num, in.pitch, C::YB, C::ZA)) !=
          cudaSuccess ||
      (e = make_slab_map(&tmL, in.label, g.nx, g.ny, g.nz, g.num, in.pitch, C::YB, C::ZL)) !=
          cudaSuccess)
    return e;
  TmaParams p{};
  p.sv = subject_view(g, in, out, div, partial, pl);
  p.err = err;
  p.timeout_ns = 2000000000ull;
  p.withhold_cta = -1;
  p.item_end = pl.groups * pl.tiles;
  if ((e = launch_runs(runs, pl.ctas, tmA, tmL, p, stats, evaluated, stream)) != cudaSuccess) return e;
  return pl.groups > 1 ? launch_combine_groups(g, partial, pl.groups, out, stream) : cudaSuccess;
}
}  // namespace

cudaError_t fuse_runs_plan(const Geometry &g, const OffsetRuns &runs, size_t partial_limit,
                           FusePlan *plan) {
  *plan = FusePlan{};
  const int ns = 2 * runs.reach + 1;
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaErrorInvalidValue;
  // the tile's cost for a whole window of this reach, by the list's share of it; the runs are
  // shorter, so that the first planes of each weigh more
  const double cost = 1.2 * kTileCost[runs.reach - 1][2] * runs.count / ((double)ns * ns * ns);
  const int sms = sm_count();
  switch (runs.reach) {
    case 1: plan_hw<6, 1>(g, sms, cost, partial_limit, plan, false); break;
    case 2: plan_hw<6, 2>(g, sms, cost, partial_limit, plan, false); break;
    default: plan_hw<6, 3>(g, sms, cost, partial_limit, plan, false); break;
  }
  return cudaSuccess;
}

cudaError_t launch_fuse_runs(const Geometry &g, const SlabInputs &in, float *out, double div,
                             float *partial, int *err, const FusePlan &pl, const OffsetRuns &runs,
                             unsigned long long *stats, unsigned long long evaluated,
                             cudaStream_t s) {
  switch (runs.reach) {
    case 1: return launch_runs_hw<6, 1>(g, in, out, div, partial, err, pl, runs, stats, evaluated, s);
    case 2: return launch_runs_hw<6, 2>(g, in, out, div, partial, err, pl, runs, stats, evaluated, s);
    case 3: return launch_runs_hw<6, 3>(g, in, out, div, partial, err, pl, runs, stats, evaluated, s);
    default: return cudaErrorInvalidValue;
  }
}

TileShape fuse_tile_shape(const Geometry &g) {
  using T = TileOf<0, 5>;
  TileShape t{};
  t.out_y = kOutY;
  t.xc = kWarps * T::RX;
  t.zt = 2 * T::TZ;
  if (g.ix > 0 && g.iy > 0 && g.iz > 0) {
    t.tiles_y = (g.iy + kOutY - 1) / kOutY;
    t.tiles_x = (g.ix + t.xc - 1) / t.xc;
    t.tiles_z = (g.iz + t.zt - 1) / t.zt;
  }
  return t;
}

namespace {

// One masked item per pair of flagged atlases of every tile with a non-empty mask (any order:
// each item writes its own partial slot).
__global__ void masked_items_kernel(const uint32_t *__restrict__ masks, int ntiles,
                                    int *__restrict__ items, int *__restrict__ count) {
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntiles; t += gridDim.x * blockDim.x) {
    const uint32_t m = masks[t];
    if (!m) continue;
    const int pairs = (__popc(m) + 1) / 2;
    const int at = atomicAdd(count, pairs);
    for (int k = 0; k < pairs; ++k) items[at + k] = (k << 24) | t;
  }
}

// Adds the pair slots of every interior voxel of a masked tile into acc_p / acc_w, in pair order.
__global__ void masked_combine_kernel(const uint32_t *__restrict__ masks, const TileShape ts,
                                      int nx, int ny, int nz, int lo, long long nvox,
                                      const float *__restrict__ partial, float *__restrict__ acc_p,
                                      float *__restrict__ acc_w) {
  const int ix = nx - 2 * lo, iy = ny - 2 * lo, iz = nz - 2 * lo;
  const long long total = (long long)ix * iy * iz;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const int yi = (int)(i % iy);
    const long long r = i / iy;
    const int xi = (int)(r % ix), zi = (int)(r / ix);
    const int t = ((zi / ts.zt) * ts.tiles_x + xi / ts.xc) * ts.tiles_y + yi / ts.out_y;
    const uint32_t m = masks[t];
    if (!m) continue;
    const long long v = (long long)(zi + lo) * nx * ny + (long long)(xi + lo) * ny + (yi + lo);
    float p = acc_p[v], w = acc_w[v];
    for (int k = 0; k < (__popc(m) + 1) / 2; ++k) {
      p += partial[(2LL * k) * nvox + v];
      w += partial[(2LL * k + 1) * nvox + v];
    }
    acc_p[v] = p;
    acc_w[v] = w;
  }
}

}  // namespace

cudaError_t launch_fuse_masked(const Geometry &g, const SlabInputs &in, double div, int atlas_base,
                               const uint32_t *masks, int *items, int *count, float *partial,
                               float *acc_p, float *acc_w, int *err, cudaStream_t stream) {
  if (g.hw != 5 || atlas_base < 0 || atlas_base >= g.num) return cudaErrorInvalidValue;
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaSuccess;
  using T = TileOf<0, 5>;
  using C = Cfg<5, T::RX, T::TZ>;
  cudaError_t e;
  CUtensorMap tmA, tmL;
  if ((e = make_slab_map(&tmA, in.atlas, g.nx, g.ny, g.nz, g.num, in.pitch, C::YB, C::ZA)) !=
      cudaSuccess)
    return e;
  if ((e = make_slab_map(&tmL, in.label, g.nx, g.ny, g.nz, g.num, in.pitch, C::YB, C::ZL)) !=
      cudaSuccess)
    return e;
  const TileShape ts = fuse_tile_shape(g);
  const int ntiles = ts.tiles_y * ts.tiles_x * ts.tiles_z;
  if (ntiles >= (1 << 24)) return cudaErrorInvalidValue;  // items pack the tile in 24 bits
  if ((e = cudaMemsetAsync(count, 0, sizeof(int), stream)) != cudaSuccess) return e;
  masked_items_kernel<<<(ntiles + 255) / 256, 256, 0, stream>>>(masks, ntiles, items, count);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  FusePlan pl{};
  pl.tiles_y = ts.tiles_y;
  pl.tiles_x = ts.tiles_x;
  pl.tiles_z = ts.tiles_z;
  pl.tiles = ntiles;
  pl.groups = 2;  // partial slots (the pair of each item), not a plan's atlas groups
  pl.atlas_groups = pl.splits = 1;
  TmaParams p{};
  p.sv = subject_view(g, in, nullptr, div, partial, pl);
  p.sv.atlas_base = atlas_base;
  p.sv.atlas_mask = masks;
  p.err = err;
  p.timeout_ns = 2000000000ull;
  p.withhold_cta = -1;
  if ((e = launch_list(sm_count(), tmA, tmL, p, items, count, stream)) != cudaSuccess) return e;
  masked_combine_kernel<<<sm_count() * 8, 256, 0, stream>>>(masks, ts, g.nx, g.ny, g.nz, g.lo,
                                                            g.nvox(), partial, acc_p, acc_w);
  return cudaGetLastError();
}

cudaError_t fuse_tma_plan(const Geometry &g, int set, size_t partial_limit, FusePlan *plan) {
  *plan = FusePlan{};
  if (g.hw < 1 || g.hw > 5 || set < 0 || set >= kTileSets) return cudaErrorInvalidValue;
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaSuccess;
  const int sms = sm_count();
  if (set != 0) {
    plan_internal(g, set, sms, kTileCost[g.hw - 1][0], partial_limit, plan);
    return cudaSuccess;
  }
  double best = -1.0;
  for (int k = 0; k < 4; ++k) {
    FusePlan p{};
    const double t =
        plan_internal(g, kTileChoices[k], sms, kTileCost[g.hw - 1][k], partial_limit, &p);
    if (best >= 0.0 && t >= best) continue;
    best = t;
    *plan = p;
  }
  return cudaSuccess;
}

int fuse_tma_planes_read(const Geometry &g, const FusePlan &info, int ztiles) {
  // z-tile tz reads the atlas MRI slab [2 tz TZ, 2 tz TZ + 2 TZ + 2 + 2 HW) (its first output
  // plane minus the box and window reach), the CT slab and the input taps lie inside it
  const long long n = (long long)ztiles * 2 * info.tz + 2 + 2 * g.hw;
  return ztiles <= 0 ? 0 : (int)(n < g.nz ? n : g.nz);
}

cudaError_t launch_fuse_tma(const Geometry &g, const SlabInputs &in, float *out, double div,
                            float *partial, int *err, const LaunchHooks &wt, const FusePlan &plan,
                            cudaStream_t stream) {
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaSuccess;
  return launch_any(g, in, out, div, partial, err, wt, plan, -1, -1, stream);
}

cudaError_t launch_fuse_tma_items(const Geometry &g, const SlabInputs &in, float *out, double div,
                                  float *partial, int *err, const FusePlan &plan, int item_begin,
                                  int item_end, cudaStream_t stream) {
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaSuccess;
  if (item_begin < 0) return cudaErrorInvalidValue;
  const LaunchHooks wt{0, nullptr, nullptr};
  return launch_any(g, in, out, div, partial, err, wt, plan, item_begin, item_end, stream);
}

cudaError_t launch_fuse_tma_combine(const Geometry &g, const float *partial, const FusePlan &plan,
                                    float *out, int z_begin, int z_end, cudaStream_t stream) {
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaSuccess;
  if (plan.groups < 2) return cudaErrorInvalidValue;
  return launch_combine_groups(g, partial, plan.groups, out, z_begin, z_end, stream);
}

namespace {
// One warp per row (grid-stride over rows), so that no element index is divided by the row
// length; PAIRS copies 8-byte pairs (even ny and 8-byte aligned sources; the destinations' pitch
// is a multiple of 4 floats). Rows past `rows` are the second stack's: one launch for both (two cost
// 4 us more of a call at 97x85x53, 3 atlases, NH 5: 106.6 us, 102.4 in one, timed in turn).
template <bool PAIRS>
__global__ void pitch_copy_kernel(const float *__restrict__ src0, float *__restrict__ dst0,
                                  const float *__restrict__ src1, float *__restrict__ dst1,
                                  long long rows, int stacks, int ny, int pitch) {
  const int lane = threadIdx.x & 31;
  const long long nwarps = ((long long)gridDim.x * blockDim.x) >> 5;
  for (long long i = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < rows * stacks;
       i += nwarps) {
    const bool second = i >= rows;
    const long long r = second ? i - rows : i;
    const float *s = (second ? src1 : src0) + r * ny;
    float *d = (second ? dst1 : dst0) + r * pitch;
    if constexpr (PAIRS) {
      const float2 *s2 = reinterpret_cast<const float2 *>(s);
      float2 *d2 = reinterpret_cast<float2 *>(d);
#pragma unroll 4
      for (int c = lane; c < ny / 2; c += 32) d2[c] = s2[c];
    } else {
#pragma unroll 4
      for (int c = lane; c < ny; c += 32) d[c] = s[c];
    }
  }
}

cudaError_t launch_pitch(const float *src0, float *dst0, const float *src1, float *dst1,
                         long long rows, int stacks, int ny, int pitch, cudaStream_t stream) {
  if (rows <= 0) return cudaSuccess;
  const int sms = sm_count();
  auto at = [](const void *p, unsigned n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
  const bool pairs = ny % 2 == 0 && pitch % 4 == 0 && at(src0, 8) && at(dst0, 16) &&
                     (stacks == 1 || (at(src1, 8) && at(dst1, 16)));
  auto kern = pairs ? pitch_copy_kernel<true> : pitch_copy_kernel<false>;
  kern<<<sms * 8, 256, 0, stream>>>(src0, dst0, src1, dst1, rows, stacks, ny, pitch);
  return cudaGetLastError();
}
}  // namespace

cudaError_t launch_pitch_copy(const float *src, float *dst, long long rows, int ny, int pitch,
                              cudaStream_t stream) {
  return launch_pitch(src, dst, nullptr, nullptr, rows, 1, ny, pitch, stream);
}

cudaError_t launch_pitch_copy_pair(const float *src0, float *dst0, const float *src1, float *dst1,
                                   long long rows, int ny, int pitch, cudaStream_t stream) {
  return launch_pitch(src0, dst0, src1, dst1, rows, 2, ny, pitch, stream);
}

}  // namespace pct
