// Plain FP32 patch-based multi-atlas fusion for sm_100a, atlas slabs staged by TMA.
//
// Same arithmetic contract as the reference (MultiAtlasPatchBasedSegmentationOpenMP +
// PatchSimilarity, NewPatchedBrainPureC.cpp:1184-1212,1350-1449), in FP32:
//     SSD(x,d) = sum_{p in 3x3x3} (I(x+p) - A_a(x+d+p))^2,   w = exp(-SSD/div)
//     out(x)   = sum_{a,d} w*L_a(x+d) / sum_{a,d} w            (NaN rule of :1325-1331)
//
// Work decomposition
//  * A warp owns 30 (y) x RX (x) x 2*TZ (z) output voxels. Lanes run along the contiguous y
//    axis (lanes 1..30 own outputs, lanes 0/31 carry the y-halo). For one offset d the SSD of
//    all voxels is a 3x3x3 box sum of D_d = (I - A_d)^2: each lane box-sums its RX+2 rows x
//    TZ+2 planes in registers along x and z, and the y-box is two warp shuffles.
//  * The thread's two z-halves are packed into float2 and run on the paired FP32 instructions
//    (add/mul/fma .f32x2): same lane throughput as scalar FP32, half the issue slots.
//  * dw is the innermost offset loop: stepping dw shifts the atlas planes by one, so the atlas
//    window (TZ+2 planes x RX+2 rows per half) lives in registers as a ring and each step reads
//    one new plane. The step loop is unrolled one ring period at a time (not the whole window)
//    to keep the kernel inside the instruction cache.
//  * A CTA is 4 warps stacked along x. Its atlas MRI and atlas CT rows (one x-row = a z x y
//    slab) sit in two shared-memory rings indexed by x. Each du step needs one new row of each;
//    one thread issues it with cp.async.bulk.tensor (TMA, no multicast) one step ahead, and the
//    step's readers wait on an mbarrier (transaction-count completion, ping-pong pair). Every
//    per-thread shared-memory read is one LDS with an immediate offset.
//  * TMA zero-fills coordinates outside the volume, so tiles need no clamping: out-of-volume
//    rows/planes/lanes only ever feed voxels outside the interior, which are never stored.
//  * CTAs are persistent over the tile list.
//  * Every mbarrier wait is bounded (globaltimer); on timeout the CTA records an error code,
//    stops at the next CTA barrier, drains its own in-flight copies (bounded) and returns.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "pct_internal.h"
#include "pct_ptx.cuh"

namespace pct {
namespace {

using namespace ptx;

constexpr int kOutY = 30;
constexpr int kWarps = 4;
constexpr int kThreads = kWarps * 32;
constexpr float kDblEpsilonF = 2.220446049250313080847e-16f;

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 mul2(float2 a, float2 b) { return __fmul2_rn(a, b); }
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }

__device__ __forceinline__ float fuse_result(float product, float sum_weight) {
  return (fabsf(product) > kDblEpsilonF && fabsf(sum_weight) > kDblEpsilonF)
             ? __fdiv_rn(product, sum_weight)
             : __int_as_float(0x7fc00000);
}

// ---------------------------------------------------------------- geometry of one variant

// LIST: an offset list of reach HW in a volume of any half window, so that a tile's slab may start at
// any y modulo 4 (the plain kernel's start at 30 ty: 0 or 2).
template <int HW, int RX, int TZ, bool LIST = false>
struct Cfg {
  static constexpr int NQ = TZ + 2;          // D planes per half
  static constexpr int NR = RX + 2;          // D rows per warp
  static constexpr int NS = 2 * HW + 1;      // offsets per axis
  static constexpr int XC = kWarps * RX;     // output rows per CTA
  // y extent of a slab row: lanes span 32 positions, +-HW for dv, +2 for the 16-byte
  // alignment of the TMA start coordinate (tile starts are 30*ty, i.e. 0 or 2 mod 4).
  static constexpr int YB = ((LIST ? 35 : 34) + 2 * HW + 3) / 4 * 4;
  static constexpr int ZA = 2 * TZ + 2 + 2 * HW;  // atlas MRI planes per slab row
  static constexpr int ZL = 2 * TZ + 2 * HW;      // atlas CT planes per slab row
  static constexpr int RA = XC + 3;               // MRI ring: XC+2 rows in use + 1 prefetch
  static constexpr int RL = XC + 1;               // CT ring: XC rows in use + 1 prefetch
  static constexpr uint32_t ROW_A = ZA * YB * 4;  // TMA transaction bytes per row
  static constexpr uint32_t ROW_L = ZL * YB * 4;
  static constexpr uint32_t SLOT_A = (ROW_A + 127) / 128 * 128;
  static constexpr uint32_t SLOT_L = (ROW_L + 127) / 128 * 128;
  static constexpr uint32_t PLANE = YB * 4;       // bytes between planes of a slab row
  static constexpr int SMEM = 128 + 128 + RA * SLOT_A + RL * SLOT_L;  // + alignment slack
  // LIST: the threads' sums of whole atlases, behind the rings
  static constexpr int SUMS = LIST ? kThreads * 4 * RX * TZ * (int)sizeof(float) : 0;
  static constexpr int NCH = (NS + NQ - 1) / NQ;  // ring periods per dw sweep
  static constexpr int OFF = NCH * NQ - NS;       // virtual steps skipped in the first period
};

// One subject as the kernels see it.
struct SubjectView {
  const float *img;   // input MRI, reference layout
  float *out;         // fused output, reference layout (interior written)
  float *partial;     // groups > 1: [groups][2][nvox] partial (product, sum_weight) sums
  const CUtensorMap *tmA, *tmL;  // atlas MRI / CT slab maps (param or global space)
  int nx, ny, nz, nxy;
  long long nvox;
  float scale;        // sqrt(log2(e)/div): taps are scaled so that the box sum is SSD*log2(e)/div
  int tiles_y, tiles_x, ntiles;
  int groups, atlases_per_group;  // items = groups * ntiles (group-major)
  int splits;         // groups per atlas group: each takes a range of the window's x offsets
  int hw, lo;         // half window of this subject (batched kernel dispatch), first interior index
  int item_begin;     // first global item of this subject (batched kernel)
  int atlas_base;     // first atlas of group 0 (a single-atlas launch over a tile list)
  float *acc_p, *acc_w;  // non-null: add each voxel's (product, sum_weight) into these instead
  // non-null (masked items): item = pair << 24 | tile, over the atlases atlas_base + i for the
  // set bits i of atlas_mask[tile], two per pair in bit order; pair k's sums go to partial slot k
  const uint32_t *atlas_mask;
};

struct TmaParams {
  SubjectView sv;
  int item_begin, item_end;  // the work items this launch covers (group-major numbering)
  int *err;           // device status word (0 = ok)
  unsigned long long timeout_ns;
  int withhold_cta;   // testing hook: this CTA withholds its first copies (-1 = none)
};

// One dw sweep (all dw for fixed atlas, du, dv) of the thread's voxels.
template <int HW, int RX, int TZ>
__device__ __forceinline__ void sweep_dw(const float2 (&In)[TZ + 2][RX + 2], float2 (&P)[TZ][RX],
                                         float2 (&W)[TZ][RX], const uint32_t (&rowA)[RX + 2],
                                         const uint32_t (&rowL)[RX], const float2 scale2) {
  using C = Cfg<HW, RX, TZ>;
  constexpr int NQ = C::NQ, NR = C::NR;
  float2 Aw[NQ][NR];  // logical plane q at virtual step v lives in slot (q + v) % NQ
#pragma unroll
  for (int q = 0; q < NQ - 1; ++q)
#pragma unroll
    for (int r = 0; r < NR; ++r)
      Aw[(q + C::OFF) % NQ][r] = make_float2(lds_f32(rowA[r] + q * C::PLANE),
                                             lds_f32(rowA[r] + (TZ + q) * C::PLANE));
#pragma unroll 1
  for (int c = 0; c < C::NCH; ++c) {
#pragma unroll
    for (int jj = 0; jj < NQ; ++jj) {
      if (jj < C::OFF && c == 0) continue;
      const uint32_t so = (uint32_t)(c * NQ + jj - C::OFF) * C::PLANE;  // real step s = dw + HW
      {
        constexpr int qn = NQ - 1;
        const int sn = (qn + jj) % NQ;
#pragma unroll
        for (int r = 0; r < NR; ++r)
          Aw[sn][r] = make_float2(lds_f32(rowA[r] + so + qn * C::PLANE),
                                  lds_f32(rowA[r] + so + (TZ + qn) * C::PLANE));
      }
      // x-box of D = s^2 (A - I)^2 per plane
      float2 g[NQ][RX];
#pragma unroll
      for (int q = 0; q < NQ; ++q) {
        const int sq = (q + jj) % NQ;
        float2 D[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
          const float2 d = fma2(Aw[sq][r], scale2, In[q][r]);  // s * (A - I)
          D[r] = mul2(d, d);
        }
#pragma unroll
        for (int x = 0; x < RX; x += 2) {
          if (x + 1 < RX) {
            const float2 mid = add2(D[x + 1], D[x + 2]);
            g[q][x] = add2(D[x], mid);
            g[q][x + 1] = add2(mid, D[x + 3]);
          } else {
            g[q][x] = add2(add2(D[x], D[x + 1]), D[x + 2]);
          }
        }
      }
      // z-box, y-box (warp shuffles), weight, accumulate
#pragma unroll
      for (int x = 0; x < RX; ++x) {
#pragma unroll
        for (int q = 0; q < TZ; q += 2) {
          float2 S[2];
          if (q + 1 < TZ) {
            const float2 mid = add2(g[q + 1][x], g[q + 2][x]);
            S[0] = add2(g[q][x], mid);
            S[1] = add2(mid, g[q + 3][x]);
          } else {
            S[0] = add2(add2(g[q][x], g[q + 1][x]), g[q + 2][x]);
          }
#pragma unroll
          for (int k = 0; k < 2; ++k) {
            if (q + k >= TZ) break;
            const float2 cc = S[k];
            const float2 lft = make_float2(__shfl_up_sync(0xffffffffu, cc.x, 1),
                                           __shfl_up_sync(0xffffffffu, cc.y, 1));
            const float2 rgt = make_float2(__shfl_down_sync(0xffffffffu, cc.x, 1),
                                           __shfl_down_sync(0xffffffffu, cc.y, 1));
            const float2 e = add2(add2(cc, lft), rgt);  // SSD * log2(e) / div
            const float2 w = make_float2(ex2_approx(-e.x), ex2_approx(-e.y));
            const float2 lab = make_float2(lds_f32(rowL[x] + so + (q + k) * C::PLANE),
                                           lds_f32(rowL[x] + so + (TZ + q + k) * C::PLANE));
            P[q + k][x] = fma2(w, lab, P[q + k][x]);
            W[q + k][x] = add2(W[q + k][x], w);
          }
        }
      }
    }
  }
}

// ------------------------------------------------------------- y-pair layout (LY = 1)
//
// Same warp tile (30 y x RX x x 2*TZ z) and the same shared-memory slabs as above, mapped
// differently: half-warp h = lane / 16 owns the z planes [z0 + h*TZ, z0 + h*TZ + TZ), and lane
// j = lane % 16 owns the two adjacent y positions (y0 - 1 + 2j, y0 + 2j), packed in a float2.
//  * y-box: each output needs one neighbour value from each side (the left lane's .y, the right
//    lane's .x): 2 shuffles per voxel pair instead of 4.
//  * x-box: the squares are folded into the first additions as FMAs
//    (g = d0*d0 + (d1*d1 + d2*d2) with the inner pair shared by two outputs), 6 instructions per
//    plane of 3 outputs instead of 5 multiplies + 5 adds.
//    The three additions are m = S.x + S.y and one packed (m, m) + (left, right): what bounds the
//    loop is the issue of operands, and a packed instruction with at most two distinct operand
//    pairs costs the same two cycles as two scalar ones but loads the two halves of the FMA pipe
//    equally (scalar additions pile up on one half: 72.6 % against 61.8 % busy). With the shared
//    loads visible to the compiler and the warp index known to be uniform, NH 11 at 222x222x112,
//    10 atlases takes 28.4 ms (29.2 ms before; 1965 MHz).
//  * labels ride a register ring like the atlas planes: one new plane per dw step.
//  * a pair's shared-memory address is 8-byte aligned for every other dv (the parity of
//    dv + HW): those sweeps load pairs with one 64-bit LDS, the others with two 32-bit LDS.

// (plain loads, not volatile asm: the compiler may then move them across the arithmetic)
__device__ __forceinline__ float shared_f32(uint32_t addr) {
  return *static_cast<const float *>(__cvta_shared_to_generic(addr));
}

template <bool AL>
__device__ __forceinline__ float2 lds_pair(uint32_t addr) {
  if constexpr (AL) {
    return *static_cast<const float2 *>(__cvta_shared_to_generic(addr));
  } else {
    return make_float2(shared_f32(addr), shared_f32(addr + 4));
  }
}

// g[x] = d[x]^2 + d[x+1]^2 + d[x+2]^2 for x < RX, two outputs at a time sharing d[x+1]^2 + d[x+2]^2.
template <int RX>
__device__ __forceinline__ void xbox_squares(const float2 (&d)[RX + 2], float2 (&g)[RX]) {
  float2 u = make_float2(0.f, 0.f);
#pragma unroll
  for (int x = 0; x < RX; x += 2) {
    if (x + 1 < RX) {
      u = mul2(d[x + 2], d[x + 2]);
      const float2 m = fma2(d[x + 1], d[x + 1], u);
      g[x] = fma2(d[x], d[x], m);
      g[x + 1] = fma2(d[x + 3], d[x + 3], m);
    } else if (x >= 2) {  // odd RX: u holds d[x]^2 from the previous pair
      g[x] = fma2(d[x + 2], d[x + 2], fma2(d[x + 1], d[x + 1], u));
    } else {
      g[x] = fma2(d[x], d[x], fma2(d[x + 1], d[x + 1], mul2(d[x + 2], d[x + 2])));
    }
  }
}

// One offset of the lane's voxels, y-pair layout: step jj of a ring period (compile-time), slab
// plane offset so. Atlas plane t (= step + D plane) and label plane t (= step + output plane) live
// in ring slot (jj + plane) % NQ.
template <int HW, int RX, int TZ, bool AL, bool LR, bool LIST = false>
__device__ __forceinline__ void step_yp(const float2 (&In)[TZ + 2][RX + 2], float2 (&P)[TZ][RX],
                                        float2 (&W)[TZ][RX], float2 (&Aw)[TZ + 2][RX + 2],
                                        float2 (&Lw)[TZ + 2][RX],
                                        const uint32_t (&rowA)[RX + 2], const uint32_t (&rowL)[RX],
                                        const uint32_t so, const int jj, const float2 scale2) {
  using C = Cfg<HW, RX, TZ, LIST>;
  constexpr int NQ = C::NQ, NR = C::NR;
        {
          const int sa = (jj + NQ - 1) % NQ;
  #pragma unroll
          for (int r = 0; r < NR; ++r)
            Aw[sa][r] = lds_pair<AL>(rowA[r] + so + (NQ - 1) * C::PLANE);
          if constexpr (LR) {
            const int sl = (jj + TZ - 1) % NQ;
  #pragma unroll
            for (int r = 0; r < RX; ++r)
              Lw[sl][r] = lds_pair<AL>(rowL[r] + so + (TZ - 1) * C::PLANE);
          }
        }
        // Output planes two at a time: the x-box of D = (s A - s I)^2 for the planes they need
        // (computed once, as late as possible, to keep few x-box sums live), then the z-box, the
        // y-box (half-warp shuffles), the weight and the accumulators.
        float2 g[NQ][RX];
  #pragma unroll
        for (int q = 0; q < TZ; q += 2) {
  #pragma unroll
          for (int pq = (q == 0 ? 0 : q + 2); pq < (q + 4 < NQ ? q + 4 : NQ); ++pq) {
            const int sq = (pq + jj) % NQ;
            float2 d[NR];
  #pragma unroll
            for (int r = 0; r < NR; ++r) d[r] = fma2(Aw[sq][r], scale2, In[pq][r]);  // s * (A - I)
            xbox_squares<RX>(d, g[pq]);
          }
  #pragma unroll
          for (int x = 0; x < RX; ++x) {
            float2 S[2];
            if (q + 1 < TZ) {
              const float2 mid = add2(g[q + 1][x], g[q + 2][x]);
              S[0] = add2(g[q][x], mid);
              S[1] = add2(mid, g[q + 3][x]);
            } else {
              S[0] = add2(add2(g[q][x], g[q + 1][x]), g[q + 2][x]);
            }
  #pragma unroll
            for (int k = 0; k < 2; ++k) {
              if (q + k >= TZ) break;
              const float2 cc = S[k];
              const float lft = __shfl_up_sync(0xffffffffu, cc.y, 1, 16);
              const float rgt = __shfl_down_sync(0xffffffffu, cc.x, 1, 16);
              const float m = cc.x + cc.y;
              const float2 e = add2(make_float2(m, m), make_float2(lft, rgt));
              const float2 w = make_float2(ex2_approx(-e.x), ex2_approx(-e.y));
              const float2 lab = LR ? Lw[(q + k + jj) % NQ][x]
                                    : lds_pair<AL>(rowL[x] + so + (q + k) * C::PLANE);
              P[q + k][x] = fma2(w, lab, P[q + k][x]);
              W[q + k][x] = add2(W[q + k][x], w);
            }
          }
        }
}

// One dw sweep (all dw for fixed atlas, du, dv) of the lane's voxels, y-pair layout.
// rowA[r] / rowL[r]: the lane's pair in plane 0 of its half's slab rows, at this dv.
template <int HW, int RX, int TZ, bool AL, bool LR>
__device__ __forceinline__ void sweep_dw_yp(const float2 (&In)[TZ + 2][RX + 2],
                                            float2 (&P)[TZ][RX], float2 (&W)[TZ][RX],
                                            const uint32_t (&rowA)[RX + 2],
                                            const uint32_t (&rowL)[RX], const float2 scale2) {
  using C = Cfg<HW, RX, TZ>;
  constexpr int NQ = C::NQ, NR = C::NR;
  // (plane t lives in slot (t + OFF) % NQ: virtual step v = c*NQ + jj, slot (jj + plane) % NQ)
  float2 Aw[NQ][NR];
  float2 Lw[NQ][RX];
#pragma unroll
  for (int t = 0; t < NQ - 1; ++t)
#pragma unroll
    for (int r = 0; r < NR; ++r) Aw[(t + C::OFF) % NQ][r] = lds_pair<AL>(rowA[r] + t * C::PLANE);
  if constexpr (LR) {
#pragma unroll
    for (int t = 0; t < TZ - 1; ++t)
#pragma unroll
      for (int r = 0; r < RX; ++r)
        Lw[(t + C::OFF) % NQ][r] = lds_pair<AL>(rowL[r] + t * C::PLANE);
  }
#pragma unroll 1
  for (int c = 0; c < C::NCH; ++c) {
#pragma unroll
    for (int jj = 0; jj < NQ; ++jj) {
      if (jj < C::OFF && c == 0) continue;
      const uint32_t so = (uint32_t)(c * NQ + jj - C::OFF) * C::PLANE;  // real step s = dw + HW
      step_yp<HW, RX, TZ, AL, LR>(In, P, W, Aw, Lw, rowA, rowL, so, jj, scale2);
    }
  }
}

// The same sweep over the `len` planes from w0 on only (an offset list's run of dw for one du, dv).
template <int HW, int RX, int TZ, bool AL>
__device__ __forceinline__ void sweep_run_yp(const float2 (&In)[TZ + 2][RX + 2],
                                             float2 (&P)[TZ][RX], float2 (&W)[TZ][RX],
                                             const uint32_t (&rowA)[RX + 2],
                                             const uint32_t (&rowL)[RX], const int len,
                                             const float2 scale2) {
  using C = Cfg<HW, RX, TZ, true>;
  constexpr int NQ = C::NQ, NR = C::NR;
  float2 Aw[NQ][NR];
  float2 Lw[NQ][RX];
#pragma unroll
  for (int t = 0; t < NQ - 1; ++t)
#pragma unroll
    for (int r = 0; r < NR; ++r) Aw[t][r] = lds_pair<AL>(rowA[r] + t * C::PLANE);
#pragma unroll 1
  for (int c = 0; c < len; c += NQ) {
#pragma unroll
    for (int jj = 0; jj < NQ; ++jj) {
      if (jj > 0 && c + jj >= len) return;
      const uint32_t so = (uint32_t)(c + jj) * C::PLANE;
      step_yp<HW, RX, TZ, AL, false, true>(In, P, W, Aw, Lw, rowA, rowL, so, jj, scale2);
    }
  }
}

// Pipeline state of one CTA, carried across its work items.
struct Pipe {
  uint32_t base;              // 128-byte aligned start of the dynamic shared memory
  uint32_t gstep;             // steps taken: barrier gstep&1, phase (gstep>>1)&1
  bool armed_next;            // thread 0: a prefetch is in flight on barrier (gstep+1)&1
  volatile int *abort_flag;
};

// Processes work item `item` (tile x atlas group) of subject `sv` with register tile (RX, TZ) in
// layout LY (0: z-halves packed; 1: y-pairs, labels read per use; 2: y-pairs, labels in a
// register ring). Returns false when a bounded wait gave up (the CTA must stop).
// With `runs` (y-pairs, labels read per use) an item evaluates that offset list instead of the whole
// window, and HW is the reach of the list rather than the volume's half window.
template <int HW, int RX, int TZ, int LY, bool MASKED = false, bool LIST = false>
__device__ __forceinline__ bool run_item(const SubjectView &sv, int item, Pipe &pp, int *err,
                                         unsigned long long timeout_ns, int withhold_cta,
                                         const OffsetRuns *runs = nullptr) {
  using C = Cfg<HW, RX, TZ, LIST>;
  constexpr int NQ = C::NQ, NR = C::NR, NS = C::NS;
  const uint32_t bar0 = pp.base, bar1 = pp.base + 8;
  const uint32_t ringA = pp.base + 128;
  const uint32_t ringL = ringA + C::RA * C::SLOT_A;
  // (the shuffle tells the compiler that the warp index, and every ring address made from it, is
  // uniform over the warp)
  const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int lo = LIST ? sv.lo : HW + 1;
  const float2 scale2 = make_float2(sv.scale, sv.scale);
  int grp, t, a_first, natl;
  int j0 = 0, nj = NS;  // the item's x offsets du = j - HW, j in [j0, j0 + nj)
  uint32_t later = 0;  // masked items: the pair's atlases after the current one (bits)
  if constexpr (MASKED) {
    grp = (int)((uint32_t)item >> 24);
    t = item & 0xffffff;
    uint32_t m = sv.atlas_mask[t];
    for (int k = 0; k < 2 * grp; ++k) m &= m - 1;  // drop the earlier pairs' atlases
    natl = min(2, __popc(m));
    a_first = sv.atlas_base + __ffs(m) - 1;
    later = m & (m - 1);
  } else {
    grp = item / sv.ntiles;
    t = item - grp * sv.ntiles;
    const int ag = grp / sv.splits, part = grp - ag * sv.splits;
    a_first = sv.atlas_base + ag * sv.atlases_per_group;
    natl = sv.atlases_per_group;
    j0 = part * NS / sv.splits;
    nj = (part + 1) * NS / sv.splits - j0;
  }
  const int T = natl * nj;  // du steps per item (atlas-major)
  const int ty = t % sv.tiles_y;
  t /= sv.tiles_y;
  const int txc = t % sv.tiles_x;
  const int tz = t / sv.tiles_x;
  const int y0 = lo + ty * kOutY, X0 = lo + txc * C::XC, z0 = lo + tz * (2 * TZ);
  const int y = y0 - 1 + lane;
  const int yb = y0 - 1 - HW;      // first y of the slab (>= 0)
  const int e = yb & 3;
  const int ybox = yb - e;         // TMA start, 16-byte aligned
  const int xw = X0 + warp * RX;   // this warp's first output row
  const int xA = X0 - 1 - HW, zA = z0 - 1 - HW;  // MRI slab origin (row k=0)
  const int xL = X0 - HW, zL = z0 - HW;          // CT slab origin
  // y-pair layout: half-warp hh stacks in z, lane jj owns y positions yp, yp + 1.
  const int hh = lane >> 4, jj = lane & 15;
  const int yp = y0 - 1 + 2 * jj;
  const uint32_t lane_off = LY == 0 ? (uint32_t)(lane + HW + e) * 4u
                                    : (uint32_t)(2 * jj + HW + e) * 4u + hh * TZ * C::PLANE;

  // Input patch values, negated and scaled (D = (s A + In)^2 = s^2 (A - I)^2), zero outside.
  float2 In[NQ][NR];
#pragma unroll
  for (int q = 0; q < NQ; ++q)
#pragma unroll
    for (int r = 0; r < NR; ++r) {
      float v[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const int zz = (LY == 0 ? z0 + k * TZ : z0 + hh * TZ) - 1 + q, xx = xw - 1 + r;
        const int yy = LY == 0 ? y : yp + k;
        v[k] = (zz < sv.nz && xx < sv.nx && yy < sv.ny)
                   ? -__ldg(sv.img + (long long)zz * sv.nxy + (long long)xx * sv.ny + yy) * sv.scale
                   : 0.f;
      }
      In[q][r] = make_float2(v[0], v[1]);
    }
  float2 P[TZ][RX], W[TZ][RX];
#pragma unroll
  for (int q = 0; q < TZ; ++q)
#pragma unroll
    for (int r = 0; r < RX; ++r) {
      P[q][r] = make_float2(0.f, 0.f);
      W[q][r] = make_float2(0.f, 0.f);
    }

  // A list is short, so its sums are worth keeping short too: once 64 offsets or more are summed at
  // the end of an atlas they are added to the thread's own sums in shared memory (one thread's
  // column, no conflicts) and start again, as if each atlas had been summed by itself.
  int summed = 0;
  bool kept = false;
  const uint32_t sums = ringL + C::RL * C::SLOT_L + (uint32_t)tid * 4u;
  auto keep_sums = [&](bool restart) {
#pragma unroll
    for (int q = 0; q < TZ; ++q)
#pragma unroll
      for (int r = 0; r < RX; ++r)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
          float2 &v = k ? W[q][r] : P[q][r];
          float *at = static_cast<float *>(__cvta_shared_to_generic(
              sums + (uint32_t)(((q * RX + r) * 2 + k) * 2 * kThreads * 4)));
          if (kept) v = make_float2(at[0] + v.x, at[kThreads] + v.y);
          if (restart) {
            at[0] = v.x;
            at[kThreads] = v.y;
            v = make_float2(0.f, 0.f);
          }
        }
  };

  int a = a_first;
  for (int i = 0; i < T; ++i, ++pp.gstep) {
    const int ai = i / nj, j = j0 + i - ai * nj;
    if constexpr (MASKED) {
      if (j == 0 && i > 0) {  // the pair's second atlas
        a = sv.atlas_base + __ffs(later) - 1;
        later &= later - 1;
      }
    } else {
      a = a_first + ai;
    }
    __syncthreads();  // every warp is done with step i-1: its ring rows may be refilled
    if (*pp.abort_flag) return false;
    const uint32_t gstep = pp.gstep;
    if (tid == 0) {
      fence_proxy_async_smem();
      // Testing hook: withhold the first window of this CTA so that the wait below runs out.
      const bool withhold = (int)blockIdx.x == withhold_cta && gstep == 0;
      if (j == j0 && !withhold) {  // atlas start: the whole window for this step
        const uint32_t b = (gstep & 1) ? bar1 : bar0;
        mbar_arrive_expect_tx(b, (C::XC + 2) * C::ROW_A + C::XC * C::ROW_L);
        for (int k = j; k < j + C::XC + 2; ++k)
          tma_load_4d(ringA + (k % C::RA) * C::SLOT_A, sv.tmA, b, ybox, xA + k, zA, a);
        for (int k = j; k < j + C::XC; ++k)
          tma_load_4d(ringL + (k % C::RL) * C::SLOT_L, sv.tmL, b, ybox, xL + k, zL, a);
      }
      pp.armed_next = false;
      if (j + 1 < j0 + nj) {  // prefetch the one new row of each ring for step i+1
        const uint32_t b = ((gstep + 1) & 1) ? bar1 : bar0;
        mbar_arrive_expect_tx(b, C::ROW_A + C::ROW_L);
        const int ka = j + C::XC + 2, kl = j + C::XC;
        tma_load_4d(ringA + (ka % C::RA) * C::SLOT_A, sv.tmA, b, ybox, xA + ka, zA, a);
        tma_load_4d(ringL + (kl % C::RL) * C::SLOT_L, sv.tmL, b, ybox, xL + kl, zL, a);
        pp.armed_next = true;
      }
    }
    const bool ok = mbar_wait_bounded((gstep & 1) ? bar1 : bar0, (gstep >> 1) & 1, timeout_ns);
    if (!__all_sync(0xffffffffu, ok)) {
      if (lane == 0) {
        atomicExch(err, 1);
        *pp.abort_flag = 1;
      }
      continue;  // the next CTA barrier sees the flag
    }
    // Ring rows of this thread for step (a, du = j - HW).
    uint32_t rowA[NR], rowL[RX];
#pragma unroll
    for (int r = 0; r < NR; ++r)
      rowA[r] = ringA + (uint32_t)((warp * RX + r + j) % C::RA) * C::SLOT_A + lane_off;
#pragma unroll
    for (int r = 0; r < RX; ++r)
      rowL[r] = ringL + (uint32_t)((warp * RX + r + j) % C::RL) * C::SLOT_L + lane_off;
    if constexpr (LIST) {
      static_assert(LY == 1, "offset lists run in the y-pair layout");
#pragma unroll 1
      for (int sv2 = 0; sv2 < NS; ++sv2) {
        const int len = runs->len[j][sv2];
        if (len == 0) continue;
        const uint32_t at = (uint32_t)((sv2 - HW) * 4) + runs->w0[j][sv2] * C::PLANE;
        uint32_t ra[NR], rl[RX];
#pragma unroll
        for (int r = 0; r < NR; ++r) ra[r] = rowA[r] + at;
#pragma unroll
        for (int r = 0; r < RX; ++r) rl[r] = rowL[r] + at;
        if ((sv2 + e) & 1)  // the pairs' 8-byte alignment also follows the slab's start
          sweep_run_yp<HW, RX, TZ, false>(In, P, W, ra, rl, len, scale2);
        else
          sweep_run_yp<HW, RX, TZ, true>(In, P, W, ra, rl, len, scale2);
      }
      if (j == j0 + nj - 1 && i + 1 < T && (summed += runs->count) >= 64) {
        keep_sums(true);
        kept = true;
        summed = 0;
      }
    } else if constexpr (LY == 0) {
#pragma unroll 1
      for (int dv = -HW; dv <= HW; ++dv) {
        uint32_t ra[NR], rl[RX];
#pragma unroll
        for (int r = 0; r < NR; ++r) ra[r] = rowA[r] + (uint32_t)(dv * 4);
#pragma unroll
        for (int r = 0; r < RX; ++r) rl[r] = rowL[r] + (uint32_t)(dv * 4);
        sweep_dw<HW, RX, TZ>(In, P, W, ra, rl, scale2);
      }
    } else {
      // Pairs are 8-byte aligned when dv + HW is even: those sweeps first, then the others (the
      // order of the offsets only changes the FP32 summation order).
#pragma unroll 1
      for (int sv2 = 0; sv2 < NS; sv2 += 2) {
        uint32_t ra[NR], rl[RX];
#pragma unroll
        for (int r = 0; r < NR; ++r) ra[r] = rowA[r] + (uint32_t)((sv2 - HW) * 4);
#pragma unroll
        for (int r = 0; r < RX; ++r) rl[r] = rowL[r] + (uint32_t)((sv2 - HW) * 4);
        sweep_dw_yp<HW, RX, TZ, true, LY == 2>(In, P, W, ra, rl, scale2);
      }
#pragma unroll 1
      for (int sv2 = 1; sv2 < NS; sv2 += 2) {
        uint32_t ra[NR], rl[RX];
#pragma unroll
        for (int r = 0; r < NR; ++r) ra[r] = rowA[r] + (uint32_t)((sv2 - HW) * 4);
#pragma unroll
        for (int r = 0; r < RX; ++r) rl[r] = rowL[r] + (uint32_t)((sv2 - HW) * 4);
        sweep_dw_yp<HW, RX, TZ, false, LY == 2>(In, P, W, ra, rl, scale2);
      }
    }
  }
  __syncthreads();  // a timeout in the item's last step is seen here
  if (*pp.abort_flag) return false;
  if constexpr (LIST) {
    if (kept) keep_sums(false);
  }

#pragma unroll
  for (int k = 0; k < 2; ++k) {
    // LY 0: k is the z half, the lane's y is y; LY 1: k is the y of the pair, the half is hh.
    const int yy = LY == 0 ? y : yp + k;
    if (yy < y0 || yy >= y0 + kOutY || yy >= sv.ny - lo) continue;
#pragma unroll
    for (int q = 0; q < TZ; ++q) {
      const int z = (LY == 0 ? z0 + k * TZ : z0 + hh * TZ) + q;
      if (z >= sv.nz - lo) continue;
#pragma unroll
      for (int r = 0; r < RX; ++r) {
        const int x = xw + r;
        if (x >= sv.nx - lo) continue;
        const float pr = k ? P[q][r].y : P[q][r].x;
        const float sw = k ? W[q][r].y : W[q][r].x;
        const long long v = (long long)z * sv.nxy + (long long)x * sv.ny + yy;
        if (sv.acc_p) {
          sv.acc_p[v] += pr;
          sv.acc_w[v] += sw;
        } else if (sv.groups == 1) {
          sv.out[v] = fuse_result(pr, sw);
        } else {
          sv.partial[(2LL * grp) * sv.nvox + v] = pr;
          sv.partial[(2LL * grp + 1) * sv.nvox + v] = sw;
        }
      }
    }
  }
  return true;
}

__device__ __forceinline__ Pipe pipe_init(unsigned char *smem_raw) {
  Pipe pp;
  pp.base = (smem_u32(smem_raw) + 127u) & ~127u;
  pp.gstep = 0;
  pp.armed_next = false;
  pp.abort_flag =
      reinterpret_cast<volatile int *>(smem_raw + (pp.base + 16 - smem_u32(smem_raw)));
  if (threadIdx.x == 0) {
    mbar_init(pp.base, 1);
    mbar_init(pp.base + 8, 1);
    *pp.abort_flag = 0;
    fence_mbarrier_init();
  }
  __syncthreads();
  return pp;
}

// After an abort, let this CTA's own outstanding copies land (bounded) before exiting: those of
// the step whose wait timed out (gstep-1) and the prefetch armed during it, if any.
__device__ __forceinline__ void pipe_drain(const Pipe &pp, unsigned long long timeout_ns) {
  if (threadIdx.x != 0) return;
  const uint32_t bar0 = pp.base, bar1 = pp.base + 8;
  const uint32_t s = pp.gstep - 1;
  mbar_wait_bounded((s & 1) ? bar1 : bar0, (s >> 1) & 1, timeout_ns);
  if (pp.armed_next)
    mbar_wait_bounded((pp.gstep & 1) ? bar1 : bar0, (pp.gstep >> 1) & 1, timeout_ns);
}

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

// Register tiles (x rows RX, z planes per half TZ, layout LY, CTAs per SM MB) by half window, in
// sets the autotuner chooses between. Set 0 is the fastest measured shape per window on one B200
// (222x222x112, 10 atlases): y-pairs (3,4) for NH 7 and 11, y-pairs with the label ring (3,3)
// for NH 9. Set 1 is the z-pair layout (3,4), set 2 the z-pair (3,3)/(4,2) tiles, set 3 y-pairs
// with the label ring (3,4), set 4 y-pairs (2,3) at three CTAs per SM (168 registers).
template <int SET, int HW> struct TileOf { static constexpr int RX = 3, TZ = 4, LY = 1, MB = 1; };
template <> struct TileOf<0, 4> { static constexpr int RX = 3, TZ = 3, LY = 2, MB = 1; };
template <> struct TileOf<0, 2> { static constexpr int RX = 3, TZ = 3, LY = 1, MB = 1; };
template <> struct TileOf<0, 1> { static constexpr int RX = 4, TZ = 2, LY = 1, MB = 1; };
template <int HW> struct TileOf<1, HW> { static constexpr int RX = 3, TZ = 4, LY = 0, MB = 1; };
template <> struct TileOf<1, 2> { static constexpr int RX = 3, TZ = 3, LY = 0, MB = 1; };
template <> struct TileOf<1, 1> { static constexpr int RX = 4, TZ = 2, LY = 0, MB = 1; };
template <int HW> struct TileOf<2, HW> { static constexpr int RX = 4, TZ = 2, LY = 0, MB = 1; };
template <> struct TileOf<2, 5> { static constexpr int RX = 3, TZ = 3, LY = 0, MB = 1; };
template <> struct TileOf<2, 2> { static constexpr int RX = 3, TZ = 3, LY = 0, MB = 1; };
template <int HW> struct TileOf<3, HW> { static constexpr int RX = 3, TZ = 4, LY = 2, MB = 1; };
template <> struct TileOf<3, 1> { static constexpr int RX = 4, TZ = 2, LY = 2, MB = 1; };
template <int HW> struct TileOf<4, HW> { static constexpr int RX = 2, TZ = 3, LY = 1, MB = 3; };
// Further y-pair tiles, which set 0 of the single-subject kernel chooses between by the volume's
// shape (kTileCost): (2,5), (2,6) and (2,4).
template <int HW> struct TileOf<5, HW> { static constexpr int RX = 2, TZ = 5, LY = 1, MB = 1; };
template <int HW> struct TileOf<6, HW> { static constexpr int RX = 2, TZ = 6, LY = 1, MB = 1; };
template <int HW> struct TileOf<7, HW> { static constexpr int RX = 2, TZ = 4, LY = 1, MB = 1; };

// The batched kernel's tiles: one kernel holds the tile code of three windows beside the walk over
// the subject table, and the register tiles that fill 255 registers by themselves spill there (500
// bytes of spill loads with set 0's). Set 0 takes y-pairs (2,4): 250 registers, no spills. Six
// subjects of 64..160 x 64..160 x 48..96, 2..8 atlases, NH 7/9/11: 7.73 ms against 8.73; (2,5) for
// NH 11 7.83, (2,6) 7.87; sixteen such subjects 24.6 ms against 28.6.
template <int SET, int HW> struct BatchTileOf : TileOf<SET, HW> {};
template <int HW> struct BatchTileOf<0, HW> : TileOf<7, HW> {};
template <int SET, int HW>
constexpr int smem_of() {
  return Cfg<HW, BatchTileOf<SET, HW>::RX, BatchTileOf<SET, HW>::TZ>::SMEM;
}
template <int SET>
constexpr int batch_smem() {
  return smem_of<SET, 5>() > smem_of<SET, 4>()
             ? (smem_of<SET, 5>() > smem_of<SET, 3>() ? smem_of<SET, 5>() : smem_of<SET, 3>())
             : (smem_of<SET, 4>() > smem_of<SET, 3>() ? smem_of<SET, 4>() : smem_of<SET, 3>());
}

struct BatchParams {
  const SubjectView *subjects;  // device array, sorted by half window (largest first)
  int nsub;
  int total_items;
  int *err;
  int *next;  // items taken beyond each CTA's first (zero at launch)
  unsigned long long timeout_ns;
};

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

// ---------------------------------------------------------------- host side

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
// scheduler takes 0.61 of the time of two sharing it; 0.85 measured behind a full round), plus what
// each item spends on its windows, taps and stores and, with partial sums, the combine. Within 10 %
// of the measured times for 17 shapes from 48x40x30 to 222x222x112, every tile and split; the plan
// chosen is 0..2 % behind the best of them on 14 of the 17, 11 % at worst.
double expected_us(const Geometry &g, const FusePlan &pl, int slots, double voxel_ns, int natl,
                   int splits, int groups) {
  const double rounds = (double)pl.tiles * groups / slots;
  const double full = std::floor(rounds), rem = rounds - full;
  const double voxels = (double)kOutY * kWarps * pl.rx * 2 * pl.tz;
  const double round = 1e-3 * slots * voxels * voxel_ns * natl / splits;  // items of average length
  const double longest = round * splits * ((g.nh + splits - 1) / splits) / g.nh;
  double t = 0.0;
  if (full < 1.0)
    t = (rem <= 0.5 ? 0.61 : 1.0) * longest;
  else if (rem > 0.0)
    t = std::min((full + (rem <= 0.5 ? 0.85 : 1.0)) * round, (rounds + 0.4) * round) + longest - round;
  else
    t = full * round + longest - round;
  t += std::max(1.0, rounds) * (6.0 + 1.0 * natl);
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
  } else if (pl.groups < 2 || item_begin >= item_end || item_end > pl.groups * pl.tiles) {
    return cudaErrorInvalidValue;  // an item range needs partial sums and a later combine
  }
  auto kern = fuse_tma_kernel<HW, T::RX, T::TZ, T::LY, T::MB>;
  cudaError_t e;
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM)) !=
      cudaSuccess)
    return e;
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
  if (wt.start && (e = cudaEventRecord(wt.start, stream)) != cudaSuccess) return e;
  kern<<<blocks, kThreads, C::SMEM, stream>>>(tmA, tmL, p);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if (wt.stop && (e = cudaEventRecord(wt.stop, stream)) != cudaSuccess) return e;
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
  pl->groups = pl->atlas_groups = pl->splits = 1;  // many subjects fill the grid; no partial sums
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

  constexpr int smem = batch_smem<SET>();
  auto kern = fuse_batch_kernel<SET>;
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) !=
      cudaSuccess)
    return e;
  int per_sm = 1;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem)) !=
      cudaSuccess)
    return e;
  if (per_sm < 1) return cudaErrorLaunchOutOfResources;
  const int slots = sm_count() * per_sm;
  setup->params_ready = true;
  setup->items = total;
  setup->blocks = total < slots ? total : slots;
  setup->smem = smem;
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
  switch (setup.set) {
    case 0: fuse_batch_kernel<0><<<setup.blocks, kThreads, setup.smem, stream>>>(bp); break;
    case 1: fuse_batch_kernel<1><<<setup.blocks, kThreads, setup.smem, stream>>>(bp); break;
    case 2: fuse_batch_kernel<2><<<setup.blocks, kThreads, setup.smem, stream>>>(bp); break;
    case 3: fuse_batch_kernel<3><<<setup.blocks, kThreads, setup.smem, stream>>>(bp); break;
    case 4: fuse_batch_kernel<4><<<setup.blocks, kThreads, setup.smem, stream>>>(bp); break;
    default: return cudaErrorInvalidValue;
  }
  const cudaError_t e = cudaGetLastError();
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
  auto kern = fuse_runs_kernel<HW, T::RX, T::TZ>;
  cudaError_t e;
  constexpr int smem = C::SMEM + C::SUMS;
  static_assert(2 * (smem + 1024) <= 228 * 1024, "2 CTAs per SM");
  if ((e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) !=
      cudaSuccess)
    return e;
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
  kern<<<pl.ctas, kThreads, smem, stream>>>(tmA, tmL, p, runs, stats, evaluated);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
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
  kern<<<sm_count() * per_sm, kThreads, C::SMEM, stream>>>(tmA, tmL, p, items, count);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
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

cudaError_t launch_fuse_tma_items(const Geometry &g, const SlabInputs &in, double div,
                                  float *partial, int *err, const FusePlan &plan, int item_begin,
                                  int item_end, cudaStream_t stream) {
  if (g.ix <= 0 || g.iy <= 0 || g.iz <= 0) return cudaSuccess;
  if (item_begin < 0) return cudaErrorInvalidValue;
  const LaunchHooks wt{0, nullptr, nullptr};
  return launch_any(g, in, nullptr, div, partial, err, wt, plan, item_begin, item_end, stream);
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
// 11 us of a 107 us call at 97x85x53, 3 atlases, NH 5; 102 us in one).
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
