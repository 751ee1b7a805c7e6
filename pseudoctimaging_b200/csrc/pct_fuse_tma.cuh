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
//
// The kernels are compiled to one object per register tile (pct_fuse_set.cu, pct_fuse_batch.cu) and one
// for the two list forms (pct_fuse_list.cu): the driver loads an object's whole device code at the first
// launch from it, so a process that fuses one volume loads five kernels and not all 49. First call of a
// process on 64x64x32: 2.9 ms; 25 with one object, 16 with that and 31 kernels. pct_fuse_tma.cu plans
// and launches.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "pct_internal.h"
#include "pct_ptx.cuh"

namespace pct {
namespace fuse {

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

// Register tiles (x rows RX, z planes per half TZ, layout LY, CTAs per SM MB) by half window, in
// sets the autotuner chooses between. Set 0 was the fastest of sets 0 to 4 per window on one B200
// (222x222x112, 10 atlases): y-pairs (3,4) for NH 7 and 11, y-pairs with the label ring (3,3)
// for NH 9; of sets 5 to 7, which it chooses between by shape, the best takes 1 to 8 % less per voxel
// (kTileCost).
// Set 1 is the z-pair layout (3,4), set 2 the z-pair (3,3)/(4,2) tiles, set 3 y-pairs with the label
// ring (3,4), set 4 y-pairs (2,3) at three CTAs per SM (168 registers).
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

// ---------------------------------------------------------------- launches

// The items [p.item_begin, p.item_end) of one subject on `blocks` CTAs, half window hw in 1..5.
template <int SET>
cudaError_t launch_tiles(int hw, int blocks, const CUtensorMap &tmA, const CUtensorMap &tmL,
                         const TmaParams &p, const LaunchHooks &wt, cudaStream_t stream);
// The batched kernel: its CTAs per SM, and its launch.
template <int SET>
cudaError_t batch_ctas_per_sm(int *per_sm);
template <int SET>
cudaError_t launch_batch_items(const BatchParams &bp, int blocks, cudaStream_t stream);
// An offset list (set 6's tiles) and the masked items of the learned form's fallback (NH = 11, set 0's
// tile, as many CTAs as fit).
cudaError_t launch_runs(const OffsetRuns &runs, int blocks, const CUtensorMap &tmA,
                        const CUtensorMap &tmL, const TmaParams &p, unsigned long long *stats,
                        unsigned long long evaluated, cudaStream_t stream);
cudaError_t launch_list(int sms, const CUtensorMap &tmA, const CUtensorMap &tmL, const TmaParams &p,
                        const int *items, const int *count, cudaStream_t stream);

}  // namespace fuse
}  // namespace pct
