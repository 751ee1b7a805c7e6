// Training side of the learned proposal: exact targets, forward/backward, Adam.
//
// Targets: for a sampled (subject, atlas, voxel) the plain method's SSD of every one of the 11^3
// offsets is computed directly in FP32 (the same 27-tap arithmetic as the path), the 32 smallest
// are kept (ties broken by offset order) and turned into one distribution per axis: the share of
// the 32 that has each dw, du and dv.
//
// Training: one CTA takes a few samples at a time. A sample's two 9^3 patches (scaled input MRI and
// atlas MRI) are staged in shared memory and the whole network runs there: forward through the
// four valid 3x3x3 convolutions and the three heads, softmax cross-entropy per axis against the
// targets, and backward. Weights are read as BF16 (the inference precision); the math and the
// gradients are FP32. Each CTA sums its samples' gradients (weights in registers, the rest in
// shared memory) and adds them to the global FP32 gradient once. Adam then updates FP32 master weights and re-rounds the BF16 copy.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "pct_internal.h"
#include "pct_learned.h"

namespace pct {
namespace learned {
namespace {

constexpr int kTrainThreads = 384;
constexpr int kN1 = 7 * 7 * 7, kN2 = 5 * 5 * 5, kN3 = 3 * 3 * 3, kNX = 9 * 9 * 9;

struct SubjectRef {
  const float *img;
  const float *atlas;
  int nx, ny, nz, num;
};

// ---------------------------------------------------------------- targets

__global__ void targets_kernel(const SubjectRef *__restrict__ subs, const int *__restrict__ samples,
                               int n, float *__restrict__ targets, short *__restrict__ top_out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = samples[3 * i], a = samples[3 * i + 1], vox = samples[3 * i + 2];
  const SubjectRef sr = subs[s];
  const int nxy = sr.nx * sr.ny;
  const long long nvox = (long long)nxy * sr.nz;
  const float *img = sr.img;
  const float *A = sr.atlas + (long long)a * nvox;
  float in[27];
  {
    int k = 0;
    for (int dz = -1; dz <= 1; ++dz)
      for (int dx = -1; dx <= 1; ++dx)
        for (int dy = -1; dy <= 1; ++dy) in[k++] = __ldg(img + vox + dz * nxy + dx * sr.ny + dy);
  }
  float best[kTopK];
  short idx[kTopK];
  int cnt = 0;
  for (int o = 0; o < kAxis * kAxis * kAxis; ++o) {
    const int dw = o / (kAxis * kAxis) - 5, du = (o / kAxis) % kAxis - 5, dv = o % kAxis - 5;
    const int c = vox + dw * nxy + du * sr.ny + dv;
    float ssd = 0.f;
    int k = 0;
    for (int pz = -1; pz <= 1; ++pz)
      for (int px = -1; px <= 1; ++px)
        for (int py = -1; py <= 1; ++py) {
          const float d = in[k++] - __ldg(A + c + pz * nxy + px * sr.ny + py);
          ssd = fmaf(d, d, ssd);
        }
    if (cnt < kTopK || ssd < best[cnt - 1]) {  // insertion into the sorted top-32
      int j = cnt < kTopK ? cnt++ : kTopK - 1;
      while (j > 0 && best[j - 1] > ssd) {
        best[j] = best[j - 1];
        idx[j] = idx[j - 1];
        --j;
      }
      best[j] = ssd;
      idx[j] = (short)o;
    }
  }
  float *t = targets + (long long)i * kHeads;
  for (int j = 0; j < kHeads; ++j) t[j] = 0.f;
  for (int j = 0; j < kTopK; ++j) {
    const int o = idx[j];
    t[o / (kAxis * kAxis)] += 1.0f / kTopK;
    t[kAxis + (o / kAxis) % kAxis] += 1.0f / kTopK;
    t[2 * kAxis + o % kAxis] += 1.0f / kTopK;
    if (top_out) top_out[(long long)i * kTopK + j] = idx[j];
  }
}

// ---------------------------------------------------------------- forward / backward
//
// What bounds the pass is FP32 arithmetic (3.8 M multiply-adds per sample) fed from shared memory,
// so every phase works on a register tile that uses each value it loads several times. A CTA of 12
// warps takes kTS samples at a time; activations are channels-last ([position][16]), weights
// [tap][ci][co], so that four channels are one 16-byte load:
//  * forward and input gradients: a thread owns one output row along y and four channels; a step
//    loads the input row once for its three y taps. The forward sums start at the bias and run over
//    input channels, then taps, one after the other: a pre-activation near zero changes its side of
//    the ReLU with the order of its sum, and one of those moves the gradient by 1e-6. (Channels in
//    groups of four, conv3 and conv4 in partial sums: 1.21 ms, and other sides taken.)
//  * weight gradients: a warp owns the 16 x 16 x 3 (co, ci, ky) weights of one (kz, kx), 24 per
//    lane, and keeps their sums in registers over all samples of the CTA (conv2: 12 loads for 120
//    multiply-adds per row); nine warps take conv2 while the other three take conv3.
// The gradient of conv1's output overwrites that output, and conv3's likewise, once the weight
// gradients that read it are done. 4,096 samples: 13.8 ms with one output per thread and the
// gradients in shared memory, 1.28 ms now (gradients read back, whole call).

constexpr int kTS = 3;  // samples per CTA pass: what fits beside the weights in 227 KB

struct SampleSmem {
  float x0[kCin * kNX + 2];  // scaled input patches [ci][z][x][y]
  float a1[kN1 * kC];        // conv1's output, later its gradient ([position][channel], rotated)
  float a2[kN2 * kC];        // (rotated as well)
  float a3[kN3 * kC];        // conv3's output, later its gradient
  float d2[kN2 * kC];
  float a4[kC], d4[kC];
  float logits[36], dlog[36];
};
constexpr int kSmallB = 0, kSmallH = 4 * kC, kSmallHB = kSmallH + kHeads * kC;
constexpr int kSmall = kSmallHB + kHeads;  // biases, heads, head biases

struct TrainSmem {
  float w1[27][kCin][kC];
  float w[3][27][kC][kC];  // conv2..conv4 (conv2 and conv3 with wgroup)
  __align__(16) float small[kSmall];   // biases [4][16], heads [33][16], head biases [33]
  __align__(16) float gsmall[kSmall];  // this CTA's gradient sums of the same
  __align__(16) SampleSmem s[kTS];
  float loss;
};
static_assert(sizeof(TrainSmem) <= 227 * 1024, "shared memory");
static_assert(sizeof(SampleSmem) % 16 == 0 && offsetof(TrainSmem, s) % 16 == 0 &&
                  offsetof(SampleSmem, a1) % 16 == 0 && offsetof(SampleSmem, d2) % 16 == 0 &&
                  offsetof(SampleSmem, d4) % 16 == 0,
              "16-byte rows");

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ float get(const float4 &v, int c) {
  return c == 0 ? v.x : c == 1 ? v.y : c == 2 ? v.z : v.w;
}
__device__ __forceinline__ void axpy(float (&acc)[4], float a, const float4 &w) {
  acc[0] = fmaf(a, w.x, acc[0]);
  acc[1] = fmaf(a, w.y, acc[1]);
  acc[2] = fmaf(a, w.z, acc[2]);
  acc[3] = fmaf(a, w.w, acc[3]);
}
__device__ __forceinline__ float dot(const float4 &a, const float4 &b, float acc) {
  return fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc))));
}

// Place of the four-channel group cog of row ci of conv2's and conv3's weights: rotated within the
// row by the row's own group, so that the four lanes that read four groups of one row (forward) and
// the four that read one group of four rows (input gradients) both hit different banks. (Without:
// half of all shared wavefronts were conflicts, 1.62 ms for the 4,096 samples.)
__device__ __forceinline__ int wgroup(int ci, int cog) { return 4 * (cog ^ (ci >> 2)); }

// Place of channel group g in row `row` (z * S + x) of a1 and a2: rotated by the row, so that lanes on
// consecutive rows that read one channel (forward) hit different banks.
__device__ __forceinline__ int agroup(int row, int g) { return 4 * (g ^ ((row >> 1) & 3)); }

// One output row (SO positions along y, row (z, x)) and channels [4 cg, 4 cg + 4) of a 16 -> 16
// convolution, added to acc in the order of the input channels and, within one, of the taps.
template <int SI, int SO>
__device__ __forceinline__ void conv_row(const float (&w)[27][kC][kC], const float *in, int z, int x,
                                         int cg, float (&acc)[SO][4]) {
#pragma unroll 1
  for (int ci = 0; ci < kC; ++ci) {
    const int wg = wgroup(ci, cg);
#pragma unroll 3
    for (int kzx = 0; kzx < 9; ++kzx) {
      const int r = (z + kzx / 3) * SI + x + kzx % 3;
      const float *row = in + r * SI * kC + agroup(r, ci >> 2) + (ci & 3);
      float v[SO + 2];
#pragma unroll
      for (int y = 0; y < SO + 2; ++y) v[y] = row[y * kC];
#pragma unroll
      for (int ky = 0; ky < 3; ++ky) {
        const float4 wv = ld4(&w[kzx * 3 + ky][ci][wg]);
#pragma unroll
        for (int y = 0; y < SO; ++y) axpy(acc[y], v[y + ky], wv);
      }
    }
  }
}

// One input row (SI positions along y, row (z, x)) and input channels [4 cg, 4 cg + 4) of the
// gradient with respect to a 16 -> 16 convolution's input, dz its output's gradient.
template <int SI, int SO>
__device__ __forceinline__ void grad_row(const float (&w)[27][kC][kC], const float *dz, int z, int x,
                                         int cg, float (&acc)[SI][4]) {
#pragma unroll
  for (int y = 0; y < SI; ++y)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[y][c] = 0.f;
  const int kz0 = max(0, z - SO + 1), kz1 = min(2, z), kx0 = max(0, x - SO + 1), kx1 = min(2, x);
#pragma unroll 1
  for (int kz = kz0; kz <= kz1; ++kz)
#pragma unroll 1
    for (int kx = kx0; kx <= kx1; ++kx)
#pragma unroll 1
      for (int g = 0; g < 4; ++g) {
        const float *row = dz + ((z - kz) * SO + x - kx) * SO * kC + 4 * g;
        float4 v[SO];
#pragma unroll
        for (int y = 0; y < SO; ++y) v[y] = ld4(row + y * kC);
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          float4 wv[4];
#pragma unroll
          for (int c = 0; c < 4; ++c)
            wv[c] = ld4(&w[(kz * 3 + kx) * 3 + ky][4 * cg + c][wgroup(4 * cg, g)]);
          // (four multiply-adds in a row share one operand: three fresh ones each take 1.6 cycles)
#pragma unroll
          for (int y = 0; y < SO; ++y)
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
              for (int c = 0; c < 4; ++c)
                acc[y + ky][c] = fmaf(get(v[y], k), get(wv[c], k), acc[y + ky][c]);
        }
      }
}

// Rows (z * SI + x) of the input-gradient phases by how many (kz, kx) reach them, 9 first: a warp's
// lanes then take the same number of steps, and the long warps spread over the schedulers. (In
// plain order every warp held a row with the longest loops: conv2's phase was 31 % of the whole
// pass; 4,096 samples 1.33 ms, 1.23 with the order.)
__constant__ unsigned char kRowOrder7[49] = {
    16, 17, 18, 23, 24, 25, 30, 31, 32, 15, 19, 22, 26, 29, 33, 9, 10, 11, 37, 38, 39, 8, 12, 36, 40,
    14, 20, 21, 27, 28, 34, 2, 3, 4, 44, 45, 46, 7, 13, 35, 41, 1, 5, 43, 47, 0, 6, 42, 48};
__constant__ unsigned char kRowOrder5[25] = {
    12, 11, 13, 7, 17, 6, 8, 16, 18, 10, 14, 2, 22, 5, 9, 15, 19, 1, 3, 21, 23, 0, 4, 20, 24};

// Adds one sample's share of the weight gradients of one (kz, kx): acc[ky][2 co][4 ci] of the
// lane's co pair and ci group.
template <int SI, int SO>
__device__ __forceinline__ void weight_rows(const float *in, const float *dz, int kz, int kx, int lane,
                                            float *acc) {
  const int cop = 2 * (lane >> 2), cig = lane & 3;
#pragma unroll 1
  for (int r = 0; r < SO * SO; ++r) {
    const int z = r / SO, x = r - z * SO;
    const int ri = (z + kz) * SI + x + kx;
    const float *row = in + ri * SI * kC + agroup(ri, cig);
    const float *drow = dz + r * SO * kC + cop;
    float4 v[SO + 2];
#pragma unroll
    for (int y = 0; y < SO + 2; ++y) v[y] = ld4(row + y * kC);
#pragma unroll
    for (int y = 0; y < SO; ++y) {
      const float2 d = *reinterpret_cast<const float2 *>(drow + y * kC);
#pragma unroll
      for (int ky = 0; ky < 3; ++ky)
#pragma unroll
        for (int o = 0; o < 2; ++o)
#pragma unroll
          for (int c = 0; c < 4; ++c)
            acc[ky * 8 + o * 4 + c] = fmaf(o ? d.y : d.x, get(v[y + ky], c), acc[ky * 8 + o * 4 + c]);
    }
  }
}

// Adds the channel sums of n positions to g[16] (one warp).
__device__ __forceinline__ void bias_sum(const float *d, int n, int lane, float *g) {
  float acc = 0.f;
  for (int p = lane >> 4; p < n; p += 2) acc += d[p * kC + (lane & 15)];
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);
  if (lane < kC) g[lane] += acc;
}

__global__ void __launch_bounds__(kTrainThreads, 1)
    train_kernel(const SubjectRef *__restrict__ subs, const int *__restrict__ samples,
                 const float *__restrict__ targets, int begin, int count,
                 const __nv_bfloat16 *__restrict__ wbf, float *__restrict__ grad,
                 float *__restrict__ loss_sum) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TrainSmem &S = *reinterpret_cast<TrainSmem *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < 27 * kCin * kC; i += kTrainThreads) {
    const int k = i / (kCin * kC), ci = (i / kC) % kCin, co = i % kC;
    S.w1[k][ci][co] = __bfloat162float(wbf[kW1 + (co * kCin + ci) * 27 + k]);
  }
  for (int l = 0; l < 3; ++l) {
    const int off = l == 0 ? kW2 : l == 1 ? kW3 : kW4;
    for (int i = tid; i < 27 * kC * kC; i += kTrainThreads) {
      const int k = i / (kC * kC), ci = (i / kC) % kC, co = i % kC;
      S.w[l][k][ci][l < 2 ? wgroup(ci, co >> 2) + (co & 3) : co] =
          __bfloat162float(wbf[off + (co * kC + ci) * 27 + k]);
    }
  }
  auto small_param = [](int i) {  // flat parameter index of a small one
    if (i >= kSmallHB) return kHB + i - kSmallHB;
    if (i >= kSmallH) return kH + i - kSmallH;
    const int l = i / kC;
    return (l == 0 ? kB1 : l == 1 ? kB2 : l == 2 ? kB3 : kB4) + i % kC;
  };
  for (int i = tid; i < kSmall; i += kTrainThreads) {
    S.small[i] = __bfloat162float(wbf[small_param(i)]);
    S.gsmall[i] = 0.f;
  }
  if (tid == 0) S.loss = 0.f;
  // Gradient sums in registers. Warps 0-8: conv2's (kz, kx) = warp in R[0, 24) and two of conv1's
  // 18 (ci, kz, kx) in R[24, 48); warps 9-11: conv3's three (warp - 9, kx). conv4: R4, flat index
  // tid + kTrainThreads * i of [tap][ci][co].
  float R[72], R4[18];
#pragma unroll
  for (int i = 0; i < 72; ++i) R[i] = 0.f;
#pragma unroll
  for (int i = 0; i < 18; ++i) R4[i] = 0.f;
  static_assert(27 * kC * kC == 18 * kTrainThreads && kTrainThreads == 384, "conv4 gradients");

  const int first = (int)((long long)count * blockIdx.x / gridDim.x);
  const int last = (int)((long long)count * (blockIdx.x + 1) / gridDim.x);
  for (int base = first; base < last; base += kTS) {
    const int ns = min(kTS, last - base);
    __syncthreads();  // the previous samples' buffers are free
    for (int e = tid; e < ns * kCin * kNX; e += kTrainThreads) {
      const int si = e / (kCin * kNX), q = e % (kCin * kNX), c = q / kNX, p = q % kNX;
      const int smp = begin + base + si;
      const int a = samples[3 * smp + 1], vox = samples[3 * smp + 2];
      const SubjectRef sr = subs[samples[3 * smp]];
      const int nxy = sr.nx * sr.ny;
      const int z = p / 81 - 4, x = (p / 9) % 9 - 4, y = p % 9 - 4;
      const float *src = c == 0 ? sr.img : sr.atlas + (long long)a * nxy * sr.nz;
      S.s[si].x0[q] = __ldg(src + vox + z * nxy + x * sr.ny + y) * kInScale;
    }
    __syncthreads();
    // conv1
    for (int t = tid; t < ns * 49 * 4; t += kTrainThreads) {
      const int cg = t & 3, si = (t >> 2) / 49, row = (t >> 2) % 49, z = row / 7, x = row % 7;
      float acc[7][4];
      const float4 b = ld4(S.small + kSmallB + 4 * cg);
#pragma unroll
      for (int y = 0; y < 7; ++y) acc[y][0] = b.x, acc[y][1] = b.y, acc[y][2] = b.z, acc[y][3] = b.w;
#pragma unroll 1
      for (int q = 0; q < 18; ++q) {
        const int ci = q / 9, kzx = q % 9;
        const float *src = S.s[si].x0 + ci * kNX + ((z + kzx / 3) * 9 + x + kzx % 3) * 9;
        float v[9];
#pragma unroll
        for (int y = 0; y < 9; ++y) v[y] = src[y];
#pragma unroll
        for (int ky = 0; ky < 3; ++ky) {
          const float4 wv = ld4(&S.w1[kzx * 3 + ky][ci][4 * cg]);
#pragma unroll
          for (int y = 0; y < 7; ++y) axpy(acc[y], v[y + ky], wv);
        }
      }
      float *dst = S.s[si].a1 + row * 7 * kC + agroup(row, cg);
#pragma unroll
      for (int y = 0; y < 7; ++y)
        *reinterpret_cast<float4 *>(dst + y * kC) =
            make_float4(fmaxf(acc[y][0], 0.f), fmaxf(acc[y][1], 0.f), fmaxf(acc[y][2], 0.f),
                        fmaxf(acc[y][3], 0.f));
    }
    __syncthreads();
    // conv2
    if (tid < ns * 25 * 4) {
      const int cg = tid & 3, si = (tid >> 2) / 25, row = (tid >> 2) % 25;
      float acc[5][4];
      const float4 b = ld4(S.small + kSmallB + kC + 4 * cg);
#pragma unroll
      for (int y = 0; y < 5; ++y) acc[y][0] = b.x, acc[y][1] = b.y, acc[y][2] = b.z, acc[y][3] = b.w;
      conv_row<7, 5>(S.w[0], S.s[si].a1, row / 5, row % 5, cg, acc);
      float *dst = S.s[si].a2 + row * 5 * kC + agroup(row, cg);
#pragma unroll
      for (int y = 0; y < 5; ++y)
        *reinterpret_cast<float4 *>(dst + y * kC) =
            make_float4(fmaxf(acc[y][0], 0.f), fmaxf(acc[y][1], 0.f), fmaxf(acc[y][2], 0.f),
                        fmaxf(acc[y][3], 0.f));
    }
    __syncthreads();
    // conv3
    if (tid < ns * 9 * 4) {
      const int cg = tid & 3, si = (tid >> 2) / 9, row = (tid >> 2) % 9;
      float acc[3][4];
      const float4 b = ld4(S.small + kSmallB + 2 * kC + 4 * cg);
#pragma unroll
      for (int y = 0; y < 3; ++y) acc[y][0] = b.x, acc[y][1] = b.y, acc[y][2] = b.z, acc[y][3] = b.w;
      conv_row<5, 3>(S.w[1], S.s[si].a2, row / 3, row % 3, cg, acc);
#pragma unroll
      for (int y = 0; y < 3; ++y)
        *reinterpret_cast<float4 *>(S.s[si].a3 + (row * 3 + y) * kC + 4 * cg) =
            make_float4(fmaxf(acc[y][0], 0.f), fmaxf(acc[y][1], 0.f), fmaxf(acc[y][2], 0.f),
                        fmaxf(acc[y][3], 0.f));
    }
    __syncthreads();
    // conv4
    if (tid < ns * kC) {
      const int si = tid / kC, co = tid % kC;
      const float *w4 = &S.w[2][0][0][0], *a3 = S.s[si].a3;
      float acc = S.small[kSmallB + 3 * kC + co];
      for (int ci = 0; ci < kC; ++ci)
#pragma unroll
        for (int k = 0; k < 27; ++k) acc = fmaf(w4[(k * kC + ci) * kC + co], a3[k * kC + ci], acc);
      S.s[si].a4[co] = fmaxf(acc, 0.f);
    }
    __syncthreads();
    if (tid < ns * kHeads) {
      const int si = tid / kHeads, o = tid % kHeads;
      float acc = S.small[kSmallHB + o];
      for (int c = 0; c < kC; ++c) acc = fmaf(S.small[kSmallH + o * kC + c], S.s[si].a4[c], acc);
      S.s[si].logits[o] = acc;
    }
    __syncthreads();
    // softmax cross-entropy per axis: dlogits = softmax - target
    if (tid < 3 * ns) {
      const int si = tid / 3, h = tid % 3;
      const float *t = targets + (long long)(begin + base + si) * kHeads + h * kAxis;
      const float *lg = S.s[si].logits + h * kAxis;
      float m = -1e30f;
      for (int j = 0; j < kAxis; ++j) m = fmaxf(m, lg[j]);
      float z = 0.f;
      for (int j = 0; j < kAxis; ++j) z += __expf(lg[j] - m);
      const float lz = __logf(z) + m;
      float l = 0.f;
      for (int j = 0; j < kAxis; ++j) {
        const float lp = lg[j] - lz;
        l -= t[j] * lp;
        S.s[si].dlog[h * kAxis + j] = __expf(lp) - t[j];
      }
      atomicAdd(&S.loss, l);
    }
    __syncthreads();
    // heads: dH, dhb, d4
    for (int e = tid; e < kHeads * kC; e += kTrainThreads) {
      float acc = S.gsmall[kSmallH + e];
      for (int si = 0; si < ns; ++si) acc = fmaf(S.s[si].dlog[e / kC], S.s[si].a4[e % kC], acc);
      S.gsmall[kSmallH + e] = acc;
    }
    if (tid < kHeads)
      for (int si = 0; si < ns; ++si) S.gsmall[kSmallHB + tid] += S.s[si].dlog[tid];
    if (tid >= 64 && tid < 64 + ns * kC) {
      const int si = (tid - 64) / kC, c = (tid - 64) % kC;
      float acc = 0.f;
      for (int o = 0; o < kHeads; ++o)
        acc = fmaf(S.small[kSmallH + o * kC + c], S.s[si].dlog[o], acc);
      S.s[si].d4[c] = S.s[si].a4[c] > 0.f ? acc : 0.f;
    }
    __syncthreads();
    // conv4: weight gradients, then the input's gradient over its activation
    for (int si = 0; si < ns; ++si) {
      const float d = S.s[si].d4[tid & 15];  // kTrainThreads is a multiple of 16
#pragma unroll
      for (int i = 0; i < 18; ++i)
        R4[i] = fmaf(d, S.s[si].a3[(tid + kTrainThreads * i) >> 4], R4[i]);
      if (tid < kC) S.gsmall[kSmallB + 3 * kC + tid] += S.s[si].d4[tid];
    }
    __syncthreads();
    for (int e = tid; e < ns * kN3 * kC; e += kTrainThreads) {
      const int si = e / (kN3 * kC), q = e % (kN3 * kC);
      const float *wr = &S.w[2][0][0][0] + q * kC;
      float acc = 0.f;
#pragma unroll
      for (int g = 0; g < 4; ++g) acc = dot(ld4(wr + 4 * g), ld4(S.s[si].d4 + 4 * g), acc);
      S.s[si].a3[q] = S.s[si].a3[q] > 0.f ? acc : 0.f;
    }
    __syncthreads();
    // conv3's input gradient
    if (tid < ns * 25 * 4) {
      const int cg = tid & 3, si = (tid >> 2) % ns, row = kRowOrder5[(tid >> 2) / ns];
      float acc[5][4];
      grad_row<5, 3>(S.w[1], S.s[si].a3, row / 5, row % 5, cg, acc);
#pragma unroll
      for (int y = 0; y < 5; ++y) {
        const float4 a = ld4(S.s[si].a2 + (row * 5 + y) * kC + agroup(row, cg));
        *reinterpret_cast<float4 *>(S.s[si].d2 + (row * 5 + y) * kC + 4 * cg) =
            make_float4(a.x > 0.f ? acc[y][0] : 0.f, a.y > 0.f ? acc[y][1] : 0.f,
                        a.z > 0.f ? acc[y][2] : 0.f, a.w > 0.f ? acc[y][3] : 0.f);
      }
    }
    __syncthreads();
    // weight gradients of conv2 (warps 0-8) and conv3 (9-11), their bias gradients
    for (int si = 0; si < ns; ++si) {
      const SampleSmem &q = S.s[si];
      if (warp < 9) {
        weight_rows<7, 5>(q.a1, q.d2, warp / 3, warp % 3, lane, R);
      } else {
#pragma unroll
        for (int kx = 0; kx < 3; ++kx) weight_rows<5, 3>(q.a2, q.a3, warp - 9, kx, lane, R + 24 * kx);
        if (warp == 9) bias_sum(q.d2, kN2, lane, S.gsmall + kSmallB + kC);
        if (warp == 10) bias_sum(q.a3, kN3, lane, S.gsmall + kSmallB + 2 * kC);
      }
    }
    __syncthreads();
    // conv2's input gradient, over conv1's output
    for (int t = tid; t < ns * 49 * 4; t += kTrainThreads) {
      const int cg = t & 3, si = (t >> 2) % ns, row = kRowOrder7[(t >> 2) / ns];
      float acc[7][4];
      grad_row<7, 5>(S.w[0], S.s[si].d2, row / 7, row % 7, cg, acc);
#pragma unroll
      for (int y = 0; y < 7; ++y) {
        float4 *a1 =
            reinterpret_cast<float4 *>(S.s[si].a1 + (row * 7 + y) * kC + agroup(row, cg));
        const float4 a = *a1;
        *a1 = make_float4(a.x > 0.f ? acc[y][0] : 0.f, a.y > 0.f ? acc[y][1] : 0.f,
                          a.z > 0.f ? acc[y][2] : 0.f, a.w > 0.f ? acc[y][3] : 0.f);
      }
    }
    __syncthreads();
    // conv1's weight gradients: a warp's two (ci, kz, kx), lanes over rows and channel groups
    if (warp < 9) {
      for (int si = 0; si < ns; ++si)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int q = 2 * warp + h, ci = q / 9, kz = q % 9 / 3, kx = q % 3;
#pragma unroll 1
          for (int row = lane >> 2; row < 49; row += 8) {
            const float *src = S.s[si].x0 + ci * kNX + ((row / 7 + kz) * 9 + row % 7 + kx) * 9;
            float v[9];
#pragma unroll
            for (int y = 0; y < 9; ++y) v[y] = src[y];
#pragma unroll
            for (int y = 0; y < 7; ++y) {
              const float4 d = ld4(S.s[si].a1 + (row * 7 + y) * kC + agroup(row, lane & 3));
#pragma unroll
              for (int ky = 0; ky < 3; ++ky)
#pragma unroll
                for (int c = 0; c < 4; ++c)
                  R[24 + h * 12 + ky * 4 + c] =
                      fmaf(get(d, c), v[y + ky], R[24 + h * 12 + ky * 4 + c]);
            }
          }
        }
    } else if (warp - 9 < ns) {
      // (three warps may add to the same channels: one sample each)
      float acc = 0.f;
      const float *d = S.s[warp - 9].a1;
      for (int p = lane >> 4; p < kN1; p += 2)
        acc += d[p * kC + agroup(p / 7, (lane & 15) >> 2) + (lane & 3)];
      acc += __shfl_xor_sync(0xffffffffu, acc, 16);
      if (lane < kC) atomicAdd(S.gsmall + kSmallB + lane, acc);
    }
  }
  __syncthreads();
  for (int i = tid; i < kSmall; i += kTrainThreads) atomicAdd(grad + small_param(i), S.gsmall[i]);
  if (tid == 0) atomicAdd(loss_sum, S.loss);
#pragma unroll
  for (int i = 0; i < 18; ++i) {
    const int e = tid + kTrainThreads * i, k = e / (kC * kC), ci = (e / kC) % kC, co = e % kC;
    atomicAdd(grad + kW4 + (co * kC + ci) * 27 + k, R4[i]);
  }
  const int cop = 2 * (lane >> 2), cig = 4 * (lane & 3);
#pragma unroll
  for (int ky = 0; ky < 3; ++ky)
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int at = ((cop + o) * kC + cig + c) * 27 + ky;
        if (warp < 9) {
          atomicAdd(grad + kW2 + at + 3 * warp, R[ky * 8 + o * 4 + c]);
        } else {
#pragma unroll
          for (int kx = 0; kx < 3; ++kx)
            atomicAdd(grad + kW3 + at + ((warp - 9) * 3 + kx) * 3, R[24 * kx + ky * 8 + o * 4 + c]);
        }
      }
  if (warp < 9) {
#pragma unroll
    for (int i = 0; i < 24; ++i) {
      float v = R[24 + i];
      for (int o = 4; o < 32; o *= 2) v += __shfl_xor_sync(0xffffffffu, v, o);
      const int q = 2 * warp + i / 12, ky = i % 12 / 4, co = 4 * (lane & 3) + i % 4;
      if (lane < 4) atomicAdd(grad + kW1 + (co * kCin + q / 9) * 27 + q % 9 * 3 + ky, v);
    }
  }
}

__global__ void adam_kernel(float *__restrict__ master, __nv_bfloat16 *__restrict__ wbf,
                            float *__restrict__ m, float *__restrict__ v,
                            float *__restrict__ grad, float scale, float lr, float b1, float b2,
                            float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kParams) return;
  const float g = grad[i] * scale;
  const float mi = b1 * m[i] + (1.f - b1) * g;
  const float vi = b2 * v[i] + (1.f - b2) * g * g;
  m[i] = mi;
  v[i] = vi;
  const float w = master[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  master[i] = w;
  wbf[i] = __float2bfloat16_rn(w);
  grad[i] = 0.f;
}

__global__ void round_weights_kernel(const float *__restrict__ master,
                                     __nv_bfloat16 *__restrict__ wbf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < kParams) wbf[i] = __float2bfloat16_rn(master[i]);
}

}  // namespace

size_t train_smem_bytes() { return sizeof(TrainSmem); }

cudaError_t launch_targets(const void *subject_refs, const int *samples, int n, float *targets,
                           short *top, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  targets_kernel<<<(n + 127) / 128, 128, 0, s>>>(static_cast<const SubjectRef *>(subject_refs),
                                                 samples, n, targets, top);
  return cudaGetLastError();
}

cudaError_t launch_train_grads(const void *subject_refs, const int *samples, const float *targets,
                               int begin, int count, const __nv_bfloat16 *wbf, float *grad,
                               float *loss_sum, cudaStream_t s) {
  if (count <= 0) return cudaSuccess;
  cudaError_t e = cudaFuncSetAttribute(train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)sizeof(TrainSmem));
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = count < sms ? count : sms;
  train_kernel<<<blocks, kTrainThreads, sizeof(TrainSmem), s>>>(
      static_cast<const SubjectRef *>(subject_refs), samples, targets, begin, count, wbf, grad,
      loss_sum);
  return cudaGetLastError();
}

cudaError_t launch_adam(float *master, __nv_bfloat16 *wbf, float *m, float *v, float *grad,
                        float grad_scale, float lr, int step, cudaStream_t s) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
  adam_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(master, wbf, m, v, grad, grad_scale, lr, b1, b2,
                                                    eps, c1, c2);
  return cudaGetLastError();
}

cudaError_t launch_round_weights(const float *master, __nv_bfloat16 *wbf, cudaStream_t s) {
  round_weights_kernel<<<(kParams + 255) / 256, 256, 0, s>>>(master, wbf);
  return cudaGetLastError();
}

size_t subject_ref_bytes() { return sizeof(SubjectRef); }

}  // namespace learned
}  // namespace pct
