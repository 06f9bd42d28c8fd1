// pruner.cu: the learned partition / mode pruner -- its features, its network (forward and
// backward), loss and optimiser, and the masks it proposes (include/celv2_pruner.h).
//
// The network is small (56,120 parameters, ~1 MFLOP per superblock), so training is bound by what
// moves between its layers. The forward pass runs all three convolutions of two samples in one CTA,
// the backward pass all three of one: the activations' BF16 copies sit in shared memory and a
// convolution's column matrix exists only as the row addresses ldmatrix is given (a zero row for the
// padding); weight gradients stay in the CTA's accumulators over up to 32 of its samples. Operands are rounded
// to BF16, mma.sync m16n8k16 with FP32 accumulators, bias and ReLU on the FP32 values, which is what the
// cache between the passes holds (the convolutions' backward masks ask its BF16 copies, zero where it is
// zero or below 2^-134). A step on 4,096 samples 2.33 -> 0.28 ms against column
// matrices written out and read back for every layer (390 MB) and weight gradients of a few CTAs.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <climits>
#include <string>

#include "celv2_pruner.h"
#include "kernels.h"

namespace celv2cu {

void set_last_error(const std::string& msg);

namespace nn {

constexpr int kF = CELV2_PRUNER_FEATURES, kOut = CELV2_PRUNER_OUTPUTS;
// parameter offsets
constexpr int kW1 = 0, kB1 = kW1 + 16 * 9, kW2 = kB1 + 16, kB2 = kW2 + 32 * 144, kW3 = kB2 + 32, kB3 = kW3 + 32 * 288,
              kW4 = kB3 + 32, kB4 = kW4 + 64 * 632, kW5 = kB4 + 64, kB5 = kW5 + kOut * 64, kParams = kB5 + kOut;
static_assert(kParams == CELV2_PRUNER_PARAMS, "parameter count");
// forward cache, floats per sample: the image, the convolutions' outputs (the last with the other
// features behind it), the hidden layer; the logits are the buffer's last
constexpr int kXs = 256, kA1 = 256 * 16, kA2 = 64 * 32, kH0 = 632, kA4 = 64, kLogits = kOut;
static_assert(kXs + kA1 + kA2 + kH0 + kA4 + kLogits + 4 <= CELV2_PRUNER_ACTS, "cache size");
// backward workspace, floats per sample: gradients at the hidden layer and at the last convolution
constexpr int kDz4 = 64, kDz3 = 512;
static_assert(kDz4 + kDz3 + 4 <= CELV2_PRUNER_WORK, "workspace size");

// The caller's buffers are floats at any address: the segments start at the first 16-byte boundary.
template <typename T>
T* aligned16(T* p) {
  return reinterpret_cast<T*>((reinterpret_cast<uintptr_t>(p) + 15) & ~uintptr_t(15));
}
struct Cache {  // the forward cache of a batch, segment by segment
  float *xs, *a1, *a2, *h0, *a4, *logits;
  Cache(float* base, long long b) {
    xs = aligned16(base);
    a1 = xs + b * kXs;
    a2 = a1 + b * kA1;
    h0 = a2 + b * kA2;
    a4 = h0 + b * kH0;
    logits = base + b * (CELV2_PRUNER_ACTS - kLogits);
  }
};

using bf16 = __nv_bfloat16;

__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float rbf(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

__device__ __forceinline__ void mma16816(float* d, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Four 8x8 matrices from shared memory, lane i giving the address of row i % 8 of matrix i / 8; T: each
// transposed on the way.
template <bool T>
__device__ __forceinline__ void ldsm4(uint32_t* r, const bf16* p) {
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  if (T)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
template <bool T>
__device__ __forceinline__ void ldsm2(uint32_t* r, const bf16* p) {  // two, lanes 0-15's addresses
  const unsigned a = (unsigned)__cvta_generic_to_shared(p);
  if (T)
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.shared.b16 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(a) : "memory");
}

constexpr int kNnThreads = 256;
// Row strides in shared memory, elements: 16 bytes more than the row, so that eight rows of a matrix
// fall into different banks (or two by two where a stride-2 convolution skips rows).
constexpr int kS1 = 24, kS2 = 40, kSw2 = 152, kSw3 = 296;

// BF16 copies of the strided convolutions' weights, all threads; the caller's barrier follows.
__device__ __forceinline__ void stage_conv_weights(const float* P, bf16* w2, bf16* w3) {
  for (int i = threadIdx.x; i < 32 * 144; i += kNnThreads) w2[i / 144 * kSw2 + i % 144] = __float2bfloat16_rn(P[kW2 + i]);
  for (int i = threadIdx.x; i < 32 * 288; i += kNnThreads) w3[i / 288 * kSw3 + i % 288] = __float2bfloat16_rn(P[kW3 + i]);
}

// The input position that tap (ky, kx) of a stride-2 convolution reads at output (oy, ox), as a row of
// the H x H activation in shared memory; its row H * H is zero and stands for the padding.
template <int H>
__device__ __forceinline__ int tap_row(int oy, int ox, int ky, int kx) {
  const int y = 2 * oy + ky - 1, x = 2 * ox + kx - 1;
  return y >= 0 && y < H && x >= 0 && x < H ? y * H + x : H * H;
}

// ---- forward: the convolutions, two samples at a time ----
struct FwdSmem {
  bf16 w2[32 * kSw2], w3[32 * kSw3];
  bf16 w1[16][kS1];          // nine taps, then zeros
  float b1[16], b2[32], b3[32];
  float x[2][18][18];        // the images, BF16-rounded, with a border of zeros
  bf16 a1[2][257][kS1], a2[2][65][kS2];
};

__global__ void __launch_bounds__(kNnThreads, 3) k_conv_forward(const float* __restrict__ P, const float* __restrict__ X,
                                                                int batch, float* xs, float* a1g, float* a2g, float* h0) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FwdSmem& S = *reinterpret_cast<FwdSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  stage_conv_weights(P, S.w2, S.w3);
  S.w1[tid >> 4][tid & 15] = __float2bfloat16_rn((tid & 15) < 9 ? P[kW1 + (tid >> 4) * 9 + (tid & 15)] : 0.f);
  if (tid < 16) S.b1[tid] = P[kB1 + tid];
  if (tid < 32) S.b2[tid] = P[kB2 + tid], S.b3[tid] = P[kB3 + tid];
  for (int i = tid; i < 2 * 18 * 18; i += kNnThreads) (&S.x[0][0][0])[i] = 0.f;
  if (tid < 2 * kS1) S.a1[tid / kS1][256][tid % kS1] = __float2bfloat16_rn(0.f);
  if (tid < 2 * kS2) S.a2[tid / kS2][64][tid % kS2] = __float2bfloat16_rn(0.f);
  __syncthreads();
  for (int b0 = 2 * blockIdx.x; b0 < batch; b0 += 2 * gridDim.x) {
    const int nb = min(2, batch - b0);
    for (int i = tid; i < nb * kF; i += kNnThreads) {
      const int s = i / kF, k = i - s * kF;
      const float v = X[(long long)(b0 + s) * kF + k];
      if (k < 256) {
        xs[(long long)(b0 + s) * kXs + k] = v;
        S.x[s][1 + (k >> 4)][1 + (k & 15)] = rbf(v);
      } else {
        h0[(long long)(b0 + s) * kH0 + 256 + k] = v;  // features 256 .. 375 behind the 512 of the convolution
      }
    }
    __syncthreads();
    const int s = warp >> 2, q = warp & 3;  // the warp's sample, and its quarter of the work
    {  // 3x3, 1 -> 16: four rows of 16 positions a warp, a row one product of its nine taps
      uint32_t w[4];
#pragma unroll
      for (int j = 0; j < 4; j++) w[j] = *reinterpret_cast<const uint32_t*>(&S.w1[(j >> 1) * 8 + g][2 * t + (j & 1) * 8]);
      const int k0 = 2 * t, k1 = 2 * t + 1;
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int y = q * 4 + i;
        uint32_t a[4];
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int x = g + 8 * h;
          a[h] = pack2(S.x[s][y + k0 / 3][x + k0 % 3], S.x[s][y + k1 / 3][x + k1 % 3]);
          a[2 + h] = t == 0 ? pack2(S.x[s][y + 2][x + 2], 0.f) : 0u;
        }
        float acc[2][4] = {};
        mma16816(acc[0], a, w[0], w[1]);
        mma16816(acc[1], a, w[2], w[3]);
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int r = y * 16 + g + 8 * h, n = j * 8 + 2 * t;
            const float v0 = fmaxf(acc[j][2 * h] + S.b1[n], 0.f), v1 = fmaxf(acc[j][2 * h + 1] + S.b1[n + 1], 0.f);
            *reinterpret_cast<uint32_t*>(&S.a1[s][r][n]) = pack2(v0, v1);
            if (s < nb) *reinterpret_cast<float2*>(a1g + (long long)(b0 + s) * kA1 + r * 16 + n) = make_float2(v0, v1);
          }
      }
    }
    __syncthreads();
    {  // 3x3 stride 2, 16 -> 32: 16 output positions a warp
      float acc[4][4] = {};
      const int pos = q * 16 + (lane & 15), kc = (lane >> 4) * 8;
      for (int k = 0; k < 9; k++) {
        uint32_t a[4], w[8];
        ldsm4<false>(a, &S.a1[s][tap_row<16>(pos >> 3, pos & 7, k / 3, k % 3)][kc]);
        const bf16* wp = S.w2 + ((lane & 7) + (lane >> 4) * 8) * kSw2 + k * 16 + ((lane >> 3) & 1) * 8;
        ldsm4<false>(w, wp);
        ldsm4<false>(w + 4, wp + 16 * kSw2);
#pragma unroll
        for (int j = 0; j < 4; j++) mma16816(acc[j], a, w[2 * j], w[2 * j + 1]);
      }
#pragma unroll
      for (int j = 0; j < 4; j++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = q * 16 + g + 8 * h, n = j * 8 + 2 * t;
          const float v0 = fmaxf(acc[j][2 * h] + S.b2[n], 0.f), v1 = fmaxf(acc[j][2 * h + 1] + S.b2[n + 1], 0.f);
          *reinterpret_cast<uint32_t*>(&S.a2[s][r][n]) = pack2(v0, v1);
          if (s < nb) *reinterpret_cast<float2*>(a2g + (long long)(b0 + s) * kA2 + r * 32 + n) = make_float2(v0, v1);
        }
    }
    __syncthreads();
    {  // 3x3 stride 2, 32 -> 32: eight channels a warp
      float acc[4] = {};
      const int pos = lane & 15, kc = (lane >> 4) * 8;
      for (int k = 0; k < 9; k++) {
        uint32_t a[4], w[4];
        const bf16* row = S.a2[s][tap_row<8>(pos >> 2, pos & 3, k / 3, k % 3)];
        ldsm4<false>(w, S.w3 + (q * 8 + (lane & 7)) * kSw3 + k * 32 + (lane >> 3) * 8);
        ldsm4<false>(a, row + kc);
        mma16816(acc, a, w[0], w[1]);
        ldsm4<false>(a, row + 16 + kc);
        mma16816(acc, a, w[2], w[3]);
      }
      if (s < nb) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int r = g + 8 * h, n = q * 8 + 2 * t;
          *reinterpret_cast<float2*>(h0 + (long long)(b0 + s) * kH0 + r * 32 + n) =
              make_float2(fmaxf(acc[2 * h] + S.b3[n], 0.f), fmaxf(acc[2 * h + 1] + S.b3[n + 1], 0.f));
        }
      }
    }
  }
}

// ---- forward: the dense layers, 32 samples a CTA ----
constexpr int kRows = 32, kKc = 128;  // samples a CTA; the first layer's inputs a step
struct DenseSmem {
  bf16 h0[kRows][648];         // inputs 632 .. 639 zero
  bf16 w4[64][kKc + 8];
  bf16 a4[kRows][72], w5[24][72];
};

__global__ void __launch_bounds__(kNnThreads) k_dense_forward(const float* __restrict__ P, const float* __restrict__ h0,
                                                              int batch, float* a4g, float* logits) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  DenseSmem& S = *reinterpret_cast<DenseSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int b0 = blockIdx.x * kRows, mt = warp & 1, np = warp >> 1;  // the warp's 16 samples, 16 outputs
#pragma unroll 5
  for (int i = tid; i < kRows * 160; i += kNnThreads) {  // four inputs at a time (h0's rows are 16-byte aligned)
    const int r = i / 160, k = 4 * (i - r * 160);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (b0 + r < batch && k < kH0) v = *reinterpret_cast<const float4*>(h0 + (long long)(b0 + r) * kH0 + k);
    *reinterpret_cast<uint2*>(&S.h0[r][k]) = make_uint2(pack2(v.x, v.y), pack2(v.z, v.w));
  }
  for (int i = tid; i < 24 * 64; i += kNnThreads) S.w5[i >> 6][i & 63] = __float2bfloat16_rn(P[kW5 + i]);
  // sums of 80 inputs, added up in FP32 (the tensor cores' accumulators round towards zero), the first and
  // the bias last
  float acc[2][4] = {}, first[2][4], sum[2][4] = {};
  for (int k0 = 0; k0 < 640; k0 += kKc) {
    __syncthreads();
#pragma unroll 16
    for (int i = tid; i < 64 * kKc; i += kNnThreads) {
      const int o = i / kKc, k = i - o * kKc;
      S.w4[o][k] = __float2bfloat16_rn(k0 + k < kH0 ? P[kW4 + o * kH0 + k0 + k] : 0.f);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kKc; k += 16) {
      uint32_t a[4], w[4];
      ldsm4<false>(a, &S.h0[mt * 16 + (lane & 15)][k0 + k + (lane >> 4) * 8]);
      ldsm4<false>(w, &S.w4[np * 16 + (lane & 7) + (lane >> 4) * 8][k + ((lane >> 3) & 1) * 8]);
      mma16816(acc[0], a, w[0], w[1]);
      mma16816(acc[1], a, w[2], w[3]);
      if ((k0 + k + 16) % 80 == 0) {
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int q = 0; q < 4; q++) {
            if (k0 + k < 80) first[j][q] = acc[j][q] + P[kB4 + np * 16 + j * 8 + 2 * t + (q & 1)];
            else sum[j][q] += acc[j][q];
            acc[j][q] = 0.f;
          }
      }
    }
  }
#pragma unroll
  for (int j = 0; j < 2; j++)
#pragma unroll
    for (int h = 0; h < 2; h++) {
      const int r = mt * 16 + g + 8 * h, n = np * 16 + j * 8 + 2 * t;
      const float v0 = fmaxf(sum[j][2 * h] + first[j][2 * h], 0.f), v1 = fmaxf(sum[j][2 * h + 1] + first[j][2 * h + 1], 0.f);
      *reinterpret_cast<uint32_t*>(&S.a4[r][n]) = pack2(v0, v1);
      if (b0 + r < batch) *reinterpret_cast<float2*>(a4g + (long long)(b0 + r) * kA4 + n) = make_float2(v0, v1);
    }
  __syncthreads();
  if (np < 3) {  // 64 -> 24
    float z[4] = {};
#pragma unroll
    for (int k = 0; k < 64; k += 16) {
      uint32_t a[4], w[2];
      ldsm4<false>(a, &S.a4[mt * 16 + (lane & 15)][k + (lane >> 4) * 8]);
      ldsm2<false>(w, &S.w5[np * 8 + (lane & 7)][k + ((lane >> 3) & 1) * 8]);
      mma16816(z, a, w[0], w[1]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = b0 + mt * 16 + g + (q >> 1) * 8, n = np * 8 + 2 * t + (q & 1);
      if (r < batch) logits[(long long)r * kOut + n] = z[q] + P[kB5 + n];
    }
  }
}

// ---- backward: the dense layers' input gradients, 32 samples a CTA ----
struct DenseBackSmem {
  bf16 dl[kRows][40], w5[32][72];  // outputs 24 .. 31 zero
  bf16 dz4[kRows][72], w4[64][kKc + 8];
};

// dz4 = dlogits W5 where the hidden unit is positive; dz3 = dz4 W4 (its first 512 inputs) where the
// convolution's output is.
__global__ void __launch_bounds__(kNnThreads) k_dense_backward(const float* __restrict__ P, const float* __restrict__ dlogits,
                                                               const float* __restrict__ a4g, const float* __restrict__ h0,
                                                               int batch, float* dz4g, float* dz3g) {
  __shared__ __align__(16) DenseBackSmem S;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int b0 = blockIdx.x * kRows, mt = warp & 1, np = warp >> 1;
  for (int i = tid; i < kRows * 32; i += kNnThreads) {
    const int r = i >> 5, k = i & 31;
    S.dl[r][k] = __float2bfloat16_rn(b0 + r < batch && k < kOut ? dlogits[(long long)(b0 + r) * kOut + k] : 0.f);
  }
  for (int i = tid; i < 32 * 64; i += kNnThreads) S.w5[i >> 6][i & 63] = __float2bfloat16_rn(i < kOut * 64 ? P[kW5 + i] : 0.f);
  __syncthreads();
  {
    float acc[2][4] = {};
#pragma unroll
    for (int k = 0; k < 32; k += 16) {
      uint32_t a[4], w[4];
      ldsm4<false>(a, &S.dl[mt * 16 + (lane & 15)][k + (lane >> 4) * 8]);
      ldsm4<true>(w, &S.w5[k + (lane & 15)][np * 16 + (lane >> 4) * 8]);
      mma16816(acc[0], a, w[0], w[1]);
      mma16816(acc[1], a, w[2], w[3]);
    }
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = mt * 16 + g + 8 * h, n = np * 16 + j * 8 + 2 * t;
        float2 m = make_float2(0.f, 0.f);
        const long long o = (long long)(b0 + r) * kA4 + n;
        if (b0 + r < batch) m = *reinterpret_cast<const float2*>(a4g + o);
        const float v0 = m.x > 0.f ? acc[j][2 * h] : 0.f, v1 = m.y > 0.f ? acc[j][2 * h + 1] : 0.f;
        *reinterpret_cast<uint32_t*>(&S.dz4[r][n]) = pack2(v0, v1);
        if (b0 + r < batch) *reinterpret_cast<float2*>(dz4g + o) = make_float2(v0, v1);
      }
  }
  for (int n0 = 0; n0 < 512; n0 += kKc) {
    __syncthreads();
#pragma unroll 16
    for (int i = tid; i < 64 * kKc; i += kNnThreads) {
      const int o = i / kKc, k = i - o * kKc;
      S.w4[o][k] = __float2bfloat16_rn(P[kW4 + o * kH0 + n0 + k]);
    }
    __syncthreads();
    float acc[4][4] = {};
#pragma unroll
    for (int k = 0; k < 64; k += 16) {
      uint32_t a[4], w[8];
      ldsm4<false>(a, &S.dz4[mt * 16 + (lane & 15)][k + (lane >> 4) * 8]);
      const bf16* wp = &S.w4[k + (lane & 15)][np * 32 + (lane >> 4) * 8];
      ldsm4<true>(w, wp);
      ldsm4<true>(w + 4, wp + 16);
#pragma unroll
      for (int j = 0; j < 4; j++) mma16816(acc[j], a, w[2 * j], w[2 * j + 1]);
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const int r = b0 + mt * 16 + g + 8 * h, n = n0 + np * 32 + j * 8 + 2 * t;
        if (r >= batch) continue;
        const float2 m = *reinterpret_cast<const float2*>(h0 + (long long)r * kH0 + n);
        *reinterpret_cast<float2*>(dz3g + (long long)r * kDz3 + n) =
            make_float2(m.x > 0.f ? acc[j][2 * h] : 0.f, m.y > 0.f ? acc[j][2 * h + 1] : 0.f);
      }
  }
}

// ---- backward: a dense layer's weight and bias gradients ----
// G[m][n] += sum over samples b of D[b][m] H[b][n] (m < M <= 64, n < N), B[m] += sum of D[b][m] (FP32). CTA
// (x, y): columns 64 x .., samples y * per ..
__global__ void __launch_bounds__(kNnThreads) k_dense_weights(const float* __restrict__ D, int M, const float* __restrict__ H,
                                                              int N, int batch, int per, float* G, float* B) {
  __shared__ __align__(16) bf16 Ds[64][72], Hs[64][72];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * 64, b1 = min(batch, (int)(blockIdx.y + 1) * per), mt = warp & 3, nh = warp >> 2;
  const int col = tid & 63;
  float acc[4][4] = {}, bias = 0.f;
  for (int b0 = blockIdx.y * per; b0 < b1; b0 += 64) {
    __syncthreads();
#pragma unroll 8
    for (int r = tid >> 6; r < 64; r += 4) {
      const long long b = b0 + r;
      const float d = b < b1 && col < M ? D[b * M + col] : 0.f;
      Ds[r][col] = __float2bfloat16_rn(d);
      Hs[r][col] = __float2bfloat16_rn(b < b1 && n0 + col < N ? H[b * N + n0 + col] : 0.f);
      bias += d;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 64; k += 16) {
      uint32_t a[4], w[8];
      ldsm4<true>(a, &Ds[k + (lane & 7) + (lane >> 4) * 8][mt * 16 + ((lane >> 3) & 1) * 8]);
      const bf16* wp = &Hs[k + (lane & 15)][nh * 32 + (lane >> 4) * 8];
      ldsm4<true>(w, wp);
      ldsm4<true>(w + 4, wp + 16);
#pragma unroll
      for (int j = 0; j < 4; j++) mma16816(acc[j], a, w[2 * j], w[2 * j + 1]);
    }
  }
#pragma unroll
  for (int j = 0; j < 4; j++)
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int m = mt * 16 + g + (q >> 1) * 8, n = n0 + nh * 32 + j * 8 + 2 * t + (q & 1);
      if (m < M && n < N) atomicAdd(G + m * N + n, acc[j][q]);
    }
  if (blockIdx.x == 0 && col < M) atomicAdd(B + col, bias);
}

// Samples a CTA of k_dense_weights takes: `least` (a multiple of 64) while that makes at most 64 CTAs of them, then more.
// Every row group of every CTA is one more FP32 addition in a row to the same bias gradient: of 65,536 samples the second
// layer's was 1.3e-6 off its sum in 64 bits with 1,024 CTAs, 5.1e-7 with 64. A chain of products stays within 2,048.
// (Four row groups added up in shared memory first cost a step on 4,096 samples 10 us of 275.)
int dense_samples(int batch, int least) {
  const int per = (int)((batch + 64LL * 64 - 1) / (64 * 64)) * 64;
  return per < least ? least : per > 2048 ? 2048 : per;
}

// ---- backward: the convolutions, a sample at a time, their weight gradients over a CTA's samples ----
// The tensor cores' accumulators round towards zero, a loss that grows with every product added, so a chain of
// theirs is at most kChain samples (for W2, with 64 positions each, 2,048 products). Up to 32 samples a CTA (9,472 on
// 148 SMs) that is all of them; CHAINS, for more, puts the sums down every 32 and starts anew, and they meet in the FP32
// atomics: 65,536 samples' gradients of one sign 5.6e-5 (W2) and 2.3e-5 (W1) low with one chain, 3.0e-6 and 2.0e-6
// with these; 16,384 samples' backward pass 447 -> 507 us. (One kernel for both costs a step on 4,096 samples 2 us of
// 269; a launch for every 9,472 samples in its place takes 530.)
constexpr int kChain = 32;
struct BackSmem {
  bf16 w2[32 * kSw2], w3[32 * kSw3];
  bf16 a1[257][kS1], a2[65][kS2], dz3[17][kS2], dz2[65][kS2], dz1[256][kS1];
  bf16 cols[256][kS1];      // the first convolution's columns (nine taps, then zeros)
  float x[18][18];
  float bias[16 + 32 + 32];
};

template <bool CHAINS>
__global__ void __launch_bounds__(kNnThreads, 2) k_conv_backward(const float* __restrict__ P, const float* __restrict__ xs,
                                                                 const float* __restrict__ a1g, const float* __restrict__ a2g,
                                                                 const float* __restrict__ dz3g, int batch, float* G) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BackSmem& S = *reinterpret_cast<BackSmem*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  stage_conv_weights(P, S.w2, S.w3);
  const bf16 zero = __float2bfloat16_rn(0.f);
  if (tid < kS1) S.a1[256][tid] = zero;
  if (tid < kS2) S.a2[64][tid] = S.dz3[16][tid] = S.dz2[64][tid] = zero;
  if (tid < 80) S.bias[tid] = 0.f;
  for (int i = tid; i < 18 * 18; i += kNnThreads) (&S.x[0][0])[i] = 0.f;
  for (int i = tid; i < 256 * 16; i += kNnThreads) S.cols[i >> 4][i & 15] = zero;
  // this warp's share: weight gradients of 16 output channels (m2) and a run of 8-column tiles
  const int m2 = warp & 1, q = warp >> 1, t2 = q < 2 ? 5 * q : 10 + 4 * (q - 2), n2 = q < 2 ? 5 : 4;
  float s3[2] = {}, s2[2] = {}, s1[4] = {};  // bias sums
  int b = blockIdx.x;
  do {
  float g3[9][4] = {}, g2[5][4] = {}, g1[2][4] = {};
  for (int i = 0; (!CHAINS || i < kChain) && b < batch; i++, b += gridDim.x) {
    __syncthreads();  // the sample before is done with
    {
      const float4* v = reinterpret_cast<const float4*>(a1g + (long long)b * kA1);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int e = tid + i * kNnThreads;
        const float4 f = v[e];
        *reinterpret_cast<uint2*>(&S.a1[e >> 2][(e & 3) * 4]) = make_uint2(pack2(f.x, f.y), pack2(f.z, f.w));
      }
      const float4* u = reinterpret_cast<const float4*>(a2g + (long long)b * kA2);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        const int e = tid + i * kNnThreads;
        const float4 f = u[e];
        *reinterpret_cast<uint2*>(&S.a2[e >> 3][(e & 7) * 4]) = make_uint2(pack2(f.x, f.y), pack2(f.z, f.w));
      }
      const float2 d = reinterpret_cast<const float2*>(dz3g + (long long)b * kDz3)[tid];
      *reinterpret_cast<uint32_t*>(&S.dz3[tid >> 4][(tid & 15) * 2]) = pack2(d.x, d.y);
      s3[0] += d.x, s3[1] += d.y;
      S.x[1 + (tid >> 4)][1 + (tid & 15)] = xs[(long long)b * kXs + tid];
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < 9; k++) S.cols[tid][k] = __float2bfloat16_rn(S.x[(tid >> 4) + k / 3][(tid & 15) + k % 3]);
    {  // W3's gradient: dz3^T (32 x 16 positions) against the columns of a2, nine tiles a warp
      uint32_t a[4];
      ldsm4<true>(a, &S.dz3[(lane & 7) + (lane >> 4) * 8][m2 * 16 + ((lane >> 3) & 1) * 8]);
      const int pos = lane & 15;
#pragma unroll
      for (int j = 0; j < 9; j++) {
        const int n = q * 9 + j, k = n >> 2;
        uint32_t w[2];
        ldsm2<true>(w, &S.a2[tap_row<8>(pos >> 2, pos & 3, k / 3, k % 3)][(n & 3) * 8]);
        mma16816(g3[j], a, w[0], w[1]);
      }
    }
    // dz2: the gradient at a2, eight channels a warp. A position of the 8 x 8 map is read by the taps
    // whose parity is its own: even rows by ky = 1 alone, odd ones by ky = 0 (from the output below) and
    // 2 (from the one above), columns likewise -- four classes of 16 positions with 1, 2, 2 and 4 taps,
    // the last to one half of the warps, the others to the other half
    {
      const int nt = warp & 3, r = lane & 15, cy = r >> 2, cx = r & 3;
      for (int c = warp < 4 ? 3 : 0; c < (warp < 4 ? 4 : 3); c++) {
        const int py = c >> 1, px = c & 1;
        float acc[4] = {};
        for (int i = 0; i <= py; i++)
          for (int j = 0; j <= px; j++) {
            // output (cy + dy, cx + dx): the tap's own for an even position, for an odd one 0 -> below / right
            const int ky = py ? 2 * i : 1, kx = px ? 2 * j : 1, oy = cy + (py && i == 0), ox = cx + (px && j == 0);
            const bf16* row = S.dz3[oy < 4 && ox < 4 ? oy * 4 + ox : 16];
            const bf16* wp = S.w3 + (lane & 15) * kSw3 + (ky * 3 + kx) * 32 + nt * 8;
            uint32_t a[4], w[2];
            float tap[4] = {};
            ldsm4<false>(a, row + (lane >> 4) * 8);
            ldsm2<true>(w, wp);
            mma16816(tap, a, w[0], w[1]);
            ldsm4<false>(a, row + 16 + (lane >> 4) * 8);
            ldsm2<true>(w, wp + 16 * kSw3);
            mma16816(tap, a, w[0], w[1]);
#pragma unroll
            for (int e = 0; e < 4; e++) acc[e] += tap[e];  // (the taps' sum in FP32)
          }
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const int pr = g + 8 * h, p = (2 * (pr >> 2) + py) * 8 + 2 * (pr & 3) + px, n = nt * 8 + 2 * t;
          const uint32_t m = *reinterpret_cast<const uint32_t*>(&S.a2[p][n]);  // (ReLU outputs: positive or zero)
          const float v0 = m & 0xffffu ? acc[2 * h] : 0.f, v1 = m >> 16 ? acc[2 * h + 1] : 0.f;
          *reinterpret_cast<uint32_t*>(&S.dz2[p][n]) = pack2(v0, v1);
          s2[0] += v0, s2[1] += v1;
        }
      }
    }
    __syncthreads();
    // W2's gradient: dz2^T (32 x 64 positions) against the columns of a1
#pragma unroll
    for (int kk = 0; kk < 4; kk++) {
      uint32_t a[4];
      ldsm4<true>(a, &S.dz2[kk * 16 + (lane & 7) + (lane >> 4) * 8][m2 * 16 + ((lane >> 3) & 1) * 8]);
      const int pos = kk * 16 + (lane & 15);
#pragma unroll
      for (int j = 0; j < 5; j++) {
        if (j >= n2) break;
        const int n = t2 + j, k = n >> 1;
        uint32_t w[2];
        ldsm2<true>(w, &S.a1[tap_row<16>(pos >> 3, pos & 7, k / 3, k % 3)][(n & 1) * 8]);
        mma16816(g2[j], a, w[0], w[1]);
      }
    }
    // dz1: the gradient at a1, 16 positions of a class (two of its eight rows) and all 16 channels a warp
    {
      const int mt = warp & 3, r = mt * 16 + (lane & 15), cy = r >> 3, cx = r & 7;
      for (int c = warp < 4 ? 3 : 0; c < (warp < 4 ? 4 : 3); c++) {
        const int py = c >> 1, px = c & 1;
        float acc[2][4] = {};
        for (int i = 0; i <= py; i++)
          for (int j = 0; j <= px; j++) {
            const int ky = py ? 2 * i : 1, kx = px ? 2 * j : 1, oy = cy + (py && i == 0), ox = cx + (px && j == 0);
            const bf16* row = S.dz2[oy < 8 && ox < 8 ? oy * 8 + ox : 64];
            const bf16* wp = S.w2 + (lane & 15) * kSw2 + (ky * 3 + kx) * 16 + (lane >> 4) * 8;
            uint32_t a[4], w[4];
            float tap[2][4] = {};
#pragma unroll
            for (int k = 0; k < 32; k += 16) {
              ldsm4<false>(a, row + k + (lane >> 4) * 8);
              ldsm4<true>(w, wp + k * kSw2);
              mma16816(tap[0], a, w[0], w[1]);
              mma16816(tap[1], a, w[2], w[3]);
            }
#pragma unroll
            for (int e = 0; e < 8; e++) acc[e >> 2][e & 3] += tap[e >> 2][e & 3];  // (the taps' sum in FP32)
          }
#pragma unroll
        for (int j = 0; j < 2; j++)
#pragma unroll
          for (int h = 0; h < 2; h++) {
            const int pr = mt * 16 + g + 8 * h, p = (2 * (pr >> 3) + py) * 16 + 2 * (pr & 7) + px, n = j * 8 + 2 * t;
            const uint32_t m = *reinterpret_cast<const uint32_t*>(&S.a1[p][n]);
            const float v0 = m & 0xffffu ? acc[j][2 * h] : 0.f, v1 = m >> 16 ? acc[j][2 * h + 1] : 0.f;
            *reinterpret_cast<uint32_t*>(&S.dz1[p][n]) = pack2(v0, v1);
            s1[2 * j] += v0, s1[2 * j + 1] += v1;
          }
      }
    }
    __syncthreads();
    // W1's gradient: dz1^T (16 x 256 positions) against the image's columns, 32 positions a warp
#pragma unroll
    for (int kk = 2 * warp; kk < 2 * warp + 2; kk++) {
      uint32_t a[4], w[4];
      ldsm4<true>(a, &S.dz1[kk * 16 + (lane & 7) + (lane >> 4) * 8][((lane >> 3) & 1) * 8]);
      ldsm4<true>(w, &S.cols[kk * 16 + (lane & 15)][(lane >> 4) * 8]);
      mma16816(g1[0], a, w[0], w[1]);
      mma16816(g1[1], a, w[2], w[3]);
    }
  }
  __syncthreads();
  // the chain's sums into the gradient vector
#pragma unroll
  for (int e = 0; e < 4; e++) {
    const int m = m2 * 16 + g + (e >> 1) * 8, c = 2 * t + (e & 1);
#pragma unroll
    for (int j = 0; j < 9; j++) atomicAdd(G + kW3 + m * 288 + (q * 9 + j) * 8 + c, g3[j][e]);
#pragma unroll
    for (int j = 0; j < 5; j++)
      if (j < n2) atomicAdd(G + kW2 + m * 144 + (t2 + j) * 8 + c, g2[j][e]);
    const int m1 = g + (e >> 1) * 8;
    atomicAdd(G + kW1 + m1 * 9 + c, g1[0][e]);
    if (c == 0) atomicAdd(G + kW1 + m1 * 9 + 8, g1[1][e]);
  }
  } while (CHAINS && b < batch);
  atomicAdd(&S.bias[48 + 2 * (tid & 15)], s3[0]), atomicAdd(&S.bias[48 + 2 * (tid & 15) + 1], s3[1]);
  atomicAdd(&S.bias[16 + (warp & 3) * 8 + 2 * t], s2[0]), atomicAdd(&S.bias[16 + (warp & 3) * 8 + 2 * t + 1], s2[1]);
#pragma unroll
  for (int j = 0; j < 4; j++) atomicAdd(&S.bias[(j >> 1) * 8 + 2 * t + (j & 1)], s1[j]);
  __syncthreads();
  if (tid < 16) atomicAdd(G + kB1 + tid, S.bias[tid]);
  if (tid < 32) atomicAdd(G + kB2 + tid, S.bias[16 + tid]), atomicAdd(G + kB3 + tid, S.bias[48 + tid]);
}

__global__ void k_bce(const float* __restrict__ z, const float* __restrict__ y, const float* __restrict__ w, int n,
                      float inv_batch, float* __restrict__ dz, float* loss) {
  __shared__ float part[256];
  float l = 0.f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float v = z[i], t = y[i], wt = w[i];
    const float sig = 1.f / (1.f + expf(-v));
    l += wt * (fmaxf(v, 0.f) - v * t + log1pf(expf(-fabsf(v))));
    dz[i] = wt * (sig - t) * inv_batch;
  }
  part[threadIdx.x] = l;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) part[threadIdx.x] += part[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, part[0] * inv_batch);
}

__global__ void k_adam(float* p, const float* __restrict__ g, float* m, float* v, int n, float lr, float b1, float b2,
                       float eps, float wd, float c1, float c2) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi, v[i] = vi;
    p[i] -= lr * ((mi / c1) / (sqrtf(vi / c2) + eps) + wd * p[i]);
  }
}

int grid_for(long long n) {
  const long long g = (n + 255) / 256;
  return (int)(g < 148 * 16 ? (g < 1 ? 1 : g) : 148 * 16);
}

// CTAs of a kernel that loops over its samples: as many as the GPU holds, at most `units`.
template <typename K>
int resident(K kernel, size_t smem, int units) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  return persistent_grid((const void*)kernel, kNnThreads, smem, units);
}

void forward(const float* P, const float* x, int batch, float* acts, cudaStream_t st) {
  Cache c(acts, batch);
  const int grid = resident(k_conv_forward, sizeof(FwdSmem), (batch + 1) / 2);
  k_conv_forward<<<grid, kNnThreads, sizeof(FwdSmem), st>>>(P, x, batch, c.xs, c.a1, c.a2, c.h0);
  const int blocks = (batch + kRows - 1) / kRows;
  resident(k_dense_forward, sizeof(DenseSmem), blocks);
  k_dense_forward<<<blocks, kNnThreads, sizeof(DenseSmem), st>>>(P, c.h0, batch, c.a4, c.logits);
}

void backward(const float* P, int batch, const float* acts, const float* dlogits, float* work, float* G,
              cudaStream_t st) {
  Cache c(const_cast<float*>(acts), batch);
  float* dz4 = aligned16(work);
  float* dz3 = dz4 + (long long)batch * kDz4;
  cudaMemsetAsync(G, 0, kParams * sizeof(float), st);  // every gradient is a sum of CTAs' sums
  const int blocks = (batch + kRows - 1) / kRows;
  k_dense_backward<<<blocks, kNnThreads, 0, st>>>(P, dlogits, c.a4, c.h0, batch, dz4, dz3);
  // the dense layers' weights: from 256 samples a CTA for the first (ten column tiles), from 64 for the second
  const int p4 = dense_samples(batch, 256), p5 = dense_samples(batch, 64);
  k_dense_weights<<<dim3((kH0 + 63) / 64, (batch + p4 - 1) / p4), kNnThreads, 0, st>>>(dz4, 64, c.h0, kH0, batch, p4,
                                                                                       G + kW4, G + kB4);
  k_dense_weights<<<dim3(1, (batch + p5 - 1) / p5), kNnThreads, 0, st>>>(dlogits, kOut, c.a4, 64, batch, p5, G + kW5,
                                                                          G + kB5);
  const auto conv = [&](auto kernel) {
    const int grid = resident(kernel, sizeof(BackSmem), batch);
    kernel<<<grid, kNnThreads, sizeof(BackSmem), st>>>(P, c.xs, c.a1, c.a2, dz3, batch, G);
  };
  const int full = resident(k_conv_backward<false>, sizeof(BackSmem), INT_MAX);
  if (batch <= (long long)full * kChain) conv(k_conv_backward<false>);
  else conv(k_conv_backward<true>);
}

}  // namespace nn

// ---- features and masks (the engine side) ----

__device__ __forceinline__ int entry_of(const NetList& l, int sb) {
  int i = 0;
  while (i + 1 < l.n && sb >= l.prefix[i + 1]) i++;
  return i;
}

// One CTA (128 threads) per superblock of the batch: the luma at level 2, the level-1 cost map per
// reference (a thread per cell and reference, rows as words where they lie inside the margins), presence
// flags and lambda (include/celv2_pruner.h).
__global__ void __launch_bounds__(128) k_features(const FrameJob* __restrict__ jobs, NetList l) {
  const int en = entry_of(l, blockIdx.x);
  const FrameJob& job = jobs[l.e[en].job];
  const int sb = blockIdx.x - l.prefix[en], tid = threadIdx.x;
  const int sby = sb / job.sb_cols, sbx = sb - sby * job.sb_cols;
  float* f = l.e[en].feats + (long long)sb * nn::kF;
  __shared__ int red[4];
  const DevPlane& l2 = job.cur.lv[2];
  const int v0 = at(l2, sby * 16 + (tid >> 4), sbx * 16 + (tid & 15));
  const int v1 = at(l2, sby * 16 + 8 + (tid >> 4), sbx * 16 + (tid & 15));
  const int sum = __reduce_add_sync(0xffffffffu, v0 + v1);  // whole numbers: exact in any order
  if ((tid & 31) == 0) red[tid >> 5] = sum;
  __syncthreads();
  const float mean = (float)(red[0] + red[1] + red[2] + red[3]) / 256.f;
  f[tid] = ((float)v0 - mean) / 64.f;
  f[128 + tid] = ((float)v1 - mean) / 64.f;
  if (tid < kMaxRefs * 16) {
    const int r = tid >> 4, cell = tid & 15;
    float v = 0.f;
    if (r < job.nrefs) {
      const int cols = job.fcols[1], rows = job.frows[1];
      const int cx = min(sbx * 4 + (cell & 3), cols - 1), cy = min(sby * 4 + (cell >> 2), rows - 1);
      const int m = job.field[r][1][cy * cols + cx], x = cx * 8 + mv_x(m), y = cy * 8 + mv_y(m);
      const DevPlane &cur = job.cur.lv[1], &ref = job.ref[r].lv[1];
      unsigned sad = 0;
      if (inside(cur, cx * 8, cy * 8, 8, 8) && inside(ref, x, y, 8, 8)) {
        const uint8_t *pc = cur.p + (long long)cy * 8 * cur.stride + cx * 8, *pr = ref.p + (long long)y * ref.stride + x;
#pragma unroll
        for (int i = 0; i < 8; i++)
#pragma unroll
          for (int h = 0; h < 2; h++)
            sad += __vsadu4(load4_pair(pc + (long long)i * cur.stride + 4 * h), load4_pair(pr + (long long)i * ref.stride + 4 * h));
      } else {
        for (int i = 0; i < 8; i++)
          for (int j = 0; j < 8; j++) sad += abs(at(cur, cy * 8 + i, cx * 8 + j) - at(ref, y + i, x + j));
      }
      v = log2f(1.f + (float)sad) / 14.f;
    }
    f[256 + tid] = v;
  }
  if (tid < kMaxRefs) f[368 + tid] = tid < job.nrefs ? 1.f : 0.f;
  if (tid == 0) f[375] = log2f((float)(job.lam > 1 ? job.lam : 1)) / 20.f;
}

void launch_features(const FrameJob* jobs, const NetList& l, cudaStream_t st) {
  if (l.prefix[l.n] > 0) k_features<<<l.prefix[l.n], 128, 0, st>>>(jobs, l);
}

// The keep word (include/celv2_decision.h) of one superblock from its logits: reference r kept
// where sigmoid >= th.ref (the likeliest reference always), intra where >= th.intra, block level l
// where >= th.level (the likeliest level always), and with intra the modes DC, V, H (their scoring
// costs next to nothing) and each other mode m where >= th.mode; everything where one of the
// reference, intra or level outputs lies within th.band of its threshold (the fallback to the full
// search).
__device__ __forceinline__ uint32_t mask_word(const float* z, int nrefs, const PrunerThresholds& th) {
  unsigned k = 0;
  int best = 0, lbest = 0;
  float pbest = -1.f, plbest = -1.f;
  bool unsure = false;
  for (int r = 0; r < nrefs; r++) {
    const float p = 1.f / (1.f + expf(-z[r]));
    if (p >= th.ref) k |= 1u << r;
    if (p > pbest) pbest = p, best = r;
    unsure |= fabsf(p - th.ref) < th.band;
  }
  k |= 1u << best;
  const float pi = 1.f / (1.f + expf(-z[7]));
  if (pi >= th.intra) k |= CELV2_KEEP_INTRA;
  unsure |= fabsf(pi - th.intra) < th.band;
  for (int l = 0; l < 4; l++) {
    const float p = 1.f / (1.f + expf(-z[8 + l]));
    if (p >= th.level) k |= CELV2_KEEP_LEVEL(l);
    if (p > plbest) plbest = p, lbest = l;
    unsure |= fabsf(p - th.level) < th.band;
  }
  k |= CELV2_KEEP_LEVEL(lbest);
  if (k & CELV2_KEEP_INTRA) {
    k |= CELV2_KEEP_MODE(0) | CELV2_KEEP_MODE(1) | CELV2_KEEP_MODE(2);
    for (int m = 3; m < kModes; m++)
      if (1.f / (1.f + expf(-z[12 + m - 3])) >= th.mode) k |= CELV2_KEEP_MODE(m);
  }
  return unsure ? 0xFFFFFFFFu : k;
}

// ---- the engine's inference: the whole network for one superblock per CTA, then its mask ----
// The same arithmetic as nn::forward (BF16 operands, FP32 sums; only the order of the sums
// differs): the 3x3 convolution 1 -> 16 and the dense layers on the CUDA cores (bf16-rounded
// operands), the two strided convolutions (85% of the FLOPs) as mma.sync m16n8k16 tiles whose A
// operand is read straight from the previous activation in shared memory (an implicit im2col).
// Weights: bf16 copies made once (infer_weights), W4 transposed so a CTA's 64 threads read rows. All the
// superblocks of a batch go in one launch, as their features do: five 1080p jobs 218 -> 123 us (a pair of
// launches a job, 510 CTAs each, left the GPU with little in flight). The sums' order is fixed: a keep word
// follows from comparisons of what they give.
namespace nn {
constexpr int kIW2 = 0, kIW3 = kIW2 + 32 * 144, kIW4 = kIW3 + 32 * 288, kIWs = kIW4 + 632 * 64;  // bf16 elements

__global__ void k_infer_weights(const float* __restrict__ P, __nv_bfloat16* __restrict__ Wb) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kIWs; i += gridDim.x * blockDim.x) {
    float v;
    if (i < kIW3) v = P[kW2 + i];
    else if (i < kIW4) v = P[kW3 + (i - kIW3)];
    else {
      const int r = i - kIW4, k = r / 64, o = r - k * 64;  // W4t[k][o] = W4[o][k]
      v = P[kW4 + o * 632 + k];
    }
    Wb[i] = __float2bfloat16_rn(v);
  }
}

__global__ void __launch_bounds__(128) k_infer(NetList l) {
  __shared__ float xr[kF];                            // the features, bf16-rounded
  __shared__ float img[18][18], w1[9][16];            // the image with a border of zeros; conv1's weights, rounded
  __shared__ __align__(16) bf16 a1[256][16];           // conv1 output, (y, x) rows, channels
  __shared__ __align__(16) bf16 a2[64][32];
  __shared__ float h0[632], a4[64], part[128];
  __shared__ float logits[kOut];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int en = entry_of(l, blockIdx.x), sb = blockIdx.x - l.prefix[en];
  const float* __restrict__ P = l.e[en].params;
  const bf16* __restrict__ Wb = static_cast<const bf16*>(l.e[en].wb);
  const float* x = l.e[en].feats + (long long)sb * kF;
  for (int i = tid; i < 18 * 18; i += 128) (&img[0][0])[i] = 0.f;
  for (int i = tid; i < 144; i += 128) w1[i % 9][i / 9] = rbf(P[kW1 + i]);
  __syncthreads();
  for (int i = tid; i < kF; i += 128) {
    const float v = rbf(x[i]);
    xr[i] = v;
    if (i < 256) img[1 + (i >> 4)][1 + (i & 15)] = v;
  }
  __syncthreads();
  // conv 3x3 1 -> 16, stride 1: a thread a channel, every eighth position (taps outside add nothing, whatever
  // the weights)
  {
    const int c = tid & 15;
    const float b = P[kB1 + c];
    float w[9];
#pragma unroll
    for (int k = 0; k < 9; k++) w[k] = w1[k][c];
    for (int p = tid >> 4; p < 256; p += 8) {
      const int y = p >> 4, xx = p & 15;
      float s = 0.f;
#pragma unroll
      for (int k = 0; k < 9; k++)
        if (!((k < 3 && y == 0) || (k >= 6 && y == 15) || (k % 3 == 0 && xx == 0) || (k % 3 == 2 && xx == 15)))
          s += img[y + k / 3][xx + k % 3] * w[k];
      a1[p][c] = __float2bfloat16_rn(fmaxf(s + b, 0.f));
    }
  }
  __syncthreads();
  // conv 3x3 16 -> 32, stride 2: rows = 64 output positions (warp w: 16w..16w+15), K = tap x 16
  {
    float acc[4][4] = {};
    const int r0 = warp * 16 + g, r1 = r0 + 8;
    for (int tap = 0; tap < 9; tap++) {
      const int ky = tap / 3, kx = tap - ky * 3;
      uint32_t a[4];
      const int iy0 = (r0 >> 3) * 2 + ky - 1, ix0 = (r0 & 7) * 2 + kx - 1;
      const int iy1 = (r1 >> 3) * 2 + ky - 1, ix1 = (r1 & 7) * 2 + kx - 1;
      const bool in0 = iy0 >= 0 && iy0 < 16 && ix0 >= 0 && ix0 < 16, in1 = iy1 >= 0 && iy1 < 16 && ix1 >= 0 && ix1 < 16;
      const uint32_t* q0 = reinterpret_cast<const uint32_t*>(a1[in0 ? iy0 * 16 + ix0 : 0]);
      const uint32_t* q1 = reinterpret_cast<const uint32_t*>(a1[in1 ? iy1 * 16 + ix1 : 0]);
      a[0] = in0 ? q0[t] : 0u, a[1] = in1 ? q1[t] : 0u, a[2] = in0 ? q0[t + 4] : 0u, a[3] = in1 ? q1[t + 4] : 0u;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t* w = reinterpret_cast<const uint32_t*>(Wb + kIW2 + (j * 8 + g) * 144 + tap * 16);
        mma16816(acc[j], a, __ldg(w + t), __ldg(w + t + 4));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int r = q < 2 ? r0 : r1, n = j * 8 + 2 * t + (q & 1);
        a2[r][n] = __float2bfloat16_rn(fmaxf(acc[j][q] + P[kB2 + n], 0.f));
      }
  }
  __syncthreads();
  // conv 3x3 32 -> 32, stride 2: 16 output positions, warp w: output channels 8w..8w+7, K = tap x 32
  {
    float acc[4] = {};
    const int r0 = g, r1 = g + 8;
    for (int s = 0; s < 18; s++) {
      const int tap = s >> 1, c0 = (s & 1) * 16, ky = tap / 3, kx = tap - ky * 3;
      uint32_t a[4];
      const int iy0 = (r0 >> 2) * 2 + ky - 1, ix0 = (r0 & 3) * 2 + kx - 1;
      const int iy1 = (r1 >> 2) * 2 + ky - 1, ix1 = (r1 & 3) * 2 + kx - 1;
      const bool in0 = iy0 >= 0 && iy0 < 8 && ix0 >= 0 && ix0 < 8, in1 = iy1 >= 0 && iy1 < 8 && ix1 >= 0 && ix1 < 8;
      const uint32_t* q0 = reinterpret_cast<const uint32_t*>(&a2[in0 ? iy0 * 8 + ix0 : 0][c0]);
      const uint32_t* q1 = reinterpret_cast<const uint32_t*>(&a2[in1 ? iy1 * 8 + ix1 : 0][c0]);
      a[0] = in0 ? q0[t] : 0u, a[1] = in1 ? q1[t] : 0u, a[2] = in0 ? q0[t + 4] : 0u, a[3] = in1 ? q1[t + 4] : 0u;
      const uint32_t* w = reinterpret_cast<const uint32_t*>(Wb + kIW3 + (warp * 8 + g) * 288 + tap * 32 + c0);
      mma16816(acc, a, __ldg(w + t), __ldg(w + t + 4));
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int r = q < 2 ? r0 : r1, n = warp * 8 + 2 * t + (q & 1);
      h0[r * 32 + n] = rbf(fmaxf(acc[q] + P[kB3 + n], 0.f));  // the dense layer reads it as BF16
    }
  }
  for (int i = tid; i < 120; i += 128) h0[512 + i] = xr[256 + i];
  __syncthreads();
  // dense 632 -> 64: thread (o, half) sums half of the row
  {
    const int o = tid & 63, half = tid >> 6;
    float s = 0.f;
#pragma unroll 16
    for (int k = half * 316; k < half * 316 + 316; k++) s += h0[k] * __bfloat162float(Wb[kIW4 + k * 64 + o]);
    part[tid] = s;
  }
  __syncthreads();
  if (tid < 64) a4[tid] = rbf(fmaxf(part[tid] + part[tid + 64] + P[kB4 + tid], 0.f));
  __syncthreads();
  // dense 64 -> kOut: warp w, lanes sum over the 64 inputs for outputs w, w + 4, ...
  for (int o = warp; o < kOut; o += 4) {
    float s = a4[lane] * rbf(P[kW5 + o * 64 + lane]) + a4[lane + 32] * rbf(P[kW5 + o * 64 + lane + 32]);
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0) logits[o] = s + P[kB5 + o];
  }
  __syncthreads();
  if (tid == 0) l.e[en].keep[sb] = mask_word(logits, l.e[en].nrefs, l.e[en].th);
}
}  // namespace nn

// bf16 copies of the convolution and dense weights the inference kernel reads (nn::kIWs elements)
size_t infer_weight_elems() { return nn::kIWs; }
void infer_weights(const float* params, void* wb, cudaStream_t st) {
  nn::k_infer_weights<<<nn::grid_for(nn::kIWs), 256, 0, st>>>(params, static_cast<__nv_bfloat16*>(wb));
}
void launch_infer(const NetList& l, cudaStream_t st) {
  if (l.prefix[l.n] > 0) nn::k_infer<<<l.prefix[l.n], 128, 0, st>>>(l);
}

}  // namespace celv2cu

using namespace celv2cu;

namespace {

int fail(const char* what, cudaError_t e) {
  set_last_error(std::string(what) + ": " + cudaGetErrorString(e));
  return CELV2_ECUDA;
}

}  // namespace

extern "C" {

int celv2_pruner_forward(const float* params, const float* x, int batch, float* acts, void* stream) {
  if (!params || !x || !acts || batch <= 0) {
    set_last_error("pruner_forward: null buffer or empty batch");
    return CELV2_EINVAL;
  }
  nn::forward(params, x, batch, acts, static_cast<cudaStream_t>(stream));
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CELV2_OK : fail("pruner_forward", e);
}

int celv2_pruner_backward(const float* params, int batch, const float* acts, const float* dlogits, float* work,
                          float* grads, void* stream) {
  if (!params || !acts || !dlogits || !work || !grads || batch <= 0) {
    set_last_error("pruner_backward: null buffer or empty batch");
    return CELV2_EINVAL;
  }
  nn::backward(params, batch, acts, dlogits, work, grads, static_cast<cudaStream_t>(stream));
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CELV2_OK : fail("pruner_backward", e);
}

int celv2_pruner_bce(const float* logits, const float* labels, const float* weights, int batch, float* dlogits,
                     float* loss, void* stream) {
  if (!logits || !labels || !weights || !dlogits || !loss || batch <= 0) {
    set_last_error("pruner_bce: null buffer or empty batch");
    return CELV2_EINVAL;
  }
  const int n = batch * nn::kOut;
  nn::k_bce<<<nn::grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(logits, labels, weights, n,
                                                                             1.f / (float)batch, dlogits, loss);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CELV2_OK : fail("pruner_bce", e);
}

int celv2_pruner_adam(float* params, const float* grads, float* m, float* v, int n, float lr, float beta1,
                      float beta2, float eps, float weight_decay, int step, void* stream) {
  if (!params || !grads || !m || !v || n <= 0 || step < 1) {
    set_last_error("pruner_adam: null buffer, empty or step < 1");
    return CELV2_EINVAL;
  }
  double c1 = 1.0, c2 = 1.0;
  for (int i = 0; i < step && i < 100000; i++) c1 *= beta1, c2 *= beta2;
  nn::k_adam<<<nn::grid_for(n), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      params, grads, m, v, n, lr, beta1, beta2, eps, weight_decay, (float)(1.0 - c1), (float)(1.0 - c2));
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? CELV2_OK : fail("pruner_adam", e);
}

}  // extern "C"
