// mlp_kernels.cuh - the conflict predictor's network: 64 -> 128 -> 128 -> 1 (ReLU, ReLU,
// sigmoid), bf16 weights, fp32 accumulation, hand-written forward, backward and Adam kernels.
//
// Layout: features X [n][64] bf16 (0/1 indicators here, exact in bf16); weights W1 [64][128],
// W2 [128][128], w3 [128] in bf16 (rounded from fp32 master copies after every step), biases
// fp32. A CTA of 256 threads works on tiles of 64 samples with every operand in shared memory;
// thread (ty, tx) = (tid / 16, tid % 16) owns samples 4ty..4ty+3 x hidden units tx + 16b
// (b < 8) of an activation tile (interleaved so a warp's weight reads hit 16 distinct banks).
// Inference (every planned transaction) runs on the tensor cores (mlp_forward_tc_kernel, tcgen05
// with fp32 accumulation); training (the probe slice, a few percent of the chunk)
// runs its fused forward + backward tile GEMMs on the FP32 pipes. Both feed layer 2 with bf16
// activations, so they compute the same network.
#pragma once
#include <cuda_bf16.h>

#include <cstdint>

namespace csmv {

constexpr int kMlpIn = 64, kMlpHid = 128, kMlpTile = 64, kMlpThreads = 256;
// fp32 master parameter block: W1 | b1 | W2 | b2 | w3 | b3 (+3 pad)
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kMlpIn * kMlpHid, kOffW2 = kOffB1 + kMlpHid,
              kOffB2 = kOffW2 + kMlpHid * kMlpHid, kOffW3 = kOffB2 + kMlpHid,
              kOffB3 = kOffW3 + kMlpHid, kMlpParams = kOffB3 + 4;

// padded row strides (floats) keep the 4-sample column reads free of bank conflicts
constexpr int kXs = kMlpIn + 1, kHs = kMlpHid + 1;

struct MlpSmem {
  float w1[kMlpIn * kMlpHid];    // [k][j]
  float w2[kMlpHid * kHs];       // [i][j], row stride kHs
  float b1[kMlpHid], b2[kMlpHid], w3[kMlpHid];
  float x[kMlpTile * kXs];       // [s][k]
  float h1[kMlpTile * kHs];      // [s][i] post-ReLU, rounded to bf16
  float h2[kMlpTile * kHs];      // [s][j] post-ReLU, then dL/dh2 pre-activation
  float dz[kMlpTile];
  float b3;
};

__device__ __forceinline__ void mlp_load_weights(MlpSmem& sm, const __nv_bfloat16* w1,
                                                 const __nv_bfloat16* w2, const __nv_bfloat16* w3,
                                                 const float* bias) {
  for (int i = threadIdx.x; i < kMlpIn * kMlpHid; i += blockDim.x) sm.w1[i] = __bfloat162float(w1[i]);
  for (int i = threadIdx.x; i < kMlpHid * kMlpHid; i += blockDim.x)
    sm.w2[(i / kMlpHid) * kHs + i % kMlpHid] = __bfloat162float(w2[i]);
  for (int i = threadIdx.x; i < kMlpHid; i += blockDim.x) {
    sm.b1[i] = bias[kOffB1 + i];
    sm.b2[i] = bias[kOffB2 + i];
    sm.w3[i] = __bfloat162float(w3[i]);
  }
  if (threadIdx.x == 0) sm.b3 = bias[kOffB3];
}

// X tile -> smem (rows beyond n are zero)
__device__ __forceinline__ void mlp_load_x(MlpSmem& sm, const __nv_bfloat16* x, uint32_t s0,
                                           uint32_t n) {
  for (int i = threadIdx.x; i < kMlpTile * kMlpIn; i += blockDim.x) {
    const uint32_t s = i / kMlpIn, k = i % kMlpIn;
    sm.x[s * kXs + k] = (s0 + s < n) ? __bfloat162float(x[(size_t)(s0 + s) * kMlpIn + k]) : 0.f;
  }
}

// Forward of one tile; leaves h1, h2 (post-ReLU) and returns z for samples ty*4.. in zq[4]
// (valid in the tx == 0 thread of each row group after the reduction).
__device__ __forceinline__ void mlp_tile_forward(MlpSmem& sm, float zq[4]) {
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  const int s0 = ty * 4;
  float acc[4][8];
  // layer 1: h1 = relu(x W1 + b1)
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[q][j] = sm.b1[tx + 16 * j];
#pragma unroll 4
  for (int k = 0; k < kMlpIn; k++) {
    float xv[4], wv[8];
#pragma unroll
    for (int q = 0; q < 4; q++) xv[q] = sm.x[(s0 + q) * kXs + k];
#pragma unroll
    for (int j = 0; j < 8; j++) wv[j] = sm.w1[k * kMlpHid + tx + 16 * j];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[q][j] = fmaf(xv[q], wv[j], acc[q][j]);
  }
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int j = 0; j < 8; j++)  // layer-2 operands are bf16, as on the tensor-core path
      sm.h1[(s0 + q) * kHs + tx + 16 * j] = __bfloat162float(__float2bfloat16_rn(fmaxf(acc[q][j], 0.f)));
  __syncthreads();
  // layer 2: h2 = relu(h1 W2 + b2)
#pragma unroll
  for (int q = 0; q < 4; q++)
#pragma unroll
    for (int j = 0; j < 8; j++) acc[q][j] = sm.b2[tx + 16 * j];
#pragma unroll 4
  for (int k = 0; k < kMlpHid; k++) {
    float hv[4], wv[8];
#pragma unroll
    for (int q = 0; q < 4; q++) hv[q] = sm.h1[(s0 + q) * kHs + k];
#pragma unroll
    for (int j = 0; j < 8; j++) wv[j] = sm.w2[k * kHs + tx + 16 * j];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int j = 0; j < 8; j++) acc[q][j] = fmaf(hv[q], wv[j], acc[q][j]);
  }
  // layer 3 partial dot products, then a reduction over the 16 tx lanes of the row group
#pragma unroll
  for (int q = 0; q < 4; q++) {
    float z = 0.f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float h = fmaxf(acc[q][j], 0.f);
      sm.h2[(s0 + q) * kHs + tx + 16 * j] = h;
      z = fmaf(h, sm.w3[tx + 16 * j], z);
    }
#pragma unroll
    for (int o = 8; o >= 1; o >>= 1) z += __shfl_xor_sync(0xFFFFFFFFu, z, o);
    zq[q] = z + sm.b3;
  }
}

__device__ __forceinline__ float mlp_sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

// Gradient of the mean binary cross-entropy over n samples, accumulated (atomicAdd) into
// grad[kMlpParams] (fp32, same packing as the master block); the summed loss into *loss.
// Grid-stride over tiles; each CTA keeps its share of dW1 and dW2 in registers across tiles.
__global__ void __launch_bounds__(kMlpThreads) mlp_grad_kernel(
    const __nv_bfloat16* __restrict__ x, const float* __restrict__ y, uint32_t n,
    const __nv_bfloat16* w1, const __nv_bfloat16* w2, const __nv_bfloat16* w3,
    const float* master, float* grad, float* loss) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MlpSmem& sm = *reinterpret_cast<MlpSmem*>(smem_raw);
  mlp_load_weights(sm, w1, w2, w3, master);
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
  const float inv_n = 1.f / (float)n;
  // register accumulators: dW2 rows i = ty*8+a, cols j = tx+16b; dW1 rows k = ty*4+a, cols
  // i = tx+16b
  float gw2[8][8], gw1[4][8];
#pragma unroll
  for (int a = 0; a < 8; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) gw2[a][b] = 0.f;
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) gw1[a][b] = 0.f;
  float gb1 = 0.f, gb2 = 0.f, gw3 = 0.f, gb3 = 0.f, lsum = 0.f;  // thread tid < 128 owns unit tid

  for (uint32_t s0 = blockIdx.x * kMlpTile; s0 < n; s0 += gridDim.x * kMlpTile) {
    __syncthreads();
    mlp_load_x(sm, x, s0, n);
    __syncthreads();
    float zq[4];
    mlp_tile_forward(sm, zq);
    if (tx == 0) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const uint32_t s = s0 + ty * 4 + q;
        float d = 0.f;
        if (s < n) {
          const float z = zq[q], t = y[s];
          d = (mlp_sigmoid(z) - t) * inv_n;
          // softplus(z) - t z, written to stay finite for large |z|
          lsum += fmaxf(z, 0.f) - t * z + log1pf(expf(-fabsf(z)));
        }
        sm.dz[ty * 4 + q] = d;
      }
    }
    __syncthreads();
    // dw3, db3, db2 partials and dh2 = dz * w3 * relu'(h2), in place over h2
    if (tid < kMlpHid) {
      float a3 = 0.f;
      for (int s = 0; s < kMlpTile; s++) a3 = fmaf(sm.dz[s], sm.h2[s * kHs + tid], a3);
      gw3 += a3;
    }
    if (tid == kMlpHid) {
      float a = 0.f;
      for (int s = 0; s < kMlpTile; s++) a += sm.dz[s];
      gb3 += a;
    }
    __syncthreads();
    for (int e = tid; e < kMlpTile * kMlpHid; e += kMlpThreads) {
      const int s = e / kMlpHid, j = e % kMlpHid;
      const float h = sm.h2[s * kHs + j];
      sm.h2[s * kHs + j] = h > 0.f ? sm.dz[s] * sm.w3[j] : 0.f;
    }
    __syncthreads();
    if (tid < kMlpHid) {
      float a = 0.f;
      for (int s = 0; s < kMlpTile; s++) a += sm.h2[s * kHs + tid];
      gb2 += a;
    }
    // dW2 += h1^T dh2
#pragma unroll 2
    for (int s = 0; s < kMlpTile; s++) {
      float hv[8], dv[8];
#pragma unroll
      for (int a = 0; a < 8; a++) hv[a] = sm.h1[s * kHs + ty * 8 + a];
#pragma unroll
      for (int b = 0; b < 8; b++) dv[b] = sm.h2[s * kHs + tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 8; a++)
#pragma unroll
        for (int b = 0; b < 8; b++) gw2[a][b] = fmaf(hv[a], dv[b], gw2[a][b]);
    }
    // dh1 = (dh2 W2^T) * relu'(h1): thread owns samples ty*4+q and units i = tx + 16*b
    float dh[4][8];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int b = 0; b < 8; b++) dh[q][b] = 0.f;
#pragma unroll 2
    for (int j = 0; j < kMlpHid; j++) {
      float dv[4], wv[8];
#pragma unroll
      for (int q = 0; q < 4; q++) dv[q] = sm.h2[(ty * 4 + q) * kHs + j];
#pragma unroll
      for (int b = 0; b < 8; b++) wv[b] = sm.w2[(tx + 16 * b) * kHs + j];
#pragma unroll
      for (int q = 0; q < 4; q++)
#pragma unroll
        for (int b = 0; b < 8; b++) dh[q][b] = fmaf(dv[q], wv[b], dh[q][b]);
    }
    __syncthreads();  // every read of h1 (dW2) and dh2 is done: dh1 replaces h1
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int b = 0; b < 8; b++) {
        const int s = ty * 4 + q, i = tx + 16 * b;
        sm.h1[s * kHs + i] = sm.h1[s * kHs + i] > 0.f ? dh[q][b] : 0.f;
      }
    __syncthreads();
    if (tid < kMlpHid) {
      float a = 0.f;
      for (int s = 0; s < kMlpTile; s++) a += sm.h1[s * kHs + tid];
      gb1 += a;
    }
    // dW1 += x^T dh1
#pragma unroll 2
    for (int s = 0; s < kMlpTile; s++) {
      float xv[4], dv[8];
#pragma unroll
      for (int a = 0; a < 4; a++) xv[a] = sm.x[s * kXs + ty * 4 + a];
#pragma unroll
      for (int b = 0; b < 8; b++) dv[b] = sm.h1[s * kHs + tx + 16 * b];
#pragma unroll
      for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 8; b++) gw1[a][b] = fmaf(xv[a], dv[b], gw1[a][b]);
    }
  }
#pragma unroll
  for (int a = 0; a < 8; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) atomicAdd(&grad[kOffW2 + (ty * 8 + a) * kMlpHid + tx + 16 * b], gw2[a][b]);
#pragma unroll
  for (int a = 0; a < 4; a++)
#pragma unroll
    for (int b = 0; b < 8; b++) atomicAdd(&grad[kOffW1 + (ty * 4 + a) * kMlpHid + tx + 16 * b], gw1[a][b]);
  if (tid < kMlpHid) {
    atomicAdd(&grad[kOffB1 + tid], gb1);
    atomicAdd(&grad[kOffB2 + tid], gb2);
    atomicAdd(&grad[kOffW3 + tid], gw3);
  }
  if (tid == kMlpHid) atomicAdd(&grad[kOffB3], gb3);
  if (tx == 0) atomicAdd(loss, lsum);
}

constexpr int kTcTile = 128;                  // samples of an inference tile
constexpr uint32_t kTcChunk = kTcTile * 128;  // 128 rows of 64 bf16: one swizzled operand block

// Byte of element (row r, column c of 64) in a SWIZZLE_128B block: 16-byte pieces XORed by row.
__host__ __device__ __forceinline__ uint32_t tc_swizzle(uint32_t r, uint32_t c) {
  return r * 128u + (((c >> 3) ^ (r & 7u)) << 4) + ((c & 7u) << 1);
}

// Parameter i's bf16 copies: as stored, and in the inference kernel's operand images (wimg, blocks
// of kTcChunk bytes: W1^T [unit][feature]; W2^T [unit][unit] in two blocks of 64 columns; the
// biases [unit][b1: 0..2, b2: 16..18] as three bf16 terms each, whose sum is the fp32 bias).
__device__ __forceinline__ void mlp_store_bf16(int i, float w, __nv_bfloat16* w1, __nv_bfloat16* w2,
                                               __nv_bfloat16* w3, unsigned char* wimg) {
  const __nv_bfloat16 h = __float2bfloat16_rn(w);
  if (i < kOffB1) {
    const uint32_t e = i - kOffW1, k = e / kMlpHid, j = e % kMlpHid;
    w1[e] = h;
    *reinterpret_cast<__nv_bfloat16*>(wimg + tc_swizzle(j, k)) = h;
  } else if (i >= kOffW2 && i < kOffB2) {
    const uint32_t e = i - kOffW2, k = e / kMlpHid, j = e % kMlpHid;
    w2[e] = h;
    *reinterpret_cast<__nv_bfloat16*>(wimg + (1u + (k >> 6)) * kTcChunk + tc_swizzle(j, k & 63u)) = h;
  } else if (i >= kOffW3 && i < kOffB3) {
    w3[i - kOffW3] = h;
  } else if (i < kOffW3) {  // a bias
    const uint32_t j = i < kOffW2 ? i - kOffB1 : i - kOffB2, c0 = i < kOffW2 ? 0u : 16u;
    const bool finite = (__float_as_uint(w) & 0x7F800000u) != 0x7F800000u;
    float rest = w;
    for (uint32_t c = 0; c < 3; c++) {  // 8 significant bits a term, truncated: exact remainders
      const float part = finite ? __uint_as_float(__float_as_uint(rest) & 0xFFFF0000u)
                                : (c ? 0.f : __bfloat162float(h));
      *reinterpret_cast<__nv_bfloat16*>(wimg + 3u * kTcChunk + tc_swizzle(j, c0 + c)) =
          __float2bfloat16_rn(part);
      rest -= part;
    }
  }
}
constexpr size_t kTcImageBytes = 4 * (size_t)kTcChunk;

// Adam on the fp32 master block, then the bf16 weight copies; clears the gradient.
__global__ void mlp_adam_kernel(float* master, float* grad, float* m, float* v, float lr,
                                float b1t, float b2t, __nv_bfloat16* w1, __nv_bfloat16* w2,
                                __nv_bfloat16* w3, unsigned char* wimg) {
  const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpParams; i += gridDim.x * blockDim.x) {
    const float g = grad[i];
    const float mi = beta1 * m[i] + (1.f - beta1) * g;
    const float vi = beta2 * v[i] + (1.f - beta2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.f - b1t), vh = vi / (1.f - b2t);
    const float w = master[i] - lr * mh / (sqrtf(vh) + eps);
    master[i] = w;
    grad[i] = 0.f;
    mlp_store_bf16(i, w, w1, w2, w3, wimg);
  }
}

__global__ void mlp_round_weights_kernel(const float* master, __nv_bfloat16* w1,
                                         __nv_bfloat16* w2, __nv_bfloat16* w3,
                                         unsigned char* wimg) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpParams; i += gridDim.x * blockDim.x) {
    const float w = master[i];
    mlp_store_bf16(i, w, w1, w2, w3, wimg);
  }
}

// ---------------------------------------------------------------------------------------------
// Inference on the 5th-generation tensor cores (tcgen05, bf16 operands, fp32 accumulators in
// tensor memory). A tile is 128 samples. One CTA per SM holds the weights (48 KB, copied as they
// lie from images kept in the operands' shared-memory layout) and runs two groups of eight warps,
// each with tiles of its own: one group's MMAs run under the other's epilogues. Thread = one
// sample's accumulator row, 64 of its 128 columns. Per tile a group
//   1. multiplies X (cp.async, two buffers ahead) by W1 and adds b1: 5 MMAs of 128 x 128 x 16;
//   2. ReLU, rounds to bf16 back into tensor memory, over the columns just read;
//   3. multiplies that, as the A operand in tensor memory, by W2 and adds b2: 9 MMAs;
//   4. starts step 1 of its next tile, then ReLU, dot product with w3, sigmoid.
// The biases are an MMA step of their own (a column of ones times the bias in three bf16 terms,
// which add up to the fp32 value): read by every row from shared memory they took as long as the
// MMAs, 2.7 cycles for a 16-byte broadcast load. The outputs of a tile are written under step 3
// of the next one.
// Bound by the MMAs (64 cycles each, 900 a tile) and the epilogues' ALU work (about as long),
// which two groups overlap only in part. 2^20 samples: 190 us with warp MMAs (mma.sync); with
// tcgen05 74 us with activations and biases in shared memory, 57 us before the issuing warps
// kept their descriptors uniform, 46 us so (of 27 us at the card's bf16 rate). One group of
// sixteen warps with double accumulators, a warp for the issue and one for the outputs: 49 us.
// Every wait on an MMA is bounded; one that runs out raises *fail and ends the CTA.
// ---------------------------------------------------------------------------------------------
constexpr int kTcGroups = 2, kTcThreads = 256 * kTcGroups;

struct MlpTcSmem {
  unsigned char w1[kTcChunk];                // W1^T [unit][feature], SWIZZLE_128B, K-major
  unsigned char w2[2 * kTcChunk];            // W2^T [unit][unit]: two blocks of 64 columns
  unsigned char bias[kTcChunk];              // [unit][terms of b1, of b2]
  unsigned char ones[kTcChunk];              // [sample][1 1 1 0 ... 0] (16 columns)
  unsigned char x[kTcGroups][2][kTcChunk];   // [sample][feature]
  float w3[kMlpHid];
  float z[kTcGroups][2][kTcTile];            // dot products over columns 64.., by tile parity
  float b3;
  uint32_t tmem;                             // base column of the accumulators
  unsigned long long bar1[kTcGroups], bar2[kTcGroups];  // completion of steps 1 and 3
  unsigned long long ready[kTcGroups];                  // step 2: the group's eight warps
};
constexpr size_t kTcSmemBytes = sizeof(MlpTcSmem) + 1024;  // operand blocks start on 1024 bytes

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
// K-major SWIZZLE_128B operand block at a 1024-byte boundary: 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr) {
  return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
// bf16 x bf16 -> fp32, both operands K-major, 128 x 128
constexpr uint32_t kTcIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

template <bool ACCUMULATE>
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
      ::"r"(d), "l"(a), "l"(b), "r"(kTcIdesc), "n"(ACCUMULATE ? 1 : 0)
      : "memory");
}
// the same, accumulating, with A in tensor memory (128 lanes x 8 columns of bf16 pairs)
__device__ __forceinline__ void tc_mma_ta(uint32_t d, uint32_t a, uint64_t b) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}"
      ::"r"(d), "r"(a), "l"(b), "r"(kTcIdesc), "n"(1)
      : "memory");
}
__device__ __forceinline__ bool elect_one() {  // one lane of the (converged) warp
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(e));
  return e != 0u;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar)
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void fence_async_shared() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// Bounded wait for the phase of parity `parity`.
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
  for (uint32_t it = 0; it < (1u << 20); it++) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// 64 consecutive fp32 columns of this thread's accumulator row, all in flight at once (a load
// takes about 250 cycles beside the MMAs; four of 16 columns in turn took 1000)
__device__ __forceinline__ void tc_load64(uint32_t taddr, uint32_t (&v)[64]) {
#pragma unroll
  for (int h = 0; h < 2; h++) {
    uint32_t* u = v + 32 * h;
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]),
          "=r"(u[7]), "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]),
          "=r"(u[14]), "=r"(u[15]), "=r"(u[16]), "=r"(u[17]), "=r"(u[18]), "=r"(u[19]),
          "=r"(u[20]), "=r"(u[21]), "=r"(u[22]), "=r"(u[23]), "=r"(u[24]), "=r"(u[25]),
          "=r"(u[26]), "=r"(u[27]), "=r"(u[28]), "=r"(u[29]), "=r"(u[30]), "=r"(u[31])
        : "r"(taddr + 32u * h));
  }
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 64; i++) asm volatile("" : "+r"(v[i]));  // used only after the wait
}
// 32 consecutive columns of it written
__device__ __forceinline__ void tc_store32(uint32_t taddr, const uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%32], "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31};"
      ::"r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]),
        "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]),
        "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
        "r"(v[29]), "r"(v[30]), "r"(v[31]), "r"(taddr)
      : "memory");
}
__device__ __forceinline__ void tc_store_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// two fp32 lanes at once
__device__ __forceinline__ unsigned long long f2_pack(uint32_t lo, uint32_t hi) {
  return ((unsigned long long)hi << 32) | lo;
}
__device__ __forceinline__ unsigned long long f2_add(unsigned long long a, unsigned long long b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ unsigned long long f2_fma(unsigned long long a, unsigned long long b,
                                                     unsigned long long c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ unsigned long long f2_relu(unsigned long long a) {
  const float lo = fmaxf(__uint_as_float((uint32_t)a), 0.f);
  const float hi = fmaxf(__uint_as_float((uint32_t)(a >> 32)), 0.f);
  return f2_pack(__float_as_uint(lo), __float_as_uint(hi));
}
// rounding of a pair to bf16 (first element in the low half), then ReLU (a NaN gives 0, as fmaxf)
__device__ __forceinline__ uint32_t relu_bf16x2(uint32_t lo, uint32_t hi) {
  uint32_t d;
  asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(__uint_as_float(hi)), "f"(__uint_as_float(lo)));
  asm("max.bf16x2 %0, %0, %1;" : "+r"(d) : "r"(0u));
  return d;
}
__device__ __forceinline__ void tc_copy16(uint32_t dst, const void* src, uint32_t bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}

// wimg: W1^T, W2^T and the biases in their shared-memory layout (kTcImageBytes).
__global__ void __launch_bounds__(kTcThreads, 1) mlp_forward_tc_kernel(
    const __nv_bfloat16* __restrict__ x, uint32_t n, const unsigned char* __restrict__ wimg,
    const __nv_bfloat16* w3, const float* master, float* __restrict__ p, uint32_t* fail) {
  extern __shared__ unsigned char smem_raw[];
  MlpTcSmem& sm = *reinterpret_cast<MlpTcSmem*>(smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u));
  const uint32_t tid = threadIdx.x, warp = tid >> 5, g = tid >> 8, gt = tid & 255u;
  const uint32_t half = gt >> 7, r = gt & 127u;  // columns 64 half .. 64 half + 63 of row r
  const uint32_t tiles = (n + kTcTile - 1) / kTcTile, step = gridDim.x * kTcGroups;
  uint32_t tile = blockIdx.x + gridDim.x * g;
  auto fetch = [&](uint32_t t, uint32_t buf) {  // X of tile t, rows beyond n zero; one copy group
    if (t < tiles) {  // 16 KB in a row: thread gt copies the 16-byte pieces gt, gt + 256, ...
      const uint32_t dst = smem_u32(sm.x[g][buf]) + tc_swizzle(gt >> 3, (gt & 7u) * 8u);
      const uint32_t s = t * kTcTile + (gt >> 3);
      const __nv_bfloat16* src = x + (size_t)s * kMlpIn + (gt & 7u) * 8u;
#pragma unroll
      for (uint32_t i = 0; i < 4; i++) {
        const bool in = s + 32u * i < n;
        tc_copy16(dst + i * 4096u, in ? src + 2048u * i : x, in ? 16u : 0u);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  for (uint32_t i = tid; i < kTcImageBytes / 16u; i += kTcThreads) tc_copy16(smem_u32(sm.w1) + i * 16u, wimg + i * 16u, 16u);
  fetch(tile, 0u);
  fetch(tile + step, 1u);
  if (tid < kTcTile) {  // 16-byte pieces 0 and 1 of every row
    *reinterpret_cast<uint4*>(sm.ones + tc_swizzle(tid, 0u)) = make_uint4(0x3F803F80u, 0x3F80u, 0u, 0u);
    *reinterpret_cast<uint4*>(sm.ones + tc_swizzle(tid, 8u)) = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid < kMlpHid) sm.w3[tid] = __bfloat162float(w3[tid]);
  if (tid == 0) sm.b3 = master[kOffB3];
  const uint32_t bar1 = smem_u32(&sm.bar1[g]), bar2 = smem_u32(&sm.bar2[g]), ready = smem_u32(&sm.ready[g]);
  if (gt == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar1) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar2) : "memory");
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 8;" ::"r"(ready) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {  // all 512 columns (one CTA per SM): 256 per group
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_u32(&sm.tmem)) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("cp.async.wait_group 1;" ::: "memory");
  fence_async_shared();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t d1 = sm.tmem + g * 256u, d2 = d1 + 128u;  // steps 1 (then its ReLU) and 3
  bool ok = true;  // a wait that runs out ends this warp's loop, and by their own bounds the others'
  uint32_t it = 0;
  // MMAs are issued by one elected lane of a converged warp, with addresses and descriptors in
  // uniform registers; a descriptor differs from its block's by a constant (16-byte units).
  // Worked out per MMA in one lane they made the issue 82 cycles an MMA, and the run wait for it.
  const uint32_t gu = __shfl_sync(0xFFFFFFFFu, g, 0), tm = __shfl_sync(0xFFFFFFFFu, sm.tmem, 0) + gu * 256u;
  const uint64_t xd = tc_desc(smem_u32(sm.x[0][0])) + gu * (2u * kTcChunk >> 4);
  const uint64_t w1d = tc_desc(smem_u32(sm.w1)), w2d = tc_desc(smem_u32(sm.w2));
  const uint64_t bd = tc_desc(smem_u32(sm.bias)), od = tc_desc(smem_u32(sm.ones));
  auto layer1 = [&](uint32_t buf) {  // by one warp
    const uint64_t xi = xd + buf * (kTcChunk >> 4);
    if (elect_one()) {
      tc_mma<false>(tm, od, bd);
#pragma unroll
      for (uint32_t k = 0; k < kMlpIn / 16; k++) tc_mma<true>(tm, xi + 2u * k, w1d + 2u * k);
      tc_commit(bar1);
    }
    __syncwarp();
  };
  const uint32_t gw = __shfl_sync(0xFFFFFFFFu, warp & 7u, 0);  // warp of the group
  if (gw == 0u && tile < tiles) layer1(0u);
  const uint32_t mine = ((warp & 3u) << 21) + 64u * half;  // this thread's lanes and columns
  float z_mine = 0.f;  // the last tile's dot product over columns 0..63 (half 0)
  // the output of tile t, both halves' sums being there
  auto finish = [&](uint32_t t, uint32_t parity) {
    const uint32_t s = t * kTcTile + r;
    if (half == 0u && s < n) p[s] = mlp_sigmoid(z_mine + sm.z[g][parity][r] + sm.b3);
  };
  for (; tile < tiles; tile += step, it++) {
    const uint32_t par = it & 1u;
    if (!(ok = __all_sync(0xFFFFFFFFu, tc_wait(bar1, par)))) break;  // the warp leaves together
    tc_fence_after();
    // ReLU, bf16, into the columns just read
    {
      uint32_t v[64], o[32];
      tc_load64(d1 + mine, v);
#pragma unroll
      for (uint32_t i = 0; i < 32; i++) o[i] = relu_bf16x2(v[2 * i], v[2 * i + 1]);
      tc_store32(d1 + mine, o);
    }
    tc_store_wait();
    asm volatile("cp.async.wait_all;" ::: "memory");  // X of the next tile
    fence_async_shared();
    tc_fence_before();
    __syncwarp();
    if ((tid & 31u) == 0u)  // (this warp has also read the last tile's step 3)
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(ready) : "memory");
    __syncwarp();
    if (gw == 0u) {
      if (!(ok = __all_sync(0xFFFFFFFFu, tc_wait(ready, par)))) break;  // all eight have
      tc_fence_after();
      if (elect_one()) {
        tc_mma<false>(tm + 128u, od, bd + 2u);
#pragma unroll
        for (uint32_t k = 0; k < kMlpHid / 16; k++)  // 16 units: 8 columns, 64 units a half
          tc_mma_ta(tm + 128u, tm + (k >> 2) * 64u + 8u * (k & 3u), w2d + (k >> 2) * (kTcChunk >> 4) + 2u * (k & 3u));
        tc_commit(bar2);
      }
      __syncwarp();
    }
    // into the buffer that step 1 has read; after the fence, which would wait for it
    fetch(tile + 2u * step, par);
    // under step 3: the last tile's outputs (every warp has arrived here, its sums stored)
    if (it && half == 0u) {
      if (!(ok = __all_sync(0xFFFFFFFFu, tc_wait(ready, par)))) break;
      finish(tile - step, par ^ 1u);
      __syncwarp();
    }
    if (!(ok = __all_sync(0xFFFFFFFFu, tc_wait(bar2, par)))) break;
    tc_fence_after();
    if (gw == 4u && tile + step < tiles) layer1(par ^ 1u);  // (the activations have been read)
    __syncwarp();
    // ReLU, dot product with w3
    unsigned long long z0 = 0ull, z1 = 0ull;
    {
      uint32_t v[64];
      tc_load64(d2 + mine, v);
      const ulonglong2* w = reinterpret_cast<const ulonglong2*>(sm.w3 + 64u * half);
#pragma unroll
      for (uint32_t i = 0; i < 16; i++) {
        const ulonglong2 ww = w[i];
        z0 = f2_fma(f2_relu(f2_pack(v[4 * i], v[4 * i + 1])), ww.x, z0);
        z1 = f2_fma(f2_relu(f2_pack(v[4 * i + 2], v[4 * i + 3])), ww.y, z1);
      }
    }
    const unsigned long long zz = f2_add(z0, z1);
    z_mine = __uint_as_float((uint32_t)zz) + __uint_as_float((uint32_t)(zz >> 32));
    if (half) sm.z[g][par][r] = z_mine;
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  if (ok && it) finish(tile - step, (it & 1u) ^ 1u);
  if (!ok) {  // once more for the MMAs in flight
    tc_wait(bar1, it & 1u);
    tc_wait(bar2, it & 1u);
    *(volatile uint32_t*)fail = 1u;
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(sm.tmem));
  }
}

}  // namespace csmv
