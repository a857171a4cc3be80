// mlp_kernels.cuh - the conflict predictor's network: 64 -> 128 -> 128 -> 1 (ReLU, ReLU,
// sigmoid), bf16 weights, fp32 accumulation, hand-written forward, backward and Adam kernels.
//
// Layout: features X [n][64] bf16 (0/1 indicators here, exact in bf16); weights W1 [64][128],
// W2 [128][128], w3 [128] in bf16 (rounded from fp32 master copies after every step), biases
// fp32.
// Inference (every planned transaction) runs on the tensor cores (mlp_forward_tc_kernel, tcgen05
// with fp32 accumulation); training (the probe slice, a few percent of the chunk) runs its fused
// forward + backward tile products on warp MMAs, with fp32 operands split into exact bf16 terms.
// Both feed layer 2 with bf16 activations, so they compute the same network.
#pragma once
#include <cuda_bf16.h>

#include <cstddef>
#include <cstdint>

namespace csmv {

constexpr int kMlpIn = 64, kMlpHid = 128, kMlpTile = 64, kMlpThreads = 512;
// fp32 master parameter block: W1 | b1 | W2 | b2 | w3 | b3 (+3 pad)
constexpr int kOffW1 = 0, kOffB1 = kOffW1 + kMlpIn * kMlpHid, kOffW2 = kOffB1 + kMlpHid,
              kOffB2 = kOffW2 + kMlpHid * kMlpHid, kOffW3 = kOffB2 + kMlpHid,
              kOffB3 = kOffW3 + kMlpHid, kMlpParams = kOffB3 + 4;

__device__ __forceinline__ float mlp_sigmoid(float z) { return 1.f / (1.f + expf(-z)); }

constexpr int kTcTile = 128;                  // samples of an inference tile
constexpr uint32_t kTcChunk = kTcTile * 128;  // 128 rows of 64 bf16: one swizzled operand block

// Byte of element (row r, column c of 64) in a SWIZZLE_128B block: 16-byte pieces XORed by row.
__host__ __device__ __forceinline__ uint32_t tc_swizzle(uint32_t r, uint32_t c) {
  return r * 128u + (((c >> 3) ^ (r & 7u)) << 4) + ((c & 7u) << 1);
}

// Parameter i's bf16 copies: W2 and w3 as stored, and operand images (wimg, blocks
// of kTcChunk bytes: W1^T [unit][feature]; W2^T [unit][unit] in two blocks of 64 columns; the
// biases [unit][b1: 0..2, b2: 16..18] as three bf16 terms each, whose sum is the fp32 bias).
__device__ __forceinline__ void mlp_store_bf16(int i, float w, __nv_bfloat16* w2,
                                               __nv_bfloat16* w3, unsigned char* wimg) {
  const __nv_bfloat16 h = __float2bfloat16_rn(w);
  if (i < kOffB1) {
    const uint32_t e = i - kOffW1, k = e / kMlpHid, j = e % kMlpHid;
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

// ---------------------------------------------------------------------------------------------
// Training: gradient of the mean binary cross-entropy over n samples, added into grad[kMlpParams]
// (fp32, packed as the master block); the summed loss into *loss.
//
// All five products run on the tensor cores (bf16 warp MMAs m16n8k16, fp32 accumulators) without
// rounding an fp32 operand: with m = (h2 > 0),
//   dW2[i][j] = w3[j] sum_s h1[s][i] (dz[s] m[s][j])      h1, m exact; dz in three bf16 terms
//   dh1[s][i] = dz[s] sum_j m[s][j] (w3[j] W2[i][j])      the products have 16 bits: two terms
//   dW1[k][i] = sum_s x[s][k] dh1[s][i]                   x exact; dh1 in three terms
// so every MMA product is exact, as fmaf's was. The tensor core truncates what it adds, which
// would bias sums; so the leading terms of each 16 samples (16 units) are summed from zero and
// added by fp32 adds, and only the lower terms, 2^8 smaller, stay in it over a tile.
//
// A CTA of 16 warps takes tiles of 64 samples; its sums stay in registers over all its tiles and
// are added to grad in 16-byte pieces. Forward, a warp has 16 samples x 32 units. Backward it has
// 16 units i of h1 and computes dh1 transposed, [i][s], whose accumulators are at once the A
// operand of dW1: dh1 never leaves the registers. Three barriers a tile; x and y of the next tile
// are loaded under the current one.
// Bound by the warp MMAs: 4096 of 2048 products a tile, which these units retire at about 512
// products a clock: 8.2 us of the 8.7 us a tile takes (other splits of the work among 8 or 16
// warps, with twice the fragment loads, took the same). A call of 52448 samples took 250 us on
// the FP32 pipes, 77 us so. Error of the gradient against 64 bits (2-norm, median of 12 to 40
// nets): 1.48e-7 of it at 52448 samples, 1.59e-7 before; of the loss 1.3e-8, 2.6e-7 before.
// ---------------------------------------------------------------------------------------------
constexpr int kGx = kMlpIn + 8, kGh = kMlpHid + 8;  // padded rows: fragment loads hit 32 banks
constexpr int kGo = kMlpHid + 4;                    // row of the staged sums (floats)

struct MlpGradSmem {
  __nv_bfloat16 w1t[kMlpHid * kGx];       // W1^T [unit][feature]
  __nv_bfloat16 w2t[kMlpHid * kGh];       // W2^T [j][i]
  __nv_bfloat16 wp[2][kMlpHid * kGh];     // w3[j] W2[i][j] as two terms, [i][j]
  __nv_bfloat16 x[2][kMlpTile * kGx];     // [s][k], two tiles
  __nv_bfloat16 h1[kMlpTile * kGh];       // [s][i]
  __nv_bfloat16 m[kMlpTile * kGh];        // [s][j] all bits set where h2 > 0, else none
  float z[4][kMlpTile];                   // layer 3, by 32 units
  float b1[kMlpHid], b2[kMlpHid], w3[kMlpHid];
  float dz[kMlpThreads / 32][kMlpTile];             // each warp its own copy
  uint32_t dzp[kMlpThreads / 32][3][kMlpTile / 2];  // the terms of dz, samples in pairs
};
static_assert(sizeof(MlpGradSmem) <= 227 * 1024, "shared memory of a CTA");
static_assert(kMlpThreads == 512 && kMlpTile == 64, "the warps' shares of a tile");

__device__ __forceinline__ uint32_t mlp_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(mlp_smem(p)) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const __nv_bfloat16* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(mlp_smem(p)) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// c += the product, summed from zero and added in fp32
__device__ __forceinline__ void mma_add(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  float u[4] = {};
  mma_bf16(u, a, b0, b1);
#pragma unroll
  for (int e = 0; e < 4; e++) c[e] += u[e];
}
// v as three bf16 terms of 8 significant bits each (their sum is v; a non-finite v is the first)
__device__ __forceinline__ void split3(float v, __nv_bfloat16 (&t)[3]) {
  const bool finite = (__float_as_uint(v) & 0x7F800000u) != 0x7F800000u;
  float rest = v;
#pragma unroll
  for (int q = 0; q < 3; q++) {
    const float part = __uint_as_float(__float_as_uint(rest) & 0xFFFF0000u);
    t[q] = finite ? __ushort_as_bfloat16((unsigned short)(__float_as_uint(part) >> 16))
                  : (q ? __ushort_as_bfloat16(0) : __float2bfloat16_rn(v));
    rest -= part;
  }
}
__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi) {
  return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}
__device__ __forceinline__ void red_add4(float* p, float4 v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}

__global__ void __launch_bounds__(kMlpThreads, 1) mlp_grad_kernel(
    const __nv_bfloat16* __restrict__ x, const float* __restrict__ y, uint32_t n,
    const unsigned char* __restrict__ wimg, const __nv_bfloat16* __restrict__ w2,
    const __nv_bfloat16* w3, const float* master, float* grad, double* loss) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MlpGradSmem& sm = *reinterpret_cast<MlpGradSmem*>(smem_raw);
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u, g = lane >> 2, t = lane & 3u;
  const uint32_t wm = warp >> 2, wn = warp & 3u;   // forward: samples 16 wm, units 32 wn
  const uint32_t wi = warp & 7u, wh = warp >> 3;   // backward: units 16 wi of h1; half of j or s
  // this lane's row and column in a load of 16 x 16: plain, and transposed for an A operand
  const uint32_t lr = lane & 15u, lc = (lane >> 4) * 8u;
  const uint32_t tr = (lane & 7u) + (lane >> 4) * 8u, tc = ((lane >> 3) & 1u) * 8u;
  const float inv_n = 1.f / (float)n;
  const bool wide = (reinterpret_cast<uintptr_t>(x) & 15u) == 0u;
  uint4 xn;      // the next tile's X: a piece of 16 bytes,
  float yn[2];   // and labels of samples lane and lane + 32
  auto fetch = [&](uint32_t s0) {
    const uint32_t s = s0 + (tid >> 3);
    const __nv_bfloat16* p = x + (size_t)s * kMlpIn + (tid & 7u) * 8u;
    xn = make_uint4(0, 0, 0, 0);
    if (s < n) {
      if (wide)
        xn = *reinterpret_cast<const uint4*>(p);
      else  // x at a 2-byte boundary
        xn = make_uint4(pack2(p[0], p[1]), pack2(p[2], p[3]), pack2(p[4], p[5]), pack2(p[6], p[7]));
    }
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) yn[h] = s0 + lane + 32u * h < n ? y[s0 + lane + 32u * h] : 0.f;
  };
  auto store_x = [&](uint32_t buf) {
    *reinterpret_cast<uint4*>(&sm.x[buf][(tid >> 3) * kGx + (tid & 7u) * 8u]) = xn;
  };
  fetch(blockIdx.x * kMlpTile);
  // the weights (unrolled: every load of a thread in flight at once)
#pragma unroll
  for (uint32_t i0 = 0; i0 < kMlpHid * 8u; i0 += kMlpThreads) {
    const uint32_t j = (i0 + tid) >> 3, q = tid & 7u;
    *reinterpret_cast<uint4*>(&sm.w1t[j * kGx + q * 8u]) = *reinterpret_cast<const uint4*>(wimg + tc_swizzle(j, q * 8u));
  }
#pragma unroll
  for (uint32_t i0 = 0; i0 < kMlpHid * 16u; i0 += kMlpThreads) {
    const uint32_t j = (i0 + tid) >> 4, q = tid & 15u;
    *reinterpret_cast<uint4*>(&sm.w2t[j * kGh + q * 8u]) =
        *reinterpret_cast<const uint4*>(wimg + (1u + (q >> 3)) * kTcChunk + tc_swizzle(j, (q & 7u) * 8u));
  }
  {
    constexpr uint32_t kRows = kMlpThreads / 16;
    const uint32_t r0 = tid >> 4, j = (tid & 15u) * 8u;
    const uint4 v4 = *reinterpret_cast<const uint4*>(w3 + j);
    uint4 in[kMlpHid / kRows];
#pragma unroll
    for (uint32_t h = 0; h < kMlpHid / kRows; h++)
      in[h] = *reinterpret_cast<const uint4*>(w2 + (r0 + h * kRows) * kMlpHid + j);
    const __nv_bfloat162* v = reinterpret_cast<const __nv_bfloat162*>(&v4);
#pragma unroll
    for (uint32_t h = 0; h < kMlpHid / kRows; h++) {
      const __nv_bfloat162* w = reinterpret_cast<const __nv_bfloat162*>(&in[h]);
#pragma unroll
      for (uint32_t e = 0; e < 4; e++) {
        __nv_bfloat16 a[3], b[3];
        split3(__bfloat162float(w[e].x) * __bfloat162float(v[e].x), a);
        split3(__bfloat162float(w[e].y) * __bfloat162float(v[e].y), b);
        for (int q = 0; q < 2; q++)
          *reinterpret_cast<uint32_t*>(&sm.wp[q][(r0 + h * kRows) * kGh + j + 2u * e]) = pack2(a[q], b[q]);
      }
    }
  }
  if (tid < kMlpHid) {
    sm.b1[tid] = master[kOffB1 + tid];
    sm.b2[tid] = master[kOffB2 + tid];
    sm.w3[tid] = __bfloat162float(w3[tid]);
  }
  const float bias3 = master[kOffB3];
  store_x(0);
  // sums over the CTA's tiles: dW2 / w3 [i][j] (16 x 64 a warp), dW1^T [i][k] (16 x 64, over half
  // of the samples), db1 of rows g and g + 8; and by the forward columns dw3 and db2 / w3
  float gw2[8][4], gw1[8][4], cb1[2] = {0.f, 0.f}, cw3[4][2], cb2[4][2], gb3 = 0.f;
  double lsum = 0.0;
#pragma unroll
  for (int q = 0; q < 8; q++)
#pragma unroll
    for (int e = 0; e < 4; e++) gw2[q][e] = gw1[q][e] = 0.f;
#pragma unroll
  for (int q = 0; q < 4; q++) cw3[q][0] = cw3[q][1] = cb2[q][0] = cb2[q][1] = 0.f;
  uint32_t buf = 0;
  for (uint32_t s0 = blockIdx.x * kMlpTile; s0 < n; s0 += gridDim.x * kMlpTile, buf ^= 1u) {
    const float yt[2] = {yn[0], yn[1]};
    const bool more = s0 + gridDim.x * kMlpTile < n;
    __syncthreads();  // x is there; the last tile's h1, m and z have been read
    if (more) fetch(s0 + gridDim.x * kMlpTile);
    const __nv_bfloat16* sx = sm.x[buf];
    float c[4][4];
    // layer 1
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 b = *reinterpret_cast<const float2*>(&sm.b1[32u * wn + 8u * q + 2u * t]);
      c[q][0] = c[q][2] = b.x;
      c[q][1] = c[q][3] = b.y;
    }
#pragma unroll
    for (uint32_t k = 0; k < kMlpIn; k += 16) {
      uint32_t a[4];
      ldsm4(a, &sx[(16u * wm + lr) * kGx + k + lc]);
#pragma unroll
      for (uint32_t q = 0; q < 4; q += 2) {  // B of two column tiles: [n][k] rows
        uint32_t b[4];
        ldsm4(b, &sm.w1t[(32u * wn + 8u * q + lr) * kGx + k + lc]);
        mma_add(c[q], a, b[0], b[2]);
        mma_add(c[q + 1], a, b[1], b[3]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<__nv_bfloat162*>(&sm.h1[(16u * wm + g + 4u * e) * kGh + 32u * wn + 8u * q + 2u * t]) =
            __floats2bfloat162_rn(fmaxf(c[q][e], 0.f), fmaxf(c[q][e + 1], 0.f));
    __syncthreads();
    // layer 2
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 b = *reinterpret_cast<const float2*>(&sm.b2[32u * wn + 8u * q + 2u * t]);
      c[q][0] = c[q][2] = b.x;
      c[q][1] = c[q][3] = b.y;
    }
#pragma unroll
    for (uint32_t k = 0; k < kMlpHid; k += 16) {
      uint32_t a[4];
      ldsm4(a, &sm.h1[(16u * wm + lr) * kGh + k + lc]);
#pragma unroll
      for (uint32_t q = 0; q < 4; q += 2) {
        uint32_t b[4];
        ldsm4(b, &sm.w2t[(32u * wn + 8u * q + lr) * kGh + k + lc]);
        mma_add(c[q], a, b[0], b[2]);
        mma_add(c[q + 1], a, b[1], b[3]);
      }
    }
    // ReLU, its mask, layer 3 (rows g and g + 8)
    float z0 = 0.f, z1 = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float2 w = *reinterpret_cast<const float2*>(&sm.w3[32u * wn + 8u * q + 2u * t]);
#pragma unroll
      for (int e = 0; e < 4; e++) c[q][e] = fmaxf(c[q][e], 0.f);
      z0 = fmaf(c[q][0], w.x, z0);
      z0 = fmaf(c[q][1], w.y, z0);
      z1 = fmaf(c[q][2], w.x, z1);
      z1 = fmaf(c[q][3], w.y, z1);
#pragma unroll
      for (int e = 0; e < 4; e += 2)
        *reinterpret_cast<uint32_t*>(&sm.m[(16u * wm + g + 4u * e) * kGh + 32u * wn + 8u * q + 2u * t]) =
            (c[q][e] > 0.f ? 0xFFFFu : 0u) | (c[q][e + 1] > 0.f ? 0xFFFF0000u : 0u);
    }
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) {
      z0 += __shfl_xor_sync(0xFFFFFFFFu, z0, o);
      z1 += __shfl_xor_sync(0xFFFFFFFFu, z1, o);
    }
    if (t == 0) {
      sm.z[wn][16u * wm + g] = z0;
      sm.z[wn][16u * wm + g + 8u] = z1;
    }
    if (more) store_x(buf ^ 1u);
    __syncthreads();
    // dz of the whole tile, in every warp (one barrier less than one warp's work for all)
#pragma unroll
    for (uint32_t h = 0; h < 2; h++) {
      const uint32_t r = lane + 32u * h;
      float d = 0.f;
      if (s0 + r < n) {
        const float z = ((sm.z[0][r] + sm.z[1][r]) + (sm.z[2][r] + sm.z[3][r])) + bias3;
        d = (mlp_sigmoid(z) - yt[h]) * inv_n;
        // softplus(z) - t z, written to stay finite for large |z|
        if (warp == 0) lsum += (double)(fmaxf(z, 0.f) - yt[h] * z + log1pf(expf(-fabsf(z))));
      }
      if (warp == 0) gb3 += d;
      sm.dz[warp][r] = d;
      __nv_bfloat16 p[3];
      split3(d, p);
#pragma unroll
      for (int q = 0; q < 3; q++) reinterpret_cast<__nv_bfloat16*>(sm.dzp[warp][q])[r] = p[q];
    }
    __syncwarp();
    const float dza = sm.dz[warp][16u * wm + g], dzb = sm.dz[warp][16u * wm + g + 8u];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int e = 0; e < 2; e++) {
        cw3[q][e] = fmaf(dza, c[q][e], fmaf(dzb, c[q][e + 2], cw3[q][e]));
        cb2[q][e] += (c[q][e] > 0.f ? dza : 0.f) + (c[q][e + 2] > 0.f ? dzb : 0.f);
      }
    // dh1^T over 32 samples: A = the terms of w3 W2 (rows i), B = m
    float lo[4][4];
#pragma unroll
    for (int q = 0; q < 4; q++)
#pragma unroll
      for (int e = 0; e < 4; e++) c[q][e] = lo[q][e] = 0.f;
#pragma unroll 2
    for (uint32_t k = 0; k < kMlpHid; k += 16) {
      uint32_t a[2][4];
      ldsm4(a[0], &sm.wp[0][(16u * wi + lr) * kGh + k + lc]);
      ldsm4(a[1], &sm.wp[1][(16u * wi + lr) * kGh + k + lc]);
#pragma unroll
      for (uint32_t q = 0; q < 4; q += 2) {
        uint32_t b[4];
        ldsm4(b, &sm.m[(32u * wh + 8u * q + lr) * kGh + k + lc]);
#pragma unroll
        for (int e = 0; e < 4; e++) b[e] &= 0x3F803F80u;  // 1.0 where the unit is on
        mma_bf16(lo[q], a[1], b[0], b[2]);
        mma_bf16(lo[q + 1], a[1], b[1], b[3]);
        mma_add(c[q], a[0], b[0], b[2]);
        mma_add(c[q + 1], a[0], b[1], b[3]);
      }
    }
    // dW1^T: A = the terms of dh1^T, B = x; 16 samples a pass
#pragma unroll
    for (uint32_t p = 0; p < 2; p++) {
      const uint32_t k = 32u * wh + 16u * p;
      uint32_t on[4], a[3][4];
      ldsm4t(on, &sm.h1[(k + tr) * kGh + 16u * wi + tc]);  // h1^T: where it is zero, dh1 is
#pragma unroll
      for (int e = 0; e < 4; e++) {  // (row g + 8 (e & 1), samples 2t, 2t + 1 + 8 (e >> 1))
        const uint32_t q = 2u * p + (e >> 1), r = 2u * (e & 1);
        const float2 d = *reinterpret_cast<const float2*>(&sm.dz[warp][k + 8u * (e >> 1) + 2u * t]);
        const float v0 = on[e] & 0x7FFFu ? d.x * (c[q][r] + lo[q][r]) : 0.f;
        const float v1 = on[e] & 0x7FFF0000u ? d.y * (c[q][r + 1] + lo[q][r + 1]) : 0.f;
        cb1[e & 1] += v0 + v1;
        __nv_bfloat16 ta[3], tb[3];
        split3(v0, ta);
        split3(v1, tb);
#pragma unroll
        for (int h = 0; h < 3; h++) a[h][e] = pack2(ta[h], tb[h]);
      }
#pragma unroll
      for (uint32_t q = 0; q < 8; q += 2) {
        uint32_t b[4];
        ldsm4t(b, &sx[(k + lr) * kGx + 8u * q + lc]);
        float u[2][4] = {};
#pragma unroll
        for (int h = 2; h >= 1; h--) {
          mma_bf16(u[0], a[h], b[0], b[1]);
          mma_bf16(u[1], a[h], b[2], b[3]);
        }
#pragma unroll
        for (int e = 0; e < 4; e++) {
          gw1[q][e] += u[0][e];
          gw1[q + 1][e] += u[1][e];
        }
        mma_add(gw1[q], a[0], b[0], b[1]);
        mma_add(gw1[q + 1], a[0], b[2], b[3]);
      }
    }
    // dW2 / w3: A = h1^T, B = m times the terms of dz
#pragma unroll
    for (uint32_t q = 0; q < 8; q += 2) {
      float u[2][4] = {};
#pragma unroll
      for (uint32_t k = 0; k < kMlpTile; k += 16) {
        uint32_t a[4], b[4];
        ldsm4t(a, &sm.h1[(k + tr) * kGh + 16u * wi + tc]);
        ldsm4t(b, &sm.m[(k + lr) * kGh + 64u * wh + 8u * q + lc]);
#pragma unroll
        for (int h = 2; h >= 0; h--) {
          const uint32_t d0 = sm.dzp[warp][h][(k >> 1) + t], d1 = sm.dzp[warp][h][(k >> 1) + t + 4u];
          if (h) {
            mma_bf16(u[0], a, b[0] & d0, b[1] & d1);
            mma_bf16(u[1], a, b[2] & d0, b[3] & d1);
          } else {
            mma_add(gw2[q], a, b[0] & d0, b[1] & d1);
            mma_add(gw2[q + 1], a, b[2] & d0, b[3] & d1);
          }
        }
      }
#pragma unroll
      for (int e = 0; e < 4; e++) {
        gw2[q][e] += u[0][e];
        gw2[q + 1][e] += u[1][e];
      }
    }
  }
  // the sums through shared memory (over the operands), then 16 bytes an add; each CTA begins at
  // another row
  __syncthreads();
  float* o2 = reinterpret_cast<float*>(sm.w2t);  // [i][j]
  float* o1 = o2 + kMlpHid * kGo;                // [k][i]
  static_assert((kMlpHid + kMlpIn) * kGo * 4 <= sizeof(sm.w2t) + sizeof(sm.wp) &&
                    offsetof(MlpGradSmem, wp) == offsetof(MlpGradSmem, w2t) + sizeof(sm.w2t),
                "staging");
#pragma unroll
  for (uint32_t q = 0; q < 8; q++) {
    const uint32_t j = 64u * wh + 8u * q + 2u * t;
    const float2 w = *reinterpret_cast<const float2*>(&sm.w3[j]);
#pragma unroll
    for (uint32_t e = 0; e < 4; e += 2)
      *reinterpret_cast<float2*>(&o2[(16u * wi + 4u * e + g) * kGo + j]) =
          make_float2(w.x * gw2[q][e], w.y * gw2[q][e + 1]);
  }
  auto each_gw1 = [&](auto&& f) {
#pragma unroll
    for (uint32_t q = 0; q < 8; q++)
#pragma unroll
      for (uint32_t e = 0; e < 4; e++)
        f(o1[(8u * q + 2u * t + (e & 1u)) * kGo + 16u * wi + g + 8u * (e >> 1)], gw1[q][e]);
  };
  if (wh == 0) each_gw1([](float& o, float v) { o = v; });
  // column sums over a warp's rows, row sums over its columns; by warps, in ov, then one add a CTA
  float* ov = reinterpret_cast<float*>(sm.x[0]);  // [wm: dw3, db2 / w3][128], [wh: db1][128]
  static_assert(10 * kMlpHid * 4 <= sizeof(sm.x), "staging");
#pragma unroll
  for (uint32_t q = 0; q < 4; q++)
#pragma unroll
    for (uint32_t e = 0; e < 2; e++) {
#pragma unroll
      for (int o = 4; o <= 16; o <<= 1) {
        cw3[q][e] += __shfl_xor_sync(0xFFFFFFFFu, cw3[q][e], o);
        cb2[q][e] += __shfl_xor_sync(0xFFFFFFFFu, cb2[q][e], o);
      }
      const uint32_t j = 32u * wn + 8u * q + 2u * t + e;
      if (g == 0) {
        ov[2u * wm * kMlpHid + j] = cw3[q][e];
        ov[(2u * wm + 1u) * kMlpHid + j] = cb2[q][e];
      }
    }
#pragma unroll
  for (uint32_t e = 0; e < 2; e++) {
#pragma unroll
    for (int o = 1; o <= 2; o <<= 1) cb1[e] += __shfl_xor_sync(0xFFFFFFFFu, cb1[e], o);
    if (t == 0) ov[(8u + wh) * kMlpHid + 16u * wi + g + 8u * e] = cb1[e];
  }
  if (warp == 0) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      gb3 += __shfl_xor_sync(0xFFFFFFFFu, gb3, o);
      lsum += __shfl_xor_sync(0xFFFFFFFFu, lsum, o);
    }
    if (lane == 0) {
      atomicAdd(&grad[kOffB3], gb3);
      atomicAdd(loss, lsum);
    }
  }
  __syncthreads();
  if (wh == 1) each_gw1([](float& o, float v) { o += v; });
  if (tid < 3u * kMlpHid) {
    const uint32_t j = tid % kMlpHid, what = tid / kMlpHid;
    auto at = [&](uint32_t r) { return ov[r * kMlpHid + j]; };
    if (what < 2u) {
      const float v = (at(what) + at(2u + what)) + (at(4u + what) + at(6u + what));
      atomicAdd(&grad[(what ? kOffB2 : kOffW3) + j], what ? sm.w3[j] * v : v);
    } else {
      atomicAdd(&grad[kOffB1 + j], at(8) + at(9));
    }
  }
  __syncthreads();
  auto add_rows = [&](float* dst, const float* src, uint32_t rows) {
    for (uint32_t i0 = tid; i0 < rows * 32u; i0 += kMlpThreads) {
      const uint32_t i = (i0 + blockIdx.x * 32u) % (rows * 32u);
      red_add4(dst + 4u * i, *reinterpret_cast<const float4*>(&src[(i >> 5) * kGo + (i & 31u) * 4u]));
    }
  };
  add_rows(grad + kOffW2, o2, kMlpHid);
  add_rows(grad + kOffW1, o1, kMlpIn);
}

// Adam on the fp32 master block, then the bf16 weight copies; clears the gradient.
__global__ void mlp_adam_kernel(float* master, float* grad, float* m, float* v, float lr,
                                float b1t, float b2t, __nv_bfloat16* w2, __nv_bfloat16* w3,
                                unsigned char* wimg) {
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
    mlp_store_bf16(i, w, w2, w3, wimg);
  }
}

__global__ void mlp_round_weights_kernel(const float* master, __nv_bfloat16* w2,
                                         __nv_bfloat16* w3, unsigned char* wimg) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < kMlpParams; i += gridDim.x * blockDim.x) {
    const float w = master[i];
    mlp_store_bf16(i, w, w2, w3, wimg);
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
