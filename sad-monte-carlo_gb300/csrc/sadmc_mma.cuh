// Device helpers of the surrogate MLP: RBF centres, SiLU, bf16 packing and the
// mma.sync m16n8k16 bf16 tensor-core instruction (FP32 accumulation).
#pragma once
#include <cuda_bf16.h>
#include <cstdint>

#include "sadmc_common.cuh"

namespace sadmc {
namespace dev {

__device__ __forceinline__ float rbf_centre(int k) { return 0.8f + (2.2f / 31.0f) * (float)k; }

// 2^x by the special-function unit; results below 2^-126 are zero.
__device__ __forceinline__ float ex2_hw(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 2^x with subnormal results.
__device__ __forceinline__ float ex2_sub(float x) {
  float y;
  asm("ex2.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// 1 / (1 + e^-z) on the special-function unit (0 once the denominator passes 2^126, the limit for
// large negative z): the kernels evaluate a few hundred per thread, and an IEEE division's length
// made their instruction fetch the limiter.  The error is far below the BF16 rounding of the
// activations.
__device__ __forceinline__ float sigmoid32(float z) {
  return rcp_hw(1.0f + ex2_hw(-z * 1.4426950408889634f));  // e^-z = 2^(-z log2 e)
}
// SiLU z / (1 + e^-z) for the batched forward and the training kernels, and its derivative.
__device__ __forceinline__ float silu32(float z) { return z * sigmoid32(z); }
// SiLU as z/2 (1 + tanh(z/2)) on the hardware tanh (tanh.approx.f32, absolute error about
// 2^-11), of c + b for two units at once: one special-function operation and an FMA in place of an
// exponential and an IEEE division.  Used by the delayed-acceptance screen only, whose value
// decides no move by itself (the exact energy makes every final decision).
__device__ __forceinline__ float tanh_hw(float x) {
  float t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(x));
  return t;
}
__device__ __forceinline__ float2 silu_fast2(float c0, float c1, float2 b) {
  const F32x2 zero = f2_pack(-0.0f, -0.0f);
  const F32x2 h = f2_mul(f2_pack(0.5f, 0.5f), f2_add(f2_pack(c0, c1), f2_pack(b.x, b.y)), zero);
  float x, y;
  f2_unpack(h, x, y);
  float2 r;
  f2_unpack(f2_fma(h, f2_pack(tanh_hw(x), tanh_hw(y)), h), r.x, r.y);
  return r;
}
__device__ __forceinline__ float dsilu32(float z) {
  const float s = sigmoid32(z);
  return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}

// D = A * B + C, m16n8k16, bf16 x bf16 -> f32
__device__ __forceinline__ void mma16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
      "{%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

}  // namespace dev
}  // namespace sadmc

namespace sadmc {
namespace dev {

// Weight layout of mlp16 in shared memory: for output unit n, the two 32-bit words a lane t
// of its quad passes to one m16n8k16 as B (K = 16 kt + 2t, 2t + 1 and 16 kt + 8 + 2t, +1) sit
// side by side, so one 64-bit load fetches them.  Units are MLP_S1 (layer 1) and MLP_S2
// (layer 2) words apart: the 8 units g of a load meet 32 different banks.
constexpr int MLP_S1 = 24, MLP_S2 = 40;
// Word index in that layout of word w (0 .. K/2 - 1) of unit n's row-major bf16 weights.
__host__ __device__ constexpr int mlp_wword(int n, int w, int stride) {
  return n * stride + (w >> 3) * 8 + 2 * (w & 3) + ((w >> 2) & 1);
}

// Surrogate energies of T tiles of 16 rows (one warp): A fragments of G from a row-major bf16
// tile in shared memory (32 bf16 = 16 words per row), weights in the mlp_wword layout and biases
// as float pairs in shared memory, SiLU in its tanh form (silu_fast2).  Rows g and g+8 of
// tile m end in ea[m] / eb[m] (in the quad's lane t == 0 and the others alike).  The tiles share
// each weight fragment that is loaded.
template <int RW, int T>  // RW: 32-bit words between consecutive rows
__device__ __forceinline__ void mlp16(const uint32_t* gtile, const uint2* sW1, const uint2* sW2,
                                      const float2* sb1, const float2* sb2, const float2* sw3,
                                      float b3, float (&ea)[T], float (&eb)[T]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  uint32_t aG[T][2][4];
#pragma unroll
  for (int m = 0; m < T; ++m) {
    const uint32_t* p = gtile + 16 * m * RW;
#pragma unroll
    for (int kt = 0; kt < 2; ++kt) {
      aG[m][kt][0] = p[g * RW + 8 * kt + t];
      aG[m][kt][1] = p[(g + 8) * RW + 8 * kt + t];
      aG[m][kt][2] = p[g * RW + 8 * kt + 4 + t];
      aG[m][kt][3] = p[(g + 8) * RW + 8 * kt + 4 + t];
    }
  }
  uint32_t h1[T][8][2];  // units 8 j + 2 t, + 1 of rows g and g + 8, as layer 2 takes them
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int n = 8 * j + g;
    const uint2 w0 = sW1[(n * MLP_S1 + 2 * t) >> 1], w1 = sW1[(n * MLP_S1 + 8 + 2 * t) >> 1];
    const float2 bb = sb1[4 * j + t];
#pragma unroll
    for (int m = 0; m < T; ++m) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
      mma16816(c, aG[m][0], w0.x, w0.y);
      mma16816(c, aG[m][1], w1.x, w1.y);
      const float2 lo = silu_fast2(c[0], c[1], bb), hi = silu_fast2(c[2], c[3], bb);
      h1[m][j][0] = pack_bf16(lo.x, lo.y);
      h1[m][j][1] = pack_bf16(hi.x, hi.y);
    }
  }
#pragma unroll
  for (int m = 0; m < T; ++m) ea[m] = eb[m] = 0.f;
#pragma unroll 2
  for (int j = 0; j < 8; ++j) {
    const int n = 8 * j + g;
    uint2 b[4];
#pragma unroll
    for (int kt = 0; kt < 4; ++kt) b[kt] = sW2[(n * MLP_S2 + 8 * kt + 2 * t) >> 1];
    const float2 bb = sb2[4 * j + t];
    const float2 ww = sw3[4 * j + t];
#pragma unroll
    for (int m = 0; m < T; ++m) {
      float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int kt = 0; kt < 4; ++kt) {
        const uint32_t a[4] = {h1[m][2 * kt][0], h1[m][2 * kt][1], h1[m][2 * kt + 1][0], h1[m][2 * kt + 1][1]};
        mma16816(c, a, b[kt].x, b[kt].y);
      }
      const float2 lo = silu_fast2(c[0], c[1], bb), hi = silu_fast2(c[2], c[3], bb);
      ea[m] = __fmaf_rn(lo.x, ww.x, ea[m]);
      ea[m] = __fmaf_rn(lo.y, ww.y, ea[m]);
      eb[m] = __fmaf_rn(hi.x, ww.x, eb[m]);
      eb[m] = __fmaf_rn(hi.y, ww.y, eb[m]);
    }
  }
#pragma unroll
  for (int m = 0; m < T; ++m) {
    ea[m] += __shfl_xor_sync(0xffffffffu, ea[m], 1);
    ea[m] += __shfl_xor_sync(0xffffffffu, ea[m], 2);
    eb[m] += __shfl_xor_sync(0xffffffffu, eb[m], 1);
    eb[m] += __shfl_xor_sync(0xffffffffu, eb[m], 2);
    ea[m] += b3;
    eb[m] += b3;
  }
}

}  // namespace dev
}  // namespace sadmc
