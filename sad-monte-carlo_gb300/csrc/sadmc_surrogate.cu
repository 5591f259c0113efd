// Learned surrogate for delayed-acceptance LJ moves: a radial-descriptor MLP
// (32 Gaussian radial basis functions per atom -> 64 -> 64 -> 1, SiLU), per-atom energies
// summed over the cluster.  The reference has no learned part; this is the surrogate the
// delayed-acceptance moves screen with, trained online on configurations the walkers
// themselves visit.
//
//   descriptor  G[i,k] = sum_{j != i} exp(-(r_ij - c_k)^2 / (2 w^2)), c_k = 0.8 + 2.2 k/31,
//               w = 0.1 (binary32)
//   forward     fifth-generation tensor cores (tcgen05.mma, BF16 operands in shared memory,
//               FP32 accumulators in tensor memory), 128-row tiles; the last layer
//               (64 -> 1) and the SiLUs in FP32.  The delayed-acceptance move kernel runs
//               the same network per walker on mma.sync fragments (sadmc_mma.cuh).
//   training    one fused kernel per tile of whole configurations: the forward, the
//               per-configuration residual, and the backward's three contractions on the
//               tensor cores (d1 = d2 W2^T; the weight gradients W2 and W1 with the bias
//               gradients from a ones column, one M = 128, N = 112, K = 128 MMA); then
//               one kernel sums the tiles in a fixed order and takes the Adam step
//   update      Adam with bias correction on FP32 master weights; bf16 copies refreshed
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "sadmc_common.cuh"
#include "sadmc_mma.cuh"
#include "sadmc_surrogate.h"
#include "sadmc_tc05.cuh"

namespace sadmc {
namespace dev {

constexpr uint32_t kPolls = 1u << 24;  // bounded mbarrier waits (never expected to run out)

// ---- descriptors -----------------------------------------------------------------------
// Descriptors, bf16 [configs * n][32] (the forward's operand), of positions [configs][n][3]
// binary32.  A lane has one radial function; the distances are computed by a lane per neighbour
// and read back as broadcasts, two pairs to a packed instruction, and a row's terms are added in
// neighbour order.  An atom's distance to itself and the padding are far outside the functions'
// reach, where the term is +0.
//
// Bound by the issue of a term's instructions, about nine, three of them for results below 2^-126.
// (Four lanes per atom with eight functions each computed the distances four times and spent 15
// instructions a term: 8192 configurations of 38 atoms 140 us, 512 configurations 13.6 us.)
struct RbfTerms {
  F32x2 mc, s2, l2e, z;
  __device__ RbfTerms(int lane) {
    const float ck = rbf_centre(lane), inv2w2 = 1.0f / (2.0f * 0.1f * 0.1f);
    mc = f2_pack(-ck, -ck);
    s2 = f2_pack(inv2w2, inv2w2);
    l2e = f2_pack(-1.4426950408889634f, -1.4426950408889634f);  // e^-x = 2^(-x log2 e)
    z = f2_pack(-0.0f, -0.0f);
  }
  // e^(-(r - c)^2 / (2 w^2)) of two distances
  __device__ __forceinline__ void operator()(float r0, float r1, float& a, float& b) const {
    const F32x2 d = f2_add(f2_pack(r0, r1), mc);
    f2_unpack(f2_mul(f2_mul(f2_mul(d, d, z), s2, z), l2e, z), a, b);
    a = ex2_sub(a);
    b = ex2_sub(b);
  }
};
__device__ __forceinline__ float distance32(float dx, float dy, float dz) {
  return sqrtf(dx * dx + dy * dy + dz * dz);
}
constexpr float kFar = 1e18f;
// A warp takes DESC_RPW atoms of a configuration: 512 configurations of 38 atoms 11.7 us.
constexpr int DESC_RPW = 4, DESC_WARPS = 4;
__global__ void __launch_bounds__(32 * DESC_WARPS) descriptor_kernel(const float* pos, int n, int configs,
                                                                     __nv_bfloat16* gq) {
  __shared__ __align__(16) float sr[DESC_WARPS][DESC_RPW][SG_MAX_ATOMS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int per = (n + DESC_RPW - 1) / DESC_RPW;
  const int u = blockIdx.x * DESC_WARPS + warp;
  const int c = u / per, i0 = (u - c * per) * DESC_RPW;
  if (c >= configs) return;  // warp-uniform
  const float* p = pos + (size_t)c * n * 3;
  float xi[DESC_RPW][3];
#pragma unroll
  for (int q = 0; q < DESC_RPW; ++q)
#pragma unroll
    for (int a = 0; a < 3; ++a) xi[q][a] = p[3 * min(i0 + q, n - 1) + a];
  const int npad = (n + 3) & ~3;
  for (int j = lane; j < npad; j += 32) {
    const int jj = min(j, n - 1);
    const float x = p[3 * jj], y = p[3 * jj + 1], z = p[3 * jj + 2];
#pragma unroll
    for (int q = 0; q < DESC_RPW; ++q) {
      const float r = distance32(x - xi[q][0], y - xi[q][1], z - xi[q][2]);
      sr[warp][q][j] = j < n && j != i0 + q ? r : kFar;
    }
  }
  __syncwarp();
  const RbfTerms term(lane);
  float g[DESC_RPW] = {};
  for (int j = 0; j < npad; j += 4) {
#pragma unroll
    for (int q = 0; q < DESC_RPW; ++q) {
      const float4 r = *reinterpret_cast<const float4*>(&sr[warp][q][j]);
      float a, b, e, f;
      term(r.x, r.y, a, b);
      term(r.z, r.w, e, f);
      g[q] += a;
      g[q] += b;
      g[q] += e;
      g[q] += f;
    }
  }
#pragma unroll
  for (int q = 0; q < DESC_RPW; ++q)
    if (i0 + q < n)
      gq[((size_t)c * n + i0 + q) * SG_RBF + lane] = __float2bfloat16_rn(g[q]);
}

// A warp takes a whole configuration and a pair's term serves both of its atoms: row j's sum over
// its lower neighbours grows in shared memory while they are the first atom, and is taken up
// when j's turn comes, so that the order of a row's terms stays.  Half the exponentials, but
// two more shared-memory accesses a pair, one warp per configuration, and n rows of sums in
// shared memory: 8192 configurations of 38 atoms 97 us (126 with descriptor_kernel), 4096 55 (65),
// 2048 36 (35), 512 29 (12).
// Row i's distances start at its own pair of atoms when i is even, else at the next one.
__host__ __device__ constexpr int pair_rows(int half) { return half * half; }  // pairs of distances of all rows
__global__ void __launch_bounds__(32 * DESC_WARPS) descriptor_pair_kernel(const float* pos, int n, int configs,
                                                                          __nv_bfloat16* gq) {
  extern __shared__ __align__(16) float dp_sm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int half = (n + 1) >> 1;  // atoms in twos
  const int c = blockIdx.x * DESC_WARPS + warp;
  if (c >= configs) return;  // warp-uniform
  float2* G = reinterpret_cast<float2*>(dp_sm) + (size_t)warp * (half * 32 + pair_rows(half));  // [atom / 2][lane]
  float2* sr = G + half * 32;
  const float* p = pos + (size_t)c * n * 3;
  for (int k = 0; k < half; ++k) G[k * 32 + lane] = make_float2(0.0f, 0.0f);
  {
    int i = 0, j = lane, len = 2 * half;  // the lane's place among the rows; j counts from the row's start
    for (int s = lane; s < 2 * pair_rows(half); s += 32) {
      while (j >= len) {
        j -= len;
        i += 1;
        len = 2 * (half - ((i + 1) >> 1));
      }
      const int a = j + 2 * ((i + 1) >> 1), aa = min(a, n - 1), ii = min(i, n - 1);
      const float r = distance32(p[3 * aa] - p[3 * ii], p[3 * aa + 1] - p[3 * ii + 1], p[3 * aa + 2] - p[3 * ii + 2]);
      reinterpret_cast<float*>(sr)[s] = a < n && a != i ? r : kFar;
      j += 32;
    }
  }
  __syncwarp();
  const RbfTerms term(lane);
  for (int i = 0; i < n; ++i) {
    const int k0 = (i + 1) >> 1;
    const float2 gi = G[(i >> 1) * 32 + lane];
    float g = i & 1 ? gi.y : gi.x;
#pragma unroll 4
    for (int k = k0; k < half; ++k) {
      const float2 r = sr[k - k0], s = G[k * 32 + lane];
      float a, b;
      term(r.x, r.y, a, b);
      g += a;
      g += b;
      float2 t;
      f2_unpack(f2_add(f2_pack(s.x, s.y), f2_pack(a, b)), t.x, t.y);
      G[k * 32 + lane] = t;
    }
    sr += half - k0;
    gq[((size_t)c * n + i) * SG_RBF + lane] = __float2bfloat16_rn(g);
  }
}

// Energies of configurations: the FP64 sum of their rows in row order.  A block stages the rows of
// SUM_CONFIGS configurations in shared memory; a thread each adds them.  The forward's timeout flag
// is read and cleared into *flag_out.
constexpr int SUM_CONFIGS = 64, SUM_THREADS = 256;
__global__ void __launch_bounds__(SUM_THREADS) config_sum_kernel(const float* e, int n, int configs, float* out,
                                                                  unsigned int* timeout, unsigned int* flag_out) {
  extern __shared__ float se[];  // [SUM_CONFIGS][n | 1]
  const int c0 = blockIdx.x * SUM_CONFIGS, nc = min(SUM_CONFIGS, configs - c0), ld = n | 1;
  int c = threadIdx.x / n, i = threadIdx.x % n;
  const int dc = SUM_THREADS / n, di = SUM_THREADS % n;
  for (int k = threadIdx.x; k < nc * n; k += SUM_THREADS) {
    se[c * ld + i] = e[(size_t)c0 * n + k];
    c += dc;
    i += di;
    if (i >= n) { i -= n; c += 1; }
  }
  __syncthreads();
  if (blockIdx.x == 0 && threadIdx.x == 0) *flag_out = atomicExch(timeout, 0u);
  if (threadIdx.x >= nc) return;
  double s = 0.0;
  for (int q = 0; q < n; ++q) s += (double)se[threadIdx.x * ld + q];
  out[c0 + threadIdx.x] = (float)s;
}

// After a bounded wait ran out, wait (bounded again) for the asynchronous work this CTA
// still has in flight before its tensor memory is freed: the weights' bulk copies
// (copies_pending) and the MMAs of the last commit (parity last_parity, if any).
__device__ void drain_async(uint64_t* wbar, bool copies_pending, uint64_t* mbar, int last_parity) {
  if (copies_pending) tc05::mbar_wait(wbar, 0, kPolls);
  if (last_parity >= 0) tc05::mbar_wait(mbar, (uint32_t)last_parity, kPolls);
}

// Forward pass on the fifth-generation tensor cores: CTAs of 4 warps, a 128-row tile at a time.
// G (128 x 32), W1^T (64 x 32), h1 (128 x 64) and W2^T (64 x 64) sit in shared memory as
// BF16 core matrices (K-major, no swizzle); thread 0 issues the tcgen05 MMAs of each
// layer (M = 128, N = 64, K = 16 per instruction) into an FP32 accumulator in tensor
// memory (layer 2's over layer 1's) and commits them to an mbarrier;
// each warp reads its 32 rows back with tcgen05.ld for the bias, SiLU and, after layer 2,
// the 64 -> 1 output in FP32.  Writes per-row energies.  A wait that runs out (it never
// should) writes NaN energies and sets *timeout when timeout is not null.
//
// Bound by the latency of its phases and the special-function unit (256 operations a row).  A CTA
// keeps its weights and tensor memory and goes over the tiles by the grid's stride, fetching the
// next G tile while it works on one; FWD_CTAS of them share an SM.  (A CTA per tile was bound by
// the rate at which an SM took new CTAs, 2.9 us each.)  311 k rows 48.6 -> 22.5 us.
constexpr int FWD_CTAS = 6;
__global__ void __launch_bounds__(128, FWD_CTAS) forward_tc_kernel(const __nv_bfloat16* gq, int rows,
                                                                   SgWeights wts, float* e_out,
                                                                   unsigned int* timeout) {
  constexpr int M = SG_TILE, CHUNKS = M * (SG_RBF / 8) / 128;  // 16-byte chunks of a G tile per thread
  __shared__ __align__(1024) uint4 sB1[SG_H1 * SG_RBF / 8];  // W1^T
  // the G tile, 4 core matrices along K, and once layer 1 is done the h1 tile, 8 along K
  __shared__ __align__(1024) uint4 sA[M * SG_H1 / 8];
  __shared__ __align__(1024) uint4 sB2[SG_H2 * SG_H1 / 8];  // W2^T
  __shared__ float sb1[SG_H1], sb2[SG_H2], sw3[SG_H2];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ __align__(8) uint64_t wbar;  // the weights' bulk copies
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int tiles = (rows + M - 1) / M;
  unsigned char* a = reinterpret_cast<unsigned char*>(sA);
  unsigned char* b1 = reinterpret_cast<unsigned char*>(sB1);
  unsigned char* b2 = reinterpret_cast<unsigned char*>(sB2);
  const uint4* G = reinterpret_cast<const uint4*>(gq);
  uint4 gv[CHUNKS];
  // chunk c: eight rows of one core matrix side by side, so that the stores meet no bank twice
  auto chunk_row = [&](int k) { const int c = tid + 128 * k; return (c & 7) + 8 * (c >> 5); };
  auto chunk_kg = [&](int k) { return ((tid + 128 * k) >> 3) & 3; };
  auto fetch = [&](int tile) {
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k) {
      const size_t row = (size_t)tile * M + chunk_row(k);
      gv[k] = tile < tiles && row < (size_t)rows ? G[row * (SG_RBF / 8) + chunk_kg(k)] : make_uint4(0, 0, 0, 0);
    }
  };
  fetch(blockIdx.x);
  for (int k = tid; k < SG_H1; k += 128) { sb1[k] = wts.b1[k]; sb2[k] = wts.b2[k]; sw3[k] = wts.w3[k]; }
  const float b3 = wts.b3[0];
  // one 64-column accumulator for both layers: the SM's 512 columns serve eight CTAs
  if (warp == 0) tc05::tmem_alloc(&tbase, SG_H1);
  constexpr uint32_t kW1Bytes = SG_H1 * SG_RBF * 2, kW2Bytes = SG_H2 * SG_H1 * 2;
  if (tid == 0) {
    tc05::mbar_init(&mbar, 1);
    tc05::mbar_init(&wbar, 1);
    // the weights come already in core-matrix order: two bulk copies by the copy engine
    tc05::mbar_expect_tx(&wbar, kW1Bytes + kW2Bytes);
    tc05::bulk_g2s(b1, wts.wc + SG_WC_W1T, kW1Bytes, &wbar);
    tc05::bulk_g2s(b2, wts.wc + SG_WC_W2T, kW2Bytes, &wbar);
  }
  constexpr uint32_t idesc = tc05::idesc_bf16(M, SG_H1);
  const int r = warp * 32 + lane;  // this thread's row of a tile
  const uint32_t lane_addr = (uint32_t)(warp * 32) << 16;
  int last_parity = -1;  // thread 0: parity of the last commit issued
  bool wok = true, ok = true;
  int tile = blockIdx.x;
  for (; tile < tiles; tile += gridDim.x) {
#pragma unroll
    for (int k = 0; k < CHUNKS; ++k)
      *reinterpret_cast<uint4*>(a + tc05::core_offset(chunk_row(k), chunk_kg(k), SG_RBF / 8)) = gv[k];
    tc05::fence_smem_async();
    tc05::fence_before();
    __syncthreads();
    tc05::fence_after();
    const uint32_t tmem = tbase;
    // layer 1: D = G W1 (two K = 16 steps, 2 core matrices = 256 bytes apart), once the
    // weights have landed; every commit is one phase of mbar, layer 1's of parity 0
    if (tid == 0 && last_parity < 0) wok = tc05::mbar_wait(&wbar, 0, kPolls);
    if (tid == 0 && wok) {
#pragma unroll
      for (int ks = 0; ks < SG_RBF / 16; ++ks)
        tc05::mma_bf16(tmem, tc05::sdesc(tc05::smem_u32(a) + 256 * ks, 128, 128 * (SG_RBF / 8)),
                       tc05::sdesc(tc05::smem_u32(b1) + 256 * ks, 128, 128 * (SG_RBF / 8)), idesc, ks > 0);
      tc05::commit(&mbar);
      last_parity = 0;
    }
    fetch(tile + gridDim.x);
    ok = __syncthreads_and(wok);
    if (ok) ok = tc05::mbar_wait(&mbar, 0, kPolls);
    tc05::fence_after();
    if (ok) {
      // bias and SiLU of layer 1, h1 into shared memory as the layer-2 A operand (loops that
      // stay rolled, for the instruction cache)
#pragma unroll 1
      for (int q = 0; q < 4; ++q) {
        float acc[16];
        tc05::ld16(tmem + lane_addr + 16 * q, acc);
        uint32_t pk[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
          const int j = 16 * q + 2 * u;
          pk[u] = pack_bf16(silu32(acc[2 * u] + sb1[j]), silu32(acc[2 * u + 1] + sb1[j + 1]));
        }
        *reinterpret_cast<uint4*>(a + tc05::core_offset(r, 2 * q, SG_H1 / 8)) = make_uint4(pk[0], pk[1], pk[2], pk[3]);
        *reinterpret_cast<uint4*>(a + tc05::core_offset(r, 2 * q + 1, SG_H1 / 8)) =
            make_uint4(pk[4], pk[5], pk[6], pk[7]);
      }
    }
    tc05::fence_smem_async();
    tc05::fence_before();
    // the CTA agrees on the layer-1 outcome before the layer-2 MMAs are issued
    ok = __syncthreads_and(ok);
    tc05::fence_after();
    // layer 2: D = h1 W2 (four K = 16 steps) over layer 1's, which every warp has read
    if (tid == 0 && ok) {
#pragma unroll
      for (int ks = 0; ks < SG_H1 / 16; ++ks)
        tc05::mma_bf16(tmem, tc05::sdesc(tc05::smem_u32(a) + 256 * ks, 128, 128 * (SG_H1 / 8)),
                       tc05::sdesc(tc05::smem_u32(b2) + 256 * ks, 128, 128 * (SG_H1 / 8)), idesc, ks > 0);
      tc05::commit(&mbar);
      last_parity = 1;
    }
    if (ok) ok = tc05::mbar_wait(&mbar, 1, kPolls);
    ok = __syncthreads_and(ok);
    tc05::fence_after();
    if (!ok) break;
    float e = 0.f;
#pragma unroll 1
    for (int h = 0; h < 4; ++h) {
      float acc[16];
      tc05::ld16(tmem + lane_addr + 16 * h, acc);
#pragma unroll
      for (int q = 0; q < 16; ++q) e += silu32(acc[q] + sb2[16 * h + q]) * sw3[16 * h + q];
    }
    e += b3;
    const size_t row = (size_t)tile * M + r;
    if (row < (size_t)rows) e_out[row] = e;
  }
  if (!ok) {
    for (; tile < tiles; tile += gridDim.x) {
      const size_t row = (size_t)tile * M + r;
      if (row < (size_t)rows) e_out[row] = __int_as_float(0x7fc00000);
    }
    if (tid == 0) {
      if (timeout) atomicOr(timeout, 1u);
      drain_async(&wbar, !wok, &mbar, last_parity);
    }
  }
  tc05::fence_before();
  __syncthreads();
  if (warp == 0) tc05::tmem_dealloc(tbase, SG_H1);
}

// ---- fused training step ------------------------------------------------------------
// Shared memory of train_tc_kernel (byte offsets from a 1024-byte aligned base).  Every
// operand is bf16 in core matrices (8 rows x 16 bytes, K-major, no swizzle):
//   A1  G tile                    [128 rows r][K = 32 k]       layer 1 A
//   B1  W1^T                      [64 n][32 k]                 layer 1 B
//   A2  h1 tile, later d2 tile    [128 r][64]                  layer 2 A, then d1's A
//   B2  W2^T                      [64 n][64 k]                 layer 2 B
//   B3  W2                        [64 k][64 n]                 d1 = d2 W2^T, B
//   A4  [d2^T ; d1^T]             [128: n then k][K = 128 r]   weight-gradient A
//   B4  [h1^T ; G^T ; 1 ; 0]      [112: k, k', ones][128 r]    weight-gradient B
constexpr uint32_t TT_A1 = 0, TT_B1 = TT_A1 + SG_TILE * SG_RBF * 2, TT_A2 = TT_B1 + SG_H1 * SG_RBF * 2,
                   TT_B2 = TT_A2 + SG_TILE * SG_H1 * 2, TT_B3 = TT_B2 + SG_H2 * SG_H1 * 2,
                   TT_A4 = TT_B3 + SG_H1 * SG_H2 * 2, TT_B4 = TT_A4 + SG_TILE * SG_TILE * 2,
                   TT_N4 = 112, TT_END = TT_B4 + TT_N4 * SG_TILE * 2;
constexpr size_t TT_SMEM = TT_END + 1024;  // + the alignment slack of the dynamic base

__device__ __forceinline__ void st_bf16(unsigned char* base, uint32_t off, float v) {
  *reinterpret_cast<__nv_bfloat16*>(base + off) = __float2bfloat16_rn(v);
}
// Byte offset of element (row, K = r) of a [rows][K = 128 r] operand.
__device__ __forceinline__ uint32_t tt_off(int row, int r) {
  return tc05::core_offset(row, r >> 3, SG_TILE / 8) + 2 * (r & 7);
}

// Sum v[0..31] over the 32 lanes of the warp by a butterfly reduce-scatter: lane l ends with the
// sum of entry l (31 shuffles).
__device__ __forceinline__ float warp_reduce_scatter32(float v[32], int lane) {
#pragma unroll
  for (int o = 16; o >= 1; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int j = 0; j < o; ++j) {
      const float keep = up ? v[o + j] : v[j];
      const float give = up ? v[j] : v[o + j];
      v[j] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0];
}

// One CTA (8 warps; thread t holds columns 32 (t / 128) .. + 31 of tile row t % 128) per tile of
// cpt = floor(128 / n) whole configurations.  Forward as forward_tc_kernel; then, with de = dL/de_row =
// 2 (E_s - E) / C for the rows of a configuration (0 for the padding rows):
//   d2 = de w3 silu'(z2)                      (FP32, then bf16 operands)
//   d1 = (d2 W2^T) silu'(z1)                  tcgen05, M = 128, N = 64, K = 64
//   [dW2^T | db2 ; dW1^T | db1] = [d2^T ; d1^T] [h1 | G | 1]
//                                             tcgen05, M = 128, N = 112, K = 128
//   dw3 = sum_r de h2, db3 = sum_r de         warp reduce-scatters
// and writes the tile's gradient sums (part[tile]) and loss sum (lpart[tile]).  Tensor
// memory: z1 in columns 0-63, z2 in 64-127, d2 W2^T in 128-191, the weight-gradient
// accumulator in 0-111 once z1 and z2 are consumed.
//
// Bound by the serial chain of its phases (a tile per SM; the MMAs themselves are short), most of it
// the elementwise work of a thread: a thread takes half a row instead of a whole one, what a
// phase needs but does not wait for (the SiLUs' derivatives) is computed before the wait.  512
// configurations of 38 atoms: 33.5 -> 16.8 us.
constexpr int TT_THREADS = 256;
__global__ void __launch_bounds__(TT_THREADS, 2) train_tc_kernel(const __nv_bfloat16* gq, const float* target,
                                                          int n, int configs, double loss_scale,
                                                          SgWeights wts, float* part, double* lpart,
                                                          unsigned int* timeout) {
  extern __shared__ unsigned char tt_raw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>(((uintptr_t)tt_raw + 1023) & ~(uintptr_t)1023);
  __shared__ float sb1[SG_H1], sb2[SG_H2], sw3[SG_H2];
  __shared__ float se[SG_TILE];       // per-row energies
  __shared__ float sde[SG_TILE];      // per-configuration dL/de
  __shared__ double sl[SG_TILE];      // per-configuration loss terms
  __shared__ float sred[8][32];       // dw3 per warp (warps 0-3 columns 0-31, 4-7 columns 32-63)
  __shared__ float sdb3[4];
  __shared__ __align__(8) uint64_t mbar;
  __shared__ __align__(8) uint64_t wbar;
  __shared__ uint32_t tbase;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int cpt = SG_TILE / n;
  const int c0 = blockIdx.x * cpt;
  const int nc = min(cpt, configs - c0);
  const int rows_t = nc * n;
  const size_t row0 = (size_t)c0 * n;
  const int r = tid & (SG_TILE - 1), half = tid >> 7;  // a warp reads its quarter of the rows
  const uint32_t base = tc05::smem_u32(sm);
  if (tid == 0) {
    tc05::mbar_init(&mbar, 1);
    tc05::mbar_init(&wbar, 1);
    constexpr uint32_t kW1 = SG_H1 * SG_RBF * 2, kW2 = SG_H2 * SG_H1 * 2;
    tc05::mbar_expect_tx(&wbar, kW1 + 2 * kW2);
    tc05::bulk_g2s(sm + TT_B1, wts.wc + SG_WC_W1T, kW1, &wbar);
    tc05::bulk_g2s(sm + TT_B2, wts.wc + SG_WC_W2T, kW2, &wbar);
    tc05::bulk_g2s(sm + TT_B3, wts.wc + SG_WC_W2, kW2, &wbar);
  }
  // G row r into A1 (K-major) and, transposed, into B4 rows 64-95; B4 row 96 = ones,
  // rows 97-111 = 0 (their columns of the weight-gradient accumulator are unused)
  {
    uint4 gv[SG_RBF / 16];
    const uint4* G = reinterpret_cast<const uint4*>(gq);
#pragma unroll
    for (int q = 0; q < SG_RBF / 16; ++q) {
      const int kg = half * (SG_RBF / 16) + q;
      gv[q] = r < rows_t ? G[(row0 + r) * (SG_RBF / 8) + kg] : make_uint4(0, 0, 0, 0);
      *reinterpret_cast<uint4*>(sm + TT_A1 + tc05::core_offset(r, kg, SG_RBF / 8)) = gv[q];
    }
    const __nv_bfloat16* gb = reinterpret_cast<const __nv_bfloat16*>(gv);
#pragma unroll
    for (int k = 0; k < SG_RBF / 2; ++k)
      *reinterpret_cast<__nv_bfloat16*>(sm + TT_B4 + tt_off(64 + half * (SG_RBF / 2) + k, r)) = gb[k];
#pragma unroll
    for (int k = 0; k < (TT_N4 - 96) / 2; ++k)
      st_bf16(sm, TT_B4 + tt_off(96 + half * ((TT_N4 - 96) / 2) + k, r), half == 0 && k == 0 ? 1.0f : 0.0f);
  }
  for (int k = tid; k < SG_H1; k += TT_THREADS) { sb1[k] = wts.b1[k]; sb2[k] = wts.b2[k]; sw3[k] = wts.w3[k]; }
  if (warp == 0) tc05::tmem_alloc(&tbase, 256);
  tc05::fence_smem_async();
  tc05::fence_before();
  __syncthreads();
  tc05::fence_after();
  const uint32_t tmem = tbase;
  const uint32_t lane_addr = (uint32_t)((warp & 3) * 32) << 16;
  const uint32_t trow = tmem + lane_addr;
  int last_parity = -1;
  // layer 1: z1 = G W1 -> columns 0-63
  const bool wok = tid == 0 ? tc05::mbar_wait(&wbar, 0, kPolls) : true;
  if (tid == 0 && wok) {
    constexpr uint32_t id = tc05::idesc_bf16(SG_TILE, SG_H1);
#pragma unroll
    for (int ks = 0; ks < SG_RBF / 16; ++ks)
      tc05::mma_bf16(tmem, tc05::sdesc(base + TT_A1 + 256 * ks, 128, 128 * (SG_RBF / 8)),
                     tc05::sdesc(base + TT_B1 + 256 * ks, 128, 128 * (SG_RBF / 8)), id, ks > 0);
    tc05::commit(&mbar);
    last_parity = 0;
  }
  bool ok = __syncthreads_and(wok);
  if (ok) ok = tc05::mbar_wait(&mbar, 0, kPolls);
  tc05::fence_after();
  // h1 = silu(z1 + b1) -> A2 (K-major) and B4 rows 0-63 (h1^T)
  if (ok) {
    float acc[32];
    tc05::ld32(trow + 32 * half, acc);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t pk[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int j = 32 * half + 8 * q + 2 * u;
        pk[u] = pack_bf16(silu32(acc[8 * q + 2 * u] + sb1[j]), silu32(acc[8 * q + 2 * u + 1] + sb1[j + 1]));
      }
      *reinterpret_cast<uint4*>(sm + TT_A2 + tc05::core_offset(r, 4 * half + q, SG_H1 / 8)) =
          make_uint4(pk[0], pk[1], pk[2], pk[3]);
      const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(pk);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<__nv_bfloat16*>(sm + TT_B4 + tt_off(32 * half + 8 * q + u, r)) = hb[u];
    }
  }
  tc05::fence_smem_async();
  tc05::fence_before();
  ok = __syncthreads_and(ok);
  tc05::fence_after();
  // layer 2: z2 = h1 W2 -> columns 64-127
  if (tid == 0 && ok) {
    constexpr uint32_t id = tc05::idesc_bf16(SG_TILE, SG_H2);
#pragma unroll
    for (int ks = 0; ks < SG_H1 / 16; ++ks)
      tc05::mma_bf16(tmem + SG_H1, tc05::sdesc(base + TT_A2 + 256 * ks, 128, 128 * (SG_H1 / 8)),
                     tc05::sdesc(base + TT_B2 + 256 * ks, 128, 128 * (SG_H1 / 8)), id, ks > 0);
    tc05::commit(&mbar);
    last_parity = 1;
  }
  if (ok) ok = tc05::mbar_wait(&mbar, 1, kPolls);
  tc05::fence_after();
  // z2 -> the layer's output terms and their derivatives; a row's energy adds its 64 terms in
  // column order, the second half's thread after the first's
  float hv[32], dv[32], e = 0.f;
  if (ok) {
    tc05::ld32(trow + SG_H1 + 32 * half, hv);
#pragma unroll
    for (int q = 0; q < 32; ++q) {
      const float z = hv[q] + sb2[32 * half + q];
      hv[q] = silu32(z);
      dv[q] = dsilu32(z);
    }
    if (half == 0) {
#pragma unroll
      for (int q = 0; q < 32; ++q) e += hv[q] * sw3[q];
      se[r] = e;
    }
  }
  __syncthreads();
  if (half == 1) {
    if (ok) {
      e = se[r];
#pragma unroll
      for (int q = 0; q < 32; ++q) e += hv[q] * sw3[32 + q];
      e += wts.b3[0];
    }
    se[r] = e;
  }
  ok = __syncthreads_and(ok);
  // per configuration: E_s = sum of its rows (FP64, row order), residual, dL/de
  if (tid < nc) {
    double s = 0.0;
    for (int i = 0; i < n; ++i) s += (double)se[tid * n + i];
    const double res = s - (double)target[c0 + tid];
    sde[tid] = (float)(2.0 * res * loss_scale);
    sl[tid] = res * res * loss_scale;
  }
  __syncthreads();
  const float de = r < rows_t ? sde[r / n] : 0.0f;
  // d2 = de w3 silu'(z2 + b2) -> A2 (the d1 MMA's A, K-major) and A4 rows 0-63 (d2^T);
  // dw3 terms de silu(z2 + b2), reduced over the warp
  if (ok) {
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      uint32_t pk[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int k = 8 * q + 2 * u, j = 32 * half + k;
        pk[u] = pack_bf16(de * sw3[j] * dv[k], de * sw3[j + 1] * dv[k + 1]);
      }
      *reinterpret_cast<uint4*>(sm + TT_A2 + tc05::core_offset(r, 4 * half + q, SG_H2 / 8)) =
          make_uint4(pk[0], pk[1], pk[2], pk[3]);
      const __nv_bfloat16* db = reinterpret_cast<const __nv_bfloat16*>(pk);
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<__nv_bfloat16*>(sm + TT_A4 + tt_off(32 * half + 8 * q + u, r)) = db[u];
    }
  }
  tc05::fence_smem_async();
  tc05::fence_before();
  ok = __syncthreads_and(ok);
  tc05::fence_after();
  // d2 W2^T -> columns 128-191
  if (tid == 0 && ok) {
    constexpr uint32_t id = tc05::idesc_bf16(SG_TILE, SG_H1);
#pragma unroll
    for (int ks = 0; ks < SG_H2 / 16; ++ks)
      tc05::mma_bf16(tmem + 128, tc05::sdesc(base + TT_A2 + 256 * ks, 128, 128 * (SG_H2 / 8)),
                     tc05::sdesc(base + TT_B3 + 256 * ks, 128, 128 * (SG_H2 / 8)), id, ks > 0);
    tc05::commit(&mbar);
    last_parity = 0;
  }
  if (ok) {  // while it runs: dw3, and silu'(z1 + b1) into dv
#pragma unroll
    for (int q = 0; q < 32; ++q) hv[q] = de * hv[q];
    sred[warp][lane] = warp_reduce_scatter32(hv, lane);
    if (half == 0) {
      float d3 = de;
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) d3 += __shfl_xor_sync(0xffffffffu, d3, o);
      if (lane == 0) sdb3[warp] = d3;
    }
    tc05::ld32(trow + 32 * half, dv);
#pragma unroll
    for (int j = 0; j < 32; ++j) dv[j] = dsilu32(dv[j] + sb1[32 * half + j]);
  }
  if (ok) ok = tc05::mbar_wait(&mbar, 0, kPolls);
  tc05::fence_after();
  // d1 = (d2 W2^T) silu'(z1 + b1) -> A4 rows 64-127 (d1^T)
  if (ok) {
    float a3[32];
    tc05::ld32(trow + 128 + 32 * half, a3);
#pragma unroll
    for (int j = 0; j < 32; ++j) st_bf16(sm, TT_A4 + tt_off(64 + 32 * half + j, r), a3[j] * dv[j]);
  }
  tc05::fence_smem_async();
  tc05::fence_before();
  ok = __syncthreads_and(ok);
  tc05::fence_after();
  // weight gradients: [d2^T ; d1^T] [h1 | G | 1 | 0] -> columns 0-111
  if (tid == 0 && ok) {
    constexpr uint32_t id = tc05::idesc_bf16(SG_TILE, TT_N4);
#pragma unroll
    for (int ks = 0; ks < SG_TILE / 16; ++ks)
      tc05::mma_bf16(tmem, tc05::sdesc(base + TT_A4 + 256 * ks, 128, 128 * (SG_TILE / 8)),
                     tc05::sdesc(base + TT_B4 + 256 * ks, 128, 128 * (SG_TILE / 8)), id, ks > 0);
    tc05::commit(&mbar);
    last_parity = 1;
  }
  if (ok) ok = tc05::mbar_wait(&mbar, 1, kPolls);
  ok = __syncthreads_and(ok);
  tc05::fence_after();
  float* P = part + (size_t)blockIdx.x * SG_NPARAM;
  if (ok) {
    float acc[32];
    if (r < 64) {  // accumulator row n = r: dW2[k][n] in columns k, db2[n] in column 96
      tc05::ld32(trow + 32 * half, acc);
#pragma unroll
      for (int j = 0; j < 32; ++j) P[SG_OFF_W2 + (32 * half + j) * SG_H2 + r] = acc[j];
      if (half == 1) {
        tc05::ld32(trow + 96, acc);
        P[SG_OFF_B2 + r] = acc[0];
      }
    } else {       // row 64 + k: dW1[k'][k] in columns 64 + k', db1[k] in column 96
      const int k = r - 64;
      tc05::ld32(trow + 64 + 32 * half, acc);
      if (half == 0) {
#pragma unroll
        for (int j = 0; j < 32; ++j) P[SG_OFF_W1 + j * SG_H1 + k] = acc[j];
      } else {
        P[SG_OFF_B1 + k] = acc[0];
      }
    }
    if (tid < SG_H2) {  // column tid: its four warps in order
      const int w0 = 4 * (tid >> 5);
      float s = sred[w0][lane];
#pragma unroll
      for (int w = 1; w < 4; ++w) s += sred[w0 + w][lane];
      P[SG_OFF_W3 + tid] = s;
    }
    if (tid == 0) {
      P[SG_OFF_B3] = sdb3[0] + sdb3[1] + sdb3[2] + sdb3[3];
      double l = 0.0;
      for (int c = 0; c < nc; ++c) l += sl[c];
      lpart[blockIdx.x] = l;
    }
  } else {
    const float nan = __int_as_float(0x7fc00000);
    for (int p = tid; p < SG_NPARAM; p += TT_THREADS) P[p] = nan;
    if (tid == 0) {
      lpart[blockIdx.x] = __longlong_as_double(0x7ff8000000000000ll);
      if (timeout) atomicOr(timeout, 1u);
      drain_async(&wbar, !wok, &mbar, last_parity);
    }
  }
  tc05::fence_before();
  __syncthreads();
  if (warp == 0) tc05::tmem_dealloc(tmem, 256);
}

// Write parameter p's bf16 copies: W1^T / W2^T row-major (mma.sync operands) and the
// tcgen05 core-matrix orders (W1^T, W2^T, W2).
__device__ __forceinline__ void refresh_one(int p, float val, __nv_bfloat16* w1t, __nv_bfloat16* w2t,
                                            __nv_bfloat16* wc) {
  const __nv_bfloat16 v = __float2bfloat16_rn(val);
  if (p >= SG_OFF_W1 && p < SG_OFF_B1) {
    const int q = p - SG_OFF_W1, k = q / SG_H1, n = q % SG_H1;  // W1[k][n]
    w1t[n * SG_RBF + k] = v;
    wc[SG_WC_W1T + (tc05::core_offset(n, k / 8, SG_RBF / 8) + 2 * (k % 8)) / 2] = v;
  } else if (p >= SG_OFF_W2 && p < SG_OFF_B2) {
    const int q = p - SG_OFF_W2, k = q / SG_H2, n = q % SG_H2;  // W2[k][n]
    w2t[n * SG_H1 + k] = v;
    wc[SG_WC_W2T + (tc05::core_offset(n, k / 8, SG_H1 / 8) + 2 * (k % 8)) / 2] = v;
    wc[SG_WC_W2 + (tc05::core_offset(k, n / 8, SG_H2 / 8) + 2 * (n % 8)) / 2] = v;
  }
}

// grad[p] = sum over tiles (fixed order) of part[t][p]; the last block sums the loss and, with
// flag_out, reads and clears the timeout flag.  With adam.step > 0, Adam (Kingma & Ba 2015) updates master[p] and the bf16 copies.
//
// Bound by the latency of the loads: eight partial sums per parameter (tiles t = k mod 8),
// combined in a fixed order, so that the result depends only on the number of tiles; warp k of a
// block takes sum k of the block's 32 parameters (one thread for all eight, in 50 blocks, left
// a chain of 21 rounds).  171 tiles: 18.2 -> 7.0 us (8.9 with the loss added in tile order).
__global__ void __launch_bounds__(256) reduce_adam_kernel(const float* part, const double* lpart, int tiles,
                                                          float* grad, double* loss, unsigned int* timeout,
                                                          unsigned int* flag_out, SgAdam adam,
                                                          __nv_bfloat16* w1t, __nv_bfloat16* w2t,
                                                          __nv_bfloat16* wc) {
  __shared__ float a[8][32];
  __shared__ double sl[8];
  if (blockIdx.x == gridDim.x - 1) {
    // a thread takes tiles t = thread mod 256, then a tree: a dependent FP64 addition is 64 clocks
    double l = 0.0;
    for (int t = threadIdx.x; t < tiles; t += 256) l += lpart[t];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if ((threadIdx.x & 31) == 0) sl[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
      *loss = ((sl[0] + sl[1]) + (sl[2] + sl[3])) + ((sl[4] + sl[5]) + (sl[6] + sl[7]));
      if (flag_out) *flag_out = atomicExch(timeout, 0u);
    }
    return;
  }
  const int k = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p = blockIdx.x * 32 + lane;
  float v = 0.f;
  if (p < SG_NPARAM) {
#pragma unroll 8
    for (int t = k; t < tiles; t += 8) v += part[(size_t)t * SG_NPARAM + p];
  }
  a[k][lane] = v;
  __syncthreads();
  if (k != 0 || p >= SG_NPARAM) return;
  const float s = ((a[0][lane] + a[1][lane]) + (a[2][lane] + a[3][lane])) +
                  ((a[4][lane] + a[5][lane]) + (a[6][lane] + a[7][lane]));
  grad[p] = s;
  if (adam.step > 0) {
    const float beta1 = 0.9f, beta2 = 0.999f, eps = 1e-8f;
    const float mm = beta1 * adam.m[p] + (1.f - beta1) * s;
    const float vv = beta2 * adam.v[p] + (1.f - beta2) * s * s;
    adam.m[p] = mm;
    adam.v[p] = vv;
    const float mh = mm / (1.f - powf(beta1, (float)adam.step));
    const float vh = vv / (1.f - powf(beta2, (float)adam.step));
    const float w = adam.master[p] - adam.lr * mh / (sqrtf(vh) + eps);
    adam.master[p] = w;
    refresh_one(p, w, w1t, w2t, wc);
  }
}

__global__ void refresh_bf16_kernel(const float* w, __nv_bfloat16* w1t, __nv_bfloat16* w2t,
                                    __nv_bfloat16* wc) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p < SG_NPARAM) refresh_one(p, w[p], w1t, w2t, wc);
}

// Copy the walkers' current configurations (LJ double-single planes) into the training
// ring as binary32 [n][3] records with their energies.
__global__ void collect_kernel(const float* lj_pos, int np, int n, const WalkerCore* cores, int walkers,
                               float* ring_pos, float* ring_e, int ring_cap, int ring_head) {
  const int w = blockIdx.x;
  if (w >= walkers) return;
  const int slot = (ring_head + w) % ring_cap;
  const float* p = lj_pos + (size_t)w * 6 * np;
  for (int j = threadIdx.x; j < n; j += blockDim.x)
    for (int a = 0; a < 3; ++a)
      ring_pos[((size_t)slot * n + j) * 3 + a] = (float)((double)p[a * np + j] + (double)p[(3 + a) * np + j]);
  if (threadIdx.x == 0) ring_e[slot] = (float)cores[w].E;
}

__device__ __forceinline__ uint64_t splitmix64(uint64_t z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void gather_kernel(const float* ring_pos, const float* ring_e, int n, int ring_count,
                              uint64_t seed, uint64_t step, int count, float* out_pos, float* out_e) {
  const int c = blockIdx.x;
  if (c >= count) return;
  const uint64_t h = splitmix64(seed ^ splitmix64(step * 0x100000001B3ull + (uint64_t)c));
  const int s = (int)((h >> 11) % (uint64_t)ring_count);
  for (int k = threadIdx.x; k < 3 * n; k += blockDim.x)
    out_pos[(size_t)c * 3 * n + k] = ring_pos[(size_t)s * 3 * n + k];
  if (threadIdx.x == 0) out_e[c] = ring_e[s];
}

__global__ void take_flag_kernel(unsigned int* flag, unsigned int* out) { *out = atomicExch(flag, 0u); }

}  // namespace dev

cudaError_t sg_descriptors(const float* pos, int n, int configs, __nv_bfloat16* gq, cudaStream_t st) {
  using namespace dev;
  // A warp per configuration from where the two kernels cross, while a block's shared memory stays
  // below 48 KB.  Up to 42 atoms six blocks share an SM and the crossing is near 2560 configurations
  // (whole predictions: 42 atoms, 2560 configurations 98 us either way, 8192 228 against 200; 13
  // atoms 49 against 47, 74 against 69); with fewer blocks the last wave weighs more, and it is near
  // 6000 (44 atoms, 3072 configurations 112 against 132 us, 8192 233 against 219; 50 atoms, 2560
  // configurations 117 against 148, 8192 284 either way).
  const int half = (n + 1) / 2;
  const size_t smem = sizeof(float2) * DESC_WARPS * (half * 32 + pair_rows(half));
  if (configs >= (smem <= 36 * 1024 ? 2560 : 6144) && smem <= 48 * 1024) {
    descriptor_pair_kernel<<<(configs + DESC_WARPS - 1) / DESC_WARPS, 32 * DESC_WARPS, smem, st>>>(pos, n, configs, gq);
  } else {
    const long long warps = (long long)configs * ((n + DESC_RPW - 1) / DESC_RPW);
    descriptor_kernel<<<(unsigned)((warps + DESC_WARPS - 1) / DESC_WARPS), 32 * DESC_WARPS, 0, st>>>(pos, n, configs, gq);
  }
  return cudaGetLastError();
}

cudaError_t sg_config_sums(const float* e, int n, int configs, float* out, unsigned int* timeout,
                           unsigned int* flag_out, cudaStream_t st) {
  dev::config_sum_kernel<<<(configs + dev::SUM_CONFIGS - 1) / dev::SUM_CONFIGS, dev::SUM_THREADS,
                           sizeof(float) * dev::SUM_CONFIGS * (n | 1), st>>>(e, n, configs, out, timeout, flag_out);
  return cudaGetLastError();
}

namespace {
// Set by the tensor-core kernels of the allocating entry points when a wait ran out
// (their energies or gradients are NaN).
__device__ unsigned int g_sg_tc_timeout;
}  // namespace

cudaError_t sg_timeout_flag(unsigned int** flag) {
  return cudaGetSymbolAddress((void**)flag, g_sg_tc_timeout);
}

cudaError_t sg_take_flag(unsigned int* flag, unsigned int* out, cudaStream_t st) {
  dev::take_flag_kernel<<<1, 1, 0, st>>>(flag, out);
  return cudaGetLastError();
}

namespace {
// Scratch of sadmc_surrogate_loss_grads_noalloc: SgScratch for SG_STATIC_ROWS rows
// (about 2 MB), one copy per device, never allocated or freed at run time.
static __device__ __align__(256) unsigned char g_sg_static_scratch[SgScratch::bytes(SG_STATIC_ROWS)];
constexpr int kStaticDevices = 64;
std::mutex g_static_mu;
void* g_static_addr[kStaticDevices] = {};
std::atomic<bool> g_train_attr[kStaticDevices] = {};
}  // namespace

cudaError_t sg_static_scratch(void** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= kStaticDevices) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lock(g_static_mu);
  if (!g_static_addr[dev]) {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_sg_static_scratch);  // with `dev` current
    if (e != cudaSuccess) return e;
    g_static_addr[dev] = p;
  }
  *out = g_static_addr[dev];
  return cudaSuccess;
}

cudaError_t sg_forward(const __nv_bfloat16* gq, int rows, const SgWeights& w, float* e,
                       unsigned int* timeout, cudaStream_t st) {
  int d = 0, sms = 0;
  cudaError_t r = cudaGetDevice(&d);
  if (r == cudaSuccess) r = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, d);
  if (r != cudaSuccess) return r;
  const int tiles = (rows + SG_TILE - 1) / SG_TILE;
  dev::forward_tc_kernel<<<std::min(tiles, sms * dev::FWD_CTAS), 128, 0, st>>>(gq, rows, w, e, timeout);
  return cudaGetLastError();
}

cudaError_t sg_prepare_train(void) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev >= 0 && dev < kStaticDevices && g_train_attr[dev].load(std::memory_order_acquire)) return cudaSuccess;
  e = cudaFuncSetAttribute(dev::train_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)dev::TT_SMEM);
  if (e == cudaSuccess && dev >= 0 && dev < kStaticDevices) g_train_attr[dev].store(true, std::memory_order_release);
  return e;
}

cudaError_t sg_train_step(const float* pos, const float* target, int configs, int n,
                          const SgWeights& w, float* grad, const SgAdam& adam, SgScratch s,
                          double* loss_dev, unsigned int* timeout, unsigned int* flag_out, cudaStream_t st) {
  if (n < 1 || n > SG_MAX_ATOMS || configs < 1) return cudaErrorInvalidValue;
  const int tiles = sg_tiles(configs, n);
  cudaError_t e = sg_prepare_train();
  if (e == cudaSuccess) e = sg_descriptors(pos, n, configs, s.gq, st);
  if (e == cudaSuccess) {
    dev::train_tc_kernel<<<tiles, dev::TT_THREADS, dev::TT_SMEM, st>>>(s.gq, target, n, configs, 1.0 / (double)configs,
                                                           w, s.part, s.lpart, timeout);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) {
    dev::reduce_adam_kernel<<<(SG_NPARAM + 31) / 32 + 1, 256, 0, st>>>(s.part, s.lpart, tiles, grad, loss_dev, timeout, flag_out,
                                                                    adam, w.w1t, w.w2t, w.wc);
    e = cudaGetLastError();
  }
  return e;
}

cudaError_t sg_refresh(const float* master, const SgWeights& w, cudaStream_t st) {
  dev::refresh_bf16_kernel<<<(SG_NPARAM + 127) / 128, 128, 0, st>>>(master, w.w1t, w.w2t, w.wc);
  return cudaGetLastError();
}

cudaError_t sg_collect(const float* lj_pos, int np, int n, const WalkerCore* cores, int walkers,
                       float* ring_pos, float* ring_e, int ring_cap, int ring_head, cudaStream_t st) {
  dev::collect_kernel<<<walkers, 64, 0, st>>>(lj_pos, np, n, cores, walkers, ring_pos, ring_e, ring_cap, ring_head);
  return cudaGetLastError();
}

cudaError_t sg_gather(const float* ring_pos, const float* ring_e, int n, int ring_count,
                      uint64_t seed, uint64_t step, int count, float* out_pos, float* out_e,
                      cudaStream_t st) {
  dev::gather_kernel<<<count, 128, 0, st>>>(ring_pos, ring_e, n, ring_count, seed, step, count, out_pos, out_e);
  return cudaGetLastError();
}

}  // namespace sadmc
