// The LJ-cluster move kernel with one or two lanes per walker (src/system/lj.rs): 32 or 16
// walkers per warp, their positions in shared memory.
//
// Why: the flat-histogram bookkeeping is FP64 and an FP64 warp instruction costs the same
// whether one lane or 32 use it; with a lane per walker each such instruction serves 32
// walkers (8 with the register kernel's 4-lane groups of 8), and the move needs no group
// shuffles at all.  The pair work, 2 (N-1) binary32 terms, runs in the walker's own lane
// (or two), at full FP32 rate.
//
// Layout: each warp holds its walkers' double-single positions in shared memory as
// [coordinate][high, low][slot pair][lane], atom j = lane + LPW * slot: a lane reads two of
// its atoms' values with one 64-bit load (conflict-free) for the packed pair terms, which
// take two atoms per instruction.  Draws, gamma and sqrt(1/t) come from tables in shared
// memory as in the register kernel.
// Measured on one GB300 (8192 LJ38 walkers, 2 lanes, SAD): 8.8 -> 4.0 us per step against
// the scalar pair terms over all 64 slots and the general bookkeeping on every move.
// Global memory keeps the register kernel's [walker][6][np] planes, so the two kernels
// continue each other's runs.
#include <cuda_runtime.h>

#include <atomic>

#include "sadmc_common.cuh"
#include "sadmc_fh.cuh"
#include "sadmc_launch.h"
#include "sadmc_lj_walker.cuh"
#include "sadmc_rng.cuh"

namespace sadmc {
namespace dev {

// 4 (s^6 - s^3), s = 1/r^2 (lj.rs:78-81) in binary32 with fused steps, of two atoms p against
// one point given as its negated double-single parts (the kernels' pair terms carry a stated
// tolerance; the FP64 re-sum and the oracle replay bound it).  Double-single differences: the
// high parts of nearby atoms subtract exactly.
__device__ __forceinline__ F32x2 lj_v32x2_fused(const F32x2 ph[3], const F32x2 pl[3], const F32x2 nh[3],
                                                const F32x2 nl[3], F32x2 z) {
  F32x2 d[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) d[c] = f2_add(f2_add(ph[c], nh[c]), f2_add(pl[c], nl[c]));
  const F32x2 r2 = f2_fma(d[0], d[0], f2_fma(d[1], d[1], f2_mul(d[2], d[2], z)));
  float a, b;
  f2_unpack(r2, a, b);
  const F32x2 s = f2_pack(rcp_hw(a), rcp_hw(b));
  const F32x2 s3 = f2_mul(f2_mul(s, s, z), s, z);
  const F32x2 n3{s3.v ^ 0x8000000080000000ull};
  return f2_mul(f2_pack(4.0f, 4.0f), f2_fma(s3, s3, n3), z);
}

// One warp's shared memory: NP-atom positions and the tables.
template <int LPW, int NP>
struct LjLaneShared {
  static constexpr int PAIRS = NP / LPW / 2;  // slot pairs per lane
  float2 pos[3][2][PAIRS][32];
  float4 hi[32], lo[32];    // displacement of the batch's moves (hi.w: the atom, as int bits)
  uint64_t u53[32];
  RateTable rate;
  double gamma[128];        // [walker][4 LPW]
  __device__ float& at(int c, int part, int slot, int ln) {
    float2& v = pos[c][part][slot >> 1][ln];
    return slot & 1 ? v.y : v.x;
  }
};

template <int LPW, int NP, int FAM>
__global__ void __launch_bounds__(128) lj_lane_kernel(MoveLaunch m, LjSys s) {
  constexpr int APL = NP / LPW;
  const int wpw = LPW == 32 ? 1 : m.walkers_per_warp;
  extern __shared__ __align__(16) unsigned char lane_smem[];
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  LjLaneShared<LPW, NP>& S = reinterpret_cast<LjLaneShared<LPW, NP>*>(lane_smem)[threadIdx.x >> 5];
  const int group = lane / LPW, glane = lane % LPW;
  const int w = warp * wpw + group;
  if (group >= wpw || w >= m.n_walkers) return;  // the collectives are over the lanes that stay
  const unsigned gmask = group_mask<LPW>(group);

  Fh<LPW, FAM, BOOK_LEAN> fh;
  fh.load(m.cores, m.P, m.B, w, gmask, glane, true);
  fh.gtab = S.gamma + group * 4 * LPW;
  fh.lean_sync();
  const int n = fh.c.n;
  const float wall_r2f = __double2float_rn(s.radius2);
  float* pw = s.pos + (size_t)w * 6 * (size_t)NP;
#pragma unroll 4
  for (int k = 0; k < APL; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int j = glane + LPW * k;
      S.at(c, 0, k, lane) = pw[c * NP + j];
      S.at(c, 1, k, lane) = pw[(3 + c) * NP + j];
    }
  // the slot pairs that hold atoms of any walker of the warp
  const int pairs = __reduce_max_sync(0xffffffffu, (n + 2 * LPW - 1) / (2 * LPW));

  DS sc = ds_from_double(fh.c.tscale);
  Every resum;
  resum.init(fh.c.moves, m.resum_interval > 0 ? (uint64_t)m.resum_interval : 0);
  Draws d{};  // of this lane's move in the batch of LPW
  auto displace = [&]() {
    const DS x = ds_scale(d.g0, sc.h, sc.l), y = ds_scale(d.g1, sc.h, sc.l), z = ds_scale(d.g2, sc.h, sc.l);
    if (LPW > 1) __syncwarp(gmask);
    S.hi[lane] = make_float4(x.h, y.h, z.h, __int_as_float((int)d.which));
    S.lo[lane] = make_float4(x.l, y.l, z.l, 0.0f);
    S.u53[lane] = d.u53;
    if (LPW > 1) __syncwarp(gmask);
  };
  const F32x2 z{s.neg_zero2};
  const uint32_t n_moves = (uint32_t)m.n_moves;
  for (uint32_t it = 0; it < n_moves; ++it) {
    const int kb = (int)(it % LPW);
    if (kb == 0) {
      d = draws_continuous<true>(m.seed, (uint32_t)w, fh.c.moves + 1 + (uint64_t)glane, (uint32_t)n, 0u);
      displace();
    }
    if (SADMC_RARE((it & 31u) == 0)) S.rate.fill<1>(fh.c.moves, lane, LPW * warp_walkers(m.n_walkers, warp, wpw));
    const double2 rate = S.rate.v[it & 31u];
    fh.begin_move(rate.y);
    // plan_move of lj.rs:365-374 and move_atom of lj.rs:86-105: the energy change summed in
    // binary32 over the walker's lanes
    const int e = group * LPW + kb;
    const float4 gh = S.hi[e], gl = S.lo[e];
    const uint64_t u53 = S.u53[e];
    const int which = __float_as_int(gh.w);
    const int wl = group * LPW + which % LPW, ws = which / LPW;
    const DS fx{S.at(0, 0, ws, wl), S.at(0, 1, ws, wl)}, fy{S.at(1, 0, ws, wl), S.at(1, 1, ws, wl)},
        fz{S.at(2, 0, ws, wl), S.at(2, 1, ws, wl)};
    const DS tx = ds_add(fx, DS{gh.x, gl.x}), ty = ds_add(fy, DS{gh.y, gl.y}), tz = ds_add(fz, DS{gh.z, gl.z});
    const bool possible = !lj_outside(tx, ty, tz, fx, fy, fz, wall_r2f, s.radius2);
    const F32x2 tnh[3] = {f2_pack(-tx.h, -tx.h), f2_pack(-ty.h, -ty.h), f2_pack(-tz.h, -tz.h)},
                tnl[3] = {f2_pack(-tx.l, -tx.l), f2_pack(-ty.l, -ty.l), f2_pack(-tz.l, -tz.l)},
                fnh[3] = {f2_pack(-fx.h, -fx.h), f2_pack(-fy.h, -fy.h), f2_pack(-fz.h, -fz.h)},
                fnl[3] = {f2_pack(-fx.l, -fx.l), f2_pack(-fy.l, -fy.l), f2_pack(-fz.l, -fz.l)};
    float dn = 0.0f, dold = 0.0f;
#pragma unroll 4
    for (int p = 0; p < pairs; ++p) {
      F32x2 ph[3], pl[3];
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float2 h = S.pos[c][0][p][lane], l = S.pos[c][1][p][lane];
        ph[c] = f2_pack(h.x, h.y);
        pl[c] = f2_pack(l.x, l.y);
      }
      float n0, n1, o0, o1;
      f2_unpack(lj_v32x2_fused(ph, pl, tnh, tnl, z), n0, n1);
      f2_unpack(lj_v32x2_fused(ph, pl, fnh, fnl, z), o0, o1);
      const int j0 = glane + LPW * 2 * p, j1 = j0 + LPW;
      const bool on0 = j0 < n && j0 != which, on1 = j1 < n && j1 != which;
      dn += on0 ? n0 : 0.0f;
      dold += on0 ? o0 : 0.0f;
      dn += on1 ? n1 : 0.0f;
      dold += on1 ? o1 : 0.0f;
    }
    const float de = group_sum<LPW>(dn - dold, 0xffffffffu);
    if (SADMC_RARE(m.trace != nullptr)) {
      const uint64_t t = fh.c.moves;
      if (glane == 0 && t > m.trace_t0 && t - m.trace_t0 <= m.trace_cap) {
        TraceRec r;
        r.e1 = fh.c.E;
        r.e2 = possible ? fh.c.E + (double)de : __longlong_as_double(0x7ff8000000000000ll);
        m.trace[(size_t)w * m.trace_cap + (t - m.trace_t0 - 1)] = r;
      }
    }
    int r = fh.lean_decide(possible, de, u53);
    if (LPW > 1) __syncwarp();  // the proposed bin is read by every lane before any stores to it
    if (SADMC_RARE(r == 2)) {
      r = fh.decide_de(possible, de, u53, rate.x) ? 1 : 0;
      fh.finish_move(r == 1);
      fh.lean_sync();
    } else {
      const int old_cur = fh.cur;
      if (r == 1) fh.lean_accept(de, rate.x);
      fh.lean_finish(old_cur);
    }
    __syncwarp();
    if (r == 1 && lane == wl) {
      S.at(0, 0, ws, wl) = tx.h; S.at(0, 1, ws, wl) = tx.l;
      S.at(1, 0, ws, wl) = ty.h; S.at(1, 1, ws, wl) = ty.l;
      S.at(2, 0, ws, wl) = tz.h; S.at(2, 1, ws, wl) = tz.l;
    }
    __syncwarp();
    if (SADMC_RARE(fh.tscale_changed)) {
      fh.tscale_changed = false;
      sc = ds_from_double(fh.c.tscale);
      displace();  // the batch's remaining moves take the new scale
    }
    if (SADMC_RARE(resum.tick())) {
      // FP64 pair sum over the double-single positions (compute_energy, lj.rs:236-244)
      double e64 = 0.0;
#pragma unroll 1
      for (int j = 0; j < n; ++j) {
        const int jl = group * LPW + j % LPW, js = j / LPW;
        const double xj = (double)S.at(0, 0, js, jl) + (double)S.at(0, 1, js, jl),
                     yj = (double)S.at(1, 0, js, jl) + (double)S.at(1, 1, js, jl),
                     zj = (double)S.at(2, 0, js, jl) + (double)S.at(2, 1, js, jl);
#pragma unroll 4
        for (int k = 0; k < APL; ++k) {
          const int i = glane + LPW * k;
          if (i < n && i > j) {
            const double dx = ((double)S.at(0, 0, k, lane) + (double)S.at(0, 1, k, lane)) - xj,
                         dy = ((double)S.at(1, 0, k, lane) + (double)S.at(1, 1, k, lane)) - yj,
                         dz = ((double)S.at(2, 0, k, lane) + (double)S.at(2, 1, k, lane)) - zj;
            const double q = 1.0 / (dx * dx + dy * dy + dz * dz);
            e64 += 4.0 * (powi6(q) - powi3(q));
          }
        }
      }
      e64 = group_sum<LPW>(e64, gmask);
      const double dr = fabs(e64 - fh.c.E);
      if (dr > fh.c.drift) fh.c.drift = dr;
      if (dr > m.drift_tol) fh.c.status |= ST_DRIFT;
      fh.set_E(e64);
      fh.grew_front = false;
      if (!fh.prepare(e64)) fh.c.status |= ST_BIN_RANGE;
      else {
        if (fh.grew_front) fh.reindex_after_growth();
        fh.move_cur(fh.gidx(e64));
      }
      fh.lean_sync();
    }
  }
#pragma unroll 4
  for (int k = 0; k < APL; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int j = glane + LPW * k;
      pw[c * NP + j] = S.at(c, 0, k, lane);
      pw[(3 + c) * NP + j] = S.at(c, 1, k, lane);
    }
  fh.store(m.cores, w);
}

template <int LPW, int NP, int FAM>
cudaError_t launch_lane(const MoveLaunch& m, const LjSys& s, cudaStream_t st) {
  const int wpb = m.warps_per_block >= 1 && m.warps_per_block <= 4 ? m.warps_per_block : 1;
  const size_t bytes = (size_t)wpb * sizeof(LjLaneShared<LPW, NP>);
  // Larger than the default 48 KB for 64-atom walkers: the limit is raised once per device
  // (host threads may race to set it; setting it twice is harmless).
  static std::atomic<bool> attr[64] = {};
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  if (device < 0 || device >= 64 || !attr[device].load(std::memory_order_acquire)) {
    e = cudaFuncSetAttribute(lj_lane_kernel<LPW, NP, FAM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(4 * sizeof(LjLaneShared<LPW, NP>)));
    if (e != cudaSuccess) return e;
    if (device >= 0 && device < 64) attr[device].store(true, std::memory_order_release);
  }
  MoveLaunch ms = m;
  ms.walkers_per_warp = spread_walkers(m.n_walkers, 32 / LPW);
  const int warps = (m.n_walkers + ms.walkers_per_warp - 1) / ms.walkers_per_warp;
  lj_lane_kernel<LPW, NP, FAM><<<(warps + wpb - 1) / wpb, 32 * wpb, bytes, st>>>(ms, s);
  return cudaGetLastError();
}

}  // namespace dev

bool lj_lane_shape(int lpw, int np) { return (lpw == 1 || lpw == 2) && (np == 32 || np == 64); }

cudaError_t launch_lj_lane(const MoveLaunch& m, const LjSys& s, int lpw, cudaStream_t st) {
#define SADMC_LANE_CASE(L, N)                                                                  \
  if (lpw == L && s.np == N)                                                                   \
    return m.method == M_SAD           ? dev::launch_lane<L, N, M_SAD>(m, s, st)                 \
           : general_method(m.method) ? dev::launch_lane<L, N, dev::FAM_GENERAL>(m, s, st)      \
                                      : dev::launch_lane<L, N, dev::FAM_ANY>(m, s, st);
  SADMC_LANE_CASE(1, 32)
  SADMC_LANE_CASE(2, 32)
  SADMC_LANE_CASE(1, 64)
  SADMC_LANE_CASE(2, 64)
#undef SADMC_LANE_CASE
  return cudaErrorInvalidConfiguration;
}

}  // namespace sadmc
