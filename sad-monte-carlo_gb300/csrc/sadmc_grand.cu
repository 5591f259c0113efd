// Grand-canonical LJ cluster with the energy-number method, many walkers per launch:
// EnergyNumberMC::move_once (src/mc/energy_number.rs:540-666) with the GrandSystem moves
// of src/system/lj.rs:291-319 (add at a uniform point of the sphere, remove a uniform
// atom by swap_remove) and translations (lj.rs:86-105, 365-374).
//
// LPW lanes per walker (32 / LPW walkers per warp): atom j in lane j % LPW of the
// walker's group, slot j / LPW, double-single positions in shared memory; pair energies in
// binary32 over double-single differences with a group reduction, every decision on the
// FP64 energy E + de as the reference takes it.  The
// (E, N) bins keep the reference's layout parameters (min, num_E, max_N) and its index
// arithmetic, including the quirks that affect results (max_S_index is not remapped
// when the layout grows; Wang-Landau's histogram is a second set of bins).
#include <cuda_runtime.h>

#include "sadmc_common.cuh"
#include "sadmc_fh.cuh"
#include "sadmc_grand.h"
#include "sadmc_grand_book.cuh"
#include "sadmc_launch.h"
#include "sadmc_lj_walker.cuh"
#include "sadmc_rng.cuh"

namespace sadmc {
namespace dev {

// What a warp keeps in shared memory: its walkers' positions, the draws of a batch of LPW moves
// per walker (one lane draws one move) and gamma.
template <int LPW, int APL>
struct GrandWarpShared {
  // [coordinate][high, low][slot pair][lane], atom j in lane j % LPW of its walker, slot j / LPW
  float2 pos[3][2][(APL + 1) / 2][32];
  float4 hi[32], lo[32];   // a translation's displacement or an add's position; hi.w the atom
                           // pick and lo.w the kind, as int bits
  ulonglong2 u[32];        // the choice's and the Metropolis test's uniforms (53 bits)
  double gamma[128];
  __device__ float& at(int c, int part, int slot, int ln) {
    float2& v = pos[c][part][slot >> 1][ln];
    return slot & 1 ? v.y : v.x;
  }
};

// A step of four LJ31 walkers was 1250 warp instructions: every lane drew every move, each kind
// of move had its own pair loop, and the bookkeeping was general.  Here a lane draws one of the
// batch's moves (an add's position too), all kinds share one packed pair loop (an add has no
// old position, a removal no new one), and an ordinary SAMC move takes the lean path.
// Bound by the warp instructions of a step, with two warps per scheduler: 4096 walkers of up to
// 31 atoms, 4096 moves, 20.9 -> 10.3 ms.  (Two blocks to an SM: left to itself the compiler keeps to
// the 168 registers of three, 12.1 ms.)
template <int LPW, int APL>
__global__ void __launch_bounds__(128, 2) lj_grand_kernel(GrandLaunch m) {
  const int wpw = LPW == 32 ? 1 : m.walkers_per_warp;
  __shared__ GrandWarpShared<LPW, APL> sh[4];
  const int lane = threadIdx.x & 31;
  const int group = lane / LPW, glane = lane % LPW;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  GrandWarpShared<LPW, APL>& S = sh[threadIdx.x >> 5];
  const int w = warp * wpw + group;
  if (group >= wpw || w >= m.n_walkers) return;  // the collectives are over the lanes that stay
  const unsigned gmask = group_mask<LPW>(group);
  GrandBook<LPW> bk;
  bk.load(m, w, glane, gmask);
  bk.gtab = S.gamma + group * 4 * LPW;
  const float wall_r2f = __double2float_rn(m.radius2);
  float* pw = m.pos + (size_t)w * 6 * (size_t)m.np;
#pragma unroll
  for (int k = 0; k < APL; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int j = glane + LPW * k;
      S.at(c, 0, k, lane) = pw[c * m.np + j];
      S.at(c, 1, k, lane) = pw[(3 + c) * m.np + j];
    }
  const DS sc = ds_from_double(m.translation_scale);
  const F32x2 z{m.neg_zero2};
  // an add's position: a uniform point of the unit ball times the radius (lj.rs:292-309)
  auto add_position = [&](uint64_t t, DS& x, DS& y, DS& zz) {
    double ux = 0, uy = 0, uz = 0;
    bool found = false;
    for (int k = 0; k < 64 && !found; ++k) {
      add_candidate(m.seed, (uint32_t)w, t, k, ux, uy, uz);
      found = ux * ux + uy * uy + uz * uz < 1.0;
    }
    x = ds_from_double(ux * m.radius);
    y = ds_from_double(uy * m.radius);
    zz = ds_from_double(uz * m.radius);
    return found;
  };
  enum { kTranslate = 0, kAdd = 1, kRemove = 2, kAddNowhere = 3 };

  Every resum;
  resum.init(bk.c.moves, m.resum_interval > 0 ? (uint64_t)m.resum_interval : 0);
  const uint32_t n_moves = (uint32_t)m.n_moves;
  for (uint32_t it = 0; it < n_moves; ++it) {
    const int kb = (int)(it % LPW);
    if (kb == 0) {
      const uint64_t td = bk.c.moves + 1 + (uint64_t)glane;
      const GrandDraws d = draws_grand(m.seed, (uint32_t)w, td);
      DS x = ds_scale(d.g0, sc.h, sc.l), y = ds_scale(d.g1, sc.h, sc.l), zz = ds_scale(d.g2, sc.h, sc.l);
      int kind = kTranslate;  // unless the choice, taken at the move, turns out add or remove
      if (d.add_bit != 0) {
        kind = kRemove;
      } else if ((int64_t)d.u_choice53 <= bk.ar_thresh) {
        kind = add_position(td, x, y, zz) ? kAdd : kAddNowhere;
      }
      __syncwarp(gmask);
      S.hi[lane] = make_float4(x.h, y.h, zz.h, __int_as_float((int)d.pick));
      S.lo[lane] = make_float4(x.l, y.l, zz.l, __int_as_float(kind));
      S.u[lane] = make_ulonglong2(d.u_choice53, d.u53);
      __syncwarp(gmask);
    }
    bk.c.moves += 1;
    const uint64_t t = bk.c.moves;
    const int e = group * LPW + kb;
    const float4 gh = S.hi[e], gl = S.lo[e];
    const ulonglong2 u = S.u[e];
    const double E1 = bk.c.E;
    const int N1 = bk.c.N;
    const uint32_t pick = (uint32_t)__float_as_int(gh.w);
    const int drawn = __float_as_int(gl.w);
    const bool translation = bk.choose(u.x);
    // the kind of the move, and -1 when it is impossible
    int kind_move = translation ? kTranslate : (drawn == kRemove ? kRemove : kAdd);
    DS tx{gh.x, gl.x}, ty{gh.y, gl.y}, tz{gh.z, gl.z};
    if (kind_move == kAdd) {
      bool found = drawn == kAdd;
      // the threshold rose since the draw: the position is still to be drawn
      if (SADMC_RARE(drawn == kTranslate)) found = add_position(t, tx, ty, tz);
      if (!found || (m.has_max_N && N1 == m.max_N) || N1 + 1 >= m.ncol || N1 >= LPW * APL) kind_move = -1;
    } else if (N1 == 0) {
      kind_move = -1;
    }
    const int which = kind_move == kAdd || N1 == 0 ? 0 : (int)mulhi_range(pick, (uint32_t)N1);
    const int wl = group * LPW + which % LPW, ws = which / LPW;
    const DS fx{S.at(0, 0, ws, wl), S.at(0, 1, ws, wl)}, fy{S.at(1, 0, ws, wl), S.at(1, 1, ws, wl)},
        fz{S.at(2, 0, ws, wl), S.at(2, 1, ws, wl)};
    if (kind_move == kTranslate) {
      // the displacement was drawn, or (an add under the threshold of its draw) not kept
      if (SADMC_RARE(drawn == kAdd || drawn == kAddNowhere)) {
        const GrandDraws d = draws_grand(m.seed, (uint32_t)w, t);
        tx = ds_scale(d.g0, sc.h, sc.l); ty = ds_scale(d.g1, sc.h, sc.l); tz = ds_scale(d.g2, sc.h, sc.l);
      }
      tx = ds_add(fx, tx); ty = ds_add(fy, ty); tz = ds_add(fz, tz);
      if (lj_outside(tx, ty, tz, fx, fy, fz, wall_r2f, m.radius2)) kind_move = -1;
    }
    // the pair terms of the new position less those of the old one
    const bool has_new = kind_move != kRemove, has_old = kind_move != kAdd;
    const int skip = has_old ? which : -1;
    float de = 0.0f;
    if constexpr (APL > 1) {
      const F32x2 tnh[3] = {f2_pack(-tx.h, -tx.h), f2_pack(-ty.h, -ty.h), f2_pack(-tz.h, -tz.h)},
                  tnl[3] = {f2_pack(-tx.l, -tx.l), f2_pack(-ty.l, -ty.l), f2_pack(-tz.l, -tz.l)},
                  fnh[3] = {f2_pack(-fx.h, -fx.h), f2_pack(-fy.h, -fy.h), f2_pack(-fz.h, -fz.h)},
                  fnl[3] = {f2_pack(-fx.l, -fx.l), f2_pack(-fy.l, -fy.l), f2_pack(-fz.l, -fz.l)};
#pragma unroll
      for (int p = 0; p < APL / 2; ++p) {
        F32x2 ph[3], pl[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const float2 h = S.pos[c][0][p][lane], l = S.pos[c][1][p][lane];
          ph[c] = f2_pack(h.x, h.y);
          pl[c] = f2_pack(l.x, l.y);
        }
        float n0, n1, o0, o1;
        f2_unpack(lj_v32x2(ph, pl, tnh, tnl, z), n0, n1);
        f2_unpack(lj_v32x2(ph, pl, fnh, fnl, z), o0, o1);
        const int j0 = glane + LPW * 2 * p, j1 = j0 + LPW;
        const bool on0 = j0 < N1 && j0 != skip, on1 = j1 < N1 && j1 != skip;
        de += on0 ? (has_new ? n0 : 0.0f) - (has_old ? o0 : 0.0f) : 0.0f;
        de += on1 ? (has_new ? n1 : 0.0f) - (has_old ? o1 : 0.0f) : 0.0f;
      }
    } else {
      const float px = S.at(0, 0, 0, lane), py = S.at(1, 0, 0, lane), pz = S.at(2, 0, 0, lane),
                  qx = S.at(0, 1, 0, lane), qy = S.at(1, 1, 0, lane), qz = S.at(2, 1, 0, lane);
      float dx = (px - tx.h) + (qx - tx.l), dy = (py - ty.h) + (qy - ty.l), dz = (pz - tz.h) + (qz - tz.l);
      const float vn = lj_v32(dx * dx + dy * dy + dz * dz);
      dx = (px - fx.h) + (qx - fx.l);
      dy = (py - fy.h) + (qy - fy.l);
      dz = (pz - fz.h) + (qz - fz.l);
      const float vo = lj_v32(dx * dx + dy * dy + dz * dz);
      de = glane < N1 && glane != skip ? (has_new ? vn : 0.0f) - (has_old ? vo : 0.0f) : 0.0f;
    }
    __syncwarp();
    de = group_sum<LPW>(de, 0xffffffffu);
    if (kind_move < 0) de = 0.0f;
    const bool possible = kind_move >= 0 && fabsf(de) <= 3.0e38f;
    const int N2 = !possible || translation ? N1 : (kind_move == kAdd ? N1 + 1 : N1 - 1);
    if (SADMC_RARE(m.trace && bk.lead && t > m.trace_t0 && t - m.trace_t0 <= m.trace_cap)) {
      TraceRec r;
      r.e1 = E1;
      r.e2 = possible ? E1 + (double)de : __longlong_as_double(0x7ff8000000000000ll);
      m.trace[(size_t)w * m.trace_cap + (t - m.trace_t0 - 1)] = r;
    }
    int r = bk.wl_method ? 2 : bk.lean_decide(m, possible, de, N2, u.y);
    __syncwarp();  // every lane has read the proposed bin before one lane stores to it
    if (SADMC_RARE(r == 2)) {
      r = possible && bk.decide(m, E1, N1, E1 + (double)de, N2, translation, u.y) ? 1 : 0;
      bk.finish(m, t, E1, N1);
    } else {
      bk.lean_finish(m, t, r == 1, de, N2, translation);
    }
    __syncwarp();
    if (r == 1) {
      // ConfirmSystem::confirm (lj.rs:339-358): a removal's last atom takes the removed index
      // (swap_remove)
      int dst = which;
      if (kind_move == kAdd) dst = N1;
      if (kind_move == kRemove) {
        const int ll = group * LPW + (N1 - 1) % LPW, ls = (N1 - 1) / LPW;
        tx = DS{S.at(0, 0, ls, ll), S.at(0, 1, ls, ll)};
        ty = DS{S.at(1, 0, ls, ll), S.at(1, 1, ls, ll)};
        tz = DS{S.at(2, 0, ls, ll), S.at(2, 1, ls, ll)};
      }
      if (glane == dst % LPW) {
        const int ds = dst / LPW;
        S.at(0, 0, ds, lane) = tx.h; S.at(0, 1, ds, lane) = tx.l;
        S.at(1, 0, ds, lane) = ty.h; S.at(1, 1, ds, lane) = ty.l;
        S.at(2, 0, ds, lane) = tz.h; S.at(2, 1, ds, lane) = tz.l;
      }
    }
    __syncwarp();
    if (SADMC_RARE(resum.tick())) {
      LjWalker<LPW, APL> lj;
      lj.glane = glane;
      lj.gmask = gmask;
      lj.n = bk.c.N;
#pragma unroll
      for (int k = 0; k < APL; ++k) {
        lj.x[k] = DS{S.at(0, 0, k, lane), S.at(0, 1, k, lane)};
        lj.y[k] = DS{S.at(1, 0, k, lane), S.at(1, 1, k, lane)};
        lj.z[k] = DS{S.at(2, 0, k, lane), S.at(2, 1, k, lane)};
      }
      bk.resummed(m, lj.energy64());
    }
  }
#pragma unroll
  for (int k = 0; k < APL; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int j = glane + LPW * k;
      pw[c * m.np + j] = S.at(c, 0, k, lane);
      pw[(3 + c) * m.np + j] = S.at(c, 1, k, lane);
    }
  bk.store(m.cores, w);
}

// Initial bins of every walker (energy_number.rs:474-533): the reference's one bin
// (E = 0, N = 0) has histogram 1 and round_trips 1, and Wang-Landau's histogram 1.
__global__ void grand_init_kernel(GrandLaunch m) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= m.n_walkers) return;
  const GrandCore& c = m.cores[w];
  const size_t g = (size_t)w * m.rows * m.ncol + (size_t)c.e_base * m.ncol;
  m.B.hist[g] = 1;
  m.B.round_trips[g] = 1;
  m.B.wl_hist[g] = c.kind == 2 ? 1 : 0;
  m.B.visit[g] = 0;  // generation 0, not visited
}

}  // namespace dev

#define SADMC_GRAND_CASE(L, A)                                                          \
  if (m.lanes == L && m.np == L * A) {                                                  \
    GrandLaunch ms = m;                                                                 \
    ms.walkers_per_warp = spread_walkers(m.n_walkers, 32 / L);                          \
    const int warps = (m.n_walkers + ms.walkers_per_warp - 1) / ms.walkers_per_warp;    \
    dev::lj_grand_kernel<L, A><<<(warps + 3) / 4, 128, 0, st>>>(ms);                    \
    return cudaGetLastError();                                                          \
  }

cudaError_t launch_grand_move(const GrandLaunch& m, cudaStream_t st) {
  SADMC_GRAND_CASE(32, 1) SADMC_GRAND_CASE(16, 2) SADMC_GRAND_CASE(8, 4) SADMC_GRAND_CASE(4, 8)
  SADMC_GRAND_CASE(32, 2) SADMC_GRAND_CASE(16, 4) SADMC_GRAND_CASE(8, 8)
  return cudaErrorInvalidConfiguration;
}

cudaError_t launch_grand_init(const GrandLaunch& m, cudaStream_t st) {
  dev::grand_init_kernel<<<(m.n_walkers + 127) / 128, 128, 0, st>>>(m);
  return cudaGetLastError();
}

}  // namespace sadmc
