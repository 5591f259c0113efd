// The LJ-cluster move kernel (src/system/lj.rs), many walkers per launch; included by
// the translation units that instantiate it (sadmc_lj.cu: any method; sadmc_lj_sad.cu:
// specialised for SAD).
//
// Layout: a warp packs 32/LPW walkers; walker atom j belongs to lane (j % LPW) of the
// walker's lane group, slot j / LPW, as a double-single position (hi + lo, binary32) in the
// warp's shared memory.  Per move the group computes the reference's
//   e = E + sum_{j != which} [V(|r_j - to|^2) - V(|r_j - from|^2)]      (lj.rs:86-105)
// with binary32 pair terms on double-single differences and a group shuffle reduction,
// then runs the shared flat-histogram bookkeeping.
//
// What bounds it: each walker's moves are one serial chain, and the batches this runs put
// 1.7 warps on a scheduler, so a step costs its warp instructions times about five cycles.
// Hence: an ordinary move takes the bookkeeping's lean path; the pair terms take two atoms
// per packed binary32 instruction (same roundings); draws, displacements, gamma and
// sqrt(1/t) are tables in shared memory that all lanes fill, read back with one load each
// instead of shuffles.  Measured on one GB300 (4096 LJ31 walkers, 8 lanes, SAD, past their
// first 37 k moves): 990 -> 592 warp instructions per step, 3.53 -> 1.77 us; 1024 walkers,
// two in a warp, 3.17 -> 1.51 us.  The same 4096 walkers' first 24 k moves with copies and
// descent: 98.7 -> 64.9 ms.
//
// Every resum_interval moves the energy
// is replaced by an FP64 pair sum over the double-single positions (compute_energy,
// lj.rs:236-244); the largest observed |E_incremental - E_fp64| is kept in
// WalkerCore::drift.
#pragma once
#include <cuda_runtime.h>

#include "sadmc_common.cuh"
#include "sadmc_fh.cuh"
#include "sadmc_launch.h"
#include "sadmc_rng.cuh"
#include "sadmc_lj_walker.cuh"

namespace sadmc {
namespace dev {

// The initial descent (energy.rs:840-851): downhill-only proposals of rms 0.05 on the
// descent stream until E < max_allowed_energy.
template <int LPW, int APL>
__global__ void __launch_bounds__(128) lj_descent_kernel(MoveLaunch m, LjSys s) {
  const int wpw = LPW == 32 ? 1 : m.walkers_per_warp;
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  const int group = lane / LPW, glane = lane % LPW;
  const int w = warp * wpw + group;
  if (group >= wpw || w >= m.n_walkers) return;  // the collectives are over the lanes that stay
  WalkerCore c = m.cores[w];
  LjWalker<LPW, APL> lj;
  lj.set_radius2(s.radius2);
  lj.glane = glane;
  lj.gmask = group_mask<LPW>(group);
  lj.n = c.n;
  float* pw = s.pos + (size_t)w * 6 * (size_t)s.np;
  lj.load(pw, s.np);
  const DS sc = ds_from_double(0.05);
  bool done = c.pad1 != 0;  // finished in an earlier launch
  uint64_t steps = c.pad2;
  for (uint64_t it = 0; it < m.n_moves; ++it) {
    if (__all_sync(0xffffffffu, done)) break;
    if (!done) {
      ++steps;
      Draws d = draws_continuous(m.seed, (uint32_t)w, steps, (uint32_t)lj.n, 1u);
      DS tx, ty, tz;
      float de;
      bool ok = lj.plan((int)d.which, d.g0, d.g1, d.g2, sc.h, sc.l, s.radius2, tx, ty, tz, de);
      const double e2 = c.E + (double)de;
      if (ok && finite64(e2)) {
        if (e2 < c.E) { lj.put((int)d.which, tx, ty, tz); c.E = e2; }
        if (c.E < m.descent_max) {
          // binary32 increments from overlapping starts drift; decide on the FP64 sum
          c.E = lj.energy64();
          if (c.E < m.descent_max) done = true;
        }
      }
      if (steps >= m.descent_limit) done = true;
    }
  }
  c.pad2 = steps;
  c.pad1 = done ? 1 : 0;
  double e64 = lj.energy64();
  c.E = e64;
  if (!(e64 < m.descent_max)) c.status |= ST_DESCENT_FAILED;
  else c.status &= ~(uint32_t)ST_DESCENT_FAILED;
  lj.store(pw, s.np);
  if (glane == 0) m.cores[w] = c;
}

// What a warp keeps in shared memory: its walkers' positions, and tables filled ahead by all
// lanes so that a move reads them with a few loads.
template <int LPW, int APL>
struct LjWarpShared {
  // positions [coordinate][high, low][slot pair][lane]: slots 2 p and 2 p + 1 of the lane's
  // atoms side by side, atom j in lane j % LPW of its walker, slot j / LPW
  float2 pos[3][2][(APL + 1) / 2][32];
  __device__ float& at(int c, int part, int slot, int ln) {
    float2& v = pos[c][part][slot >> 1][ln];
    return slot & 1 ? v.y : v.x;
  }
  float4 hi[32], lo[32];    // [walker][move of a batch of LPW]: displacement (high and low
                            // parts); hi.w: the atom, as int bits
  uint64_t u53[32];
  RateTable rate;
  double gamma[128];        // [walker][4 LPW]
};

// (Two blocks to an SM: left to itself the compiler may keep to the 168 registers of three and
// spill, 4096 walkers of 31 atoms, 24414 moves, 57 against 47 ms.)
template <int LPW, int APL, int FAM>
__global__ void __launch_bounds__(128, 2) lj_move_kernel(MoveLaunch m, LjSys s) {
  const int wpw = LPW == 32 ? 1 : m.walkers_per_warp;
  __shared__ LjWarpShared<LPW, APL> sh[4];
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  LjWarpShared<LPW, APL>& S = sh[threadIdx.x >> 5];
  const int group = lane / LPW, glane = lane % LPW;
  const int w = warp * wpw + group;
  if (group >= wpw || w >= m.n_walkers) return;  // the collectives are over the lanes that stay
  const unsigned gmask = group_mask<LPW>(group);

  Fh<LPW, FAM, BOOK_LEAN> fh;
  // (Stores as if they could be switched off: where the compiler sees that they are unconditional,
  // it lays the step out for the worse, 4096 fresh walkers of 31 atoms, 24414 moves, 67.6
  // against 64.8 ms.)
  fh.load(m.cores, m.P, m.B, w, gmask, glane, m.descent == 0);
  fh.gtab = S.gamma + group * 4 * LPW;
  fh.lean_sync();
  const int n = fh.c.n;
  const float wall_r2f = __double2float_rn(s.radius2);
  float* pw = s.pos + (size_t)w * 6 * (size_t)s.np;
#pragma unroll
  for (int k = 0; k < APL; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int j = glane + LPW * k;
      S.at(c, 0, k, lane) = pw[c * s.np + j];
      S.at(c, 1, k, lane) = pw[(3 + c) * s.np + j];
    }
  DS sc = ds_from_double(fh.c.tscale);
  Every resum;
  resum.init(fh.c.moves, m.resum_interval > 0 ? (uint64_t)m.resum_interval : 0);
  Draws d{};  // of this lane's move in the batch of LPW
  auto displace = [&]() {
    const DS x = ds_scale(d.g0, sc.h, sc.l), y = ds_scale(d.g1, sc.h, sc.l), z = ds_scale(d.g2, sc.h, sc.l);
    __syncwarp(gmask);
    S.hi[lane] = make_float4(x.h, y.h, z.h, __int_as_float((int)d.which));
    S.lo[lane] = make_float4(x.l, y.l, z.l, 0.0f);
    S.u53[lane] = d.u53;
    __syncwarp(gmask);
  };
  const uint32_t n_moves = (uint32_t)m.n_moves;  // launches hold at most 8192
  for (uint32_t it = 0; it < n_moves; ++it) {
    const int kb = (int)(it % LPW);
    if (kb == 0) {
      d = draws_continuous(m.seed, (uint32_t)w, fh.c.moves + 1 + (uint64_t)glane, (uint32_t)n, 0u);
      displace();
    }
    if (SADMC_RARE((it & 31u) == 0)) S.rate.fill<FAM == M_SAD ? 1 : 2>(fh.c.moves, lane, LPW * warp_walkers(m.n_walkers, warp, wpw));
    const double2 rate = S.rate.v[it & 31u];
    fh.begin_move(rate.y);
    // plan_move of lj.rs:365-374 and move_atom of lj.rs:86-105
    const int e = group * LPW + kb;
    const float4 gh = S.hi[e], gl = S.lo[e];
    const uint64_t u53 = S.u53[e];
    const int which = __float_as_int(gh.w);
    const int wl = group * LPW + which % LPW, ws = which / LPW;
    const DS fx{S.at(0, 0, ws, wl), S.at(0, 1, ws, wl)}, fy{S.at(1, 0, ws, wl), S.at(1, 1, ws, wl)},
        fz{S.at(2, 0, ws, wl), S.at(2, 1, ws, wl)};
    const DS tx = ds_add(fx, DS{gh.x, gl.x}), ty = ds_add(fy, DS{gh.y, gl.y}), tz = ds_add(fz, DS{gh.z, gl.z});
    const bool possible = !lj_outside(tx, ty, tz, fx, fy, fz, wall_r2f, s.radius2);
    // Differences of double-single positions: the high parts of two nearby atoms subtract
    // exactly (Sterbenz), so close pairs keep their full relative precision in r^2.
    float de = 0.0f;
    if constexpr (APL > 1) {  // two atoms per packed operation
      const F32x2 z{s.neg_zero2};
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
        de += j0 < n && j0 != which ? n0 - o0 : 0.0f;
        de += j1 < n && j1 != which ? n1 - o1 : 0.0f;
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
      de = glane < n && glane != which ? vn - vo : 0.0f;
    }
    de = group_sum<LPW>(de, 0xffffffffu);  // the warp's walkers take their moves together
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
    __syncwarp();  // the proposed bin is read by every lane before any stores to it
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
      LjWalker<LPW, APL> lj;
      lj.glane = glane;
      lj.gmask = gmask;
      lj.n = n;
#pragma unroll
      for (int k = 0; k < APL; ++k) {
        lj.x[k] = DS{S.at(0, 0, k, lane), S.at(0, 1, k, lane)};
        lj.y[k] = DS{S.at(1, 0, k, lane), S.at(1, 1, k, lane)};
        lj.z[k] = DS{S.at(2, 0, k, lane), S.at(2, 1, k, lane)};
      }
      const double e64 = lj.energy64();
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
#pragma unroll
  for (int k = 0; k < APL; ++k)
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const int j = glane + LPW * k;
      pw[c * s.np + j] = S.at(c, 0, k, lane);
      pw[(3 + c) * s.np + j] = S.at(c, 1, k, lane);
    }
  fh.store(m.cores, w);
}

}  // namespace dev

// Launch lj_move_kernel<LPW, APL, F> (D: lj_descent_kernel<LPW, APL>) for the (lanes per
// walker, atoms per lane) shape.
#define SADMC_LJ_CASE(L, A, F, D)                                                      \
  if (lpw == L && s.np == L * A) {                                                     \
    const int wpb = m.warps_per_block >= 1 && m.warps_per_block <= 4 ? m.warps_per_block : 4; \
    MoveLaunch ms = m;                                                                 \
    ms.walkers_per_warp = spread_walkers(m.n_walkers, 32 / L);                         \
    const int warps = (m.n_walkers + ms.walkers_per_warp - 1) / ms.walkers_per_warp;   \
    if constexpr (D) dev::lj_descent_kernel<L, A><<<(warps + wpb - 1) / wpb, 32 * wpb, 0, st>>>(ms, s); \
    else dev::lj_move_kernel<L, A, F><<<(warps + wpb - 1) / wpb, 32 * wpb, 0, st>>>(ms, s); \
    return cudaGetLastError();                                                         \
  }
#define SADMC_LJ_ALL_SHAPES(F, D)                                                      \
  SADMC_LJ_CASE(32, 1, F, D) SADMC_LJ_CASE(16, 2, F, D) SADMC_LJ_CASE(8, 4, F, D)      \
  SADMC_LJ_CASE(4, 8, F, D) SADMC_LJ_CASE(32, 2, F, D) SADMC_LJ_CASE(16, 4, F, D)      \
  SADMC_LJ_CASE(8, 8, F, D) SADMC_LJ_CASE(32, 4, F, D) SADMC_LJ_CASE(32, 8, F, D)

}  // namespace sadmc
