// 2D Ising model (src/system/ising.rs), many walkers per launch.
//
// An ordinary move takes the bookkeeping's lean path and sqrt(1/t) comes from a table in
// shared memory: 4096 walkers of 32x32 run a step in 2.45 us instead of 4.55 (SAD, eight to a
// warp).
//
// Spins are int8 in global memory, index i + j*L (ising.rs:64).  A single-spin flip
// changes E by -2 s_ij (sum of 4 periodic neighbours) (ising.rs:104-119); energies are
// integers held in FP64, so the whole chain is bit-exact.  With LPW == 1 each lane is a
// walker; with LPW == 32 one walker occupies a warp: its moves run as a serial chain on
// one lane (sadmc_ising_chain.cu) when its planes fit in shared memory, here otherwise,
// and its initial descent here.
#include <cuda_runtime.h>

#include "sadmc_common.cuh"
#include "sadmc_fh.cuh"
#include "sadmc_launch.h"
#include "sadmc_rng.cuh"

namespace sadmc {
namespace dev {

// TRIAL: the warp's walkers try the lean path as LeanTrial says.
// (Two blocks to an SM: left to itself the compiler keeps to the 168 registers of three, 4096
// walkers of 32 x 32, 8192 moves, 19.6 against 19.1 ms.)
template <int LPW, int FAM, bool TRIAL>
__global__ void __launch_bounds__(128, 2) ising_move_kernel(MoveLaunch m, IsingSys s) {
  const int wpw = LPW == 32 ? 1 : m.walkers_per_warp;
  const int lane = threadIdx.x & 31;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (warp * wpw >= m.n_walkers) return;
  const int group = lane / LPW, glane = lane % LPW;
  const int w = warp * wpw + group;
  // A lane past the warp's walkers touches no walker's memory.  It leaves the descent and a warp on
  // trial (full, or the batch's last one), and else fills the rate table with the others between the
  // moves: its FP64 chains are long for few lanes (64 walkers of 32 x 32, 8192 moves, 17.5 against
  // 13.1 ms).  The branch around such lanes in the loop keeps its code off the uniform datapath,
  // five branches a step more; a loop of their own for them was slower still (4096 walkers 16.8
  // against 17.1 ms), an empty walker in each was quicker for SAD alone (16.3; SAMC 16.5 against 12.4).
  const bool own = group < wpw && w < m.n_walkers;
  if ((TRIAL || m.descent) && !own) return;
  const unsigned gmask = group_mask<LPW>(group);
  __shared__ RateTable rates[4];
  __shared__ double gammas[4][LPW > 1 ? 128 : 1];
  Fh<LPW, FAM, BOOK_LEAN, true> fh;
  const uint64_t moves0 = m.cores[warp * wpw].moves;  // the walkers share it
  if (TRIAL || own) fh.load(m.cores, m.P, m.B, w, gmask, glane, true);
  const int L = s.L;
  int8_t* S = s.spins + (size_t)w * (size_t)L * (size_t)L;
  if (m.descent) {
    // from_params descent (energy.rs:840-851): flips on the descent stream, confirmed when
    // downhill, the energy tested against max_allowed_energy after each (so at least one
    // proposal is made); energies are exact integers.
    bool done = fh.c.pad1 != 0;
    uint64_t steps = fh.c.pad2;
    for (uint64_t it = 0; it < m.n_moves; ++it) {
      if (__all_sync(0xffffffffu, done)) break;
      if (!done) {
        ++steps;
        const Draws d = draws_ising(m.seed, (uint32_t)w, steps, (uint32_t)L, 1u);
        const int i = (int)d.which, j = (int)d.j;
        const int jp = j + 1 == L ? 0 : j + 1, jm = j == 0 ? L - 1 : j - 1;
        const int ip = i + 1 == L ? 0 : i + 1, im = i == 0 ? L - 1 : i - 1;
        const int nt = S[i + jp * L] + S[i + jm * L] + S[ip + j * L] + S[im + j * L];
        const int sij = S[i + j * L];
        const double e2 = fh.c.E - (double)(nt * sij * 2);
        if (fh.uni(e2 < fh.c.E)) {
          S[i + j * L] = (int8_t)(-sij);
          if (LPW > 1) __syncwarp(gmask);
          fh.c.E = e2;
        }
        if (fh.c.E < m.descent_max) done = true;
        if (steps >= m.descent_limit) done = true;
        done = fh.uni(done);
      }
    }
    fh.c.pad2 = steps;
    fh.c.pad1 = done ? 1 : 0;
    if (glane == 0) m.cores[w] = fh.c;
    return;
  }
  RateTable& rt = rates[threadIdx.x >> 5];
  DrawCache<LPW, true> dc;
  dc.init();
  if (TRIAL || own) {
    fh.gtab = gammas[threadIdx.x >> 5] + (LPW > 1 ? group * 4 * LPW : 0);
    fh.lean_sync();
  }
  LeanTrial trial;
  const uint32_t n_moves = (uint32_t)m.n_moves;
  for (uint32_t it = 0; it < n_moves; ++it) {
    if (SADMC_RARE((it & 31u) == 0)) {
      if (TRIAL) rt.fill<2>(moves0 + it, lane, warp_walkers(m.n_walkers, warp, wpw));
      else rt.fill<1>(moves0 + it, lane, 32);
      if (TRIAL && trial.next()) fh.lean_resync();
    }
    if (!TRIAL && !own) continue;
    const uint64_t t = fh.c.moves + 1;
    const double2 rate = rt.v[it & 31u];
    fh.begin_move(rate.y);
    const Draws d = dc.get(m.seed, (uint32_t)w, t, (uint32_t)L, gmask, glane);
    const int i = (int)d.which, j = (int)d.j;
    int jp = j + 1 == L ? 0 : j + 1, jm = j == 0 ? L - 1 : j - 1;
    int ip = i + 1 == L ? 0 : i + 1, im = i == 0 ? L - 1 : i - 1;
    const int site = i + j * L;
    const int nt = S[i + jp * L] + S[i + jm * L] + S[ip + j * L] + S[im + j * L];
    const int sij = S[site];
    const float de = (float)(-(nt * sij * 2));  // exact: |de| <= 8
    if (m.trace && glane == 0 && t > m.trace_t0 && t - m.trace_t0 <= m.trace_cap) {
      TraceRec r;
      r.e1 = fh.c.E;
      r.e2 = fh.c.E + (double)de;
      m.trace[(size_t)w * m.trace_cap + (t - m.trace_t0 - 1)] = r;
    }
    int r = TRIAL && trial.skip > 0 ? 2 : fh.lean_decide(true, de, d.u53);
    if (LPW > 1) __syncwarp();  // the proposed bin is read by every lane before any stores to it
    if (SADMC_RARE(r == 2)) {
      r = fh.decide_de(true, de, d.u53, rate.x) ? 1 : 0;
      fh.finish_move(r == 1);
      if (!TRIAL || trial.skip == 0) {
        fh.lean_sync();
        if (TRIAL) ++trial.general;
      }
    } else {
      const int old_cur = fh.cur;
      if (r == 1) fh.lean_accept(de, rate.x);
      fh.lean_finish(old_cur);
    }
    if (r == 1) {
      if (LPW > 1) __syncwarp(gmask);  // after every lane's reads
      S[site] = (int8_t)(-sij);        // all lanes of the group store the same value
      if (LPW > 1) __syncwarp(gmask);
    }
  }
  if (TRIAL || own) fh.store(m.cores, w);
}

// compute_energy (ising.rs:59-75): sum over sites of s * (s_down + s_right), exact.
__global__ void ising_energy_kernel(IsingSys s, int n_walkers, double* out) {
  const int lane = threadIdx.x & 31;
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (w >= n_walkers) return;
  const int L = s.L;
  const int8_t* S = s.spins + (size_t)w * (size_t)L * (size_t)L;
  long long e = 0;
  for (int k = lane; k < L * L; k += 32) {
    const int i1 = k % L, j1 = k / L;
    const int j2 = (j1 + 1) % L, i2 = (i1 + 1) % L;
    e += (long long)((S[i1 + j2 * L] + S[i2 + j1 * L]) * S[i1 + j1 * L]);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
  if (lane == 0) out[w] = (double)e;
}

}  // namespace dev

// Largest single-walker chain (bins, spins, tables): 200 KB of the 227 KB a block may hold.
constexpr size_t kIsingStageMax = 200 * 1024;

cudaError_t launch_ising_move(const MoveLaunch& m, const IsingSys& s, int lpw, cudaStream_t st) {
  const int wpw = spread_walkers(m.n_walkers, 32 / lpw);
  const int warps = (m.n_walkers + wpw - 1) / wpw;
  MoveLaunch ms = m;
  ms.walkers_per_warp = wpw;
  const int wpb = m.warps_per_block >= 1 && m.warps_per_block <= 4 ? m.warps_per_block : 4;
  const int blocks = (warps + wpb - 1) / wpb;
  if (lpw == 1) {
    // a full warp tries the lean path on trial (see LeanTrial): 20 000 walkers of 32 x 32, their first
    // 4096 moves, SAD 36.8 -> 30.9 ms and SAMC 16.1 -> 13.1; with eight walkers a warp the lean
    // path always pays, and the trial costs 3 %
    auto kernel = general_method(m.method)         ? dev::ising_move_kernel<1, dev::FAM_GENERAL, false>
                  : m.method == M_SAD && !m.descent ? (wpw == 32 ? dev::ising_move_kernel<1, M_SAD, true>
                                                                 : dev::ising_move_kernel<1, M_SAD, false>)
                                                    : (wpw == 32 ? dev::ising_move_kernel<1, dev::FAM_ANY, true>
                                                                 : dev::ising_move_kernel<1, dev::FAM_ANY, false>);
    kernel<<<blocks, 32 * wpb, 0, st>>>(ms, s);
  } else if (lpw == 32) {
    // a lone walker per warp: its moves as a serial chain on one lane when its planes and
    // spins fit in shared memory
    if (!m.descent && ising_chain_bytes(m.P.nbins, s.L) <= kIsingStageMax)
      return launch_ising_chain(m, s, kIsingStageMax, st);
    dev::ising_move_kernel<32, dev::FAM_ANY, false><<<blocks, 32 * wpb, 0, st>>>(ms, s);
  } else {
    return cudaErrorInvalidConfiguration;
  }
  return cudaGetLastError();
}

cudaError_t launch_ising_energy(const IsingSys& s, int n_walkers, double* out, cudaStream_t st) {
  dev::ising_energy_kernel<<<(n_walkers * 32 + 127) / 128, 128, 0, st>>>(s, n_walkers, out);
  return cudaGetLastError();
}

}  // namespace sadmc
