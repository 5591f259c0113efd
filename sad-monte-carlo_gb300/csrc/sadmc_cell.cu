// Periodic fluids with subcell lists: the subcell grid build, the FP64 energies, the
// grand-canonical WCA kernel and the launchers (the move kernel is in
// sadmc_cell_kernel.cuh; its WL and SAMC specialisations in sadmc_cell_wl.cu and
// sadmc_cell_samc.cu).
#include "sadmc_cell_kernel.cuh"

namespace sadmc {
cudaError_t launch_cell_move_wl(const MoveLaunch& m, const CellSys& s, int lpw, cudaStream_t st);
cudaError_t launch_cell_move_general(const MoveLaunch& m, const CellSys& s, int lpw, cudaStream_t st);
cudaError_t launch_cell_move_samc(const MoveLaunch& m, const CellSys& s, int lpw, cudaStream_t st);
namespace dev {

// Subcell grid of each walker (one thread per walker, atoms in index order):
// n_c = floor(L / r_cut) per axis (optcell.rs:63-73), subcell of each atom
// (optcell.rs:112-124) and the binary32 position copy.
__global__ void cell_build_kernel(const WalkerCore* cores, CellSys s, int n_walkers) {
  const int w = blockIdx.x * blockDim.x + threadIdx.x;
  if (w >= n_walkers) return;
  const int n = cores[w].n;
  const double* p = s.pos + (size_t)w * 3 * s.np;
  float4* p32 = reinterpret_cast<float4*>(s.pos32) + (size_t)w * 2 * s.np;
  int* cell_of = s.cell_of + (size_t)w * s.np;
  int* cnt = s.cell_count + (size_t)w * s.cell_cap;
  int* atoms = s.cell_atoms + (size_t)w * s.cell_cap * s.bucket;
  double L[3];
  int nc[3];
  for (int a = 0; a < 3; ++a) {
    L[a] = s.box[3 * w + a];
    nc[a] = (int)floor(L[a] / s.r_cut);
    s.ncell[3 * w + a] = nc[a];
  }
  int* status = s.build_status + w;
  *status = 0;
  if (nc[0] < 3 || nc[1] < 3 || nc[2] < 3 || nc[0] * nc[1] * nc[2] > s.cell_cap) {
    *status = ST_BAD_INPUT;
    return;
  }
  for (int c = 0; c < nc[0] * nc[1] * nc[2]; ++c) cnt[c] = 0;
  for (int i = 0; i < n; ++i) {
    const double x = p[i], y = p[s.np + i], z = p[2 * s.np + i];
    if (s.kind == SYS_WCA) put_ds<true>(p32, i, x, y, z);
    else put_ds<false>(p32, i, x, y, z);
    if (!(x >= 0.0 && x < L[0] && y >= 0.0 && y < L[1] && z >= 0.0 && z < L[2])) {
      *status = ST_BAD_INPUT;
      return;
    }
    const int cx = subcell_axis(x, L[0], nc[0]), cy = subcell_axis(y, L[1], nc[1]),
              cz = subcell_axis(z, L[2], nc[2]);
    const int c = (cx * nc[1] + cy) * nc[2] + cz;
    if (cnt[c] >= s.bucket) { *status = ST_CELL_OVERFLOW; return; }
    atoms[(size_t)c * s.bucket + cnt[c]] = i;
    cnt[c] += 1;
    cell_of[i] = c;
  }
}

// The buckets' words from their lists.
__global__ void cell_words_kernel(CellSys s, size_t cells) {
  const size_t k = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= cells) return;
  const int c = (int)(k % s.cell_cap);
  const int* nc = s.ncell + 3 * (k / s.cell_cap);
  // a walker with fewer subcells than the largest leaves the rest of its row unused
  const bool used = c < nc[0] * nc[1] * nc[2];
  s.words[k] = used ? cell_word(s.cell_atoms + k * s.bucket, min(max(s.cell_count[k], 0), s.bucket)) : 0ull;
}

// compute_energy: WCA (wca.rs:222-230) and square well (optsquare.rs:176-186) in FP64
// over the same candidate images.  One warp per walker.
template <int KIND>
__global__ void cell_energy_kernel(const WalkerCore* cores, CellSys s, int n_walkers, double* out) {
  const int lane = threadIdx.x & 31;
  const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (w >= n_walkers) return;
  const int n = cores[w].n;
  const double* p = s.pos + (size_t)w * 3 * s.np;
  const int* cell_of = s.cell_of + (size_t)w * s.np;
  const int* cnt = s.cell_count + (size_t)w * s.cell_cap;
  const int* atoms = s.cell_atoms + (size_t)w * s.cell_cap * s.bucket;
  double L[3];
  int nc[3];
  for (int a = 0; a < 3; ++a) { L[a] = s.box[3 * w + a]; nc[a] = s.ncell[3 * w + a]; }
  const double rc2 = s.r_cut * s.r_cut;
  double e = 0.0;
  long long contacts = 0;
  for (int i = lane; i < n; i += 32) {
    const double ix = p[i], iy = p[s.np + i], iz = p[2 * s.np + i];
    const int ci = cell_of[i];
    const int cx = ci / (nc[1] * nc[2]), cy = (ci / nc[2]) % nc[1], cz = ci % nc[2];
    for (int k0 = 0; k0 < 27; ++k0) {
      const int dx = k0 / 9 - 1, dy = (k0 / 3) % 3 - 1, dz = k0 % 3 - 1;
      int ux = cx + dx, uy = cy + dy, uz = cz + dz, ox = 0, oy = 0, oz = 0;
      if (ux < 0) { ux += nc[0]; ox = 1; } else if (ux >= nc[0]) { ux -= nc[0]; ox = -1; }
      if (uy < 0) { uy += nc[1]; oy = 1; } else if (uy >= nc[1]) { uy -= nc[1]; oy = -1; }
      if (uz < 0) { uz += nc[2]; oz = 1; } else if (uz >= nc[2]) { uz -= nc[2]; oz = -1; }
      const int c = (ux * nc[1] + uy) * nc[2] + uz;
      for (int q = 0; q < cnt[c]; ++q) {
        const int j = atoms[(size_t)c * s.bucket + q];
        if (j == i) continue;
        // (r1 - r2) with r2 the image of j (optcell.rs:82-89)
        const double bx = ix - (p[j] - (double)ox * L[0]);
        const double by = iy - (p[s.np + j] - (double)oy * L[1]);
        const double bz = iz - (p[2 * s.np + j] - (double)oz * L[2]);
        const double d2 = bx * bx + by * by + bz * bz;
        if (KIND == SYS_SW) { if (d2 < rc2) ++contacts; }
        else e += wca_v64(d2, rc2);
      }
    }
  }
  if (KIND == SYS_SW) {
    for (int o = 16; o > 0; o >>= 1) contacts += __shfl_xor_sync(0xffffffffu, contacts, o);
    if (lane == 0) out[w] = -(double)contacts * 0.5;
  } else {
    for (int o = 16; o > 0; o >>= 1) e += __shfl_xor_sync(0xffffffffu, e, o);
    if (lane == 0) out[w] = e * 0.5;
  }
}

// Grand-canonical WCA fluid with the energy-number method (src/mc/energy_number.rs,
// wca.rs:307-323): translations (wca.rs:342-353), adds at a uniform point of the box
// (add_atom_at, wca.rs:105-116; optcell.rs:126-130) and removals of a uniform atom
// (remove_atom_number, wca.rs:151-163; optcell.rs:177-193: swap_remove, the last atom
// takes the removed index).  LPW lanes per walker over the subcell buckets (32 by
// default: a batch of a few hundred walkers needs the warps).
//
// A step at one walker per warp was a few hundred instructions of draws on every lane and two
// chains of dependent bucket loads.  As in the move kernel: a lane draws one of a batch's moves,
// the axes run on three lanes, a bucket is one word, and a translation's two positions share
// one query when they share a subcell; an ordinary SAMC move takes the lean path.
// Bound by the chain of a step's dependent instructions and loads, with one warp per scheduler:
// 512 walkers of up to 200 atoms, 4096 moves, 28.0 -> 14.3 ms.
template <int LPW>
struct WcaGrandShared {
  float4 g[32];            // the normals and the atom pick (as int bits)
  ulonglong2 u[32];        // the choice's and the Metropolis test's uniforms (53 bits)
  double add[3][32];       // an add's position
  int kind[32];            // 0 translate, 1 add (position drawn), 2 remove, 3 add without a position
  double gamma[128];
  CellProposal prop[32 / LPW];
};

template <int LPW>
__global__ void __launch_bounds__(128) wca_grand_kernel(GrandLaunch m) {
  const int wpw = LPW == 32 ? 1 : m.walkers_per_warp;
  __shared__ WcaGrandShared<LPW> sh[4];
  const int lane = threadIdx.x & 31;
  const int group = lane / LPW, glane = lane % LPW;
  const int warp = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  WcaGrandShared<LPW>& S = sh[threadIdx.x >> 5];
  CellProposal& P = S.prop[group];
  const int w = warp * wpw + group;
  if (group >= wpw || w >= m.n_walkers) return;  // the collectives are over the lanes that stay
  const unsigned gmask = group_mask<LPW>(group);
  GrandBook<LPW> bk;
  bk.load(m, w, glane, gmask);
  bk.gtab = S.gamma + group * 4 * LPW;
  CellWalker cw;
  cw.np = m.np;
  cw.bucket = m.bucket;
  cw.p = m.pos64 + (size_t)w * 3 * m.np;
  cw.p32 = reinterpret_cast<float4*>(m.pos32) + (size_t)w * 2 * m.np;
  cw.cell_of = m.cell_of + (size_t)w * m.np;
  cw.cnt = m.cell_count + (size_t)w * m.cell_cap;
  cw.atoms = m.cell_atoms + (size_t)w * m.cell_cap * m.bucket;
  uint64_t* words = m.words + (size_t)w * m.cell_cap;
  for (int a = 0; a < 3; ++a) {
    cw.L[a] = m.box[a];
    cw.L32[a] = (float)m.box[a];
    cw.Ll32[a] = (float)(m.box[a] - (double)cw.L32[a]);
    cw.nc[a] = m.nc[a];
  }
  const double wsqr = m.r_cut * m.r_cut;
  const float wsqr32 = (float)wsqr, reach = wsqr32 + 1e-3f;
  const int ax = glane < 3 ? glane : 0;
  const double axL = m.box[ax];
  const float axL32 = (float)axL;
  const int axn = m.nc[ax];
  const int stride = ax == 0 ? cw.nc[1] * cw.nc[2] : (ax == 1 ? cw.nc[2] : 1);
  const double sc = m.translation_scale;
  // a uniform point of the box (words of add candidate 0), then put_in_cell; false: the wrap
  // gave up
  auto add_position = [&](uint64_t t, double& x, double& y, double& z) {
    const uint32_t k0 = (uint32_t)w, k1 = (uint32_t)m.seed, shi = (uint32_t)(m.seed >> 32);
    const Philox4 D = philox4x32_10(Philox4{(uint32_t)t, (uint32_t)(t >> 32), 8u, shi}, k0, k1);
    const Philox4 Q = philox4x32_10(Philox4{(uint32_t)t, (uint32_t)(t >> 32), 9u, shi}, k0, k1);
    const double s53 = 1.0 / 9007199254740992.0;
    bool bad = false;
    x = wrap_axis(cw.L[0] * ((double)u53_bits(D.x, D.y) * s53), cw.L[0], &bad);
    y = wrap_axis(cw.L[1] * ((double)u53_bits(D.z, D.w) * s53), cw.L[1], &bad);
    z = wrap_axis(cw.L[2] * ((double)u53_bits(Q.x, Q.y) * s53), cw.L[2], &bad);
  };
  // Cell::remove_atom's and add_atom_at's list operations (optcell.rs:126-193) on a bucket and its
  // word, by one lane
  auto bucket_find = [&](int c, uint64_t word, int a) {
    const int cnt = word_count(word);
    int pos = -1;
    for (int q = 0; q < cnt; ++q)
      if ((q < 4 ? word_atom(word, q) : cw.atoms[(size_t)c * cw.bucket + q]) == a) pos = q;
    return pos;
  };
  auto bucket_set = [&](int c, uint64_t word, int q, int a) {
    cw.atoms[(size_t)c * cw.bucket + q] = a;
    if (q < 4) word = (word & ~(0xfffull << (12 * q))) | ((uint64_t)a << (12 * q));
    return word;
  };
  auto bucket_count = [&](int c, uint64_t word, int cnt) {
    cw.cnt[c] = cnt;
    words[c] = (word & 0xffffffffffffull) | ((uint64_t)cnt << 48);
  };

  Every resum;
  resum.init(bk.c.moves, m.resum_interval > 0 ? (uint64_t)m.resum_interval : 0);
  const uint32_t n_moves = (uint32_t)m.n_moves;
  for (uint32_t it = 0; it < n_moves; ++it) {
    const int kb = (int)(it % LPW);
    if (kb == 0) {
      const uint64_t td = bk.c.moves + 1 + (uint64_t)glane;
      const GrandDraws d = draws_grand(m.seed, (uint32_t)w, td);
      double x = 0, y = 0, z = 0;
      int kind = 0;
      if (d.add_bit != 0) {
        kind = 2;
      } else if ((int64_t)d.u_choice53 <= bk.ar_thresh) {
        add_position(td, x, y, z);
        kind = 1;
      }
      __syncwarp(gmask);
      S.g[lane] = make_float4(d.g0, d.g1, d.g2, __int_as_float((int)d.pick));
      S.u[lane] = make_ulonglong2(d.u_choice53, d.u53);
      S.add[0][lane] = x; S.add[1][lane] = y; S.add[2][lane] = z;
      S.kind[lane] = kind;
      __syncwarp(gmask);
    }
    bk.c.moves += 1;
    const uint64_t t = bk.c.moves;
    const int e = group * LPW + kb;
    const float4 g = S.g[e];
    const ulonglong2 u = S.u[e];
    const int drawn = S.kind[e];
    const double E1 = bk.c.E;
    const int N1 = bk.c.N;
    const bool translation = bk.choose(u.x);
    // the kind of the move (0 translate, 1 add, 2 remove), and -1 when it is impossible
    int kind_move = translation ? 0 : (drawn == 2 ? 2 : 1);
    if (kind_move == 1 ? (m.has_max_N && N1 == m.max_N) || N1 >= cw.np : N1 == 0) kind_move = -1;
    const int which = kind_move == 1 || N1 == 0 ? 0 : (int)mulhi_range((uint32_t)__float_as_int(g.w), (uint32_t)N1);
    bool bad = false;
    double tax = 0.0;
    if (glane < 3 && kind_move >= 0) {
      const double f = kind_move == 1 ? 0.0 : cw.p[(size_t)ax * cw.np + which];
      tax = f;
      if (kind_move == 0) {  // plan_move: put_in_cell(from + g * scale)
        tax = wrap_axis(f + (double)(ax == 0 ? g.x : (ax == 1 ? g.y : g.z)) * sc, axL, &bad);
      } else if (kind_move == 1) {
        tax = S.add[ax][e];
        if (SADMC_RARE(drawn == 0)) {  // the threshold rose since the draw
          double x, y, z;
          add_position(t, x, y, z);
          tax = ax == 0 ? x : (ax == 1 ? y : z);
        }
      }
      P.t[ax] = tax;
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        // inside the grid even where the wrap gave up (bad: the move is impossible)
        const int cc = min(max(subcell_axis(q ? f : tax, axL, axn), 0), axn - 1);
        P.cell[q][ax] = cc * stride;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const int uu = cc + i - 1;
          const bool lo = uu < 0, hi = uu >= axn;
          CellNeighbour b;
          b.index = (uu + (lo ? axn : 0) - (hi ? axn : 0)) * stride;
          b.off = lo ? 1.0f : (hi ? -1.0f : 0.0f);
          b.shift = b.off * axL32;
          b.pad = 0;
          P.nb[q][ax][i] = b;
        }
      }
      const float th = (float)tax, fh = (float)f;
      P.nh[ax] = th; P.oh[ax] = fh;
      P.nl[ax] = (float)(tax - (double)th); P.ol[ax] = (float)(f - (double)fh);
    }
    __syncwarp();  // the proposal is stored before any lane reads it: a vote orders no memory
    const unsigned bads = __ballot_sync(0xffffffffu, bad);
    bad = (bads & gmask) != 0;
    const float4 nh = *reinterpret_cast<const float4*>(P.nh), oh = *reinterpret_cast<const float4*>(P.oh),
                 nl = *reinterpret_cast<const float4*>(P.nl), ol = *reinterpret_cast<const float4*>(P.ol);
    const int4 ni = *reinterpret_cast<const int4*>(P.cell[0]), oi = *reinterpret_cast<const int4*>(P.cell[1]);
    const bool has_new = kind_move == 0 || kind_move == 1, has_old = kind_move == 0 || kind_move == 2;
    const int new_c = has_new ? ni.x + ni.y + ni.z : 0, old_c = has_old ? oi.x + oi.y + oi.z : 0;
    const bool stay = has_new && has_old && new_c == old_c;
    const int skip = has_old ? which : -1;
    // binary32 energies of the two positions against the candidates of their 27 subcells, one
    // bucket per lane: the grand fluids are sparse (mostly empty subcells), where spreading the
    // candidates over the group costs more than it saves
    float en = 0.0f, eo = 0.0f;
    const int passes = __any_sync(0xffffffffu, has_old && !stay) ? 2 : 1;
#pragma unroll 1
    for (int p = 0; p < passes; ++p) {
      const bool wn = has_new && p == 0, wo = has_old && stay == (p == 0);
#pragma unroll 1
      for (int k = glane; k < (wn || wo ? 27 : 0); k += LPW) {
        const int kx = (k * 57) >> 9, km = k - 9 * kx, ky = (km * 11) >> 5, kz = km - 3 * ky;  // k < 27
        const CellNeighbour bx = P.nb[p][0][kx], by = P.nb[p][1][ky], bz = P.nb[p][2][kz];
        const int c = bx.index + by.index + bz.index;
        const uint64_t word = words[c];
        const int cnt = word_count(word);
#pragma unroll 1
        for (int q = 0; q < cnt; ++q) {
          const int j = q < 4 ? word_atom(word, q) : cw.atoms[(size_t)c * cw.bucket + q];
          if (j == skip) continue;
          const float4 pj = cw.p32[2 * j], pl = cw.p32[2 * j + 1];
          const float x = pj.x - bx.shift, y = pj.y - by.shift, z = pj.z - bz.shift;
          // the new position, then the old one: refined on the double-single positions when the
          // high parts put the pair within reach of the cutoff
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            const float4 qh = o ? oh : nh, ql = o ? ol : nl;
            const float dx = x - qh.x, dy = y - qh.y, dz = z - qh.z;
            if ((o ? wo : wn) && dx * dx + dy * dy + dz * dz < reach) {
              const float rx = ds_image_diff(pj.x, pl.x, qh.x, ql.x, bx.off, cw.L32[0], cw.Ll32[0]);
              const float ry = ds_image_diff(pj.y, pl.y, qh.y, ql.y, by.off, cw.L32[1], cw.Ll32[1]);
              const float rz = ds_image_diff(pj.z, pl.z, qh.z, ql.z, bz.off, cw.L32[2], cw.Ll32[2]);
              (o ? eo : en) += wca_v32(rx * rx + ry * ry + rz * rz, wsqr32);
            }
          }
        }
      }
    }
    __syncwarp();
    const float de = group_sum<LPW>(en, 0xffffffffu) - group_sum<LPW>(eo, 0xffffffffu);
    uint64_t new_word = 0;
    if (kind_move == 0 || kind_move == 1) {
      new_word = words[new_c];
      const bool full = word_count(new_word) >= cw.bucket;
      if (bad) kind_move = -1;
      else if (SADMC_RARE(full && !stay)) {
        kind_move = -1;
        bk.c.status |= ST_CELL_OVERFLOW;
      }
    }
    const bool possible = kind_move >= 0 && fabsf(de) <= 3.0e38f;
    const int N2 = !possible || translation ? N1 : (kind_move == 1 ? N1 + 1 : N1 - 1);
    if (SADMC_RARE(m.trace && bk.lead && t > m.trace_t0 && t - m.trace_t0 <= m.trace_cap)) {
      TraceRec r;
      r.e1 = E1;
      r.e2 = possible ? E1 + (double)de : __longlong_as_double(0x7ff8000000000000ll);
      m.trace[(size_t)w * m.trace_cap + (t - m.trace_t0 - 1)] = r;
    }
    int r = bk.wl_method ? 2 : bk.lean_decide(m, possible, de, N2, u.y);
    __syncwarp();  // every lane has read the proposed bin and bucket before one lane stores to it
    if (SADMC_RARE(r == 2)) {
      r = possible && bk.decide(m, E1, N1, E1 + (double)de, N2, translation, u.y) ? 1 : 0;
      bk.finish(m, t, E1, N1);
    } else {
      bk.lean_finish(m, t, r == 1, de, N2, translation);
    }
    if (r == 1) {
      // ConfirmSystem::confirm (wca.rs:276-301) on the buckets
      if (glane == 0) {
        if (has_old && !stay) {  // `which` leaves its bucket
          uint64_t word = words[old_c];
          const int cnt = word_count(word), pos = bucket_find(old_c, word, which);
          if (pos >= 0) {
            const int q = cnt - 1, last = q < 4 ? word_atom(word, q) : cw.atoms[(size_t)old_c * cw.bucket + q];
            word = bucket_set(old_c, word, pos, last);
            bucket_count(old_c, word, q);
          }
        }
        if (has_new) {
          const int a = kind_move == 0 ? which : N1;
          if (!stay) {
            const int cnt = word_count(new_word);
            bucket_count(new_c, bucket_set(new_c, new_word, cnt, a), cnt + 1);
            cw.cell_of[a] = new_c;
          }
          cw.p32[2 * a] = make_float4(nh.x, nh.y, nh.z, 0.0f);
          cw.p32[2 * a + 1] = make_float4(nl.x, nl.y, nl.z, 0.0f);
        } else if (which != N1 - 1) {
          // swap_remove: atom N1 - 1 takes index `which` (rename_neighbor, optcell.rs:419)
          const int last = N1 - 1, lc = cw.cell_of[last];
          uint64_t word = words[lc];
          const int pos = bucket_find(lc, word, last);
          if (pos >= 0) bucket_count(lc, bucket_set(lc, word, pos, which), word_count(word));
          cw.cell_of[which] = lc;
          cw.p32[2 * which] = cw.p32[2 * last];
          cw.p32[2 * which + 1] = cw.p32[2 * last + 1];
        }
      }
      if (glane < 3) {
        if (has_new) cw.p[(size_t)ax * cw.np + (kind_move == 0 ? which : N1)] = tax;
        else cw.p[(size_t)ax * cw.np + which] = cw.p[(size_t)ax * cw.np + N1 - 1];
      }
    }
    __syncwarp();
    if (SADMC_RARE(resum.tick())) {
      double es = 0.0;
      const int n = bk.c.N;
      for (int i = glane; i < n; i += LPW)
        es += pair_sum64_screened(cw, words, i, reach, [&](double r2) { return wca_v64(r2, wsqr); });
      bk.resummed(m, group_sum<LPW>(es, gmask) * 0.5);
    }
  }
  bk.store(m.cores, w);
}

}  // namespace dev

cudaError_t launch_cell_move(const MoveLaunch& m, const CellSys& s, int lpw, cudaStream_t st) {
  if (m.method == M_WL) return launch_cell_move_wl(m, s, lpw, st);
  if (m.method == M_SAMC) return launch_cell_move_samc(m, s, lpw, st);
  if (general_method(m.method)) return launch_cell_move_general(m, s, lpw, st);
  SADMC_CELL_ALL_SHAPES(M_SAD)
  return cudaErrorInvalidConfiguration;
}

cudaError_t launch_cell_build(const WalkerCore* cores, const CellSys& s, int n_walkers,
                              cudaStream_t st) {
  dev::cell_build_kernel<<<(n_walkers + 127) / 128, 128, 0, st>>>(cores, s, n_walkers);
  return cudaGetLastError();
}

cudaError_t launch_cell_words(const CellSys& s, int n_walkers, cudaStream_t st) {
  const size_t cells = (size_t)n_walkers * s.cell_cap;
  dev::cell_words_kernel<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(s, cells);
  return cudaGetLastError();
}

cudaError_t launch_cell_energy(const WalkerCore* cores, const CellSys& s, int n_walkers,
                               double* out, cudaStream_t st) {
  const int blocks = (n_walkers * 32 + 127) / 128;
  if (s.kind == SYS_SW) dev::cell_energy_kernel<SYS_SW><<<blocks, 128, 0, st>>>(cores, s, n_walkers, out);
  else dev::cell_energy_kernel<SYS_WCA><<<blocks, 128, 0, st>>>(cores, s, n_walkers, out);
  return cudaGetLastError();
}

}  // namespace sadmc

namespace sadmc {
cudaError_t launch_wca_grand_move(const GrandLaunch& m, cudaStream_t st) {
  const int lpw = m.lanes == 8 || m.lanes == 16 ? m.lanes : 32;
  GrandLaunch ms = m;
  ms.walkers_per_warp = spread_walkers(m.n_walkers, 32 / lpw);
  const int warps = (m.n_walkers + ms.walkers_per_warp - 1) / ms.walkers_per_warp;
  if (lpw == 8) dev::wca_grand_kernel<8><<<(warps + 3) / 4, 128, 0, st>>>(ms);
  else if (lpw == 16) dev::wca_grand_kernel<16><<<(warps + 3) / 4, 128, 0, st>>>(ms);
  else dev::wca_grand_kernel<32><<<(warps + 3) / 4, 128, 0, st>>>(ms);
  return cudaGetLastError();
}
}  // namespace sadmc

