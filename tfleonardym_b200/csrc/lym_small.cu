// Even-odd CG on small lattices: the whole solve of one right-hand side -- sources into
// even-odd form, FP64 reliable updates, sloppy iterations, odd sites, solution back into
// the reference layout -- in one launch, by one cluster of thread blocks.
//
// The graph form (lym_solver.cu) runs five kernels per iteration over all right-hand
// sides; on a lattice of a few thousand sites each of them is a launch and a drain
// around a microsecond of work, and every pause costs a copy and a host wait.  Here an
// iteration is five cluster barriers, the CG scalars are summed through distributed
// shared memory, and every decision the host takes between graph chunks is taken by all
// threads of the cluster from the same sums (added in block order by each block, so they
// are equal bit by bit and the control flow is uniform).  The steps, tests and stopping
// rules are cg_solve_on's.  Fields stay in the workspace (L1 / L2 resident); they are
// read with plain loads, never through the read-only path, because other blocks of the
// cluster write them between barriers.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

#include "lym_small.cuh"

namespace lym {

namespace {

namespace cg = cooperative_groups;

constexpr int kSmallThreads = 256;  // at most
constexpr int kSmallMaxCtas = 8;  // portable cluster size
// A launch cannot be interrupted, so it ends after this many iterations x sites per thread x
// waves of clusters, and the host launches the rest: half a second at the 30 to 60 us that an
// iteration with one site per thread takes at most.  A solve that converges takes some hundred
// iterations, so the usual call stays one launch.
constexpr int64_t kSmallStretch = 8192;

// --- loads of fields that the cluster writes: plain, never the read-only path -----------
template <int SP, int NCOMP>
LYM_D void load_full(const EoField& f, int rhs, int cb, cx<typename Prec<SP>::real> (&v)[NCOMP]) {
  using U = typename Prec<SP>::unit;
  constexpr int CPU = Prec<SP>::CPU;
  const U* base = reinterpret_cast<const U*>(f.data) + (size_t)rhs * f.nunits * f.Vh + cb;
  float nrm = 1.0f;
  if constexpr (SP == SP16 || SP == SPB16) nrm = f.norm[(size_t)rhs * f.Vh + cb];
#pragma unroll
  for (int u = 0; u < units_for(NCOMP, CPU); ++u) {
    const U t = base[(size_t)u * f.Vh];
    if constexpr (SP == SP64) {
      v[u] = {t.x, t.y};
    } else if constexpr (SP == SP32) {
      v[2 * u] = {t.x, t.y};
      if (2 * u + 1 < NCOMP) v[2 * u + 1] = {t.z, t.w};
    } else {
      const unsigned w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (4 * u + k < NCOMP) v[4 * u + k] = nrm * unpack2<SP>(w[k]);
    }
  }
}

// acc = hop of the field `in` at site (cb, par); flip: of gamma_d in (2 and 4 dimensions),
// or the adjoint hop (3 dimensions) -- the G5IN forms of lym_eo.cuh with a run-time switch.
template <int ND, int NC, int SP, int GP>
LYM_D void small_hop(const EoGeom& g, const HopGauge& hg, const EoField& in, int rhs, int cb, int par, bool flip,
                     cx<typename Prec<SP>::real> (&acc)[Gamma<ND>::NS][NC]) {
  using RT = typename Prec<SP>::real;
  constexpr int NS = Gamma<ND>::NS;
  const int vh = (int)g.Vh;
  const int* nb = g.nbr + par * 2 * ND * vh + cb;
#pragma unroll
  for (int a = 0; a < NS; ++a)
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[a][c] = czero<RT>();
#pragma unroll
  for (int mu = 0; mu < ND; ++mu) {
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
      const bool fwd = dir == 0;
      const int ncb = __ldg(nb + (2 * mu + dir) * vh) & 0x7fffffff;
      cx<RT> u[NC][NC];
      load_link_eo<GP, NC, false>(hg.data, hg.nunits, g.Vh, mu, fwd ? par : 1 - par, fwd ? cb : ncb, u);
      cx<RT> psi[NS * NC];
      load_full<SP, NS * NC>(in, rhs, ncb, psi);
      if constexpr (ND == 3) {
        cx<RT> p0[NC], p1[NC], h[NC], t[NC];
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          p0[c] = psi[c];
          p1[c] = psi[NC + c];
        }
        const bool pos = fwd != flip;
        if (pos) proj3<RT, NC>(mu, 1, p0, p1, h);
        else proj3<RT, NC>(mu, -1, p0, p1, h);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          t[i] = fwd ? u[i][0] * h[0] : cmul_cj(u[0][i], h[0]);
#pragma unroll
          for (int j = 1; j < NC; ++j) {
            if (fwd) cmac(t[i], u[i][j], h[j]);
            else cmac_cj(t[i], u[j][i], h[j]);
          }
        }
        if (pos) recon3<RT, NC>(mu, 1, t, acc[0], acc[1]);
        else recon3<RT, NC>(mu, -1, t, acc[0], acc[1]);
      } else {
        const RT s2 = (fwd != flip) ? RT(-1) : RT(1);
#pragma unroll
        for (int a = 0; a < NS / 2; ++a) {
          const int jb = Gamma<ND>::col(mu, a), ph = Gamma<ND>::phase(mu, a);
          cx<RT> h[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const cx<RT> l = mul_phase(ph, psi[jb * NC + c]);
            h[c] = {fma(s2, l.re, psi[a * NC + c].re), fma(s2, l.im, psi[a * NC + c].im)};
          }
          const int lph = fwd ? phase_neg(phase_conj(ph)) : phase_conj(ph);
#pragma unroll
          for (int i = 0; i < NC; ++i) {
            cx<RT> t = fwd ? u[i][0] * h[0] : cmul_cj(u[0][i], h[0]);
#pragma unroll
            for (int j = 1; j < NC; ++j) {
              if (fwd) cmac(t, u[i][j], h[j]);
              else cmac_cj(t, u[j][i], h[j]);
            }
            acc[a][i] += t;
            acc[jb][i] += mul_phase(lph, t);
          }
        }
      }
    }
  }
}

// Barrier of the cluster; a single block needs no cluster barrier, whose release waits
// for all earlier memory operations (about 0.7 us a barrier against 0.05 us).
LYM_D void cluster_sync(bool single) {
  if (single) __syncthreads();
  else cg::this_cluster().sync();
}

// Sum over the cluster: every block writes its part into every block's shared memory, and
// after the barrier (which also publishes the phase's fields) each adds them in block
// order.  Two slots in turn: a block may still be reading one while the next sum is
// written into the other; the barrier in between orders the reuse.
struct ClusterSum {
  double (*slots)[kSmallMaxCtas];
  double* warps;
  int turn;
};

LYM_D double cluster_sum(ClusterSum& cs, double v) {
  cg::cluster_group cl = cg::this_cluster();
  const unsigned rank = cl.block_rank(), n = cl.num_blocks();
  double (*slot)[kSmallMaxCtas] = cs.slots + cs.turn;
  const double w = warp_sum(v);
  if ((threadIdx.x & 31) == 0) cs.warps[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x < n) {
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < kSmallThreads / 32; ++k)
      if (k * 32 < (int)blockDim.x) s += cs.warps[k];
    if (n == 1) (*slot)[0] = s;
    else cl.map_shared_rank(&(*slot)[0], threadIdx.x)[rank] = s;
  }
  cluster_sync(n == 1);
  double t = 0.0;
  for (unsigned k = 0; k < n; ++k) t += (*slot)[k];
  cs.turn ^= 1;
  return t;
}

}  // namespace

template <int ND, int NC, int SP>
__global__ void __launch_bounds__(kSmallThreads, 1)
    small_cg_kernel(const SmallLat* __restrict__ lats, int nlat, const __grid_constant__ SmallLat one, bool resume,
                    int stop) {
  constexpr int NS = Gamma<ND>::NS, NCOMP = NS * NC;
  constexpr int GP = SP == SP64 ? SP64 : (SP == SP32 ? SP32 : SP16);
  constexpr int XP = (SP == SP16 || SP == SPB16) ? SP32 : SP;
  using RT = typename Prec<SP>::real;
  using XR = typename Prec<XP>::real;
  __shared__ double slots[2][kSmallMaxCtas];
  __shared__ double warps[kSmallThreads / 32];
  cg::cluster_group cl = cg::this_cluster();
  const int nct = (int)cl.num_blocks(), sys = (int)blockIdx.x / nct;
  const bool single = nct == 1;
  int l = 0;
  if (lats) {
    int hi = nlat - 1;
    while (l < hi) {
      const int mid = (l + hi + 1) >> 1;
      if (lats[mid].sys0 <= sys) l = mid;
      else hi = mid - 1;
    }
  }
  const SmallLat& L = lats ? lats[l] : one;
  const int rhs = sys - L.sys0;
  const int vh = (int)L.g.Vh, T = nct * (int)blockDim.x;
  const int tid = (int)cl.block_rank() * (int)blockDim.x + threadIdx.x;
  const double k = L.kappa, k2 = k * k;
  const int64_t V = 2 * (int64_t)vh;
  ClusterSum cs{slots, warps, 0};
  if (resume && !L.rep[rhs].going) return;  // all blocks of the cluster
  cluster_sync(single);  // every block of the cluster runs before its shared memory is written

  double n, bnorm2, q2 = 0.0, prev_q2 = 0.0, rr = 0.0, alpha = 0.0, pause2 = 0.0, tres = 0.0;
  int iters = 0, updates = 0, pause_iter = 0;
  bool done = false, first = true, ran = false;  // ran: iterated since the last plan
  bool going = false;
  // mode 2: r = M^dag t (t = the FP64 residual, rounded), then the plan of the next run of
  // iterations; 0: t = M p; 1: r -= alpha M^dag t, and the updates of x and p
  int mode = 2;
  if (resume) {
    const SmallReport& S = L.rep[rhs];
    // the fields are where the last launch left them, ahead of t = M p
    bnorm2 = S.bnorm2;
    prev_q2 = S.prev_q2;
    rr = S.rr;
    pause2 = S.pause2;
    tres = S.true_residual;
    iters = S.iterations;
    updates = S.updates;
    pause_iter = S.pause_iter;
    first = false;
    ran = true;
    mode = 0;
  } else {
    // sources: even-odd form (gamma_d b for the hermitian system), |b|^2
    n = 0.0;
    for (int i = tid; i < 2 * vh; i += T) {
      const int par = i >= vh, cb = par ? i - vh : i;
      int x[ND];
      const int lex = eo_coords<ND>(L.g, cb, par, x);
      cx<double> v[NCOMP];
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) {
        v[c] = ld(L.b + ((int64_t)rhs * NCOMP + c) * V + lex);
        if (L.hermitian && c >= (NS / 2) * NC) v[c] = -v[c];
        n += norm2(v[c]);
      }
      store_sp<SP64, NCOMP>(par ? L.bo : L.be, rhs, cb, v);
    }
    bnorm2 = cluster_sum(cs, n);

    // b' = b_e - kappa H_eo b_o; x = 0, so the first residual is q = b'
    n = 0.0;
    for (int i = tid; i < vh; i += T) {
      cx<double> acc[NS][NC], v[NCOMP], z[NCOMP];
      small_hop<ND, NC, SP64, SP64>(L.g, L.hg64, L.bo, rhs, i, 0, false, acc);
      load_full<SP64, NCOMP>(L.be, rhs, i, v);
      cx<RT> w[NCOMP];
      cx<XR> xz[NCOMP];
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) {
        v[c] -= k * acc[c / NC][c % NC];
        n += norm2(v[c]);
        w[c] = {(RT)v[c].re, (RT)v[c].im};
        z[c] = czero<double>();
        xz[c] = czero<XR>();
      }
      store_sp<SP64, NCOMP>(L.bp, rhs, i, v);
      store_sp<SP64, NCOMP>(L.x64, rhs, i, z);
      if constexpr (SP != SP64) store_sp<XP, NCOMP>(L.xs, rhs, i, xz);
      store_sp<SP, NCOMP>(L.t, rhs, i, w);
    }
    q2 = cluster_sum(cs, n);
  }
  const double want = L.tol * L.tol * bnorm2;
  const int limit = min(L.max_iter, stop);
  while (true) {
    const bool fwd = mode == 0;
    for (int i = tid; i < vh; i += T) {
      cx<RT> acc[NS][NC], v[NCOMP];
      small_hop<ND, NC, SP, GP>(L.g, L.hgs, fwd ? L.p : L.t, rhs, i, 1, !fwd, acc);
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) v[c] = acc[c / NC][c % NC];
      store_sp<SP, NCOMP>(L.s, rhs, i, v);
    }
    cluster_sync(single);
    n = 0.0;
    const RT a = (RT)alpha;
    for (int i = tid; i < vh; i += T) {
      cx<RT> acc[NS][NC], v[NCOMP];
      // M^dag = gamma_d M gamma_d in 2 and 4 dimensions, the adjoint hop in 3
      small_hop<ND, NC, SP, GP>(L.g, L.hgs, L.s, rhs, i, 0, ND == 3 && !fwd, acc);
      load_full<SP, NCOMP>(fwd ? L.p : L.t, rhs, i, v);
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) {
        cx<RT> h = acc[c / NC][c % NC];
        if (ND != 3 && !fwd && c >= (NS / 2) * NC) h = -h;
        v[c] -= (RT)k2 * h;
      }
      if (mode == 1) {
        cx<RT> r[NCOMP];
        load_full<SP, NCOMP>(L.r, rhs, i, r);
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) v[c] = r[c] - a * v[c];
      }
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) n += (double)v[c].re * v[c].re + (double)v[c].im * v[c].im;
      store_sp<SP, NCOMP>(fwd ? L.t : L.r, rhs, i, v);
    }
    n = cluster_sum(cs, n);

    if (mode == 0) {
      if (!(n > 0.0 && rr > 0.0)) {
        // p = 0 (or not finite): nothing left to do; the true residual decides, once
        if (!ran) break;
      } else {
        alpha = rr / n;
        mode = 1;
        continue;
      }
    } else if (mode == 1) {
      const RT beta = (RT)(n / rr);
      rr = n;
      iters += 1;
      ran = true;
      const XR xa = (XR)alpha;
      for (int i = tid; i < vh; i += T) {
        cx<RT> r[NCOMP], p[NCOMP];
        cx<XR> x[NCOMP];
        load_full<SP, NCOMP>(L.r, rhs, i, r);
        load_full<XP, NCOMP>(L.xs, rhs, i, x);
        load_full<SP, NCOMP>(L.p, rhs, i, p);
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) {
          x[c] += xa * cx<XR>{(XR)p[c].re, (XR)p[c].im};
          p[c] = r[c] + beta * p[c];
        }
        store_sp<XP, NCOMP>(L.xs, rhs, i, x);
        store_sp<SP, NCOMP>(L.p, rhs, i, p);
      }
      cluster_sync(single);
      if (!(rr < pause2 || iters >= limit || iters >= pause_iter)) {
        mode = 0;
        continue;
      }
      if (!(rr < pause2 || iters >= L.max_iter || iters >= pause_iter)) {
        going = true;
        break;
      }
    } else {
      // the plan for the next run (the rules of cg_solve_on)
      tres = bnorm2 > 0 ? sqrt(q2 / bnorm2) : 0.0;
      const bool restart = first || (prev_q2 > 0.0 && q2 > 0.25 * prev_q2);
      prev_q2 = q2;
      if (!first) updates += 1;
      if (q2 <= want || n == 0.0) {
        done = true;
        break;
      }
      const double est = n * (want / q2) * 0.25;
      rr = n;
      pause2 = SP == SP64 ? est : fmax(est, L.delta * L.delta * n);
      pause_iter = SP == SP64 ? 0x7fffffff : iters + 50;
      if (iters >= L.max_iter) break;
      if (restart) {
        for (int i = tid; i < vh; i += T) {
          cx<RT> r[NCOMP];
          load_full<SP, NCOMP>(L.r, rhs, i, r);
          store_sp<SP, NCOMP>(L.p, rhs, i, r);
        }
        cluster_sync(single);
      }
      first = ran = false;
      mode = 0;
      continue;
    }

    // reliable update: x += x_sloppy, q = b' - M x in FP64, t = q
    if constexpr (SP != SP64) {
      for (int i = tid; i < vh; i += T) {
        cx<XR> d[NCOMP];
        cx<double> x[NCOMP];
        load_full<XP, NCOMP>(L.xs, rhs, i, d);
        load_full<SP64, NCOMP>(L.x64, rhs, i, x);
#pragma unroll
        for (int c = 0; c < NCOMP; ++c) {
          x[c] += cx<double>{(double)d[c].re, (double)d[c].im};
          d[c] = czero<XR>();
        }
        store_sp<SP64, NCOMP>(L.x64, rhs, i, x);
        store_sp<XP, NCOMP>(L.xs, rhs, i, d);
      }
      cluster_sync(single);
    }
    for (int i = tid; i < vh; i += T) {
      cx<double> acc[NS][NC], v[NCOMP];
      small_hop<ND, NC, SP64, SP64>(L.g, L.hg64, L.x64, rhs, i, 1, false, acc);
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) v[c] = acc[c / NC][c % NC];
      store_sp<SP64, NCOMP>(L.s64, rhs, i, v);
    }
    cluster_sync(single);
    n = 0.0;
    for (int i = tid; i < vh; i += T) {
      cx<double> acc[NS][NC], v[NCOMP], x[NCOMP];
      small_hop<ND, NC, SP64, SP64>(L.g, L.hg64, L.s64, rhs, i, 0, false, acc);
      load_full<SP64, NCOMP>(L.bp, rhs, i, v);
      load_full<SP64, NCOMP>(L.x64, rhs, i, x);
      cx<RT> w[NCOMP];
#pragma unroll
      for (int c = 0; c < NCOMP; ++c) {
        v[c] -= x[c];
        v[c] += k2 * acc[c / NC][c % NC];
        n += norm2(v[c]);
        w[c] = {(RT)v[c].re, (RT)v[c].im};
      }
      store_sp<SP, NCOMP>(L.t, rhs, i, w);
    }
    q2 = cluster_sum(cs, n);
    mode = 2;
  }

  // x_o = b_o - kappa H_oe x_e, both parities into the reference layout
  for (int i = tid; i < vh && !going; i += T) {
    cx<double> acc[NS][NC], v[NCOMP];
    int x[ND];
    load_full<SP64, NCOMP>(L.x64, rhs, i, v);
    const int le = eo_coords<ND>(L.g, i, 0, x);
#pragma unroll
    for (int c = 0; c < NCOMP; ++c) st(L.x + ((int64_t)rhs * NCOMP + c) * V + le, v[c]);
    small_hop<ND, NC, SP64, SP64>(L.g, L.hg64, L.x64, rhs, i, 1, false, acc);
    load_full<SP64, NCOMP>(L.bo, rhs, i, v);
    const int lo = eo_coords<ND>(L.g, i, 1, x);
#pragma unroll
    for (int c = 0; c < NCOMP; ++c)
      st(L.x + ((int64_t)rhs * NCOMP + c) * V + lo, v[c] - k * acc[c / NC][c % NC]);
  }
  if (tid == 0)
    L.rep[rhs] = SmallReport{tres, iters, updates, done ? 1 : 0, going ? 1 : 0, bnorm2, prev_q2, rr, pause2, pause_iter, 0};
  cluster_sync(single);  // no block leaves while its shared memory may still be read or written
}

// ---------------------------------------------------------------------------
// host
// ---------------------------------------------------------------------------
// Where the line to the graph form lies: the measured crossovers (one B200, whole solves to
// 1e-10, kappa 0.12, the resident form's time / the graph form's).  The graph form's cost is
// launches, and with reduced precisions the host's waits at every reliable update, so the
// reduced precisions cross later; four dimensions cross earlier, by FP64 work on few SMs.
//   one lattice, FP64:  2D SU(2) 64^2 1 rhs 239 / 529 us, 128 x 64 339 / 512, 128^2 554 / 524;
//     3D SU(2) 20^3 569 / 707, 24^3 924 / 703; 4D SU(3) 4 x 4 x 8 x 8 1029 / 1391, 8^4 1269 / 1441
//     with 1 rhs and 2196 / 1903 with 16, 8^3 x 16 2440 / 1597
//   FP32 (FP16):  2D 128^2 571 / 1550 (539 / 1208); 3D 24^3 887 / 1923 (821 / 1389); 4D SU(3)
//     8^3 x 16 1971 / 3132 (1798 / 2407) with 1 rhs, 3435 / 4174 (3090 / 2983) with 16
//   The other classes, time of the graph form over this one's with 1 / 12 / 32 rhs (-: above the
//     rule): FP64 3D SU(3) 16^3 1.53 / 1.78 / 1.65, 4D SU(2) 8^4 1.47 / 1.68 / -, 2D SU(3) 64 x 128
//     1.29 / 1.75 / 1.68; FP32 4.1 / 4.5 / 3.1, 3.3 / 3.3 / 2.4 and 3.2 / 3.5 / 2.8; 64 rhs 64 x 128 1.47,
//     16^3 1.33 in FP64.
//   several lattices, whose graph form copies state per lattice at every wait: faster at
//     every size measured, 84 systems on 21 4D SU(3) lattices up to 1536 sites per parity
//     4447 / 6023 us in FP64 and 3653 / 9415 in FP32; 1024 systems on 64 lattices 1.08 (FP64) and
//     1.36 (FP32) times in 4D SU(3), 1.31 and 1.43 in 4D SU(2), 1.4 to 2.0 in 3D, 1.5 to 2.3 in 2D
bool small_applies(int nd, int nc, int sp, int64_t vh, int systems, int lattices) {
  if (lattices > 1 && vh <= 2048) return systems <= 1024;
  if (systems > 64) return false;
  if (sp == SP64) {
    if (nd == 4) return vh <= 512 || (vh <= 2048 && systems <= 12);
    return vh <= (nd == 3 && nc == 3 ? 2048 : 4096);
  }
  if (nd == 4) return vh <= 1024 || (vh <= 2048 && systems <= 24) || (vh <= 4096 && systems <= (sp == SP32 ? 40 : 12));
  return vh <= (nd == 3 && nc == 3 ? 4096 : 8192);
}

// Threads per block and blocks per cluster.  Up to 256 sites one block, whose barriers cost
// almost nothing; then one site per thread in four or eight blocks of 128 (two per SM by registers);
// above 1024 sites eight blocks of 256 while all clusters are resident at once, else of
// 128, which double the systems in flight (16^3 SU(2) FP32, 8 rhs: 379 us a solve with
// 256, 466 with 128; 16 rhs: 713 and 543).
template <int ND, int NC, int SP>
static int launch_small(int64_t vh, const SmallLat* lats, int nlat, const SmallLat& one, int systems, int round,
                        cudaStream_t st) {
  int threads = 128, ctas = 1;
  if (vh <= kSmallThreads) {
    for (threads = 64; threads < vh;) threads *= 2;
  } else {
    for (ctas = 4; ctas < kSmallMaxCtas && (int64_t)ctas * threads < vh;) ctas *= 2;  // two hold 256 sites
  }
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(systems * ctas));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = st;
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = (unsigned)ctas;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  if ((int64_t)ctas * threads < vh) {
    static std::atomic<int> resident{-1};  // clusters of eight blocks of 256 that fit at once
    int n = resident.load(std::memory_order_relaxed);
    cfg.blockDim = dim3(kSmallThreads);
    if (n < 0) {
      LYM_CUDA(cudaOccupancyMaxActiveClusters(&n, small_cg_kernel<ND, NC, SP>, &cfg));
      resident.store(n, std::memory_order_relaxed);
    }
    if (systems > n) cfg.blockDim = dim3(threads);
  }
  // 256 threads of 255 registers per SM; clusters beyond those that fit run in further waves
  const int64_t cluster = (int64_t)ctas * cfg.blockDim.x, fit = std::max<int64_t>(1, 148 * 256 / cluster);
  const int64_t waves = (systems + fit - 1) / fit, sites = (vh + cluster - 1) / cluster;
  const int64_t stop = (round + 1) * std::max<int64_t>(1, kSmallStretch / (waves * sites));
  LYM_CUDA(cudaLaunchKernelEx(&cfg, small_cg_kernel<ND, NC, SP>, lats, nlat, one, round > 0,
                              (int)std::min<int64_t>(stop, 0x7fffffff)));
  return LYM_OK;
}

int small_launch(int nd, int nc, int sp, int64_t vh, const SmallLat* lats, int nlat, const SmallLat& one, int systems,
                 int round, cudaStream_t st) {
#define LYM_SMALL(ND_, NC_)                                                                    \
  if (nd == ND_ && nc == NC_) {                                                                \
    switch (sp) {                                                                              \
      case SP64: return launch_small<ND_, NC_, SP64>(vh, lats, nlat, one, systems, round, st); \
      case SP32: return launch_small<ND_, NC_, SP32>(vh, lats, nlat, one, systems, round, st); \
      case SP16: return launch_small<ND_, NC_, SP16>(vh, lats, nlat, one, systems, round, st); \
      default: return launch_small<ND_, NC_, SPB16>(vh, lats, nlat, one, systems, round, st); \
    }                                                                                          \
  }
  LYM_SMALL(2, 2)
  LYM_SMALL(2, 3)
  LYM_SMALL(3, 2)
  LYM_SMALL(3, 3)
  LYM_SMALL(4, 2)
  LYM_SMALL(4, 3)
#undef LYM_SMALL
  set_error("unsupported (nd=%d, N=%d)", nd, nc);
  return LYM_ERR_UNSUPPORTED;
}

}  // namespace lym
