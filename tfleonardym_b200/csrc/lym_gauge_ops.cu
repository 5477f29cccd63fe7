// Gauge-side kernels in the reference layout (FP64): staples and gauge force
// (fused with the momentum update), plaquette and momenta energy reductions,
// the link update exp(eps P) U, polar reunitarisation and the fused per-link
// fermion force.  One thread per link (site, direction); every neighbour link
// is read straight from the gauge field through the reference's sup/sdn
// tables -- no shifted copies are materialised (gauge_action.py:56-91 builds
// five gathered copies per plane instead).
#include "lym_internal.cuh"
#include "lym_kernels.cuh"
#include "lym_su.cuh"

#include <mutex>

namespace lym {

// ---------------------------------------------------------------------------
// staples: S_mu(x) = sum_{nu != mu} U_nu(x) U_mu(x+nu) U_nu(x+mu)^dag
//                               + U_nu(x-nu)^dag U_mu(x-nu) U_nu(x-nu+mu)
// (gauge_action.py:56-101, staples.py:13-58)
// ---------------------------------------------------------------------------

// Row by row, so that only two neighbour links and one row are live beside the sum
// (168 registers at three blocks per SM, 128 at four, where whole products took 184 and
// left two).  Bound by the latency of its gathers: within a trajectory at 16^3 x 32 SU(3) the
// force kernel takes 95 us against 150 us with whole products (FP64 pipe 47 %, L1 52 % busy;
// the FP64 work alone is 45 us), the staples alone at 24^3 x 48 258 us against 361 us.
// FUSED: the second product accumulates straight into the sum, 36 roundings of it in 4D.
// Otherwise each staple is formed by itself and added once, six roundings: the force is
// 1.39e-16 off 64-bit-exact values (2-norm, SU(3)) and 1.80e-16 with FUSED, whole products
// 1.35e-16; FUSED serves smearing alone, whose projection outweighs it (1.1e-16 either way)
// and whose registers it saves (3 %).
// The planes one after the other: with all loads of a link free to move, ptxas gathers more of
// them ahead than the registers hold (the force in blocks of 256 spills 400 bytes and takes 20 %
// longer).  A rolled loop does it in blocks of 128 for SU(3) (2 to 5 % faster than the
// unrolled one), a pointer that depends on the sum so far does it in the others (rolled:
// 12 % slower in blocks of 256).
template <int ND, int NC, bool FUSED, bool ROLLED>
LYM_D Mat<NC> staple_sum(const int32_t* __restrict__ tab, int64_t V, const double2* __restrict__ U, int mu,
                         int64_t s, int no_dir) {
  Mat<NC> S = mzero<NC>();
  const int64_t xmu = tab[mu * V + s];
  auto plane = [&](int nu) {
    const int64_t xnu = tab[nu * V + s];
    const int64_t xmnu = tab[ND * V + nu * V + s];
    const int64_t xmnu_pmu = tab[mu * V + xmnu];
    {
      const Mat<NC> b = load_link<NC>(U, mu, xnu, V), c = load_link<NC>(U, nu, xmu, V);
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        cx<double> a[NC], r[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) a[k] = ld(U + ((int64_t)(nu * NC + i) * NC + k) * V + s);
        row_mul<NC>(r, a, b);
        if constexpr (FUSED) {
          row_mac_nd<NC>(S.m[i], r, c);
        } else {
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            cx<double> t = cmul_cj(c.m[j][0], r[0]);
#pragma unroll
            for (int k = 1; k < NC; ++k) cmac_cj(t, c.m[j][k], r[k]);
            S.m[i][j] += t;
          }
        }
      }
    }
    {
      const Mat<NC> b = load_link<NC>(U, mu, xmnu, V), c = load_link<NC>(U, nu, xmnu_pmu, V);
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        cx<double> a[NC], r[NC];
#pragma unroll
        for (int k = 0; k < NC; ++k) a[k] = conj(ld(U + ((int64_t)(nu * NC + k) * NC + i) * V + xmnu));
        row_mul<NC>(r, a, b);
        if constexpr (FUSED) {
          row_mac<NC>(S.m[i], r, c);
        } else {
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            cx<double> t = r[0] * c.m[0][j];
#pragma unroll
            for (int k = 1; k < NC; ++k) cmac(t, r[k], c.m[k][j]);
            S.m[i][j] += t;
          }
        }
      }
    }
  };
  if constexpr (ROLLED) {
#pragma unroll 1
    for (int p = 0; p < ND - 1; ++p) {
      const int nu = p + (p >= mu ? 1 : 0);
      if (nu != no_dir) plane(nu);
    }
  } else {
#pragma unroll
    for (int nu = 0; nu < ND; ++nu) {
      if (nu == mu || nu == no_dir) continue;
      if constexpr (!FUSED) asm volatile("" : "+l"(U) : "d"(S.m[0][0].re), "d"(S.m[NC - 1][NC - 1].im));
      plane(nu);
    }
  }
  return S;
}

template <int ND, int NC>
__global__ void __launch_bounds__(128, 4) staples_kernel(const int32_t* __restrict__ tab, int64_t V,
                                                         const double2* __restrict__ U, int no_dir,
                                                         double2* __restrict__ out) {
  int mu;
  int64_t s;
  if (!warp_link(ND, V, blockIdx.x, mu, s)) return;
  Mat<NC> S = (mu == no_dir) ? mzero<NC>() : staple_sum<ND, NC, false, NC == 3>(tab, V, U, mu, s, no_dir);
  store_link<NC>(out, mu, s, V, S);
}

// The per-plane staple terms themselves, in the reference's list order
// (staples.py:23-58): for direction mu, the planes (mu, nu) with nu != mu,
// no_dir in increasing nu, each giving the "up" term U_nu(x) U_mu(x+nu)
// U_nu(x+mu)^dag (sup_staple_trace) then the "down" term U_nu(x-nu)^dag
// U_mu(x-nu) U_nu(x-nu+mu) (sdn_staple_trace).  out is (nd, 2(nd-1), N, N, V);
// slot 2k / 2k+1 holds plane k's terms; the slots of an excluded direction and
// the last two slots of the others when no_dir is a direction are left as they are.
template <int ND, int NC>
__global__ void __launch_bounds__(128) staple_terms_kernel(const int32_t* __restrict__ tab, int64_t V,
                                                           const double2* __restrict__ U, int no_dir,
                                                           double2* __restrict__ out) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int mu = blockIdx.y;
  if (s >= V || mu == no_dir) return;
  constexpr int NT = 2 * (ND - 1);
  const int64_t xmu = tab[mu * V + s];
  int k = 0;
#pragma unroll
  for (int nu = 0; nu < ND; ++nu) {
    if (nu == mu || nu == no_dir) continue;
    const int64_t xnu = tab[nu * V + s];
    const int64_t xmnu = tab[ND * V + nu * V + s];
    const int64_t xmnu_pmu = tab[mu * V + xmnu];
    const Mat<NC> up = mul_nd(mul(load_link<NC>(U, nu, s, V), load_link<NC>(U, mu, xnu, V)),
                              load_link<NC>(U, nu, xmu, V));
    const Mat<NC> dn = mul(mul_dn(load_link<NC>(U, nu, xmnu, V), load_link<NC>(U, mu, xmnu, V)),
                           load_link<NC>(U, nu, xmnu_pmu, V));
    store_link<NC>(out, mu * NT + 2 * k, s, V, up);
    store_link<NC>(out, mu * NT + 2 * k + 1, s, V, dn);
    ++k;
  }
}

// F = -beta/(4N) (W^dag - W) - trace/N, W = U S^dag at one link (gauge_action.py:42-53);
// anti-Hermitian, so the upper triangle of W^dag - W gives the lower one
template <int ND, int NC, bool ROLLED>
LYM_D Mat<NC> gauge_force_link(const int32_t* __restrict__ tab, int64_t V, const double2* __restrict__ U,
                               double beta, int mu, int64_t s) {
  const Mat<NC> S = staple_sum<ND, NC, false, ROLLED>(tab, V, U, mu, s, -1);
  // the link's loads after the staples: ahead of them they would only hold registers
  asm volatile("" : "+l"(U) : "d"(S.m[0][0].re), "d"(S.m[NC - 1][NC - 1].im));
  const Mat<NC> L = load_link<NC>(U, mu, s, V);
  const double c = -0.25 * beta / NC;
  Mat<NC> F;
  double tr = 0.0;
#pragma unroll
  for (int i = 0; i < NC; ++i) {
    cx<double> w = cmul_cj(S.m[i][0], L.m[i][0]);
#pragma unroll
    for (int k = 1; k < NC; ++k) cmac_cj(w, S.m[i][k], L.m[i][k]);
    F.m[i][i] = {0.0, c * (-w.im - w.im)};
    tr += F.m[i][i].im;
#pragma unroll
    for (int j = i + 1; j < NC; ++j) {
      cx<double> x = cmul_cj(S.m[j][0], L.m[i][0]), y = cmul_cj(S.m[i][0], L.m[j][0]);
#pragma unroll
      for (int k = 1; k < NC; ++k) {
        cmac_cj(x, S.m[j][k], L.m[i][k]);
        cmac_cj(y, S.m[i][k], L.m[j][k]);
      }
      F.m[i][j] = c * (conj(y) - x);
      F.m[j][i] = -conj(F.m[i][j]);
    }
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) F.m[i][i].im -= (1.0 / NC) * tr;
  return F;
}

// F = -beta/(4N) (W^dag - W) - trace/N, W = U S^dag (gauge_action.py:42-53).
// With mom != null: out = mom + eps F instead of F (hmc.py:59-61); out may be mom (each
// thread reads its own link's momenta and writes them).
template <int ND, int NC, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == 256 ? 2 : NC == 2 ? 4 : 3)
    gauge_force_kernel(const int32_t* __restrict__ tab, int64_t V, const double2* __restrict__ U, double beta,
                       const double2* mom, double2* out, double eps) {
  int mu;
  int64_t s;
  if (!warp_link(ND, V, blockIdx.x, mu, s)) return;
  Mat<NC> F = gauge_force_link<ND, NC, NC == 3 && BLOCK == 128>(tab, V, U, beta, mu, s);
  if (mom) {
    Mat<NC> P;  // all of it before the first store: out may be mom
#pragma unroll
    for (int k = 0; k < NC * NC; ++k) {
      const double2 p = mom[(int64_t)(mu * NC * NC + k) * V + s];
      P.m[k / NC][k % NC] = {p.x, p.y};
    }
#pragma unroll
    for (int k = 0; k < NC * NC; ++k) {
      cx<double>& f = F.m[k / NC][k % NC];
      f = P.m[k / NC][k % NC] + eps * f;
    }
  }
  store_link<NC>(out, mu, s, V, F);
}

// sum_{x, mu<nu} Tr U_mu(x) U_nu(x+mu) U_mu(x+nu)^dag U_nu(x)^dag (gauge_action.py:110-113)
// A warp takes one plane of 32 sites, the planes of a site block side by side (their 24
// links in 4D are 16 distinct ones), and streams the rows of both half loops into the
// trace.  24^3 x 48 SU(3): 162 us against 195 us with a thread doing all planes of a
// site (255 registers).
template <int ND, int NC>
__global__ void __launch_bounds__(256, 2) plaquette_kernel(const int32_t* __restrict__ tab, int64_t V,
                                                           const double2* __restrict__ U, double* partials,
                                                           unsigned* counter, double* result) {
  __shared__ double sh[2 * 32];
  constexpr int NP = ND * (ND - 1) / 2;
  double v[2] = {0.0, 0.0};
  const int64_t nw = (V + 31) / 32 * NP;
  const int64_t per = (nw + gridDim.x - 1) / gridDim.x;  // a block's warps: a contiguous run of planes
  const int64_t w1 = (blockIdx.x + 1) * per < nw ? (blockIdx.x + 1) * per : nw;
  for (int64_t w = blockIdx.x * per + (threadIdx.x >> 5); w < w1; w += 8) {
    const int64_t sb = w / NP;
    int mu = 0, nu = (int)(w - sb * NP) + 1;
    while (nu >= ND) nu += ++mu + 1 - ND;  // plane index -> mu < nu
    const int64_t s = sb * 32 + (threadIdx.x & 31);
    if (s >= V) continue;
    const Mat<NC> b = load_link<NC>(U, nu, tab[mu * V + s], V), d = load_link<NC>(U, mu, tab[nu * V + s], V);
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      cx<double> p[NC], q[NC], r[NC];
#pragma unroll
      for (int k = 0; k < NC; ++k) p[k] = ld(U + ((int64_t)(mu * NC + i) * NC + k) * V + s);
      row_mul<NC>(q, p, b);
#pragma unroll
      for (int k = 0; k < NC; ++k) p[k] = ld(U + ((int64_t)(nu * NC + i) * NC + k) * V + s);
      row_mul<NC>(r, p, d);
#pragma unroll
      for (int k = 0; k < NC; ++k) {  // Tr (U_mu U_nu(x+mu)) (U_nu U_mu(x+nu))^dag
        v[0] += q[k].re * r[k].re + q[k].im * r[k].im;
        v[1] += q[k].im * r[k].re - q[k].re * r[k].im;
      }
    }
  }
  if (grid_sum<2>(v, partials, counter, sh) && threadIdx.x == 0) {
    result[0] = v[0];
    result[1] = v[1];
  }
}

// Momenta from unit normals, one thread per link, built as hmc.py:69-96 builds
// them from its draws: normals (nd, N^2-1, V) hold per direction the (re, im)
// pairs of the entries above the diagonal in row order, then the N-1 Cartan
// values; each is halved; P_ij = (re, im), P_ji = (-re, im); the diagonal is
// i times sum_i c_i H_i with the reference's diagonal generators.
template <int NC>
__global__ void __launch_bounds__(256) momenta_from_normals_kernel(int nd, int64_t V, const double* __restrict__ nrm,
                                                                   double2* __restrict__ P) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int mu = blockIdx.y;
  if (s >= V) return;
  constexpr int NG = NC * NC - 1;
  const double* n = nrm + (int64_t)mu * NG * V + s;
  Mat<NC> m;
  int k = 0;
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = i + 1; j < NC; ++j) {
      const double re = 0.5 * n[(int64_t)k * V], im = 0.5 * n[(int64_t)(k + 1) * V];
      k += 2;
      m.m[i][j] = {re, im};
      m.m[j][i] = {-re, im};
    }
  double diag[NC];
#pragma unroll
  for (int i = 0; i < NC; ++i) diag[i] = 0.0;
#pragma unroll
  for (int i = 1; i < NC; ++i) {
    const double r = 0.5 * n[(int64_t)k * V];
    ++k;
    const double di = (double)i;
#pragma unroll
    for (int j = 0; j < i; ++j) diag[j] += r / sqrt(di * (di + 1.0) / 2.0);
    diag[i] += -r * (di * sqrt(2.0 / (di * (di + 1.0))));
  }
#pragma unroll
  for (int i = 0; i < NC; ++i) m.m[i][i] = {0.0, diag[i]};
  store_link<NC>(P, mu, s, V, m);
}

// -Re sum Tr P^2 (hmc.py:170-176)
template <int NC>
__global__ void __launch_bounds__(256) momenta_energy_kernel(int64_t nlinks, int64_t V,
                                                             const double2* __restrict__ P, double* partials,
                                                             unsigned* counter, double* result) {
  __shared__ double sh[32];
  double v[1] = {0.0};
  for (int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; l < nlinks; l += (int64_t)gridDim.x * blockDim.x) {
    const int mu = (int)(l / V);
    const int64_t s = l - mu * V;
    Mat<NC> p = load_link<NC>(P, mu, s, V);
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < NC; ++j) v[0] -= (p.m[i][j] * p.m[j][i]).re;
  }
  if (grid_sum<1>(v, partials, counter, sh) && threadIdx.x == 0) result[0] = v[0];
}

// out = y + a x (out may be y)
__global__ void axpy_real_kernel(int64_t n, const double2* y, const double2* __restrict__ x, double a, double2* out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double2 yv = y[i], xv = x[i];
    out[i] = make_double2(yv.x + a * xv.x, yv.y + a * xv.y);
  }
}

// ---------------------------------------------------------------------------
// exp of an anti-Hermitian matrix (the HMC momenta, hmc.py:69-96)
// ---------------------------------------------------------------------------

// sin(w)/w with its series near zero
LYM_D double sinc(double w) {
  if (fabs(w) < 0.05) {
    double w2 = w * w;
    return 1.0 - w2 / 6.0 * (1.0 - w2 / 20.0 * (1.0 - w2 / 42.0 * (1.0 - w2 / 72.0)));
  }
  return sin(w) / w;
}

// exp(t) of the trace part; momenta are traceless up to rounding, where four terms of the
// series are exact to rounding (|t|^5 / 120 < 1e-17)
LYM_D cx<double> exp_trace(cx<double> t) {
  if (norm2(t) < 1e-8) {
    cx<double> r = {1.0 + 0.25 * t.re, 0.25 * t.im};
    r = cx<double>{1.0, 0.0} + (1.0 / 3.0) * (t * r);
    r = cx<double>{1.0, 0.0} + 0.5 * (t * r);
    return cx<double>{1.0, 0.0} + t * r;
  }
  const double e = exp(t.re);
  double sn, cs;
  sincos(t.im, &sn, &cs);
  return {e * cs, e * sn};
}

// exp(X) for 2x2 X = t 1 + X0, X0 traceless: X0^2 = -det(X0) 1 (Cayley-Hamilton),
// so exp(X0) = cos(a) 1 + sinc(a) X0 with a^2 = det(X0) (>= 0 for anti-Hermitian X0).
LYM_D Mat<2> expm(const Mat<2>& X) {
  cx<double> t = 0.5 * trace(X);
  Mat<2> X0 = X;
  X0.m[0][0] -= t;
  X0.m[1][1] -= t;
  double a2 = det(X0).re;
  double a = sqrt(fmax(a2, 0.0));
  double c = cos(a), sc = sinc(a);
  Mat<2> R;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) R.m[i][j] = sc * X0.m[i][j];
  R.m[0][0].re += c;
  R.m[1][1].re += c;
  // exp(t) with t = i phi for anti-Hermitian X (real part kept for generality)
  return mscale(exp_trace(t), R);
}

// exp(X) for 3x3 anti-Hermitian X: X = t 1 + i Q with Q Hermitian traceless,
// exp(i Q) = f0 + f1 Q + f2 Q^2 with the closed-form coefficients of
// Morningstar & Peardon, Phys. Rev. D 69 (2004) 054501, eqs. (23)-(34).
LYM_D Mat<3> expm(const Mat<3>& X) {
  cx<double> t = (1.0 / 3.0) * trace(X);
  Mat<3> Q;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      cx<double> x = X.m[i][j];
      if (i == j) x -= t;
      Q.m[i][j] = {x.im, -x.re};  // -i x
    }
  Mat<3> Q2 = mul(Q, Q);
  const double c1 = 0.5 * trace(Q2).re;
  cx<double> f0, f1, f2;
  if (c1 < 1e-12) {
    // exp(iQ) = 1 + iQ - Q^2/2 + O(|Q|^3) with |Q| < 1e-6
    f0 = {1.0, 0.0};
    f1 = {0.0, 1.0};
    f2 = {-0.5, 0.0};
  } else {
    double c0 = det(Q).re;
    const bool neg = c0 < 0;
    if (neg) c0 = -c0;
    const double c13 = c1 / 3.0, r13 = sqrt(c13);
    const double c0max = 2.0 * c13 * r13;
    double ratio = c0 / c0max;
    ratio = fmin(1.0, fmax(-1.0, ratio));
    const double theta = acos(ratio);
    double st3, ct3;
    sincos(theta / 3.0, &st3, &ct3);
    const double u = r13 * ct3;
    const double w = sqrt(c1) * st3;
    const double u2 = u * u, w2 = w * w;
    double s2u, c2u, su, cu;
    sincos(u, &su, &cu);
    // by itself: from su and cu the drift is 1.55e-16 off exact values instead of 1.45e-16
    sincos(2.0 * u, &s2u, &c2u);
    const cx<double> e2iu{c2u, s2u}, emiu{cu, -su};
    const double cw = cos(w), xi0 = sinc(w);
    cx<double> h0 = (u2 - w2) * e2iu + emiu * cx<double>{8.0 * u2 * cw, 2.0 * u * (3.0 * u2 + w2) * xi0};
    cx<double> h1 = (2.0 * u) * e2iu - emiu * cx<double>{2.0 * u * cw, -(3.0 * u2 - w2) * xi0};
    cx<double> h2 = e2iu - emiu * cx<double>{cw, 3.0 * u * xi0};
    const double d = 1.0 / (9.0 * u2 - w2);
    f0 = d * h0;
    f1 = d * h1;
    f2 = d * h2;
    if (neg) {  // f_j(-c0) = (-1)^j conj(f_j(c0))
      f0 = conj(f0);
      f1 = -conj(f1);
      f2 = conj(f2);
    }
  }
  const cx<double> et = exp_trace(t);
  f0 = et * f0;
  f1 = et * f1;
  f2 = et * f2;
  Mat<3> R;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      R.m[i][j] = f1 * Q.m[i][j];
      cmac(R.m[i][j], f2, Q2.m[i][j]);
    }
#pragma unroll
  for (int i = 0; i < 3; ++i) R.m[i][i] += f0;
  return R;
}

// |d|^(-1/N)
template <int NC>
LYM_D double inv_root(double d2) { return NC == 2 ? rsqrt(sqrt(d2)) : rcbrt(sqrt(d2)); }

// A Hermitian 3 x 3 matrix: its diagonal, and (0,1), (0,2), (1,2)
struct Herm3 {
  double d[3];
  cx<double> a, b, c;
};

// U^dag U
LYM_D Herm3 gram(const Mat<3>& U) {
  Herm3 H{};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
#pragma unroll
    for (int j = 0; j < 3; ++j) H.d[j] += norm2(U.m[k][j]);
    cmac_cj(H.a, U.m[k][0], U.m[k][1]);
    cmac_cj(H.b, U.m[k][0], U.m[k][2]);
    cmac_cj(H.c, U.m[k][1], U.m[k][2]);
  }
  return H;
}

// U <- U (a0 + a1 K + a2 K^2); with ADD, U + that, rounding a small correction once
template <bool ADD>
LYM_D void times_quadratic(Mat<3>& U, const Herm3& K, double a0, double a1, double a2) {
  const double na = norm2(K.a), nb = norm2(K.b), nc = norm2(K.c);
  Herm3 P;
  P.d[0] = fma(a2, fma(K.d[0], K.d[0], na + nb), fma(a1, K.d[0], a0));
  P.d[1] = fma(a2, fma(K.d[1], K.d[1], na + nc), fma(a1, K.d[1], a0));
  P.d[2] = fma(a2, fma(K.d[2], K.d[2], nb + nc), fma(a1, K.d[2], a0));
  P.a = fma(a2, K.d[0] + K.d[1], a1) * K.a + a2 * cmul_cj(K.c, K.b);
  P.b = fma(a2, K.d[0] + K.d[2], a1) * K.b + a2 * (K.a * K.c);
  P.c = fma(a2, K.d[1] + K.d[2], a1) * K.c + a2 * cmul_cj(K.a, K.b);
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    const cx<double> x = U.m[i][0], y = U.m[i][1], z = U.m[i][2];
    cx<double> t = P.d[0] * x, u = P.d[1] * y, v = P.d[2] * z;
    cmac_cj(t, P.a, y);
    cmac_cj(t, P.b, z);
    cmac(u, x, P.a);
    cmac_cj(u, P.c, z);
    cmac(v, x, P.b);
    cmac(v, y, P.c);
    U.m[i][0] = ADD ? x + t : t;
    U.m[i][1] = ADD ? y + u : u;
    U.m[i][2] = ADD ? z + v : v;
  }
}

// U <- U p(U^dag U) near the unitary polar factor, p the quadratic through x^(-1/2) at the three
// eigenvalues of U^dag U.  Any p positive there keeps the polar factor, and the product is formed
// in FP64, so the eigenvalues (the trigonometric solution of the characteristic cubic) and p's
// coefficients (divided differences of x^(-1/2), closed forms in the square roots) need no more
// than FP32: they set how close the step lands, about 1e-7.  False, U as it was, where the
// smallest eigenvalue is under 0.05 of the mean (beyond, the quadratic's cancellations would show) or the matrix is not finite.
LYM_D bool polar_step_exact(Mat<3>& U) {
  Herm3 K = gram(U);
  const double m = (K.d[0] + K.d[1] + K.d[2]) * (1.0 / 3.0), inv = 1.0 / m;
#pragma unroll
  for (int j = 0; j < 3; ++j) K.d[j] = fma(K.d[j], inv, -1.0);
  K.a = inv * K.a;
  K.b = inv * K.b;
  K.c = inv * K.c;
  const float d0 = (float)K.d[0], d1 = (float)K.d[1], d2 = (float)K.d[2];
  const cx<float> a{(float)K.a.re, (float)K.a.im}, b{(float)K.b.re, (float)K.b.im}, c{(float)K.c.re, (float)K.c.im};
  const float na = norm2(a), nb = norm2(b), nc = norm2(c);
  const float q = (d0 * d0 + d1 * d1 + d2 * d2 + 2.f * (na + nb + nc)) * (1.f / 6.f);
  const cx<float> ac = a * c;
  const float dt = d0 * d1 * d2 + 2.f * (ac.re * b.re + ac.im * b.im) - d0 * nc - d1 * nb - d2 * na;
  const float h = sqrtf(q);
  const float r = q > 1e-16f ? fminf(1.f, fmaxf(-1.f, dt / (2.f * q * h))) : 0.f;
  const float phi = acosf(r) * (1.f / 3.f);
  const float k1 = 2.f * h * cosf(phi), k3 = 2.f * h * cosf(phi + 2.0943951f), k2 = -k1 - k3;
  if (!(1.f + k3 > 0.05f) || !(k1 < 3.f)) return false;
  const float s1 = sqrtf(1.f + k1), s2 = sqrtf(1.f + k2), s3 = sqrtf(1.f + k3);
  const float f12 = -1.f / (s1 * s2 * (s1 + s2));
  const float f123 = (s1 + s2 + s3) / (s1 * s2 * s3 * (s1 + s2) * (s2 + s3) * (s1 + s3));
  const double sc = rsqrt(m);
  times_quadratic<false>(U, K, sc * (double)(1.f / s1 - f12 * k1 + f123 * k1 * k2),
                         sc * (double)(f12 - f123 * (k1 + k2)), sc * (double)f123);
  return true;
}

// One step of third order, U <- U (1 - E/2 + 3 E^2/8), E = U^dag U - 1; |E|^2
LYM_D double polar_step_near(Mat<3>& U) {
  Herm3 E = gram(U);
#pragma unroll
  for (int j = 0; j < 3; ++j) E.d[j] -= 1.0;
  times_quadratic<true>(U, E, 0.0, -0.5, 0.375);
  return E.d[0] * E.d[0] + E.d[1] * E.d[1] + E.d[2] * E.d[2] + 2.0 * (norm2(E.a) + norm2(E.b) + norm2(E.c));
}

// Unitary polar factor by the scaled Newton iteration
// U <- (g U + U^{-dag} / g) / 2, g = |det U|^{-1/N} (Higham, "Functions of
// Matrices", sec. 8.6), then division by the principal det^{1/N}
// (smearing.py:17-31 computes X (X^dag X)^{-1/2} / det^{1/N} via sqrtm).
// The iteration converges quadratically, |U_{k+1} - U| <= |U_k - U|^2 / 2 near the end, so
// a step of squared length 1e-17 leaves an error of 1e-17 and is the last.
template <int NC>
LYM_D Mat<NC> polar_newton(const Mat<NC>& X) {
  Mat<NC> Uk = X;
  cx<double> d = det(Uk);
  for (int it = 0; it < 40; ++it) {
    const double d2 = norm2(d);
    // the scale only speeds up the approach: near |det U| = 1 it is left at 1
    const double g = fabs(d2 - 1.0) < 1e-2 ? 1.0 : inv_root<NC>(d2);
    const double hg = 0.5 * g, hi = 0.5 / (g * d2);
    const Mat<NC> C = cofactors(Uk);  // U^{-dag} = conj(C) / conj(d) = conj(C) d / |d|^2
    const cx<double> w = hi * d;
    double diff = 0.0;
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        cx<double> n = cmul_cj(C.m[i][j], w);
        n.re = fma(hg, Uk.m[i][j].re, n.re);
        n.im = fma(hg, Uk.m[i][j].im, n.im);
        diff += norm2(n - Uk.m[i][j]);
        Uk.m[i][j] = n;
      }
    d = det(Uk);
    if (diff < 1e-17) break;
  }
  const cx<double> r = principal_root(d, NC);
  return mscale(cdiv(cx<double>{1.0, 0.0}, r), Uk);
}

// out of line: few links take it, and inlined it costs the others registers
__device__ __noinline__ Mat<3> polar_newton3(Mat<3> X) { return polar_newton<3>(X); }

// d^(-1/3), principal root, for d on the unit circle to 1e-5: the angle in FP32, then Newton steps
// on w^3 = d in FP64, w^(-2) from conj(w)^2 (each squares the distance: 1e-7, 1e-14, 1e-28)
LYM_D cx<double> inv_cube_root_unit(cx<double> d) {
  float sn, cs;
  sincosf(atan2f((float)d.im, (float)d.re) * (1.f / 3.f), &sn, &cs);
  cx<double> w{cs, sn};
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const cx<double> w2 = w * w;
    const double f = (3.0 - 2.0 * norm2(w)) * (1.0 / 3.0);
    w = (2.0 / 3.0) * w + f * cmul_cj(w2, d);
  }
  return conj(w);
}

// SU(3) starts from polar_step_exact and one third-order step, which leaves 5/16 |E|^3 <= 1e-17
// where |E|^2 < 1e-11; the Newton steps then only serve ill-conditioned matrices.  The two cost
// about 400 FP64 operations against 230 for each of five Newton steps: smearing step at
// 24^3 x 48 459 us against 558 us, errors against 64-bit polar factors the same (rms 7e-16,
// unitarity 2.8e-16).
template <int NC>
LYM_D Mat<NC> polar_su(const Mat<NC>& X) {
  if constexpr (NC == 3) {
    Mat<3> U = X;
    if (polar_step_exact(U) && polar_step_near(U) < 1e-11) return mscale(inv_cube_root_unit(det(U)), U);
    return polar_newton3(X);
  } else {
    return polar_newton<NC>(X);
  }
}

template <int NC>
__global__ void __launch_bounds__(128) update_links_kernel(int64_t nlinks, int64_t V, const double2* U,
                                                           const double2* __restrict__ P, double eps, int reunit,
                                                           double2* out) {
  const int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= nlinks) return;
  const int mu = (int)(l / V);
  const int64_t s = l - mu * V;
  Mat<NC> p = load_link<NC>(P, mu, s, V), u;
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const double2 t = U[((int64_t)(mu * NC + i) * NC + j) * V + s];  // out may be U
      u.m[i][j] = {t.x, t.y};
    }
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) p.m[i][j] = eps * p.m[i][j];
  Mat<NC> r = mul(expm(p), u);
  if (reunit) r = polar_su<NC>(r);
  store_link<NC>(out, mu, s, V, r);
}

template <int NC>
__global__ void __launch_bounds__(128) unitary_projection_kernel(int64_t nlinks, int64_t V,
                                                                 const double2* __restrict__ in,
                                                                 double2* __restrict__ out) {
  const int64_t l = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (l >= nlinks) return;
  const int mu = (int)(l / V);
  const int64_t s = l - mu * V;
  store_link<NC>(out, mu, s, V, polar_su<NC>(load_link<NC>(in, mu, s, V)));
}

// One APE smearing step (smearing.py:34-51) per link: the staples without direction no_dir,
// the fat link (rho / 6) S + (1 - rho) U (rho U + (1 - rho) U for no_dir) and its projection,
// so the staples and the fat links never reach memory.  FP64-bound (the projection).
// 24^3 x 48 SU(3): 459 us against 1108 us in separate passes (staples, four scaled
// sums with their copies, projection).
template <int ND, int NC, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == 256 ? 2 : 4)
    smear_kernel(const int32_t* __restrict__ tab, int64_t V, const double2* __restrict__ U, cx<double> rho, int no_dir,
                 double2* __restrict__ out) {
  int mu;
  int64_t s;
  if (!warp_link(ND, V, blockIdx.x, mu, s)) return;
  const cx<double> one{1.0, 0.0};
  Mat<NC> F;
  if (mu == no_dir) {
    F = mscale(rho, load_link<NC>(U, mu, s, V));
  } else {
    F = mscale(cx<double>{rho.re / 6, rho.im / 6}, staple_sum<ND, NC, true, false>(tab, V, U, mu, s, no_dir));
  }
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) cmac(F.m[i][j], one - rho, ld(U + ((int64_t)(mu * NC + i) * NC + j) * V + s));
  store_link<NC>(out, mu, s, V, polar_su<NC>(F));
}

// ---------------------------------------------------------------------------
// fermion force (dirac.py:525-565, fermion_action.py:64-93)
//
// For link (mu, x), with V_m = U_mu(x) Y_m(x+mu) (colour matvec per spin row m):
//   A = sum_m conj(X_m(x)) (x) (P+ V)_m ,  B = sum_m conj(V_m) (x) (P- X(x))_m
//   L(X, Y)_{ut} = kappa/2 [A_{tu} - B_{tu} - delta_{ut} (Tr A - Tr B)/N]
// which is the reference's sum over generators T^k_{ij} T^k_{ut} written with
// the SU(N) completeness relation sum_k T^k_ij T^k_ut = (d_it d_ju - d_ij d_ut/N)/2.
// P+- = (1 -+ gamma_mu), multiplied by gamma_d when hermitian.  The projectors have rank
// ns/2: over the upper rows a, with x+- = X_a +- g_a X_ja and v+- = U (Y_a +- g_a Y_ja)(x+mu),
//   hermitian:  A = sum_a conj(x+) (x) v-,   B = A^dag (one outer product per row)
//   plain:      A = sum_a conj(x-) (x) v-,   B = sum_a conj(v+) (x) x+
// so a link and pole costs ns/2 matvecs and outer products per ordering instead of ns
// matvecs, two full projections and 2 ns outer products, which spilled.  Each pole's terms are
// summed by themselves and added with its weight: straight into the sum, every product is rounded
// against all poles before it (SU(3), 4 poles: 2.4e-16 off exact values instead of 1.8e-16).  The sum
// waits in shared memory, where registers would spill.  12^3 x 24 SU(3), 8 poles: 95 us against
// 336 us, 16^4, 10 poles: 174 us against 620 us (three blocks per SM); bound by the four spinor
// gathers per link and pole.
// ---------------------------------------------------------------------------
constexpr int kMaxForceTerms = 64;
struct ForceTerms {
  double alpha[kMaxForceTerms];
};

// one upper row of psi_a + s g_a psi_ja at site x
template <int ND, int NC>
LYM_D void half_row(const double2* __restrict__ f, int mu, int a, bool plus, int64_t V, int64_t x,
                    cx<double> (&h)[NC]) {
  const bool im = gamma_imag<ND>(mu);
  const double g = plus ? gamma_sign<ND>(mu, a) : -gamma_sign<ND>(mu, a);
  const double2* pu = f + (int64_t)a * NC * V + x;
  const double2* pl = f + (int64_t)Gamma<ND>::col(mu, a) * NC * V + x;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    h[c] = ld(pu + c * V);
    add_gamma(h[c], g, im, ld(pl + c * V));
  }
}

template <int ND, int NC, bool HERM>
__global__ void __launch_bounds__(128, 3) fermion_force_kernel(
    const int32_t* __restrict__ tab, int64_t V, int Lt, double kappa, double bcr, double bci,
    const double2* __restrict__ U, int nterms, ForceTerms terms, const double2* __restrict__ X,
    const double2* __restrict__ Y, int symmetric, double scale, double2* __restrict__ force) {
  constexpr int NS = Gamma<ND>::NS;
  int mu;
  int64_t s;
  if (!warp_link(ND, V, blockIdx.x, mu, s)) return;
  const int64_t y = tab[mu * V + s];
  Mat<NC> u = load_link<NC>(U, mu, s, V);
  if (mu == ND - 1 && (s % Lt) == Lt - 1) u = mscale(cx<double>{bcr, bci}, u);
  __shared__ double2 sum[NC * NC][128];  // over the poles: w (A - B), hermitian: w A
#pragma unroll
  for (int i = 0; i < NC * NC; ++i) sum[i][threadIdx.x] = make_double2(0.0, 0.0);
  Mat<NC> K;
  const int64_t vec = (int64_t)NS * NC * V;
  for (int k = 0; k < nterms; ++k) {
    const double w = 0.5 * kappa * terms.alpha[k];
    K = mzero<NC>();
    for (int side = 0; side < (symmetric ? 2 : 1); ++side) {
      const double2* P = (side == 0 ? X : Y) + k * vec;  // L(P, Q): P at x, Q at x + mu
      const double2* Q = (side == 0 ? Y : X) + k * vec;
#pragma unroll
      for (int c = 0; c < (HERM ? NS / 2 : NS); ++c) {
        const bool plus = c >= NS / 2;  // the B term of the plain projector
        const int a = plus ? c - NS / 2 : c;
        cx<double> h[NC], q[NC];
        half_row<ND, NC>(P, mu, a, HERM || plus, V, s, h);
        half_row<ND, NC>(Q, mu, a, plus, V, y, q);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          cx<double> v = u.m[i][0] * q[0];
#pragma unroll
          for (int l = 1; l < NC; ++l) cmac(v, u.m[i][l], q[l]);
          if (plus) v = -v;
#pragma unroll
          for (int j = 0; j < NC; ++j) {
            if (plus) cmac_cj(K.m[i][j], v, h[j]);  // conj(v)_i x_j
            else cmac_cj(K.m[j][i], h[j], v);       // conj(x)_j v_i
          }
        }
      }
    }
#pragma unroll
    for (int i = 0; i < NC * NC; ++i) {
      double2& o = sum[i][threadIdx.x];
      const cx<double> t = K.m[i / NC][i % NC];
      o = make_double2(fma(w, t.re, o.x), fma(w, t.im, o.y));
    }
  }
#pragma unroll
  for (int i = 0; i < NC * NC; ++i) K.m[i / NC][i % NC] = {sum[i][threadIdx.x].x, sum[i][threadIdx.x].y};
  if constexpr (HERM) {
    Mat<NC> D;
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < NC; ++j) D.m[i][j] = K.m[i][j] - conj(K.m[j][i]);
    K = D;
  }
  const cx<double> tr = (1.0 / NC) * trace(K);
#pragma unroll
  for (int i = 0; i < NC; ++i) K.m[i][i] -= tr;
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      double2* o = force + ((int64_t)(mu * NC + i) * NC + j) * V + s;
      st(o, ld(o) + scale * K.m[j][i]);
    }
}

// ---------------------------------------------------------------------------
// A kick and the drift that follows it: mom_out = mom + eps_p F(U), then
// U_out = exp(eps_u mom_out) U, link by link in one pass (the force reads the old links of
// the neighbours, so the new ones go to another field).  The momenta and the link are not
// read again by a second kernel: 16^3 x 32 SU(3) 128.1 us against 145.6 us in two, 4^4 8.1 against
// 9.6, 1024^2 333 against 393; SU(2) 16^3 x 32 56.5 against 61.8.
// ---------------------------------------------------------------------------
template <int ND, int NC, int BLOCK>
__global__ void __launch_bounds__(BLOCK, BLOCK == 256 ? 2 : NC == 2 ? 4 : 3)
    kick_drift_kernel(const int32_t* __restrict__ tab, int64_t V, const double2* __restrict__ U, double beta,
                      const double2* mom, double eps_p, double eps_u, double2* mom_out, double2* __restrict__ U_out) {
  int mu;
  int64_t s;
  if (!warp_link(ND, V, blockIdx.x, mu, s)) return;
  const Mat<NC> F = gauge_force_link<ND, NC, NC == 3 && BLOCK == 128>(tab, V, U, beta, mu, s);
  Mat<NC> P;  // all of it before the first store: mom_out may be mom
#pragma unroll
  for (int k = 0; k < NC * NC; ++k) {
    const double2 p = mom[(int64_t)(mu * NC * NC + k) * V + s];
    P.m[k / NC][k % NC] = cx<double>{p.x, p.y} + eps_p * F.m[k / NC][k % NC];
  }
  store_link<NC>(mom_out, mu, s, V, P);
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) P.m[i][j] = eps_u * P.m[i][j];
  store_link<NC>(U_out, mu, s, V, mul(expm(P), load_link<NC>(U, mu, s, V)));
}

// ---------------------------------------------------------------------------
// The gauge part of an HMC step on many lattices at once (builder-defined: the
// reference runs one lattice per process, hmc.py:218-246): momenta P += eps_p F(U)
// for every link of every lattice in one launch, then U <- exp(eps_u P) U in a
// second (the force reads neighbouring links, so all forces come first).  The
// lattices' descriptors travel as the kernel parameter; every lattice owns a
// contiguous range of blocks (nd x its site blocks) and a block finds its lattice
// by binary search over the range starts.  Any mix of (nd, N) in one launch.
// ---------------------------------------------------------------------------
struct HmcLat {
  const int32_t* tab;
  double2* U;
  double2* P;
  int64_t V;
  double beta;
  int nd, nc;
  int b0;  // first block of this lattice
};
constexpr int kHmcMaxLat = 256;
struct HmcTable {
  int n;
  double eps;
  HmcLat l[kHmcMaxLat];
};

LYM_D int hmc_lat_of(const HmcTable& t, int b) {
  int lo = 0, hi = t.n - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (t.l[mid].b0 <= b) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

template <int ND, int NC>
LYM_D void hmc_kick_link(const HmcLat& L, double eps, int mu, int64_t s) {
  const Mat<NC> F = gauge_force_link<ND, NC, NC == 3>(L.tab, L.V, L.U, L.beta, mu, s);
  Mat<NC> P = load_link<NC>(L.P, mu, s, L.V);
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) P.m[i][j] += eps * F.m[i][j];
  store_link<NC>(L.P, mu, s, L.V, P);
}

template <int NC>
LYM_D void hmc_drift_link(const HmcLat& L, double eps, int mu, int64_t s) {
  const Mat<NC> e = expm(mscale(cx<double>{eps, 0.0}, load_link<NC>(L.P, mu, s, L.V)));
  store_link<NC>(L.U, mu, s, L.V, mul(e, load_link<NC>(L.U, mu, s, L.V)));
}

// kick = 1: momenta from the force; 0: links from the momenta
__global__ void __launch_bounds__(128) hmc_multi_kernel(const __grid_constant__ HmcTable t, int kick) {
  const HmcLat& L = t.l[hmc_lat_of(t, blockIdx.x)];
  int mu;
  int64_t s;
  if (!warp_link(L.nd, L.V, blockIdx.x - L.b0, mu, s)) return;
  if (kick) {
    switch (L.nd * 10 + L.nc) {
      case 22: hmc_kick_link<2, 2>(L, t.eps, mu, s); break;
      case 23: hmc_kick_link<2, 3>(L, t.eps, mu, s); break;
      case 32: hmc_kick_link<3, 2>(L, t.eps, mu, s); break;
      case 33: hmc_kick_link<3, 3>(L, t.eps, mu, s); break;
      case 42: hmc_kick_link<4, 2>(L, t.eps, mu, s); break;
      default: hmc_kick_link<4, 3>(L, t.eps, mu, s); break;
    }
  } else if (L.nc == 2) {
    hmc_drift_link<2>(L, t.eps, mu, s);
  } else {
    hmc_drift_link<3>(L, t.eps, mu, s);
  }
}

// ---------------------------------------------------------------------------
// dispatch
// ---------------------------------------------------------------------------
#define LYM_DISPATCH_ND_NC(nd, nc, CALL)                                              \
  do {                                                                                \
    if ((nd) == 2 && (nc) == 2) { constexpr int ND = 2, NC = 2; CALL; }               \
    else if ((nd) == 2 && (nc) == 3) { constexpr int ND = 2, NC = 3; CALL; }          \
    else if ((nd) == 3 && (nc) == 2) { constexpr int ND = 3, NC = 2; CALL; }          \
    else if ((nd) == 3 && (nc) == 3) { constexpr int ND = 3, NC = 3; CALL; }          \
    else if ((nd) == 4 && (nc) == 2) { constexpr int ND = 4, NC = 2; CALL; }          \
    else if ((nd) == 4 && (nc) == 3) { constexpr int ND = 4, NC = 3; CALL; }          \
    else { set_error("unsupported (nd=%d, N=%d)", (nd), (nc)); return LYM_ERR_UNSUPPORTED; } \
  } while (0)

// Link kernels whose 4D SU(3) form at 128 registers is worth blocks of eight warps: 64 sites
// and their directions share an SM's L1, and the block's rows of loads go out together.  From
// three waves of sixteen warps per SM on: force / kick and drift / smear in us with 256 | 128
// threads (launches in a row, random links), 16^3 x 32 85.3 / 128.0 / 106.1 | 90.0 / 141.4 / 121.5, 16^4 42.7 / 66.9 / 53.1 |
// 45.3 / 72.8 / 61.1; below, 12^3 x 24 29.5 / 48.1 / 37.5 | 28.5 / 45.8 / 41.0, 8^4 7.9 / 11.7 /
// 10.3 | 5.9 / 9.6 / 9.1.  SU(2) and fewer dimensions gain nothing (24^4 SU(2) 94.7 / 145.6 /
// 146 | 92.4 / 142.1 / 140).
constexpr int64_t kWideFrom = 3 * 16 * 148;  // warps
#define LYM_LINK_LAUNCH(KERNEL, lat, nc, st, ...)                                                                \
  do {                                                                                                           \
    if ((lat)->nd == 4 && (nc) == 3 && ((lat)->V + 31) / 32 * 4 >= kWideFrom) {                                  \
      KERNEL<4, 3, 256><<<warp_link_grid(4, (lat)->V, 256), 256, 0, (st)>>>(__VA_ARGS__);                        \
    } else {                                                                                                     \
      LYM_DISPATCH_ND_NC((lat)->nd, (nc), (KERNEL<ND, NC, 128><<<warp_link_grid(ND, (lat)->V, 128), 128, 0, (st)>>>( \
                                              __VA_ARGS__)));                                                    \
    }                                                                                                            \
  } while (0)

}  // namespace lym

using namespace lym;

extern "C" {

int lym_staple_terms(const lym_lattice* lat, int nc, const void* gauge, int no_direction, void* terms,
                     void* stream) {
  LYM_REQUIRE(lat && gauge && terms, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(gauge != terms, LYM_ERR_BAD_ARG, "gauge and terms must not alias");
  cudaStream_t st = (cudaStream_t)stream;
  dim3 grid(grid_for(lat->V, 128), lat->nd);
  LYM_DISPATCH_ND_NC(lat->nd, nc, (staple_terms_kernel<ND, NC><<<grid, 128, 0, st>>>(
                                      lat->d_tab, lat->V, (const double2*)gauge, no_direction, (double2*)terms)));
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_staples(const lym_lattice* lat, int nc, const void* gauge, int no_direction, void* staples,
                void* stream) {
  LYM_REQUIRE(lat && gauge && staples, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(gauge != staples, LYM_ERR_BAD_ARG, "gauge and staples must not alias");
  const unsigned grid = warp_link_grid(lat->nd, lat->V, 128);
  cudaStream_t st = (cudaStream_t)stream;
  LYM_DISPATCH_ND_NC(lat->nd, nc, (staples_kernel<ND, NC><<<grid, 128, 0, st>>>(
                                      lat->d_tab, lat->V, (const double2*)gauge, no_direction, (double2*)staples)));
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

// force: out = F; kick: out = mom + eps F
static int gauge_force(const lym_lattice* lat, int nc, double beta, const void* gauge, const void* mom, void* out,
                       double eps, cudaStream_t st) {
  LYM_LINK_LAUNCH(gauge_force_kernel, lat, nc, st, lat->d_tab, lat->V, (const double2*)gauge, beta,
                  (const double2*)mom, (double2*)out, eps);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_gauge_force(const lym_lattice* lat, int nc, double beta, const void* gauge, void* force, void* momenta,
                    double eps, void* stream) {
  LYM_REQUIRE(lat && gauge && (force || momenta), LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(gauge != force && gauge != momenta, LYM_ERR_BAD_ARG, "outputs must not alias the gauge field");
  return gauge_force(lat, nc, beta, gauge, momenta, momenta ? momenta : force, eps, (cudaStream_t)stream);
}

int lym_gauge_kick(const lym_lattice* lat, int nc, double beta, const void* gauge, const void* momenta, double eps,
                   void* out, void* stream) {
  LYM_REQUIRE(lat && gauge && momenta && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(gauge != out, LYM_ERR_BAD_ARG, "out must not alias the gauge field");
  return gauge_force(lat, nc, beta, gauge, momenta, out, eps, (cudaStream_t)stream);
}

int lym_gauge_kick_drift(const lym_lattice* lat, int nc, double beta, const void* gauge, const void* momenta,
                         double eps_p, double eps_u, void* momenta_out, void* gauge_out, void* stream) {
  LYM_REQUIRE(lat && gauge && momenta && momenta_out && gauge_out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(gauge != gauge_out && gauge != momenta_out && momenta_out != gauge_out && momenta != gauge_out,
              LYM_ERR_BAD_ARG, "the new links and momenta need fields of their own");
  cudaStream_t st = (cudaStream_t)stream;
  LYM_LINK_LAUNCH(kick_drift_kernel, lat, nc, st, lat->d_tab, lat->V, (const double2*)gauge, beta,
                  (const double2*)momenta, eps_p, eps_u, (double2*)momenta_out, (double2*)gauge_out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_plaquette_sum(const lym_lattice* lat, int nc, const void* gauge, double* out, void* stream) {
  LYM_REQUIRE(lat && gauge && out, LYM_ERR_BAD_ARG, "null argument");
  Scratch* s;
  int rc = scratch_get(&s);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(host_reduce_mutex());
  const int slot = 1;
  cudaStream_t st = (cudaStream_t)stream;
  unsigned nb = reduction_blocks((lat->V + 31) / 32 * 32 * (lat->nd * (lat->nd - 1) / 2), 256);
  double* part = s->partials + (size_t)slot * Scratch::kMaxBlocks * Scratch::kMaxVals;
  double* res = s->results + slot * Scratch::kMaxVals;
  LYM_DISPATCH_ND_NC(lat->nd, nc, (plaquette_kernel<ND, NC><<<nb, 256, 0, st>>>(
                                      lat->d_tab, lat->V, (const double2*)gauge, part, s->counters + slot, res)));
  LYM_CHECK_LAUNCH();
  LYM_CUDA(cudaMemcpyAsync(s->host + slot * Scratch::kMaxVals, res, 2 * sizeof(double), cudaMemcpyDeviceToHost, st));
  LYM_CUDA(cudaStreamSynchronize(st));
  out[0] = s->host[slot * Scratch::kMaxVals];
  out[1] = s->host[slot * Scratch::kMaxVals + 1];
  return LYM_OK;
}

int lym_momenta_from_normals(int nd, int nc, int64_t volume, const double* normals, void* momenta, void* stream) {
  LYM_REQUIRE(normals && momenta && nd >= 1 && nd <= LYM_MAX_ND && volume >= 0, LYM_ERR_BAD_ARG, "bad argument");
  LYM_REQUIRE(nc == 2 || nc == 3, LYM_ERR_UNSUPPORTED, "N must be 2 or 3");
  if (volume == 0) return LYM_OK;
  cudaStream_t st = (cudaStream_t)stream;
  const dim3 grid(grid_for(volume, 256), nd);
  if (nc == 2)
    momenta_from_normals_kernel<2><<<grid, 256, 0, st>>>(nd, volume, normals, (double2*)momenta);
  else
    momenta_from_normals_kernel<3><<<grid, 256, 0, st>>>(nd, volume, normals, (double2*)momenta);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_momenta_energy(int nd, int nc, int64_t volume, const void* momenta, double* out, void* stream) {
  LYM_REQUIRE(momenta && out && nd >= 1 && nd <= LYM_MAX_ND && volume >= 0, LYM_ERR_BAD_ARG, "bad argument");
  LYM_REQUIRE(nc == 2 || nc == 3, LYM_ERR_UNSUPPORTED, "N must be 2 or 3");
  Scratch* s;
  int rc = scratch_get(&s);
  if (rc) return rc;
  std::lock_guard<std::mutex> lk(host_reduce_mutex());
  const int slot = 1;
  cudaStream_t st = (cudaStream_t)stream;
  const int64_t nl = (int64_t)nd * volume;
  unsigned nb = reduction_blocks(nl, 256);
  double* part = s->partials + (size_t)slot * Scratch::kMaxBlocks * Scratch::kMaxVals;
  double* res = s->results + slot * Scratch::kMaxVals;
  if (nc == 2)
    momenta_energy_kernel<2><<<nb, 256, 0, st>>>(nl, volume, (const double2*)momenta, part, s->counters + slot, res);
  else
    momenta_energy_kernel<3><<<nb, 256, 0, st>>>(nl, volume, (const double2*)momenta, part, s->counters + slot, res);
  LYM_CHECK_LAUNCH();
  LYM_CUDA(cudaMemcpyAsync(s->host + slot * Scratch::kMaxVals, res, sizeof(double), cudaMemcpyDeviceToHost, st));
  LYM_CUDA(cudaStreamSynchronize(st));
  out[0] = s->host[slot * Scratch::kMaxVals];
  return LYM_OK;
}

int lym_momenta_kick(int64_t n, const void* momenta, const void* force, double eps, void* out, void* stream) {
  LYM_REQUIRE(n >= 0 && momenta && force && out, LYM_ERR_BAD_ARG, "null argument");
  if (n == 0) return LYM_OK;
  axpy_real_kernel<<<reduction_blocks(n, 256) * 4, 256, 0, (cudaStream_t)stream>>>(
      n, (const double2*)momenta, (const double2*)force, eps, (double2*)out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_update_momenta(int64_t n, void* momenta, const void* force, double eps, void* stream) {
  return lym_momenta_kick(n, momenta, force, eps, momenta, stream);
}

int lym_gauge_hmc_step_multi(int nlat, const lym_lattice* const* lats, const int* nc, const double* betas,
                             void* const* gauges, void* const* momenta, double eps_p, double eps_u, void* stream) {
  LYM_REQUIRE(nlat >= 1 && nlat <= kHmcMaxLat, LYM_ERR_BAD_ARG, "nlat must be in [1, %d]", kHmcMaxLat);
  LYM_REQUIRE(lats && nc && betas && gauges && momenta, LYM_ERR_BAD_ARG, "null argument");
  HmcTable t;
  t.n = nlat;
  int64_t blocks = 0;
  for (int l = 0; l < nlat; ++l) {
    LYM_REQUIRE(lats[l] && gauges[l] && momenta[l], LYM_ERR_BAD_ARG, "null argument (lattice %d)", l);
    LYM_REQUIRE(nc[l] == 2 || nc[l] == 3, LYM_ERR_UNSUPPORTED, "N must be 2 or 3 (lattice %d)", l);
    LYM_REQUIRE(lats[l]->nd >= 2 && lats[l]->nd <= 4, LYM_ERR_UNSUPPORTED, "nd must be 2, 3 or 4 (lattice %d)", l);
    LYM_REQUIRE(lats[l]->V >= 1, LYM_ERR_BAD_ARG, "empty lattice %d", l);
    LYM_REQUIRE(gauges[l] != momenta[l], LYM_ERR_BAD_ARG, "gauge and momenta alias (lattice %d)", l);
    for (int k = 0; k < l; ++k)  // two lattices on one buffer would race in the same launch
      LYM_REQUIRE(gauges[k] != gauges[l] && momenta[k] != momenta[l] && gauges[k] != momenta[l] &&
                      momenta[k] != gauges[l],
                  LYM_ERR_BAD_ARG, "lattices %d and %d share a buffer", k, l);
    t.l[l] = HmcLat{lats[l]->d_tab, (double2*)gauges[l], (double2*)momenta[l], lats[l]->V, betas[l], lats[l]->nd,
                    nc[l], (int)blocks};
    blocks += warp_link_grid(lats[l]->nd, lats[l]->V, 128);
  }
  LYM_REQUIRE(blocks < (int64_t(1) << 31), LYM_ERR_UNSUPPORTED, "too many links for one launch");
  cudaStream_t st = (cudaStream_t)stream;
  t.eps = eps_p;
  hmc_multi_kernel<<<(unsigned)blocks, 128, 0, st>>>(t, 1);
  LYM_CHECK_LAUNCH();
  t.eps = eps_u;
  hmc_multi_kernel<<<(unsigned)blocks, 128, 0, st>>>(t, 0);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_link_drift(int nd, int nc, int64_t volume, const void* gauge, const void* momenta, double eps,
                   int reunitarize, void* out, void* stream) {
  LYM_REQUIRE(gauge && momenta && out && nd >= 1 && nd <= LYM_MAX_ND && volume >= 0, LYM_ERR_BAD_ARG, "bad argument");
  if (volume == 0) return LYM_OK;
  const int64_t nl = (int64_t)nd * volume;
  cudaStream_t st = (cudaStream_t)stream;
  if (nc == 2)
    update_links_kernel<2><<<grid_for(nl, 128), 128, 0, st>>>(nl, volume, (const double2*)gauge,
                                                              (const double2*)momenta, eps, reunitarize, (double2*)out);
  else if (nc == 3)
    update_links_kernel<3><<<grid_for(nl, 128), 128, 0, st>>>(nl, volume, (const double2*)gauge,
                                                              (const double2*)momenta, eps, reunitarize, (double2*)out);
  else {
    set_error("N=%d not supported", nc);
    return LYM_ERR_UNSUPPORTED;
  }
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_update_links(int nd, int nc, int64_t volume, void* gauge, const void* momenta, double eps, int reunitarize,
                     void* stream) {
  return lym_link_drift(nd, nc, volume, gauge, momenta, eps, reunitarize, gauge, stream);
}

int lym_ape_smear(const lym_lattice* lat, int nc, const void* gauge, double rho_re, double rho_im, int no_direction,
                  void* out, void* stream) {
  LYM_REQUIRE(lat && gauge && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(gauge != out, LYM_ERR_BAD_ARG, "gauge and out must not alias");
  cudaStream_t st = (cudaStream_t)stream;
  LYM_LINK_LAUNCH(smear_kernel, lat, nc, st, lat->d_tab, lat->V, (const double2*)gauge, cx<double>{rho_re, rho_im},
                  no_direction, (double2*)out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_unitary_projection(int nd, int nc, int64_t volume, const void* in, void* out, void* stream) {
  LYM_REQUIRE(in && out && nd >= 1 && nd <= LYM_MAX_ND && volume >= 0, LYM_ERR_BAD_ARG, "bad argument");
  if (volume == 0) return LYM_OK;
  const int64_t nl = (int64_t)nd * volume;
  cudaStream_t st = (cudaStream_t)stream;
  if (nc == 2)
    unitary_projection_kernel<2><<<grid_for(nl, 128), 128, 0, st>>>(nl, volume, (const double2*)in, (double2*)out);
  else if (nc == 3)
    unitary_projection_kernel<3><<<grid_for(nl, 128), 128, 0, st>>>(nl, volume, (const double2*)in, (double2*)out);
  else {
    set_error("N=%d not supported", nc);
    return LYM_ERR_UNSUPPORTED;
  }
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_fermion_force(const lym_lattice* lat, int nc, double kappa, int hermitian, double bc_re, double bc_im,
                      const void* gauge, int nterms, const double* alphas, const void* X, const void* Y,
                      int symmetric, double scale, void* force, void* stream) {
  LYM_REQUIRE(lat && gauge && alphas && X && Y && force, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(nterms >= 1 && nterms <= kMaxForceTerms, LYM_ERR_BAD_ARG, "nterms must be in [1, %d]",
              kMaxForceTerms);
  if (lat->nd != 2 && lat->nd != 4) {
    set_error("Number of dimensions %d not supported for fermions!", lat->nd);
    return LYM_ERR_UNSUPPORTED;
  }
  ForceTerms t;
  for (int i = 0; i < kMaxForceTerms; ++i) t.alpha[i] = i < nterms ? alphas[i] : 0.0;
  const unsigned grid = warp_link_grid(lat->nd, lat->V, 128);
  cudaStream_t st = (cudaStream_t)stream;
  const int Lt = lat->dims[lat->nd - 1];
#define LYM_FF(ND_, NC_, H_)                                                                        \
  fermion_force_kernel<ND_, NC_, H_><<<grid, 128, 0, st>>>(lat->d_tab, lat->V, Lt, kappa, bc_re, bc_im, \
                                                           (const double2*)gauge, nterms, t,          \
                                                           (const double2*)X, (const double2*)Y,      \
                                                           symmetric, scale, (double2*)force)
  if (lat->nd == 2 && nc == 2) { if (hermitian) LYM_FF(2, 2, true); else LYM_FF(2, 2, false); }
  else if (lat->nd == 2 && nc == 3) { if (hermitian) LYM_FF(2, 3, true); else LYM_FF(2, 3, false); }
  else if (lat->nd == 4 && nc == 2) { if (hermitian) LYM_FF(4, 2, true); else LYM_FF(4, 2, false); }
  else if (lat->nd == 4 && nc == 3) { if (hermitian) LYM_FF(4, 3, true); else LYM_FF(4, 3, false); }
  else {
    set_error("N=%d not supported", nc);
    return LYM_ERR_UNSUPPORTED;
  }
#undef LYM_FF
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// gauge observables (measurements.py:46-290): link products along paths, slice sums
// ---------------------------------------------------------------------------
namespace lym {

static int64_t lat_stride(const lym_lattice* lat, int d) {
  int64_t s = 1;
  for (int e = d + 1; e < lat->nd; ++e) s *= lat->dims[e];
  return s;
}

constexpr int kMaxPathSteps = 256;
struct PathSteps {
  signed char step[kMaxPathSteps];  // +(mu+1): U_mu(y), y += mu;  -(mu+1): y -= mu, U_mu(y)^dag
};

// One thread per starting site: M = product of the links along the path; writes
// Tr M (trace = 1, out (V) complex) or M (out (N, N, V)).  The first link is taken as it
// is and the last one enters the trace directly (n - 2 products and a trace for n links).
// Bound by the latency of its dependent gathers: occupancy counts, so one link is held
// at a time.  24^3 x 48 SU(3): 4 links 49 us against 54 us, 8 links 74 us against 84 us.
template <int NC>
__global__ void __launch_bounds__(128) path_kernel(const int32_t* __restrict__ tab, int nd, int64_t V,
                                                   const double2* __restrict__ U, int nsteps, PathSteps path,
                                                   int want_trace, double2* __restrict__ out) {
  const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (x >= V) return;
  int64_t y = x;
  Mat<NC> m = mident<NC>();
  for (int k = 0; k < nsteps; ++k) {
    const int s = path.step[k];
    const int mu = (s > 0 ? s : -s) - 1;
    const int64_t nx = tab[(s > 0 ? mu : nd + mu) * V + y];
    const Mat<NC> l = load_link<NC>(U, mu, s > 0 ? y : nx, V);  // U_mu(y), or U_mu(y - mu) entering as its dagger
    y = nx;
    if (k == 0) {
      m = s > 0 ? l : mdag(l);
    } else if (want_trace && k == nsteps - 1) {
      cx<double> t = czero<double>();
#pragma unroll
      for (int i = 0; i < NC; ++i) {  // a diagonal element by itself: the trace is rounded N times, not 2 N^2
        cx<double> d = s > 0 ? m.m[i][0] * l.m[0][i] : cmul_cj(l.m[i][0], m.m[i][0]);
#pragma unroll
        for (int j = 1; j < NC; ++j) {
          if (s > 0) cmac(d, m.m[i][j], l.m[j][i]);
          else cmac_cj(d, l.m[i][j], m.m[i][j]);
        }
        t += d;
      }
      st(out + x, t);
      return;
    } else if (s > 0) {
      m = mul(m, l);
    } else {
      m = mul_nd(m, l);
    }
  }
  if (want_trace) {
    st(out + x, trace(m));
  } else {
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int j = 0; j < NC; ++j) st(out + ((int64_t)i * NC + j) * V + x, m.m[i][j]);
  }
}

// t += conj(r) . q, the product of the rows formed by itself
template <int NC>
LYM_D void add_dot(cx<double>& t, const cx<double> (&r)[NC], const cx<double> (&q)[NC]) {
  cx<double> d = cmul_cj(r[0], q[0]);
#pragma unroll
  for (int k = 1; k < NC; ++k) cmac_cj(d, r[k], q[k]);
  t += d;
}

// plaq(x), square(x) = sum over the planes without direction `skip` of the traces of the
// 1 x 1 and 2 x 2 loops from x (measurements.py:197-290), each loop as its two halves
// (Tr P Q^dag), all planes of a site in one thread: ten distinct links per plane, no
// per-plane fields.  24^3 x 48 SU(3), three planes: 235 us against 1130 us for the six paths and
// their sums.
template <int NC>
__global__ void __launch_bounds__(128, 3) plane_loops_kernel(const int32_t* __restrict__ tab, int nd, int64_t V,
                                                             const double2* __restrict__ U, int skip,
                                                             double2* __restrict__ plaq, double2* __restrict__ square) {
  const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (x >= V) return;
  cx<double> tp = czero<double>(), ts = czero<double>();
#pragma unroll 1
  for (int a = 0; a < nd; ++a)
#pragma unroll 1
    for (int b = a + 1; b < nd; ++b) {
      if (a == skip || b == skip) continue;
      const int64_t xa = tab[a * V + x], xb = tab[b * V + x], xaa = tab[a * V + xa], xbb = tab[b * V + xb];
      const int64_t xaab = tab[b * V + xaa], xbba = tab[a * V + xbb];
      cx<double> loop = czero<double>();
      {
        const Mat<NC> b1 = load_link<NC>(U, b, xa, V), c1 = load_link<NC>(U, a, xb, V);
#pragma unroll
        for (int i = 0; i < NC; ++i) {
          cx<double> p[NC], q[NC], r[NC];
#pragma unroll
          for (int k = 0; k < NC; ++k) p[k] = ld(U + ((int64_t)(a * NC + i) * NC + k) * V + x);
          row_mul<NC>(q, p, b1);
#pragma unroll
          for (int k = 0; k < NC; ++k) p[k] = ld(U + ((int64_t)(b * NC + i) * NC + k) * V + x);
          row_mul<NC>(r, p, c1);
          add_dot<NC>(loop, r, q);
        }
      }
      tp += loop;
      loop = czero<double>();
      Mat<NC> p = mul(load_link<NC>(U, a, x, V), load_link<NC>(U, a, xa, V));
      p = mul(p, load_link<NC>(U, b, xaa, V));
      p = mul(p, load_link<NC>(U, b, xaab, V));
      Mat<NC> q = mul(load_link<NC>(U, b, x, V), load_link<NC>(U, b, xb, V));
      q = mul(q, load_link<NC>(U, a, xbb, V));
      const Mat<NC> l = load_link<NC>(U, a, xbba, V);
#pragma unroll
      for (int i = 0; i < NC; ++i) {
        cx<double> r[NC];
        row_mul<NC>(r, q.m[i], l);
        add_dot<NC>(loop, r, p.m[i]);
      }
      ts += loop;
    }
  st(plaq + x, tp);
  st(square + x, ts);
}

// Trace of the links once around direction d: by the cyclic invariance of the trace it is
// the same from every site of a line, so a line is multiplied once -- kPolySeg threads
// each take a segment -- and its trace written to all of its sites, where the general
// path multiplies the line from each of its L_d sites.  24^3 x 48 SU(3), 48 links:
// 39 us against 319 us.
constexpr int kPolySeg = 4;
template <int NC>
__global__ void __launch_bounds__(32 * kPolySeg) loop_kernel(int64_t nlines, int64_t V, int64_t stride, int L,
                                                             int mu, const double2* __restrict__ U,
                                                             double2* __restrict__ out) {
  __shared__ cx<double> part[kPolySeg][NC * NC][32];
  __shared__ cx<double> tr[32];
  const int tx = threadIdx.x & 31, seg = threadIdx.x >> 5;
  const int64_t line = blockIdx.x * (int64_t)32 + tx;
  // line -> its first site: coordinates slower than d, then the faster ones
  const int64_t x0 = line / stride * (stride * L) + line % stride;
  const int q = (L + kPolySeg - 1) / kPolySeg, k0 = seg * q, k1 = k0 + q < L ? k0 + q : L;
  Mat<NC> m = mident<NC>();
  if (line < nlines && k0 < k1) {
    m = load_link<NC>(U, mu, x0 + k0 * stride, V);
    for (int k = k0 + 1; k < k1; ++k) m = mul(m, load_link<NC>(U, mu, x0 + k * stride, V));
  }
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) part[seg][i * NC + j][tx] = m.m[i][j];
  __syncthreads();
  if (seg == 0) {
    for (int g = 1; g < kPolySeg; ++g) {
      Mat<NC> n;
#pragma unroll
      for (int i = 0; i < NC; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) n.m[i][j] = part[g][i * NC + j][tx];
      m = mul(m, n);
    }
    tr[tx] = trace(m);
  }
  __syncthreads();
  if (line < nlines)
    for (int k = k0; k < k1; ++k) st(out + x0 + k * stride, tr[tx]);
}

// out[2z], out[2z+1] = sum of f(x) over the sites with x_dir = z (and, when
// mask_len > 0, x_mask = 0); x_d = (x / stride_d) mod L_d for the lexicographic
// index with the last coordinate fastest.  The cluster walks its slice's sites only
// (24^3 x 48: 6 us against 712 us for one block per slice that tested every site of
// the lattice).
__global__ void __cluster_dims__(kSliceCtas, 1, 1) __launch_bounds__(kSliceThreads)
    slice_sum_kernel(uint32_t per, uint32_t stride, uint32_t L, uint32_t mask_stride, uint32_t mask_len,
                     const double2* __restrict__ f, double* __restrict__ out) {
  const uint32_t z = blockIdx.x / kSliceCtas, rank = blockIdx.x % kSliceCtas;
  double re = 0.0, im = 0.0;
  for (uint32_t j = rank * kSliceThreads + threadIdx.x; j < per; j += kSliceCtas * kSliceThreads) {
    const uint32_t x = (j / stride) * (L * stride) + z * stride + j % stride;
    if (mask_len > 0 && (x / mask_stride) % mask_len != 0) continue;
    const double2 v = f[x];
    re += v.x;
    im += v.y;
  }
  cluster_pair_sum(re, im, out + 2 * z);
}

// out[2k], out[2k+1] = sum_x conj(f(x + k dir)) f(x) for k = 0 .. L/2, and the complex
// conjugate for L - k (substitute x -> x - k): a cluster per k.
__global__ void __cluster_dims__(kSliceCtas, 1, 1) __launch_bounds__(kSliceThreads)
    shift_dots_kernel(uint32_t V, uint32_t stride, uint32_t L, const double2* __restrict__ f,
                      double* __restrict__ out) {
  const uint32_t k = blockIdx.x / kSliceCtas, rank = blockIdx.x % kSliceCtas;
  double re = 0.0, im = 0.0;
#pragma unroll 4
  for (uint32_t x = rank * kSliceThreads + threadIdx.x; x < V; x += kSliceCtas * kSliceThreads) {
    const uint32_t z = (x / stride) % L;
    const uint32_t y = z + k < L ? x + k * stride : x - (L - k) * stride;
    const double2 a = f[y], b = f[x];
    re += a.x * b.x + a.y * b.y;
    im += a.x * b.y - a.y * b.x;
  }
  cluster_pair_sum(re, im, out + 2 * k);
  if (rank == 0 && threadIdx.x == 0 && k > 0 && L - k != k) {
    out[2 * (L - k)] = out[2 * k];
    out[2 * (L - k) + 1] = -out[2 * k + 1];
  }
}

}  // namespace lym

extern "C" int lym_path_product(const lym_lattice* lat, int nc, const void* gauge, int nsteps, const int* steps,
                                int trace, void* out, void* stream) {
  using namespace lym;
  LYM_REQUIRE(lat && gauge && out && (steps || nsteps == 0), LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(nsteps >= 0 && nsteps <= kMaxPathSteps, LYM_ERR_BAD_ARG, "at most %d steps", kMaxPathSteps);
  PathSteps p{};
  for (int k = 0; k < nsteps; ++k) {
    const int s = steps[k];
    LYM_REQUIRE(s != 0 && (s > 0 ? s : -s) <= lat->nd, LYM_ERR_BAD_ARG, "step %d out of range", s);
    p.step[k] = (signed char)s;
  }
  dim3 grid(grid_for(lat->V, 128));
  cudaStream_t st = (cudaStream_t)stream;
  // once around one direction: the trace is the same along the line
  const int d = nsteps > 0 ? steps[0] - 1 : -1;
  bool around = trace && d >= 0 && nsteps == lat->dims[d];
  for (int k = 1; k < nsteps && around; ++k) around = steps[k] == steps[0];
  if (around && (nc == 2 || nc == 3)) {
    const int64_t nlines = lat->V / nsteps;
    const unsigned lg = grid_for(nlines, 32);
    if (nc == 2)
      loop_kernel<2><<<lg, 32 * kPolySeg, 0, st>>>(nlines, lat->V, lat_stride(lat, d), nsteps, d, (const double2*)gauge,
                                                   (double2*)out);
    else
      loop_kernel<3><<<lg, 32 * kPolySeg, 0, st>>>(nlines, lat->V, lat_stride(lat, d), nsteps, d, (const double2*)gauge,
                                                   (double2*)out);
    LYM_CHECK_LAUNCH();
    return LYM_OK;
  }
  if (nc == 2)
    path_kernel<2><<<grid, 128, 0, st>>>(lat->d_tab, lat->nd, lat->V, (const double2*)gauge, nsteps, p, trace != 0,
                                         (double2*)out);
  else if (nc == 3)
    path_kernel<3><<<grid, 128, 0, st>>>(lat->d_tab, lat->nd, lat->V, (const double2*)gauge, nsteps, p, trace != 0,
                                         (double2*)out);
  else {
    set_error("N=%d not supported", nc);
    return LYM_ERR_UNSUPPORTED;
  }
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

extern "C" int lym_plane_loops(const lym_lattice* lat, int nc, const void* gauge, int skip_direction, void* plaquettes,
                               void* squares, void* stream) {
  using namespace lym;
  LYM_REQUIRE(lat && gauge && plaquettes && squares, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(nc == 2 || nc == 3, LYM_ERR_UNSUPPORTED, "N=%d not supported", nc);
  const unsigned grid = grid_for(lat->V, 128);
  cudaStream_t st = (cudaStream_t)stream;
  if (nc == 2)
    plane_loops_kernel<2><<<grid, 128, 0, st>>>(lat->d_tab, lat->nd, lat->V, (const double2*)gauge, skip_direction,
                                                (double2*)plaquettes, (double2*)squares);
  else
    plane_loops_kernel<3><<<grid, 128, 0, st>>>(lat->d_tab, lat->nd, lat->V, (const double2*)gauge, skip_direction,
                                                (double2*)plaquettes, (double2*)squares);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

extern "C" int lym_slice_sums(const lym_lattice* lat, int direction, int mask_direction, const void* field,
                              double* out, void* stream) {
  using namespace lym;
  LYM_REQUIRE(lat && field && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(direction >= 0 && direction < lat->nd && mask_direction < lat->nd, LYM_ERR_BAD_ARG,
              "direction out of range");
  const int L = lat->dims[direction];
  const int mask_len = mask_direction >= 0 ? lat->dims[mask_direction] : 0;
  slice_sum_kernel<<<L * kSliceCtas, kSliceThreads, 0, (cudaStream_t)stream>>>(
      (uint32_t)(lat->V / L), (uint32_t)lat_stride(lat, direction), L,
      (uint32_t)(mask_direction >= 0 ? lat_stride(lat, mask_direction) : 1), mask_len, (const double2*)field, out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

extern "C" int lym_shift_dots(const lym_lattice* lat, int direction, const void* field, double* out, void* stream) {
  using namespace lym;
  LYM_REQUIRE(lat && field && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(direction >= 0 && direction < lat->nd, LYM_ERR_BAD_ARG, "direction %d out of range", direction);
  const int L = lat->dims[direction];
  shift_dots_kernel<<<(L / 2 + 1) * kSliceCtas, kSliceThreads, 0, (cudaStream_t)stream>>>(
      (uint32_t)lat->V, (uint32_t)lat_stride(lat, direction), L, (const double2*)field, out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}
