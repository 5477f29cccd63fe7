// Adjoint-representation Wilson fermions: operator, adjoint links and fermion
// force (reference dirac.py:358-370, 380-456, 525-565; lie_generators.py).
//
// Spinors are matrix valued, (ns, N, N, V) complex128 planes in the reference
// layout; the adjoint links are (nd, N^2-1, N^2-1, V).  The generator basis is
// the reference's (lie_generators.py:3-17, T^a = lambda^a / 2 in its order), so
// lym_adjoint_links reproduces the reference's fermion_gauge_field entry by
// entry; the force does not depend on the basis.
#include <cmath>

#include "lym_internal.cuh"
#include "lym_su.cuh"

namespace lym {

namespace {

constexpr int kAdjBlock = 128;

// fundamental generator a, element (i, j), in the reference's basis and order
template <int NC>
LYM_D cx<double> gen(int a, int i, int j);

template <>
LYM_D cx<double> gen<2>(int a, int i, int j) {
  // Pauli / 2: sigma_x, sigma_y, sigma_z
  if (a == 0) return {(i != j) ? 0.5 : 0.0, 0.0};
  if (a == 1) return {0.0, (i == 0 && j == 1) ? -0.5 : ((i == 1 && j == 0) ? 0.5 : 0.0)};
  return {(i == j) ? (i == 0 ? 0.5 : -0.5) : 0.0, 0.0};
}

template <>
LYM_D cx<double> gen<3>(int a, int i, int j) {
  // lambda_1, lambda_4, lambda_6, lambda_2, lambda_5, lambda_7, lambda_3, lambda_8 (each / 2)
  const int lo = i < j ? i : j, hi = i < j ? j : i;
  if (a < 6) {
    const int pi = (a % 3 == 0) ? 0 : ((a % 3 == 1) ? 0 : 1);
    const int pj = (a % 3 == 0) ? 1 : ((a % 3 == 1) ? 2 : 2);
    if (lo != pi || hi != pj) return {0.0, 0.0};
    if (a < 3) return {0.5, 0.0};
    return {0.0, i < j ? -0.5 : 0.5};
  }
  if (i != j) return {0.0, 0.0};
  if (a == 6) return {i == 0 ? 0.5 : (i == 1 ? -0.5 : 0.0), 0.0};
  const double s3 = 0.5 / sqrt(3.0);
  return {i == 2 ? -2.0 * s3 : s3, 0.0};
}

// The block's copies of the generators, built once per block in shared memory.
template <int NC>
struct AdjTables {
  static constexpr int A = NC * NC - 1;
  cx<double> T[A][NC][NC];
};

template <int NC>
LYM_D void build_tables(AdjTables<NC>& tb) {
  constexpr int A = NC * NC - 1;
  for (int e = threadIdx.x; e < A * NC * NC; e += blockDim.x) {
    const int a = e / (NC * NC), i = (e / NC) % NC, j = e % NC;
    tb.T[a][i][j] = gen<NC>(a, i, j);
  }
  __syncthreads();
}

// U_mu(site), or U_mu(site)^dag when !fwd
template <int NC>
LYM_D Mat<NC> load_hop_link(const double2* __restrict__ U, int mu, int64_t site, int64_t V, bool fwd) {
  Mat<NC> r;
  const double2* base = U + (int64_t)mu * NC * NC * V + site;
  const double s = fwd ? 1.0 : -1.0;
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      const cx<double> t = ld(base + (fwd ? i * NC + j : j * NC + i) * V);
      r.m[i][j] = {t.re, s * t.im};
    }
  return r;
}

LYM_D size_t adj_index(int s, int i, int j, int NC, int64_t V, int64_t x) {
  return ((size_t)(s * NC + i) * NC + j) * V + x;
}

}  // namespace

// ---------------------------------------------------------------------------
// operator: one thread per (site, upper spin row a, vector); in 4D the two threads of
// a site are lanes l and l + 16 of one warp (16 consecutive sites per warp).
//
// Row a of the upper half spinor h = psi_a - s g_a psi_ja feeds the output rows a and
// j_a, where j_a is 3 - a (mu = 0, 1) or 2 + a (mu = 2, 3): after mu = 1 the two threads
// swap their lower rows, which makes the partner's 3 - (1 - a) this thread's 2 + a, so
// two rows are live at a time.  No spinor value is loaded by both threads; the link is,
// from the same addresses of the same instruction.  (A thread per colour row loaded the
// whole neighbour spinor N times.)  Latency-bound at 8 warps per SM (255 registers);
// 16^4 SU(3): 45 us against 75 us, the FP64 work alone is 13 us.  Three or four blocks per
// SM spill and take 59 and 87 us; a real loop over the directions 54 to 62 us.
// LR: the left links are another field than the right ones.
// ---------------------------------------------------------------------------
template <int ND, int NC, bool HERM, bool LR>
__global__ void __launch_bounds__(kAdjBlock, 2) wilson_adjoint_kernel(
    const int32_t* __restrict__ tab, int V, int Lt, double kappa, double bcr, double bci,
    const double2* __restrict__ UL, const double2* __restrict__ UR, const double2* __restrict__ in,
    double2* __restrict__ out) {
  constexpr int NS = Gamma<ND>::NS, NA = NS / 2;  // NA threads per site
  constexpr int SW = 32 / NA;                     // sites per warp
  const int lane = threadIdx.x & 31;
  const int a = NA == 2 ? lane >> 4 : 0;
  const int xs = (int)(blockIdx.x * (kAdjBlock / 32) + (threadIdx.x >> 5)) * SW + (lane % SW);
  const int x = xs < V ? xs : V - 1;  // every lane takes part in the exchange below
  const size_t vec = (size_t)NS * NC * NC * V;
  const double2* psi = in + blockIdx.y * vec;
  double2* res = out + blockIdx.y * vec;
  const cx<double> bc{bcr, bci};
  Mat<NC> up = mzero<NC>(), low = mzero<NC>();

  // forward M = U(x), backward M = U(x - mu)^dag, both o = M h M^dag
#pragma unroll
  for (int md = 0; md < 2 * ND; ++md) {
    const int mu = md >> 1;
    const bool fwd = (md & 1) == 0;
    if (NA == 2 && md == 4) {
#pragma unroll
      for (int i = 0; i < NC; ++i)
#pragma unroll
        for (int l = 0; l < NC; ++l) {
          low.m[i][l].re = __shfl_xor_sync(0xffffffffu, low.m[i][l].re, 16);
          low.m[i][l].im = __shfl_xor_sync(0xffffffffu, low.m[i][l].im, 16);
        }
    }
    const int y = tab[(fwd ? 0 : ND) * V + mu * V + x];
    const int site = fwd ? x : y;  // the link's site: x forward, x - mu backward
    const bool boundary = mu == ND - 1 && (fwd ? (x % Lt) == Lt - 1 : (x % Lt) == 0);
    const double sg = fwd ? 1.0 : -1.0;
    const bool im = gamma_imag<ND>(mu);
    const double g = gamma_sign<ND>(mu, a);
    Mat<NC> h;
    {
      const double2* pu = psi + adj_index(a, 0, 0, NC, V, y);
      const double2* pl = psi + adj_index(Gamma<ND>::col(mu, a), 0, 0, NC, V, y);
#pragma unroll
      for (int k = 0; k < NC * NC; ++k) {
        cx<double> t = ld(pu + (size_t)k * V);
        add_gamma(t, -sg * g, im, ld(pl + (size_t)k * V));
        h.m[k / NC][k % NC] = t;
      }
    }
    const Mat<NC> r = load_hop_link<NC>(UR, mu, site, V, fwd);
    Mat<NC> ll;
    if constexpr (LR) ll = load_hop_link<NC>(UL, mu, site, V, fwd);
    else ll = r;
#pragma unroll
    for (int i = 0; i < NC; ++i) {
      cx<double> w[NC];
      row_mul<NC>(w, ll.m[i], h);
      if (boundary) {
#pragma unroll
        for (int l = 0; l < NC; ++l) w[l] = (fwd ? bc : conj(bc)) * w[l];
      }
      cx<double> o[NC];
#pragma unroll
      for (int l = 0; l < NC; ++l) o[l] = czero<double>();
      row_mac_nd<NC>(o, w, r);
#pragma unroll
      for (int l = 0; l < NC; ++l) {
        up.m[i][l] += o[l];
        add_gamma(low.m[i][l], im ? sg * g : -sg * g, im, o[l]);  // -s conj(g) o
      }
    }
  }
  if (xs >= V) return;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const Mat<NC>& acc = half ? low : up;
#pragma unroll
    for (int i = 0; i < NC; ++i)
#pragma unroll
      for (int l = 0; l < NC; ++l) {
        const size_t k = adj_index(half * (NS / 2) + a, i, l, NC, V, x);
        cx<double> v = ld(psi + k) + kappa * acc.m[i][l];
        if (HERM && half) v = -v;
        st(res + k, v);
      }
  }
}

// ---------------------------------------------------------------------------
// adjoint links V^{ab} = 2 Tr(T_a U T_b U^dag), one thread per (site, mu)
// ---------------------------------------------------------------------------
template <int NC>
__global__ void __launch_bounds__(kAdjBlock) adjoint_links_kernel(int nd, int64_t V, int Lt, double bcr, double bci,
                                                                  const double2* __restrict__ U,
                                                                  double2* __restrict__ out) {
  constexpr int A = NC * NC - 1;
  __shared__ AdjTables<NC> tb;
  build_tables<NC>(tb);
  const int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int mu = blockIdx.y;
  if (x >= V) return;
  Mat<NC> u = load_link<NC>(U, mu, x, V);
  const bool boundary = mu == nd - 1 && (x % Lt) == Lt - 1;
  const cx<double> f = boundary ? cx<double>{bcr, bci} : cx<double>{1.0, 0.0};
  for (int b = 0; b < A; ++b) {
    Mat<NC> tbm;
#pragma unroll
    for (int p = 0; p < NC; ++p)
#pragma unroll
      for (int q = 0; q < NC; ++q) tbm.m[p][q] = tb.T[b][p][q];
    const Mat<NC> w = mul_nd(mul(u, tbm), u);  // U T_b U^dag
    for (int a = 0; a < A; ++a) {
      cx<double> t = czero<double>();
#pragma unroll
      for (int p = 0; p < NC; ++p)
#pragma unroll
        for (int q = 0; q < NC; ++q) t += tb.T[a][p][q] * w.m[q][p];
      st(out + ((size_t)(mu * A + a) * A + b) * V + x, f * (2.0 * t));
    }
  }
}

// ---------------------------------------------------------------------------
// fermion force: one thread per (site, mu)
//
// The reference contracts adjoint components (dirac.py:547-560):
//   c_k = sum_ij TA^k_ij sum_m [conj(X_m)_i (P+ Z)_mj - conj(Z_m)_i (P- X)_mj],  Z = V Y(x + mu)
// with TA^k_ij = -2 Tr([T_k, T_i] T_j), and the force is sum_k c_k T_k.  In matrices,
// Z = U Y U^dag, and by the completeness of the T_k (2 sum_k T_k Tr(T_k C) = C for
// traceless C) the whole contraction is
//   sum_k c_k T_k = -sum_m ([X_m^dag, (P+ Z)_m] - [Z_m^dag, (P- X)_m])
// (the trace parts of X and Z drop out of the commutators; Y's is removed first).
// The projectors have rank two: with h+- = X_a +- g_a X_ja and z+- = U (Y_a +- g_a Y_ja) U^dag
// over the upper rows a,
//   gamma_d (1 -+ gamma):  -sum_a (K_a - K_a^dag),  K_a = h+^dag z-  - z- h+^dag
//   (1 -+ gamma):          -sum_a ([h-^dag, z-] - [z+^dag, h+])
// so a pole costs 16 (hermitian) N x N products per link instead of the (N^2-1)-component
// contraction through local memory (the neighbour loads now bound it): 8^3 x 16 SU(3), 4 poles: 34 us
// against 870 us.  Off exact values (80-bit, 2-norm): 2.2e-16, the component form 4.6e-16.
// ---------------------------------------------------------------------------
constexpr int kMaxAdjForceTerms = 32;
struct AdjForceTerms {
  double alpha[kMaxAdjForceTerms];
};

// psi_a + s g_a psi_ja at site x
template <int ND, int NC>
LYM_D Mat<NC> adj_half(const double2* __restrict__ f, int mu, int a, bool plus, int64_t V, int64_t x) {
  const bool im = gamma_imag<ND>(mu);
  const double g = plus ? gamma_sign<ND>(mu, a) : -gamma_sign<ND>(mu, a);
  const double2* pu = f + adj_index(a, 0, 0, NC, V, x);
  const double2* pl = f + adj_index(Gamma<ND>::col(mu, a), 0, 0, NC, V, x);
  Mat<NC> h;
#pragma unroll
  for (int k = 0; k < NC * NC; ++k) {
    cx<double> t = ld(pu + k * V);
    add_gamma(t, g, im, ld(pl + k * V));
    h.m[k / NC][k % NC] = t;
  }
  return h;
}

template <int NC>
LYM_D void remove_trace(Mat<NC>& m) {
  const cx<double> t = (1.0 / NC) * trace(m);
#pragma unroll
  for (int i = 0; i < NC; ++i) m.m[i][i] -= t;
}

// K += w [h^dag, z]
template <int NC>
LYM_D void commutator_mac(Mat<NC>& K, double w, const Mat<NC>& h, const Mat<NC>& z) {
#pragma unroll
  for (int i = 0; i < NC; ++i)
#pragma unroll
    for (int j = 0; j < NC; ++j) {
      cx<double> t = cmul_cj(h.m[0][i], z.m[0][j]);
#pragma unroll
      for (int k = 1; k < NC; ++k) cmac_cj(t, h.m[k][i], z.m[k][j]);
#pragma unroll
      for (int k = 0; k < NC; ++k) {  // - z_ik conj(h_jk)
        const cx<double> n = -z.m[i][k];
        cmac_cj(t, h.m[j][k], n);
      }
      K.m[i][j] += w * t;
    }
}

// In 4D the two upper rows of a link are two threads, lanes l and l + 16 of a warp (16
// sites), added by a shuffle at the end: the poles of a link are a serial chain of loads,
// and the small lattices of this force leave the chip half empty with a thread per link.
template <int ND, int NC, bool HERM>
__global__ void __launch_bounds__(kAdjBlock, 2) adjoint_force_kernel(
    const int32_t* __restrict__ tab, int64_t V, int Lt, double kappa, double bcr, double bci,
    const double2* __restrict__ U, int nterms, AdjForceTerms terms, const double2* __restrict__ X,
    const double2* __restrict__ Y, int symmetric, double scale, double2* __restrict__ force) {
  constexpr int NS = Gamma<ND>::NS, NA = NS / 2, SW = 32 / NA;
  const int lane = threadIdx.x & 31, a = NA == 2 ? lane >> 4 : 0;
  const int64_t wid = (int64_t)blockIdx.x * (kAdjBlock / 32) + (threadIdx.x >> 5), sb = wid / ND;
  const int mu = (int)(wid - sb * ND);  // the directions of a site block run side by side
  const int64_t xs = sb * SW + lane % SW;
  const int64_t x = xs < V ? xs : V - 1;  // every lane takes part in the shuffle
  const int64_t y = tab[mu * V + x];
  const Mat<NC> u = load_link<NC>(U, mu, x, V);
  const bool boundary = mu == ND - 1 && (x % Lt) == Lt - 1;
  const cx<double> f = boundary ? cx<double>{bcr, bci} : cx<double>{1.0, 0.0};
  Mat<NC> K = mzero<NC>();
  const size_t vec = (size_t)NS * NC * NC * V;
  for (int term = 0; term < nterms; ++term) {
    const double w = kappa * terms.alpha[term];
    for (int side = 0; side < (symmetric ? 2 : 1); ++side) {
      const double2* P = (side == 0 ? X : Y) + term * vec;  // L(P, Q): P at x, Q at x + mu
      const double2* Q = (side == 0 ? Y : X) + term * vec;
#pragma unroll 1
      for (int c = 0; c < (HERM ? 1 : 2); ++c) {
        const bool plus = c == 1;  // the second commutator of the plain projector
        Mat<NC> q = adj_half<ND, NC>(Q, mu, a, plus, V, y);
        remove_trace<NC>(q);  // the components have no trace part, whatever U is
        const Mat<NC> h = adj_half<ND, NC>(P, mu, a, HERM || plus, V, x);
        Mat<NC> z = mul_nd(mul(u, q), u);
        if (boundary) z = mscale(f, z);
        if (HERM || !plus) commutator_mac<NC>(K, w, h, z);
        else commutator_mac<NC>(K, -w, z, h);
      }
    }
  }
  if constexpr (NA == 2) {
#pragma unroll
    for (int p = 0; p < NC; ++p)
#pragma unroll
      for (int q = 0; q < NC; ++q) {
        K.m[p][q].re += __shfl_xor_sync(0xffffffffu, K.m[p][q].re, 16);
        K.m[p][q].im += __shfl_xor_sync(0xffffffffu, K.m[p][q].im, 16);
      }
  }
  if (xs >= V || a != 0) return;
#pragma unroll
  for (int p = 0; p < NC; ++p)
#pragma unroll
    for (int q = 0; q < NC; ++q) {
      const cx<double> t = HERM ? conj(K.m[q][p]) - K.m[p][q] : -K.m[p][q];
      double2* o = force + ((int64_t)(mu * NC + p) * NC + q) * V + x;
      st(o, ld(o) + scale * t);
    }
}

}  // namespace lym

using namespace lym;

extern "C" {

int lym_wilson_apply_adjoint(const lym_lattice* lat, int nc, double kappa, int hermitian, double bc_re,
                             double bc_im, const void* gauge_left, const void* gauge, int nvec, const void* in,
                             void* out, void* stream) {
  LYM_REQUIRE(lat && gauge_left && gauge && in && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(in != out, LYM_ERR_BAD_ARG, "in and out must not alias");
  LYM_REQUIRE(nvec >= 1 && nvec <= 65535, LYM_ERR_BAD_ARG, "nvec out of range");
  if (lat->nd != 2 && lat->nd != 4) {
    set_error("Number of dimensions %d not supported for fermions!", lat->nd);
    return LYM_ERR_UNSUPPORTED;
  }
  LYM_REQUIRE(nc == 2 || nc == 3, LYM_ERR_UNSUPPORTED, "N=%d not supported (2 or 3)", nc);
  const int per_block = lat->nd == 4 ? kAdjBlock / 2 : kAdjBlock;  // sites
  dim3 grid(grid_for(lat->V, per_block), nvec);
  cudaStream_t st = (cudaStream_t)stream;
  const int Lt = lat->dims[lat->nd - 1];
  const bool lr = gauge_left != gauge;
#define LYM_ADJ(ND_, NC_, H_, LR_)                                                                         \
  wilson_adjoint_kernel<ND_, NC_, H_, LR_><<<grid, kAdjBlock, 0, st>>>(                                    \
      lat->d_tab, (int)lat->V, Lt, kappa, bc_re, bc_im, (const double2*)gauge_left, (const double2*)gauge, \
      (const double2*)in, (double2*)out)
#define LYM_ADJ_H(ND_, NC_)                                              \
  do {                                                                   \
    if (hermitian) {                                                     \
      if (lr) LYM_ADJ(ND_, NC_, true, true);                             \
      else LYM_ADJ(ND_, NC_, true, false);                               \
    } else {                                                             \
      if (lr) LYM_ADJ(ND_, NC_, false, true);                            \
      else LYM_ADJ(ND_, NC_, false, false);                              \
    }                                                                    \
  } while (0)
  if (lat->nd == 2 && nc == 2) LYM_ADJ_H(2, 2);
  else if (lat->nd == 2 && nc == 3) LYM_ADJ_H(2, 3);
  else if (lat->nd == 4 && nc == 2) LYM_ADJ_H(4, 2);
  else LYM_ADJ_H(4, 3);
#undef LYM_ADJ_H
#undef LYM_ADJ
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_adjoint_links(const lym_lattice* lat, int nc, double bc_re, double bc_im, const void* gauge, void* out,
                      void* stream) {
  LYM_REQUIRE(lat && gauge && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(nc == 2 || nc == 3, LYM_ERR_UNSUPPORTED, "N=%d not supported (2 or 3)", nc);
  dim3 grid(grid_for(lat->V, kAdjBlock), lat->nd);
  cudaStream_t st = (cudaStream_t)stream;
  const int Lt = lat->dims[lat->nd - 1];
  if (nc == 2)
    adjoint_links_kernel<2><<<grid, kAdjBlock, 0, st>>>(lat->nd, lat->V, Lt, bc_re, bc_im, (const double2*)gauge,
                                                        (double2*)out);
  else
    adjoint_links_kernel<3><<<grid, kAdjBlock, 0, st>>>(lat->nd, lat->V, Lt, bc_re, bc_im, (const double2*)gauge,
                                                        (double2*)out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

int lym_fermion_force_adjoint(const lym_lattice* lat, int nc, double kappa, int hermitian, double bc_re,
                              double bc_im, const void* gauge, int nterms, const double* alphas, const void* X,
                              const void* Y, int symmetric, double scale, void* force, void* stream) {
  LYM_REQUIRE(lat && gauge && alphas && X && Y && force, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(nterms >= 1 && nterms <= kMaxAdjForceTerms, LYM_ERR_BAD_ARG, "nterms must be in [1, %d]",
              kMaxAdjForceTerms);
  if (lat->nd != 2 && lat->nd != 4) {
    set_error("Number of dimensions %d not supported for fermions!", lat->nd);
    return LYM_ERR_UNSUPPORTED;
  }
  LYM_REQUIRE(nc == 2 || nc == 3, LYM_ERR_UNSUPPORTED, "N=%d not supported (2 or 3)", nc);
  AdjForceTerms t;
  for (int i = 0; i < kMaxAdjForceTerms; ++i) t.alpha[i] = i < nterms ? alphas[i] : 0.0;
  const int sites = lat->nd == 4 ? 16 : 32;  // per warp and direction
  const unsigned grid = grid_for((lat->V + sites - 1) / sites * lat->nd, kAdjBlock / 32);
  cudaStream_t st = (cudaStream_t)stream;
  const int Lt = lat->dims[lat->nd - 1];
#define LYM_AF(ND_, NC_, H_)                                                                            \
  adjoint_force_kernel<ND_, NC_, H_><<<grid, kAdjBlock, 0, st>>>(lat->d_tab, lat->V, Lt, kappa, bc_re,    \
                                                                 bc_im, (const double2*)gauge, nterms, t, \
                                                                 (const double2*)X, (const double2*)Y,    \
                                                                 symmetric, scale, (double2*)force)
  if (lat->nd == 2 && nc == 2) { if (hermitian) LYM_AF(2, 2, true); else LYM_AF(2, 2, false); }
  else if (lat->nd == 2 && nc == 3) { if (hermitian) LYM_AF(2, 3, true); else LYM_AF(2, 3, false); }
  else if (lat->nd == 4 && nc == 2) { if (hermitian) LYM_AF(4, 2, true); else LYM_AF(4, 2, false); }
  else { if (hermitian) LYM_AF(4, 3, true); else LYM_AF(4, 3, false); }
#undef LYM_AF
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}

}  // extern "C"

// ---------------------------------------------------------------------------
// slice sums of the pion correlator (fermion_measurements.py:76-90)
// ---------------------------------------------------------------------------
namespace lym {

// out[2z], out[2z+1] = sum over the vectors and the sites with x_dir = z of
// sum_{spin,colour} conj(S) S (fundamental, (ns, N, V) per vector) or
// sum_{spin,c,d} conj(S_cd) S_dc (adjoint, (ns, N, N, V)); a cluster of blocks per slice,
// each adding its sites in a fixed order (deterministic).  One block per slice left most
// of the chip idle: 16^3 x 32 SU(3), 12 vectors, time slices: 93 us against 1049 us.
__global__ void __cluster_dims__(kSliceCtas, 1, 1) __launch_bounds__(kSliceThreads)
    timeslice_sums_kernel(int64_t V, uint32_t stride, uint32_t L, int nvec, int ns, int nc, int adjoint,
                          const double2* __restrict__ in, double* __restrict__ out) {
  const uint32_t z = blockIdx.x / kSliceCtas, rank = blockIdx.x % kSliceCtas;
  const uint32_t per = (uint32_t)(V / L);
  const int ncomp = adjoint ? nc * nc : nc;
  const int64_t planes = (int64_t)nvec * ns * ncomp;
  double re = 0.0, im = 0.0;
  for (uint32_t j = rank * kSliceThreads + threadIdx.x; j < per; j += kSliceCtas * kSliceThreads) {
    const double2* base = in + ((j / stride) * (L * stride) + z * stride + j % stride);
    if (!adjoint) {
#pragma unroll 4
      for (int64_t p = 0; p < planes; ++p) {
        const cx<double> a = ld(base + p * V);
        re += a.re * a.re + a.im * a.im;
      }
    } else {
      for (int64_t p = 0; p < planes; p += ncomp)
        for (int c = 0; c < nc; ++c)
          for (int d = 0; d < nc; ++d) {
            const cx<double> t = cmul_cj(ld(base + (p + c * nc + d) * V), ld(base + (p + d * nc + c) * V));
            re += t.re;
            im += t.im;
          }
    }
  }
  cluster_pair_sum(re, im, out + 2 * z);
}

}  // namespace lym

extern "C" int lym_timeslice_sums(const lym_lattice* lat, int direction, int nvec, int ns, int nc, int adjoint,
                                  const void* in, double* out, void* stream) {
  using namespace lym;
  LYM_REQUIRE(lat && in && out, LYM_ERR_BAD_ARG, "null argument");
  LYM_REQUIRE(direction >= 0 && direction < lat->nd, LYM_ERR_BAD_ARG, "direction %d out of range", direction);
  LYM_REQUIRE(nvec >= 1 && ns >= 1 && nc >= 1, LYM_ERR_BAD_ARG, "bad sizes");
  int64_t stride = 1;
  for (int d = direction + 1; d < lat->nd; ++d) stride *= lat->dims[d];
  const int L = lat->dims[direction];
  timeslice_sums_kernel<<<L * kSliceCtas, kSliceThreads, 0, (cudaStream_t)stream>>>(lat->V, (uint32_t)stride, L, nvec, ns, nc, adjoint != 0,
                                                            (const double2*)in, out);
  LYM_CHECK_LAUNCH();
  return LYM_OK;
}
