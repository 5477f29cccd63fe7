// Small SU(N) matrix algebra (N = 2, 3) in registers, FP64, and what the per-link and
// per-slice kernels share.
#pragma once

#include <cooperative_groups.h>

#include "lym_internal.cuh"

namespace lym {

template <int N>
struct Mat {
  cx<double> m[N][N];
};

// reference gauge layout (nd, N, N, V): element (mu, i, j, s)
template <int N>
LYM_D Mat<N> load_link(const double2* __restrict__ U, int mu, int64_t s, int64_t V) {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) r.m[i][j] = ld(U + ((int64_t)(mu * N + i) * N + j) * V + s);
  return r;
}

template <int N>
LYM_D void store_link(double2* __restrict__ U, int mu, int64_t s, int64_t V, const Mat<N>& a) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) st(U + ((int64_t)(mu * N + i) * N + j) * V + s, a.m[i][j]);
}

template <int N>
LYM_D Mat<N> mzero() {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) r.m[i][j] = czero<double>();
  return r;
}

template <int N>
LYM_D Mat<N> mident() {
  Mat<N> r = mzero<N>();
#pragma unroll
  for (int i = 0; i < N; ++i) r.m[i][i] = {1.0, 0.0};
  return r;
}

// Thread -> link for the kernels that read neighbouring links: warp w of the grid takes
// direction w mod nd of the 32 sites of site block w / nd, so the directions of a site run
// side by side in one block and the links they share (44 distinct links per site in 4D
// against 76 loads) meet in L1; with the direction as the slow grid index every direction
// streamed the field through L2 on its own.
LYM_D bool warp_link(int nd, int64_t V, int64_t block, int& mu, int64_t& s) {
  const int64_t w = block * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t sb = w / nd;
  mu = (int)(w - sb * nd);
  s = sb * 32 + (threadIdx.x & 31);
  return s < V;
}
inline unsigned warp_link_grid(int nd, int64_t V, int block) { return grid_for((V + 31) / 32 * nd, block / 32); }

// A B
template <int N>
LYM_D Mat<N> mul(const Mat<N>& a, const Mat<N>& b) {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      cx<double> t = a.m[i][0] * b.m[0][j];
#pragma unroll
      for (int k = 1; k < N; ++k) cmac(t, a.m[i][k], b.m[k][j]);
      r.m[i][j] = t;
    }
  return r;
}

// A B^dag
template <int N>
LYM_D Mat<N> mul_nd(const Mat<N>& a, const Mat<N>& b) {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      cx<double> t = cmul_cj(b.m[j][0], a.m[i][0]);
#pragma unroll
      for (int k = 1; k < N; ++k) cmac_cj(t, b.m[j][k], a.m[i][k]);
      r.m[i][j] = t;
    }
  return r;
}

// r = a B for a row vector a
template <int N>
LYM_D void row_mul(cx<double> (&r)[N], const cx<double> (&a)[N], const Mat<N>& b) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    r[j] = a[0] * b.m[0][j];
#pragma unroll
    for (int k = 1; k < N; ++k) cmac(r[j], a[k], b.m[k][j]);
  }
}
// s += a B
template <int N>
LYM_D void row_mac(cx<double> (&s)[N], const cx<double> (&a)[N], const Mat<N>& b) {
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int k = 0; k < N; ++k) cmac(s[j], a[k], b.m[k][j]);
}
// s += a B^dag
template <int N>
LYM_D void row_mac_nd(cx<double> (&s)[N], const cx<double> (&a)[N], const Mat<N>& b) {
#pragma unroll
  for (int j = 0; j < N; ++j)
#pragma unroll
    for (int k = 0; k < N; ++k) cmac_cj(s[j], b.m[j][k], a[k]);
}

// A^dag B
template <int N>
LYM_D Mat<N> mul_dn(const Mat<N>& a, const Mat<N>& b) {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) {
      cx<double> t = cmul_cj(a.m[0][i], b.m[0][j]);
#pragma unroll
      for (int k = 1; k < N; ++k) cmac_cj(t, a.m[k][i], b.m[k][j]);
      r.m[i][j] = t;
    }
  return r;
}

template <int N>
LYM_D void madd(Mat<N>& a, const Mat<N>& b) {
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) a.m[i][j] += b.m[i][j];
}

template <int N>
LYM_D Mat<N> mscale(cx<double> s, const Mat<N>& a) {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) r.m[i][j] = s * a.m[i][j];
  return r;
}

template <int N>
LYM_D Mat<N> mdag(const Mat<N>& a) {
  Mat<N> r;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) r.m[i][j] = conj(a.m[j][i]);
  return r;
}

template <int N>
LYM_D cx<double> trace(const Mat<N>& a) {
  cx<double> t = czero<double>();
#pragma unroll
  for (int i = 0; i < N; ++i) t += a.m[i][i];
  return t;
}

template <int N>
LYM_D double fro2(const Mat<N>& a) {
  double t = 0;
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int j = 0; j < N; ++j) t += norm2(a.m[i][j]);
  return t;
}

LYM_D cx<double> det(const Mat<2>& a) { return a.m[0][0] * a.m[1][1] - a.m[0][1] * a.m[1][0]; }
LYM_D cx<double> det(const Mat<3>& a) {
  return a.m[0][0] * (a.m[1][1] * a.m[2][2] - a.m[1][2] * a.m[2][1]) -
         a.m[0][1] * (a.m[1][0] * a.m[2][2] - a.m[1][2] * a.m[2][0]) +
         a.m[0][2] * (a.m[1][0] * a.m[2][1] - a.m[1][1] * a.m[2][0]);
}

// cofactor matrix C: inverse(A) = C^T / det(A)
LYM_D Mat<2> cofactors(const Mat<2>& a) {
  Mat<2> r;
  r.m[0][0] = a.m[1][1];
  r.m[0][1] = -a.m[1][0];
  r.m[1][0] = -a.m[0][1];
  r.m[1][1] = a.m[0][0];
  return r;
}
LYM_D Mat<3> cofactors(const Mat<3>& a) {
  Mat<3> r;
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      const int i1 = (i + 1) % 3, i2 = (i + 2) % 3, j1 = (j + 1) % 3, j2 = (j + 2) % 3;
      cx<double> t = a.m[i1][j1] * a.m[i2][j2];
      cmac(t, -a.m[i1][j2], a.m[i2][j1]);
      r.m[i][j] = t;
    }
  return r;
}

// principal N-th root of a non-zero complex number (matches numpy's z ** (1/N))
LYM_D cx<double> principal_root(cx<double> z, int n) {
  double r = sqrt(z.re * z.re + z.im * z.im);
  double ph = atan2(z.im, z.re);
  double rr = pow(r, 1.0 / n);
  double s, c;
  sincos(ph / n, &s, &c);
  return {rr * c, rr * s};
}

LYM_D cx<double> cdiv(cx<double> a, cx<double> b) {
  double n = norm2(b);
  return {(a.re * b.re + a.im * b.im) / n, (a.im * b.re - a.re * b.im) / n};
}

// Sums over lattice slices and shifted products, a cluster of kSliceCtas blocks per sum:
// every block adds its part in a fixed order, block 0 of the cluster adds the parts in
// block order through distributed shared memory, so the result is deterministic and needs
// no scratch that two streams could share.
constexpr int kSliceCtas = 8, kSliceThreads = 512;

LYM_D void cluster_pair_sum(double re, double im, double* out) {
  __shared__ double sh[2 * 32];
  __shared__ double mine[2];
  double v[2] = {re, im};
  block_sum<2>(v, sh);
  if (threadIdx.x == 0) {
    mine[0] = v[0];
    mine[1] = v[1];
  }
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  cl.sync();
  if (cl.block_rank() == 0 && threadIdx.x == 0) {
    double a = 0.0, b = 0.0;
    for (int r = 0; r < kSliceCtas; ++r) {
      const double* o = cl.map_shared_rank(mine, r);
      a += o[0];
      b += o[1];
    }
    out[0] = a;
    out[1] = b;
  }
  cl.sync();  // no block leaves while its part may still be read
}

}  // namespace lym
