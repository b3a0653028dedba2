// The clover term: field strength, the term's 6x6 blocks with their inverses,
// and its molecular-dynamics force.  FP64 throughout, on the resident links
// with all three rows stored (GaugeArrays::d18): threads take consecutive
// half-sites of one parity, so link loads are coalesced.
#include <cstdint>

#include "internal.h"

namespace iro {

using M3d = Su3<double>;

// C = A B, A B^dag, A^dag B
__device__ __forceinline__ M3d m3_mul(const M3d& A, const M3d& B) {
  M3d C;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      C.e[a][b] = A.e[a][0] * B.e[0][b] + A.e[a][1] * B.e[1][b] + A.e[a][2] * B.e[2][b];
  return C;
}
__device__ __forceinline__ M3d m3_mul_nd(const M3d& A, const M3d& B) {
  M3d C;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      C.e[a][b] = mul_cj(A.e[a][0], B.e[b][0]) + mul_cj(A.e[a][1], B.e[b][1]) + mul_cj(A.e[a][2], B.e[b][2]);
  return C;
}
__device__ __forceinline__ M3d m3_mul_dn(const M3d& A, const M3d& B) {
  M3d C;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b)
      C.e[a][b] = cj_mul(A.e[0][a], B.e[0][b]) + cj_mul(A.e[1][a], B.e[1][b]) + cj_mul(A.e[2][a], B.e[2][b]);
  return C;
}
__device__ __forceinline__ M3d m3_dag(const M3d& A) {
  M3d C;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) C.e[a][b] = conjx(A.e[b][a]);
  return C;
}
__device__ __forceinline__ void m3_add(M3d& A, const M3d& B) {
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) A.e[a][b] = A.e[a][b] + B.e[a][b];
}

// A site and the steps from it in lexicographic index (x fastest); all extents
// are even, so a step also flips the parity at the periodic wrap, and the
// half-site index of a lexicographic index is its half.
struct Site {
  int p, lex;
  int c[4];
};
__device__ __forceinline__ Site site_of(const Geom& g, int hs, int p) {
  const Coord c = coord_of(g, hs, p);
  return Site{p, c.x + g.L[0] * c.row, {c.x, c.y, c.z, c.t}};
}
__device__ __forceinline__ int step(const Geom& g, const Site& s, int d, int sign) {
  const int x = d == 0 ? s.c[0] : d == 1 ? s.c[1] : d == 2 ? s.c[2] : s.c[3];
  const int stride = d == 0 ? 1 : d == 1 ? g.L[0] : d == 2 ? 2 * g.sz : 2 * g.st;
  const int n = g.L[d];
  if (sign > 0) return x + 1 == n ? -(n - 1) * stride : stride;
  return x == 0 ? (n - 1) * stride : -stride;
}
// link mu of the site `off` away from s (odd: an odd number of steps)
__device__ __forceinline__ M3d link_at(const double2* __restrict__ d18, int64_t vh, const Site& s, int off,
                                       int odd, int mu) {
  M3d U;
  const double2* q = link_chunk0<9>(d18, vh, s.p ^ odd, mu, (s.lex + off) >> 1);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    const double2 v = __ldg(q + 32 * k);
    U.e[k / 3][k % 3] = {v.x, v.y};
  }
  return U;
}

// A traceless anti-hermitian 3x3 matrix as 9 reals: the imaginary diagonal,
// then re, im of (0,1), (0,2), (1,2).  tah(M) is (M - M^dag)/2 without trace.
__device__ __forceinline__ void tah(const M3d& M, double f[9]) {
  const double tr = (M.e[0][0].im + M.e[1][1].im + M.e[2][2].im) / 3.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) f[i] = M.e[i][i].im - tr;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
    f[3 + 2 * k] = 0.5 * (M.e[i][j].re - M.e[j][i].re);
    f[4 + 2 * k] = 0.5 * (M.e[i][j].im + M.e[j][i].im);
  }
}
__device__ __forceinline__ M3d tah_matrix(const double f[9]) {
  M3d M;
#pragma unroll
  for (int i = 0; i < 3; ++i) M.e[i][i] = {0.0, f[i]};
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const int i = k == 2 ? 1 : 0, j = k == 0 ? 1 : 2;
    M.e[i][j] = {f[3 + 2 * k], f[4 + 2 * k]};
    M.e[j][i] = {-f[3 + 2 * k], f[4 + 2 * k]};
  }
  return M;
}

// v(y) = Vup(y)^dag - Vdn(y)^dag of Staples::fieldStrength
// (lib/Measurements/GaugeM/staples.cpp:596-597, 641-643) at the site y that is
// `o` away from s; dm, dn, dnm: the steps +mu (from y), +nu, -nu
__device__ __forceinline__ M3d leaves(const double2* __restrict__ d18, int64_t vh, const Site& s, int o,
                                      int odd, int dm, int dn, int dnm, int mu, int nu) {
  // U_nu(y+mu) U_mu(y+nu)^dag U_nu(y)^dag
  M3d a = m3_mul_nd(link_at(d18, vh, s, o + dm, odd ^ 1, nu), link_at(d18, vh, s, o + dn, odd ^ 1, mu));
  a = m3_mul_nd(a, link_at(d18, vh, s, o, odd, nu));
  // (U_mu(y-nu) U_nu(y-nu+mu))^dag U_nu(y-nu)
  M3d b = m3_mul(link_at(d18, vh, s, o + dnm, odd ^ 1, mu), link_at(d18, vh, s, o + dnm + dm, odd, nu));
  b = m3_mul_dn(b, link_at(d18, vh, s, o + dnm, odd ^ 1, nu));
#pragma unroll
  for (int i = 0; i < 3; ++i)
#pragma unroll
    for (int j = 0; j < 3; ++j) a.e[i][j] = a.e[i][j] - b.e[i][j];
  return a;
}

// F_{mu nu}(s) (Staples::fieldStrength, staples.cpp:587-666): a quarter of the
// traceless anti-hermitian part of U_mu(x) v(x) + v(x-mu) U_mu(x-mu)
__device__ __forceinline__ void field_strength_at(const Geom& g, const double2* __restrict__ d18,
                                                  const Site& s, int mu, int nu, double f[9]) {
  const int64_t vh = g.Vh;
  const int dm = step(g, s, mu, 1), dmm = step(g, s, mu, -1), dn = step(g, s, nu, 1), dnm = step(g, s, nu, -1);
  M3d M = m3_mul(link_at(d18, vh, s, 0, 0, mu), leaves(d18, vh, s, 0, 0, dm, dn, dnm, mu, nu));
  // from x - mu, the step +mu leads back to x
  m3_add(M, m3_mul(leaves(d18, vh, s, dmm, 1, -dmm, dn, dnm, mu, nu), link_at(d18, vh, s, dmm, 1, mu)));
  tah(M, f);
#pragma unroll
  for (int k = 0; k < 9; ++k) f[k] *= 0.25;
}

__global__ void __launch_bounds__(128) field_strength_kernel(Geom g, const double2* d18, int mu, int nu,
                                                             double* out) {
  const int hs = blockIdx.x * blockDim.x + threadIdx.x;
  if (hs >= g.Vh) return;
  const Site s = site_of(g, hs, blockIdx.y);
  double f[9];
  field_strength_at(g, d18, s, mu, nu, f);
  const M3d M = tah_matrix(f);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    out[18 * int64_t(s.lex) + 2 * k] = M.e[k / 3][k % 3].re;
    out[18 * int64_t(s.lex) + 2 * k + 1] = M.e[k / 3][k % 3].im;
  }
}

cudaError_t launch_field_strength(const Geom& g, const double2* d18, int mu, int nu, double* out,
                                  cudaStream_t st) {
  field_strength_kernel<<<dim3((g.Vh + 127) / 128, 2), 128, 0, st>>>(g, d18, mu, nu, out);
  return cudaGetLastError();
}

// ---- the term's blocks -----------------------------------------------------------------
// Hermitian 6x6 matrix: real diagonal and upper triangle (CloverBlock).
using Block = CloverBlock<double>;

// Element (i, j), i != j, of a block, either side of the diagonal
__device__ __forceinline__ Cx<double> at(const Block& B, int i, int j) {
  return i < j ? B.o[tri(i, j)] : conjx(B.o[tri(j, i)]);
}

// B <- B^-1 by the symmetric sweep operator (Beaton 1964; Goodnight, "A tutorial
// on the SWEEP operator", The American Statistician 33 (1979)): sweeping every
// diagonal element of a Hermitian matrix leaves -B^-1, and each sweep keeps it
// Hermitian, so 36 reals live in registers.  The pivots are the diagonal
// elements in order; false when one is below half of the largest element it
// would eliminate (the term is 1 plus a small matrix: this is for very rough
// fields), where the caller pivots instead.
__device__ __forceinline__ bool invert_sweep(Block& B) {
  bool fine = true;
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    double big = 0.0;
#pragma unroll
    for (int i = k + 1; i < 6; ++i) {
      const Cx<double> v = at(B, i, k);
      big = fmax(big, v.re * v.re + v.im * v.im);
    }
    fine = fine && B.d[k] != 0.0 && 4.0 * B.d[k] * B.d[k] >= big;
    const double inv = 1.0 / B.d[k];
    Cx<double> col[6];  // a_ik / a_kk
#pragma unroll
    for (int i = 0; i < 6; ++i)
      if (i != k) col[i] = inv * at(B, i, k);
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      if (i == k) continue;
      const Cx<double> v = at(B, i, k);
      B.d[i] -= v.re * col[i].re + v.im * col[i].im;
#pragma unroll
      for (int j = i + 1; j < 6; ++j)
        if (j != k) B.o[tri(i, j)] = B.o[tri(i, j)] - mul_cj(col[i], at(B, j, k));
    }
#pragma unroll
    for (int i = 0; i < 6; ++i) {
      if (i < k) B.o[tri(i, k)] = col[i];
      if (i > k) B.o[tri(k, i)] = conjx(col[i]);
    }
    B.d[k] = -inv;
  }
#pragma unroll
  for (int k = 0; k < 6; ++k) B.d[k] = -B.d[k];
#pragma unroll
  for (int k = 0; k < 15; ++k) B.o[k] = {-B.o[k].re, -B.o[k].im};
  return fine;
}

// The same by Gauss-Jordan elimination with partial pivoting; false when singular
__device__ __noinline__ bool invert_pivoted(Block& B) {
  Cx<double> a[6][6], inv[6][6];
  for (int i = 0; i < 6; ++i)
    for (int j = 0; j < 6; ++j) {
      a[i][j] = i == j ? Cx<double>{B.d[i], 0.0} : at(B, i, j);
      inv[i][j] = {i == j ? 1.0 : 0.0, 0.0};
    }
  for (int c = 0; c < 6; ++c) {
    int piv = c;
    double best = a[c][c].re * a[c][c].re + a[c][c].im * a[c][c].im;
    for (int r = c + 1; r < 6; ++r) {
      const double m = a[r][c].re * a[r][c].re + a[r][c].im * a[r][c].im;
      if (m > best) {
        best = m;
        piv = r;
      }
    }
    if (!(best > 0.0)) return false;
    if (piv != c)
      for (int j = 0; j < 6; ++j) {
        Cx<double> t = a[c][j]; a[c][j] = a[piv][j]; a[piv][j] = t;
        t = inv[c][j]; inv[c][j] = inv[piv][j]; inv[piv][j] = t;
      }
    const double den = a[c][c].re * a[c][c].re + a[c][c].im * a[c][c].im;
    const Cx<double> rp = {a[c][c].re / den, -a[c][c].im / den};
    for (int j = 0; j < 6; ++j) {
      a[c][j] = a[c][j] * rp;
      inv[c][j] = inv[c][j] * rp;
    }
    for (int r = 0; r < 6; ++r) {
      if (r == c) continue;
      const Cx<double> f = a[r][c];
      for (int j = 0; j < 6; ++j) {
        a[r][j] = a[r][j] - f * a[c][j];
        inv[r][j] = inv[r][j] - f * inv[c][j];
      }
    }
  }
  for (int i = 0; i < 6; ++i) {
    B.d[i] = inv[i][i].re;
    for (int j = i + 1; j < 6; ++j)
      B.o[tri(i, j)] = {0.5 * (inv[i][j].re + inv[j][i].re), 0.5 * (inv[i][j].im - inv[j][i].im)};
  }
  return true;
}

// Block `blk` of half-site hs of parity p in every storage precision: values
// 36 blk .. 36 blk + 35 of the site's 72 (the diagonal, then the triangle)
__device__ __forceinline__ void store_block(void* const arr[3][2], int p, int hs, int blk, const Block& B) {
  double v[36];
#pragma unroll
  for (int i = 0; i < 6; ++i) v[i] = B.d[i];
#pragma unroll
  for (int k = 0; k < 15; ++k) {
    v[6 + 2 * k] = B.o[k].re;
    v[7 + 2 * k] = B.o[k].im;
  }
  double2* d = chunk0<36>(static_cast<double2*>(arr[0][p]), hs) + 32 * 18 * blk;
#pragma unroll
  for (int k = 0; k < 18; ++k) d[32 * k] = make_double2(v[2 * k], v[2 * k + 1]);
  float4* f = chunk0<18>(static_cast<float4*>(arr[1][p]), hs) + 32 * 9 * blk;
#pragma unroll
  for (int k = 0; k < 9; ++k)
    f[32 * k] = make_float4(float(v[4 * k]), float(v[4 * k + 1]), float(v[4 * k + 2]), float(v[4 * k + 3]));
  // FP16: 9 chunks of 8 halves over both blocks; chunk 4 is half of each
  uint32_t h[18];
#pragma unroll
  for (int k = 0; k < 18; ++k) h[k] = pack_h2(float(v[2 * k]), float(v[2 * k + 1]));
  uint4* q = chunk0<9>(static_cast<uint4*>(arr[2][p]), hs);
  uint2* mid = reinterpret_cast<uint2*>(q + 32 * 4) + blk;
  if (blk == 0) {
#pragma unroll
    for (int k = 0; k < 4; ++k) q[32 * k] = make_uint4(h[4 * k], h[4 * k + 1], h[4 * k + 2], h[4 * k + 3]);
    *mid = make_uint2(h[16], h[17]);
  } else {
    *mid = make_uint2(h[0], h[1]);
#pragma unroll
    for (int k = 0; k < 4; ++k)
      q[32 * (5 + k)] = make_uint4(h[2 + 4 * k], h[3 + 4 * k], h[4 + 4 * k], h[5 + 4 * k]);
  }
}

__constant__ int8_t c_plane[6][2] = {{1, 2}, {2, 0}, {0, 1}, {3, 0}, {3, 1}, {3, 2}};

// A = 1 - kappa csw sum_k F_k (i sigma_k) (Dirac_Clover::set_csw,
// lib/Dirac_ops/dirac_clover.cpp:139-162, isigma_* :221-329) as its two 6x6
// blocks on phi+- and their inverses.  With G_j = F_j -+ F_{j+3} the block is
//   1 - kappa csw [[i G_2, i G_0 + G_1], [i G_0 - G_1, -i G_2]].
// A CTA takes 96 half-sites: warp k forms plane k's field strength of all of
// them into shared memory, then each thread owns one block: it is formed,
// stored, inverted in registers and stored again.
//
// Bound by the FP64 pipe (10 matrix products a plane and site) and the stores
// (2016 B a site).  One thread per site over Format_G links, with 64-bit index
// divisions and the blocks in local memory, took 4.84 ms at 24^3x48;
// 1.08 ms now.
constexpr int kBuildSites = 96;
constexpr int kBuildThreads = 192;
__global__ void __launch_bounds__(kBuildThreads, 2) clover_build_kernel(Geom g, const double2* __restrict__ d18,
                                                                        double kc, CloverArrays ca,
                                                                        int* singular) {
  __shared__ double F[6][9][kBuildSites];
  const int p = blockIdx.y;
  const int base = blockIdx.x * kBuildSites;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (int grp = 0; grp < kBuildSites / 32; ++grp) {
    const int hs = base + 32 * grp + lane;
    if (hs >= g.Vh) break;
    double f[9];
    field_strength_at(g, d18, site_of(g, hs, p), c_plane[warp][0], c_plane[warp][1], f);
#pragma unroll
    for (int k = 0; k < 9; ++k) F[warp][k][32 * grp + lane] = f[k];
  }
  __syncthreads();
  const int blk = threadIdx.x / kBuildSites, sl = threadIdx.x - blk * kBuildSites;
  const int hs = base + sl;
  if (hs >= g.Vh) return;
  // G_j = F_j - s F_{j+3}, s = +1 for phi+ and -1 for phi-
  const double sg = blk == 0 ? 1.0 : -1.0;
  double G[3][9];
#pragma unroll
  for (int j = 0; j < 3; ++j)
#pragma unroll
    for (int k = 0; k < 9; ++k) G[j][k] = F[j][k][sl] - sg * F[j + 3][k][sl];
  const M3d G0 = tah_matrix(G[0]), G1 = tah_matrix(G[1]), G2 = tah_matrix(G[2]);
  Block B;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    // -kc (i G_2)_ii = kc Im (G_2)_ii
    B.d[i] = 1.0 + kc * G2.e[i][i].im;
    B.d[3 + i] = 1.0 - kc * G2.e[i][i].im;
#pragma unroll
    for (int j = i + 1; j < 3; ++j) {
      const Cx<double> t = kc * mul_mi(G2.e[i][j]);
      B.o[tri(i, j)] = t;
      B.o[tri(3 + i, 3 + j)] = {-t.re, -t.im};
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) B.o[tri(i, 3 + j)] = kc * (mul_mi(G0.e[i][j]) - G1.e[i][j]);
  }
  store_block(ca.A, p, hs, blk, B);
  Block I = B;
  if (!invert_sweep(I)) {
    I = B;
    if (!invert_pivoted(I)) atomicExch(singular, 1);
  }
  store_block(ca.Ainv, p, hs, blk, I);
}

cudaError_t launch_clover_build(const Geom& g, const double2* d18, double kappa_csw, CloverArrays ca,
                                int* singular, cudaStream_t st) {
  clover_build_kernel<<<dim3((g.Vh + kBuildSites - 1) / kBuildSites, 2), kBuildThreads, 0, st>>>(
      g, d18, kappa_csw, ca, singular);
  return cudaGetLastError();
}

// ---- the term's force --------------------------------------------------------------------
// Dirac_Clover::md_force (lib/Dirac_ops/dirac_clover.cpp:356-367; its block
// md_force_block :369-532) adds to the Wilson force the derivative of the
// clover term T f = -kappa csw sum_k (i sigma_k (x) F_k) f, F_k = 0.25 TA(Q_k),
// Q_k(x) the four leaves at x in the plane of k (Staples::fieldStrength,
// staples.cpp:587-666), TA the traceless anti-hermitian part.  TA is
// self-adjoint for Re Tr, so
//   Re(zeta^dag T eta) = -kappa csw / 4 sum_{x,k} Re Tr(Q_k(x) Lambda_k(x)),
//   Lambda_k(x) = TA(sum_{s,t} (i sigma_k)_{st} eta_t(x) zeta_s(x)^dag).
// A plaquette through the link U = U_rho(y) is a leaf of its four corners, each
// with that corner's Lambda inserted in the loop (Lambda^dag = -Lambda makes the
// two orientations agree), so with the rest of the loop from y + rho back to y
// as A B C the link's force is, in the convention of the Wilson force
// (Re Tr(X F_mu(x)) = d/de Re(zeta^dag D(U_mu(x) -> (1 + e X) U_mu(x)) eta)),
//   +- U [ L1 A B C + A L2 B C + A B L3 C + A B C L4 ],
// L1 .. L4 the corners' Lambda from y + rho on: + for the plaquette on the side
// of +nu when rho is the plane's first direction, - on the other side, both
// reversed when it is the second.

// i sigma_k (k = Bx, By, Bz, Ex, Ey, Ez; Dirac_Clover::isigma_{23,31,12,41,42,43},
// dirac_clover.cpp:221-329): row s has one entry, i^phase at column perm
template <int K, int S>
struct ISigma {
  static constexpr int perm = K < 2 ? (S ^ 1) : K == 2 ? S : K < 5 ? 3 - S : (S ^ 2);
  static constexpr int phase = K == 0   ? 1
                               : K == 1 ? ((S & 1) ? 2 : 0)
                               : K == 2 ? ((S & 1) ? 3 : 1)
                               : K == 3 ? 3
                               : K == 4 ? ((S & 1) ? 0 : 2)
                                        : ((S & 1) ? 1 : 3);
};
template <int PHASE>
__device__ __forceinline__ Cx<double> times_phase(Cx<double> v) {
  return PHASE == 0 ? v : PHASE == 1 ? mul_i(v) : PHASE == 2 ? Cx<double>{-v.re, -v.im} : mul_mi(v);
}

template <int K>
__device__ __forceinline__ void lambda_plane(const Cx<double> et[12], const Cx<double> zt[12], double f[9]) {
  M3d M;
#pragma unroll
  for (int b = 0; b < 3; ++b)
#pragma unroll
    for (int a = 0; a < 3; ++a)
      M.e[b][a] = times_phase<ISigma<K, 0>::phase>(mul_cj(et[3 * ISigma<K, 0>::perm + b], zt[a])) +
                  times_phase<ISigma<K, 1>::phase>(mul_cj(et[3 * ISigma<K, 1>::perm + b], zt[3 + a])) +
                  times_phase<ISigma<K, 2>::phase>(mul_cj(et[3 * ISigma<K, 2>::perm + b], zt[6 + a])) +
                  times_phase<ISigma<K, 3>::phase>(mul_cj(et[3 * ISigma<K, 3>::perm + b], zt[9 + a]));
  tah(M, f);
}

// Lambda_k(x) as 9 reals each: lam[((k * 9 + q) * 2 + parity) * Vh + half-site]
__global__ void __launch_bounds__(128) clover_lambda_kernel(Geom g, SpinorPtr e0, SpinorPtr e1, SpinorPtr z0,
                                                            SpinorPtr z1, double* __restrict__ lam) {
  const int hs = blockIdx.x * blockDim.x + threadIdx.x;
  if (hs >= g.Vh) return;
  const int p = blockIdx.y;
  Cx<double> et[12], zt[12];
  SpinorIO<PREC_DOUBLE>::load(p ? e1 : e0, hs, et);
  SpinorIO<PREC_DOUBLE>::load(p ? z1 : z0, hs, zt);
  double* out = lam + size_t(p) * g.Vh + hs;
  const size_t V = 2 * size_t(g.Vh);
  auto put = [&](int k, const double f[9]) {
#pragma unroll
    for (int q = 0; q < 9; ++q) out[(size_t(k) * 9 + q) * V] = f[q];
  };
  double f[9];
  lambda_plane<0>(et, zt, f); put(0, f);
  lambda_plane<1>(et, zt, f); put(1, f);
  lambda_plane<2>(et, zt, f); put(2, f);
  lambda_plane<3>(et, zt, f); put(3, f);
  lambda_plane<4>(et, zt, f); put(4, f);
  lambda_plane<5>(et, zt, f); put(5, f);
}

__device__ __forceinline__ M3d lambda_at(const double* __restrict__ lam, int64_t vh, int k, const Site& s,
                                         int off, int odd) {
  const double* q = lam + (size_t(k) * 9 * 2 + (s.p ^ odd)) * vh + ((s.lex + off) >> 1);
  double f[9];
#pragma unroll
  for (int j = 0; j < 9; ++j) f[j] = __ldg(q + size_t(j) * 2 * vh);
  return tah_matrix(f);
}

// L1 A B C + A L2 B C + A B L3 C + A B C L4 of the plaquette of U_rho(y) on the
// +nu (UP) or -nu side; dr: the step +rho, dn: the step to that side
template <bool UP>
__device__ __forceinline__ M3d plaquette_force(const double2* __restrict__ d18, const double* __restrict__ lam,
                                               int64_t vh, const Site& s, int dr, int dn, int rho, int nu, int k) {
  // A = U_nu(y+rho), B = U_rho(y+nu)^dag, C = U_nu(y)^dag on the +nu side;
  // A = U_nu(y+rho-nu)^dag, B = U_rho(y-nu)^dag, C = U_nu(y-nu) on the other
  M3d P, AB;
  {
    M3d A = link_at(d18, vh, s, UP ? dr : dr + dn, UP ? 1 : 0, nu);
    if (!UP) A = m3_dag(A);
    P = m3_mul(lambda_at(lam, vh, k, s, dr, 1), A);
    m3_add(P, m3_mul(A, lambda_at(lam, vh, k, s, dr + dn, 0)));
    const M3d B = link_at(d18, vh, s, dn, 1, rho);
    AB = m3_mul_nd(A, B);
    P = m3_mul_nd(P, B);
  }
  m3_add(P, m3_mul(AB, lambda_at(lam, vh, k, s, dn, 1)));
  const M3d C = link_at(d18, vh, s, UP ? 0 : dn, UP ? 0 : 1, nu);
  P = UP ? m3_mul_nd(P, C) : m3_mul(P, C);
  AB = UP ? m3_mul_nd(AB, C) : m3_mul(AB, C);
  m3_add(P, m3_mul(AB, lambda_at(lam, vh, k, s, 0, 0)));
  return P;
}

// plane of directions (rho, nu)
__constant__ int8_t c_plane_of[4][4] = {{-1, 2, 1, 3}, {2, -1, 0, 4}, {1, 0, -1, 5}, {3, 4, 5, -1}};

// One thread per link: F_rho(y) += w times its six plaquettes' terms, in a
// fixed order.  Bound by the FP64 pipe: 8 matrix products a plaquette, 49 a
// link.  Summing the 24 occurrences of a link in the leaves one by one (144
// products a link, on 144-byte Format_G links) took 1.14 ms at 16^3x32;
// 0.37 ms now (Lambda 0.088 -> 0.017 ms).
__global__ void __launch_bounds__(128, 2) clover_force_kernel(Geom g, const double2* __restrict__ d18,
                                                              const double* __restrict__ lam, double w,
                                                              double* __restrict__ F) {
  const int hs = blockIdx.x * blockDim.x + threadIdx.x;
  if (hs >= g.Vh) return;
  const int rho = blockIdx.z;
  const int64_t vh = g.Vh;
  const Site s = site_of(g, hs, blockIdx.y);
  const int dr = step(g, s, rho, 1);
  M3d acc;
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) acc.e[a][b] = {0.0, 0.0};
#pragma unroll 1
  for (int j = 1; j < 4; ++j) {
    const int nu = (rho + j) & 3;
    const int k = c_plane_of[rho][nu];
    const double sg = c_plane[k][0] == rho ? 1.0 : -1.0;
    const M3d up = plaquette_force<true>(d18, lam, vh, s, dr, step(g, s, nu, 1), rho, nu, k);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) acc.e[a][b] = acc.e[a][b] + sg * up.e[a][b];
    const M3d dn = plaquette_force<false>(d18, lam, vh, s, dr, step(g, s, nu, -1), rho, nu, k);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) acc.e[a][b] = acc.e[a][b] - sg * dn.e[a][b];
  }
  const M3d R = m3_mul(link_at(d18, vh, s, 0, 0, rho), acc);
  double2* Fp = reinterpret_cast<double2*>(F) + 9 * (int64_t(s.lex) + 2 * vh * rho);
#pragma unroll
  for (int k = 0; k < 9; ++k) {
    double2 f = Fp[k];
    f.x += w * R.e[k / 3][k % 3].re;
    f.y += w * R.e[k / 3][k % 3].im;
    Fp[k] = f;
  }
}

cudaError_t launch_clover_force(const Geom& g, const double2* d18, SpinorPtr e0, SpinorPtr e1, SpinorPtr z0,
                                SpinorPtr z1, double w, double* lam, double* F, cudaStream_t st) {
  const int n = (g.Vh + 127) / 128;
  clover_lambda_kernel<<<dim3(n, 2), 128, 0, st>>>(g, e0, e1, z0, z1, lam);
  clover_force_kernel<<<dim3(n, 2, 4), 128, 0, st>>>(g, d18, lam, w, F);
  return cudaGetLastError();
}

}  // namespace iro
