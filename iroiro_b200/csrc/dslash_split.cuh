// The hopping stencil with a site's eight neighbour terms formed by eight warps:
// a group of 32 elements (sites times right-hand sides) per pass of a
// 256-thread block, warp d loading, projecting and multiplying neighbour d, the
// sums over the directions and the epilogue (as hop_kernel's) by spin in warps
// 0-3, the clover product by chirality in warps 4-5.  For lattices too small to
// fill the device with a thread per site, where a launch is the latency of
// that thread's walk over its neighbours.
#pragma once

#include "dslash.cuh"

namespace iro {
namespace split {

constexpr int kThreads = 256;

// ---- loads at the L2 level: other blocks' writes of the same launch must be seen ------
__device__ __forceinline__ void load_co(const SpinorPtr& s, int i, Cx<double> v[12]) {
  const double2* p = chunk0<12>(static_cast<const double2*>(s.data), i);
#pragma unroll
  for (int k = 0; k < 12; ++k) {
    const double2 d = __ldcg(p + 32 * k);
    v[k] = {d.x, d.y};
  }
}
__device__ __forceinline__ void load_co(const SpinorPtr& s, int i, Cx<float> v[12]) {
  const float4* p = chunk0<6>(static_cast<const float4*>(s.data), i);
#pragma unroll
  for (int k = 0; k < 6; ++k) {
    const float4 d = __ldcg(p + 32 * k);
    v[2 * k] = {d.x, d.y};
    v[2 * k + 1] = {d.z, d.w};
  }
}
__device__ __forceinline__ float load_co_w(const SpinorPtr& s, int i, uint32_t f[12]) {
  const uint4* p = chunk0<3>(static_cast<const uint4*>(s.data), i);
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const uint4 d = __ldcg(p + 32 * k);
    f[4 * k] = d.x;
    f[4 * k + 1] = d.y;
    f[4 * k + 2] = d.z;
    f[4 * k + 3] = d.w;
  }
  return __ldcg(s.norm + uint32_t(i));
}

// the three colours of spin `sp` of element i
template <int SP>
struct SpinIO;
template <>
struct SpinIO<PREC_DOUBLE> {
  __device__ __forceinline__ static double2* at(const SpinorPtr& s, int i, int k) {
    return chunk0<12>(static_cast<double2*>(s.data), i) + 32 * k;
  }
  __device__ __forceinline__ static void load(const SpinorPtr& s, int i, int sp, Cx<double> v[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double2 d = __ldcg(at(s, i, 3 * sp + c));
      v[c] = {d.x, d.y};
    }
  }
  __device__ __forceinline__ static void store(const SpinorPtr& s, int i, int sp, const Cx<double> v[3], float) {
#pragma unroll
    for (int c = 0; c < 3; ++c) *at(s, i, 3 * sp + c) = make_double2(v[c].re, v[c].im);
  }
};
template <>
struct SpinIO<PREC_SINGLE> {
  __device__ __forceinline__ static float2* at(const SpinorPtr& s, int i, int k) {
    return reinterpret_cast<float2*>(chunk0<6>(static_cast<float4*>(s.data), i) + 32 * (k >> 1)) + (k & 1);
  }
  __device__ __forceinline__ static void load(const SpinorPtr& s, int i, int sp, Cx<float> v[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float2 d = __ldcg(at(s, i, 3 * sp + c));
      v[c] = {d.x, d.y};
    }
  }
  __device__ __forceinline__ static void store(const SpinorPtr& s, int i, int sp, const Cx<float> v[3], float) {
#pragma unroll
    for (int c = 0; c < 3; ++c) *at(s, i, 3 * sp + c) = make_float2(v[c].re, v[c].im);
  }
};
template <>
struct SpinIO<PREC_HALF> {
  __device__ __forceinline__ static uint32_t* at(const SpinorPtr& s, int i, int k) {
    return reinterpret_cast<uint32_t*>(chunk0<3>(static_cast<uint4*>(s.data), i) + 32 * (k >> 2)) + (k & 3);
  }
  __device__ __forceinline__ static void load(const SpinorPtr& s, int i, int sp, Cx<float> v[3]) {
    const float n = __ldcg(s.norm + i);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const float2 d = unpack_h2(__ldcg(at(s, i, 3 * sp + c)));
      v[c] = {n * d.x, n * d.y};
    }
  }
  // n: the largest component of the whole element (SpinorIO<PREC_HALF>::store_scaled)
  __device__ __forceinline__ static void store(const SpinorPtr& s, int i, int sp, const Cx<float> v[3], float n) {
    if (!(n >= 1e-37f)) n = 0.f;
    const float inv = n > 0.f ? 1.0f / n : 0.f;
#pragma unroll
    for (int c = 0; c < 3; ++c) *at(s, i, 3 * sp + c) = pack_h2(v[c].re * inv, v[c].im * inv);
    if (sp == 0) s.norm[i] = n;
  }
};

// one 6x6 block of a site
__device__ __forceinline__ void load_block(const CloverPtr& c, int i, int b, CloverBlock<double>& B) {
  const double2* q = chunk0<36>(static_cast<const double2*>(c.data), i) + 32 * 18 * b;
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double2 d = __ldg(q + 32 * k);
    B.d[2 * k] = d.x;
    B.d[2 * k + 1] = d.y;
  }
#pragma unroll
  for (int k = 0; k < 15; ++k) {
    const double2 d = __ldg(q + 32 * (3 + k));
    B.o[k] = {d.x, d.y};
  }
}
__device__ __forceinline__ void unpack_block(const float* v, CloverBlock<float>& B) {
#pragma unroll
  for (int k = 0; k < 6; ++k) B.d[k] = v[k];
#pragma unroll
  for (int k = 0; k < 15; ++k) B.o[k] = {v[6 + 2 * k], v[7 + 2 * k]};
}
template <int SP>
__device__ __forceinline__ void load_block(const CloverPtr& c, int i, int b, CloverBlock<float>& B) {
  if constexpr (SP == PREC_SINGLE) {
    const float4* q = chunk0<18>(static_cast<const float4*>(c.data), i) + 32 * 9 * b;
    float v[36];
#pragma unroll
    for (int k = 0; k < 9; ++k) {
      const float4 d = __ldg(q + 32 * k);
      v[4 * k] = d.x;
      v[4 * k + 1] = d.y;
      v[4 * k + 2] = d.z;
      v[4 * k + 3] = d.w;
    }
    unpack_block(v, B);
  } else {
    // block b owns values 36 b .. of the 72: chunks 4b .. 4b + 4, the middle one shared
    const uint4* q = chunk0<9>(static_cast<const uint4*>(c.data), i) + 32 * 4 * b;
    float v[40];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const uint4 d = __ldg(q + 32 * k);
      const float2 x = unpack_h2(d.x), y = unpack_h2(d.y), z = unpack_h2(d.z), w = unpack_h2(d.w);
      v[8 * k] = x.x; v[8 * k + 1] = x.y; v[8 * k + 2] = y.x; v[8 * k + 3] = y.y;
      v[8 * k + 4] = z.x; v[8 * k + 5] = z.y; v[8 * k + 6] = w.x; v[8 * k + 7] = w.y;
    }
    if (b == 0) {
      unpack_block(v, B);
    } else {
      unpack_block(v + 4, B);
    }
  }
}

// ---- one neighbour's term: the link times the projected half spinor ------------------
// The direction is data: which spins and phases the projector (1 - S gamma_mu)
// takes (project / reconstruct of dslash.cuh) come from small tables in shared
// memory and the link is transposed by its addresses, so that the eight warps
// run the same few instructions.  With a copy of the code per direction (as
// hop_kernel) a phase was bound by instruction fetch: 6600 cycles for one group
// of sites, of which the loads take ~1000.
template <typename R>
struct DirTab {
  R a, re0, im0, re1, im1;  // h0 = a f0 + (re0 + i im0) b0, h1 = a f1 + (re1 + i im1) b1
  int swap;                 // (b0, b1) = (f3, f2) instead of (f2, f3)
};
template <typename R>
struct SpinTab {
  R re, im;  // the output spin's weight on half spinor `src`
  int src;
};

template <typename R>
__device__ __forceinline__ void fill_tables(DirTab<R> dir[2][8], SpinTab<R> spin[2][8][4]) {
  const int t = threadIdx.x;
  if (t >= 16) return;
  const int dag = t >> 3, d = t & 7, mu = d >> 1;
  const R S = ((d & 1) == 0) != (dag != 0) ? R(1) : R(-1);
  const R z = R(0), o = R(1);
  DirTab<R> D{o, z, z, z, z, mu < 2};
  SpinTab<R> T[4] = {{o, z, 0}, {o, z, 1}, {z, z, 0}, {z, z, 0}};
  if (mu == 0) {
    D.im0 = D.im1 = S;
    T[2] = {z, -S, 1};
    T[3] = {z, -S, 0};
  } else if (mu == 1) {
    D.re0 = S;
    D.re1 = -S;
    T[2] = {-S, z, 1};
    T[3] = {S, z, 0};
  } else if (mu == 2) {
    D.im0 = S;
    D.im1 = -S;
    T[2] = {z, -S, 0};
    T[3] = {z, S, 1};
  } else {
    D.a = S > z ? z : R(2);
    D.re0 = D.re1 = S > z ? R(2) : z;
    T[0].re = T[1].re = S > z ? z : o;
    T[2] = {S > z ? o : z, z, 0};
    T[3] = {S > z ? o : z, z, 1};
  }
  dir[dag][d] = D;
  for (int k = 0; k < 4; ++k) spin[dag][d][k] = T[k];
}

// V = U (forward) or U^dag (backward) of link (par, mu, site)
template <int SP, typename R>
__device__ __forceinline__ void load_link(const GaugePtr& g, int par, int mu, int site, bool fwd, Su3<R>& V) {
  if constexpr (SP == PREC_DOUBLE) {  // three stored rows: chunk 3 a + b
    const double2* q = link_chunk0<9>(static_cast<const double2*>(g.a), g.Vh, par, mu, site);
    const double s = fwd ? 1.0 : -1.0;
    const int ra = fwd ? 96 : 32, rb = fwd ? 32 : 96;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const double2 v = __ldg(q + ra * a + rb * b);
        V.e[a][b] = {v.x, s * v.y};
      }
  } else {
    Su3<R> U;
    GaugeIO<SP, 12>::load(g, par, mu, site, U);
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) V.e[a][b] = fwd ? U.e[a][b] : conjx(U.e[b][a]);
  }
}

// The half spinor of (1 - S gamma_mu) f
template <typename R>
__device__ __forceinline__ void project(const DirTab<R>& T, const Cx<R> f[12], Cx<R> h[6]) {
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const Cx<R> b0 = T.swap ? f[9 + c] : f[6 + c], b1 = T.swap ? f[6 + c] : f[9 + c];
    h[c] = {T.a * f[c].re + T.re0 * b0.re - T.im0 * b0.im, T.a * f[c].im + T.re0 * b0.im + T.im0 * b0.re};
    h[3 + c] = {T.a * f[3 + c].re + T.re1 * b1.re - T.im1 * b1.im, T.a * f[3 + c].im + T.re1 * b1.im + T.im1 * b1.re};
  }
}

template <int SP>
__device__ __forceinline__ void dir_term(const GaugePtr& gauge, const SpinorPtr& in, int par, int mu, int site,
                                         bool fwd, int e, uint32_t vh,
                                         const DirTab<typename SpinorIO<SP>::Real>& T,
                                         Cx<typename SpinorIO<SP>::Real> g[6]) {
  using R = typename SpinorIO<SP>::Real;
  if constexpr (SP == PREC_HALF) {
    // FP16 words, projected and multiplied in FP32; the element's norm is left
    // to the result.  (Projecting in packed FP16, as dslash_mix.cuh does, rounds
    // the half spinors once more and saves no time: a clover solve on 8^3x16
    // takes 2.8 ms either way.)
    uint32_t u[9], f[12];
    load_link_w(gauge, uint32_t(par * 4 + mu) * vh + uint32_t(site), u);
    const float n = load_co_w(in, e, f);
    Su3<float> V;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int b = 0; b < 3; ++b) {
        const float2 v = unpack_h2(fwd ? u[3 * a + b] : u[3 * b + a]);
        V.e[a][b] = {v.x, fwd ? v.y : -v.y};
      }
    Cx<float> v[12], h[6];
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const float2 w = unpack_h2(f[k]);
      v[k] = {w.x, w.y};
    }
    project(T, v, h);
    su3_mul(V, h, g);
#pragma unroll
    for (int k = 0; k < 6; ++k) g[k] = n * g[k];
  } else {
    Su3<R> V;
    Cx<R> f[12], h[6];
    load_co(in, e, f);
    load_link<SP>(gauge, par, mu, site, fwd, V);
    project(T, f, h);
    su3_mul(V, h, g);
  }
}

// half-site index of neighbour d (x+, x-, y+, ...) of half-site hs (neighbours())
__device__ __forceinline__ int neighbour(const Geom& g, const Coord& c, int hs, int d) {
  if (d < 2) {
    const int x = d == 0 ? (c.x + 1 == g.L[0] ? 0 : c.x + 1) : (c.x == 0 ? g.L[0] - 1 : c.x - 1);
    return c.row * g.Lxh + (x >> 1);
  }
  const int mu = d >> 1;
  const int v = mu == 1 ? c.y : mu == 2 ? c.z : c.t;
  const int s = mu == 1 ? g.sy : mu == 2 ? g.sz : g.st;
  const int n = mu == 1 ? g.L[1] : mu == 2 ? g.L[2] : g.L[3];
  if ((d & 1) == 0) return v + 1 == n ? hs - (n - 1) * s : hs + s;
  return v == 0 ? hs + (n - 1) * s : hs - s;
}

template <typename R>
struct Shared {
  DirTab<R> dir[2][8];       // by dagger and direction
  SpinTab<R> spin[2][8][4];  // and output spin
  Cx<R> g[8][6][32];         // the eight half-spinor terms of the group's elements
  Cx<R> acc[12][32];         // the hopping sum (clover inverse only)
  Cx<R> cl[2][6][32];        // the two chiralities of a clover product
  float big[4][32];          // largest component per spin (FP16 stores)
};

// One group: lane's element e (site hs of parity p, `act` if it exists), its
// neighbour nb in the warp's direction at right-hand side r:
//   out = scale H in through the epilogue, stored to `out`, or, with `subtract`,
//   out -= alpha (that).
// Returns the warp's spin part of |what is stored|^2 (warps 0-3).  Ends with a
// block barrier.
template <int SP>
__device__ __forceinline__ double group(const GaugePtr& gauge, uint32_t vh,
                                        Shared<typename SpinorIO<SP>::Real>& sm, const SpinorPtr& in,
                                        const SpinorPtr& own, const SpinorPtr& out, const CloverPtr& cl, int epi,
                                        int dag, typename SpinorIO<SP>::Real scale, bool subtract,
                                        typename SpinorIO<SP>::Real alpha, bool act, int p, int hs, int e, int nb,
                                        int nrhs, int r) {
  using R = typename SpinorIO<SP>::Real;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double sum = 0.0;
  // the own-site inputs of the epilogue, requested with the neighbours
  Cx<R> xv[3], rv[3];
  if (warp < 4 && act) {
    if (epi == EPI_XPAY) SpinIO<SP>::load(own, e, warp, xv);
    if (subtract) SpinIO<SP>::load(out, e, warp, rv);
  }
  if (act) {
    const bool fwd = (warp & 1) == 0;
    Cx<R> g[6];
    dir_term<SP>(gauge, in, fwd ? p : 1 - p, warp >> 1, fwd ? hs : nb, fwd, nb * nrhs + r, vh, sm.dir[dag][warp], g);
#pragma unroll
    for (int j = 0; j < 6; ++j) sm.g[warp][j][lane] = g[j];
  }
  __syncthreads();
  Cx<R> a[3];
  if (warp < 4 && act) {
    // forward and backward terms in two chains
    Cx<R> b[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = b[c] = {R(0), R(0)};
#pragma unroll
    for (int d = 0; d < 8; ++d) {
      const SpinTab<R> T = sm.spin[dag][d][warp];
      Cx<R>* x = d & 1 ? b : a;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const Cx<R> v = sm.g[d][3 * T.src + c][lane];
        x[c] = {x[c].re + (T.re * v.re - T.im * v.im), x[c].im + (T.re * v.im + T.im * v.re)};
      }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = a[c] + b[c];
#pragma unroll
    for (int c = 0; c < 3; ++c) a[c] = scale * a[c];
    if (epi == EPI_SCALE_CLOV) {
#pragma unroll
      for (int c = 0; c < 3; ++c) sm.acc[3 * warp + c][lane] = a[c];
    }
  }
  if (epi == EPI_SCALE_CLOV || epi == EPI_XPAY_CLOV) {
    if (epi == EPI_SCALE_CLOV) __syncthreads();
    if ((warp == 4 || warp == 5) && act) {
      // chirality b of the clover product (clover_apply)
      const int b = warp - 4;
      const R sg = b == 0 ? R(1) : R(-1);
      Cx<R> v[12], x[6], z[6];
      if (epi == EPI_SCALE_CLOV) {
#pragma unroll
        for (int k = 0; k < 12; ++k) v[k] = sm.acc[k][lane];
      } else if constexpr (SP == PREC_HALF) {
        uint32_t w[12];
        const float n = load_co_w(own, e, w);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          const float2 f = unpack_h2(w[k]);
          v[k] = {n * f.x, n * f.y};
        }
      } else {
        load_co(own, e, v);
      }
#pragma unroll
      for (int k = 0; k < 6; ++k) x[k] = v[k] + sg * v[6 + k];
      CloverBlock<R> B;
      if constexpr (SP == PREC_DOUBLE) load_block(cl, hs, b, B);
      else load_block<SP>(cl, hs, b, B);
      herm6(B, x, z);
#pragma unroll
      for (int k = 0; k < 6; ++k) sm.cl[b][k][lane] = z[k];
    }
    __syncthreads();
  }
  float big = 0.f;
  if (warp < 4 && act) {
    if (epi == EPI_SCALE_CLOV || epi == EPI_XPAY_CLOV) {
      const int k0 = 3 * (warp & 1);
      const R sg = warp < 2 ? R(1) : R(-1);
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const Cx<R> v = R(0.5) * (sm.cl[0][k0 + c][lane] + sg * sm.cl[1][k0 + c][lane]);
        a[c] = epi == EPI_SCALE_CLOV ? v : v + a[c];
      }
    } else if (epi == EPI_XPAY) {
#pragma unroll
      for (int c = 0; c < 3; ++c) a[c] = xv[c] + a[c];
    }
    if (subtract) {
#pragma unroll
      for (int c = 0; c < 3; ++c) a[c] = rv[c] - alpha * a[c];
    }
    R s2 = R(0);
#pragma unroll
    for (int c = 0; c < 3; ++c) s2 += a[c].re * a[c].re + a[c].im * a[c].im;
    sum += double(s2);
    if constexpr (SP == PREC_HALF) {
#pragma unroll
      for (int c = 0; c < 3; ++c) big = fmaxf(big, fmaxf(fabsf(a[c].re), fabsf(a[c].im)));
      sm.big[warp][lane] = big;
    }
  }
  if constexpr (SP == PREC_HALF) {
    __syncthreads();
    if (warp < 4 && act)
      big = fmaxf(fmaxf(sm.big[0][lane], sm.big[1][lane]), fmaxf(sm.big[2][lane], sm.big[3][lane]));
  }
  if (warp < 4 && act) SpinIO<SP>::store(out, e, warp, a, big);
  __syncthreads();  // the shared terms are read before the next group's are written
  return sum;
}

}  // namespace split
}  // namespace iro
