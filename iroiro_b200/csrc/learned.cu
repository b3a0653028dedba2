// Gauge-equivariant learned preconditioner: parallel-transport convolution
// (PTC) layers and their gradients.
//
// A layer maps C_in colour-vector channels to C_out channels on every site of
// the full lattice:
//     out_o(x) = sum_{d=0..8} sum_i W_d[o][i] (T_d in_i)(x)
// with T_0 the identity and, for d = 1 + 2*mu + s,
//     T_{+mu} f(x) = U_mu(x) f(x+mu),   T_{-mu} f(x) = U_mu(x-mu)^dag f(x-mu),
// so the layer commutes with gauge transformations (the weights act on the
// channel index only, the links on colour).  A Wilson spinor is 4 channels
// (its spins).  The reference has no learned part; this follows the
// parallel-transport convolutions of Lehner & Wettig, "Gauge-equivariant
// neural networks as preconditioners in lattice QCD", PRD 108 (2023).
//
// Forward kernel: every warp works alone on tiles of 32 sites = 96 rows (site,
// colour).  Per displacement it transports the input channels on the CUDA
// cores (lane = site), stages them as BF16 rows in shared memory and multiplies
// them with the displacement's weights on the tensor cores (mma.sync, BF16 x
// BF16 -> FP32, the accumulators in registers over all nine displacements),
// then stores the output channels in FP32.  The contraction is small (K = 8 or
// 16 per displacement and a few output columns): what bounds a layer is the
// latency of the gathers.  A block-wide version, nine warps building one
// operand for tcgen05.mma in tensor memory, spent its time at the block's
// barriers: (4,4,4,4) at 32^3x64 1.30 ms, 0.95 ms now; (4,16,16,16,4) at
// 24^3x48 1.74 and 1.31 ms.
//
// Backward: the gradient of the input is a layer of the same kind on dY, with
// adjoint weights and the displacements reversed (T_{+mu}^dag = T_{-mu}), so it
// runs in the forward kernels; dB = A^T dY is summed in FP32 over a tile and in
// FP64 over the tiles, with a deterministic reduction over the CTAs.
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "dslash_pair.cuh"
#include "internal.h"
#include "iroiro_b200.h"

namespace iro {

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// K and N of the packed real weights B[n][k]: k = (2d + re/im) CIN + i, n = 2o +
// re/im, padded to multiples of 16
template <int CIN, int COUT>
struct Ptc {
  static constexpr int KF = 18 * CIN;
  static constexpr int KP = (KF + 15) / 16 * 16;
};

// Feature element (site s, channel o, colour a) of a V-site field.  Channels
// are stored in pairs, structure-of-arrays over sites in 16-byte units: pair
// q = o/2 and colour a occupy the float4 row (3q + a)*V + s holding
// (re o=2q, re o=2q+1, im o=2q, im o=2q+1).  A warp reading one row for 32
// consecutive (or uniformly shifted) sites is coalesced, and a row is
// directly the packed FP32x2 operand pair of the two channels.
__host__ __device__ __forceinline__ size_t fidx(int s, int o, int a, int V) {
  return (size_t((o >> 1) * 3 + a) * V + s) * 4 + (o & 1);
}
__device__ __forceinline__ float2 feat_get(const float2* f, int s, int o, int a, int V) {
  const float* p = reinterpret_cast<const float*>(f) + fidx(s, o, a, V);
  return make_float2(p[0], p[2]);
}
__device__ __forceinline__ void feat_set(float2* f, int s, int o, int a, int V, float2 v) {
  float* p = reinterpret_cast<float*>(f) + fidx(s, o, a, V);
  p[0] = v.x;
  p[2] = v.y;
}

struct PtcGeo {
  Geom g;
  GaugePtr gauge;  // FP32 two-row links
  int V;
  const int* skip;  // forward only: when set and nonzero the launch does nothing
};

// ---- forward ----------------------------------------------------------------------
// The CIN channel vectors of site s transported along displacement d, as
// BF16 words: wre/wim[colour][q] hold the real/imaginary parts of channels
// 2q, 2q+1.  Channels are handled in pairs in the packed FP32x2 arithmetic
// (su3_row).
template <int CIN>
__device__ __forceinline__ void transport_words(const PtcGeo& G, const float2* __restrict__ in, int s,
                                                int d, uint32_t wre[3][CIN / 2],
                                                uint32_t wim[3][CIN / 2]) {
  constexpr int NW = CIN / 2;
  const int Vh = G.g.Vh;
  const int p = s >= Vh ? 1 : 0;
  const int hs = s - p * Vh;
  int src = s;
  Su3<float> U;
  bool fwd = true;
  int mu = 0, n = hs;
  if (d > 0) {
    const Coord c = coord_of(G.g, hs, p);
    int nb[8];
    neighbours(G.g, c, hs, nb);
    mu = (d - 1) >> 1;
    fwd = ((d - 1) & 1) == 0;
    n = nb[d - 1];
    src = (1 - p) * Vh + n;
  }
  // channels 2q, 2q+1 of the source site, one float4 row per colour (see fidx)
  const float4* f4 = reinterpret_cast<const float4*>(in) + src;
  const size_t V = size_t(G.V);
  // all of the job's feature rows requested at once (into L1), so that the
  // loads below, which the register budget spreads over the channel
  // pairs, find them there instead of each pair waiting on memory
#pragma unroll
  for (int q = 0; q < 3 * NW; ++q) asm volatile("prefetch.global.L1 [%0];" ::"l"(f4 + q * V));
  if (d > 0) {
    if (fwd)
      GaugeIO<PREC_SINGLE, 12>::load(G.gauge, p, mu, hs, U);
    else
      GaugeIO<PREC_SINGLE, 12>::load(G.gauge, 1 - p, mu, n, U);
  }
#pragma unroll
  for (int q = 0; q < NW; ++q) {
    const float4 a = __ldg(f4 + (3 * q) * V), b = __ldg(f4 + (3 * q + 1) * V),
                 e = __ldg(f4 + (3 * q + 2) * V);
    const Cp h0 = {make_float2(a.x, a.y), make_float2(a.z, a.w)};
    const Cp h1 = {make_float2(b.x, b.y), make_float2(b.z, b.w)};
    const Cp h2 = {make_float2(e.x, e.y), make_float2(e.z, e.w)};
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      Cp w;
      if (d == 0)
        w = r == 0 ? h0 : (r == 1 ? h1 : h2);
      else if (fwd)
        w = su3_row<false>(U, r, h0, h1, h2);
      else
        w = su3_row<true>(U, r, h0, h1, h2);
      const __nv_bfloat162 br = __floats2bfloat162_rn(w.re.x, w.re.y);
      const __nv_bfloat162 bi = __floats2bfloat162_rn(w.im.x, w.im.y);
      wre[r][q] = *reinterpret_cast<const uint32_t*>(&br);
      wim[r][q] = *reinterpret_cast<const uint32_t*>(&bi);
    }
  }
}

constexpr int kFwdSites = 32;

// First site of forward tile `tile`: even and odd tiles alternate (tile 2k is
// even-parity half-sites [32k, 32k + 32), tile 2k + 1 the same odd ones), so
// that a feature or link read as a neighbour by one parity's tiles is read
// again as the centre of the other parity's tiles shortly after, from L2.
// Tiling the even sites before the odd ones read each of them from DRAM twice
// (8->8 layer at 24^3x48: 512 MB of DRAM reads per launch, 261 MB now, the
// input features and links once).
// (The volume is a multiple of 64, so each parity is a whole number of tiles.)
__device__ __forceinline__ int fwd_tile_site0(const PtcGeo& G, int tile) {
  return (tile & 1) * G.g.Vh + (tile >> 1) * kFwdSites;
}
constexpr int kDbThreads = 288;

// ---- backward: dB[n][k] = sum over rows (site, colour) of dY[row][n] A[row][k] ------
// c (16x8, FP32) += a (16x16) b (16x8), BF16
__device__ __forceinline__ void mma_16816(float c[4], const uint32_t a[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Weight gradient of a layer.  Persistent CTAs of 9 warps loop over tiles of
// 32 sites.  Warp d transports the tile's input channels along displacement d
// (as the forward kernel, rounded to BF16) and multiplies its own 2*CIN columns
// of A with the tile's FP32 dY: per colour the 32 sites are the contraction
// index, and lane (ng, kg) holds a TN x TK block of the sum in registers, its
// operands read from shared memory.
//
// The sum of a tile (96 rows) is FP32 with FMAs; tiles are added in FP64, in
// the CTA's own block of `partial`, in the order of the tiles, and the CTAs in
// block order.  The tensor cores take the same products faster (a 16->16 layer
// at 16^3x32 147 us, 277 us here; a training step of (4,16,16,16,4) 1.19 and
// 1.51 ms), but truncate their FP32 sums: the error was one-sided and grew with
// the volume, on unit links against a 64-bit sum of the same operands 2.6e-7 at
// 8^3x16, 3.4e-6 at 16^3x32, 1.7e-5 at 24^3x48, where it is 3.3e-8 here, the
// rounding of the result.
//
// Bound by the operand loads from shared memory (L1 busy 78 %) and the FMAs.
// Blocks of 4 x 8 with BF16 rows of A, half the loads, took the same time.
template <int CIN, int COUT>
struct PtcDb {
  static constexpr int NF = 2 * COUT;
  static constexpr int CH = CIN < 8 ? CIN : 8;    // channels transported at a time (registers)
  static constexpr int NH = CIN / CH;
  static constexpr int KC = 2 * CH;               // columns staged at a time: re, then im
  static constexpr int TN = NF * KC >= 128 ? 4 : 2;
  static constexpr int TK = NF * KC / (32 * TN);
  static constexpr int NG = NF / TN;              // lane = kg * NG + ng
  static constexpr int NACC = NH * TN * TK;       // entries of a lane over all columns
  static constexpr int YS = NF * 4 + 16;          // bytes of a dY row (padded: conflict-free)
  static constexpr int AS = KC * 4 + 16;          // bytes of an A row (as above)
  static constexpr int Y_BYTES = 96 * YS;
  static constexpr int A_BYTES = 32 * AS;         // one colour of one warp
  static constexpr int SMEM = 2 * Y_BYTES + 9 * A_BYTES;
};

// N consecutive floats of shared memory
template <int N>
__device__ __forceinline__ void lds(const unsigned char* p, float v[N]) {
  if constexpr (N == 4) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x;
    v[1] = x.y;
    v[2] = x.z;
    v[3] = x.w;
  } else if constexpr (N == 2) {
    const float2 x = *reinterpret_cast<const float2*>(p);
    v[0] = x.x;
    v[1] = x.y;
  } else {
    v[0] = *reinterpret_cast<const float*>(p);
  }
}
__device__ __forceinline__ float2 bf16_pair(uint32_t w) {
  return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}

template <int CIN, int COUT>
__global__ void __launch_bounds__(kDbThreads, 2) ptc_db_kernel(PtcGeo G, const float2* __restrict__ in,
                                                             const float2* __restrict__ dy,
                                                             double* __restrict__ partial, int ntiles) {
  using S = PtcDb<CIN, COUT>;
  constexpr int NW = S::CH / 2;
  extern __shared__ __align__(1024) unsigned char smem[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ng = lane % S::NG, kg = lane / S::NG;
  unsigned char* As = smem + 2 * S::Y_BYTES + warp * S::A_BYTES;
  double* sums = partial + (size_t(blockIdx.x) * 9 + warp) * S::NACC * 32 + lane;
  for (int tile = blockIdx.x, it = 0; tile < ntiles; tile += gridDim.x, ++it) {
    const int site0 = fwd_tile_site0(G, tile);
    unsigned char* Y = smem + (it & 1) * S::Y_BYTES;
    // dY of the tile: float4 row (3q + colour) of 32 sites -> columns 4q .. 4q+3
    // (re 2q, re 2q+1, im 2q, im 2q+1) of rows 32 colour + site
    for (int j = threadIdx.x; j < 32 * 3 * (COUT / 2); j += kDbThreads) {
      const int sl = j & 31, qa = j >> 5;
      const int q = qa / 3, a = qa - 3 * q;
      *reinterpret_cast<float4*>(Y + (32 * a + sl) * S::YS + 16 * q) =
          __ldg(reinterpret_cast<const float4*>(dy) + size_t(qa) * G.V + site0 + sl);
    }
#pragma unroll 1
    for (int h = 0; h < S::NH; ++h) {
      uint32_t wre[3][NW], wim[3][NW];
      transport_words<S::CH>(G, in + size_t(24 * h) * G.V, site0 + lane, warp, wre, wim);
      // one barrier a tile: the other dY buffer is written next, and this one
      // again only after every warp has passed the next tile's barrier
      if (h == 0) __syncthreads();
      float acc[S::TN][S::TK];
#pragma unroll
      for (int n = 0; n < S::TN; ++n)
#pragma unroll
        for (int k = 0; k < S::TK; ++k) acc[n][k] = 0.f;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        __syncwarp();
        unsigned char* row = As + lane * S::AS;
#pragma unroll
        for (int q = 0; q < NW; q += 2) {
          const float2 r0 = bf16_pair(wre[a][q]), r1 = bf16_pair(wre[a][q + 1]);
          const float2 i0 = bf16_pair(wim[a][q]), i1 = bf16_pair(wim[a][q + 1]);
          *reinterpret_cast<float4*>(row + 8 * q) = make_float4(r0.x, r0.y, r1.x, r1.y);
          *reinterpret_cast<float4*>(row + 4 * S::CH + 8 * q) = make_float4(i0.x, i0.y, i1.x, i1.y);
        }
        __syncwarp();
        const unsigned char* yp = Y + 32 * a * S::YS + 4 * S::TN * ng;
        const unsigned char* ap = As + 4 * S::TK * kg;
#pragma unroll 8
        for (int r = 0; r < 32; ++r) {
          float yv[S::TN], av[S::TK];
          lds<S::TN>(yp + r * S::YS, yv);
          lds<S::TK>(ap + r * S::AS, av);
#pragma unroll
          for (int n = 0; n < S::TN; ++n)
#pragma unroll
            for (int k = 0; k < S::TK; ++k) acc[n][k] += yv[n] * av[k];
        }
      }
      double* p = sums + size_t(h) * S::TN * S::TK * 32;
#pragma unroll
      for (int n = 0; n < S::TN; ++n)
#pragma unroll
        for (int k = 0; k < S::TK; ++k) {
          double* e = p + (n * S::TK + k) * 32;
          *e = it == 0 ? double(acc[n][k]) : *e + double(acc[n][k]);
        }
    }
  }
}

// Deterministic sum over the CTAs' blocks of sums: 8 threads take every 8th
// block of one entry, and their sums are added in order.  An entry is (warp,
// column block h, n, k of the lane's block, lane) of ptc_db_kernel; its place in
// dB[n][k]: column np = 4q + j of dY is output n = 2o + re/im with o = 2q +
// (j & 1), re/im = j >> 1; A's column is the real or imaginary part of a channel.
constexpr int kSumSlices = 8;
template <int CIN, int COUT>
__global__ void __launch_bounds__(32 * kSumSlices) sum_partials_kernel(const double* __restrict__ partial,
                                                                       int nparts, float* out) {
  using S = PtcDb<CIN, COUT>;
  constexpr int n = 9 * S::NACC * 32;  // a multiple of 32
  __shared__ double sm[kSumSlices][32];
  const int lane = threadIdx.x, q = blockIdx.x * 32 + lane, sl = threadIdx.y;
  double acc = 0.0;
#pragma unroll 8
  for (int t = sl; t < nparts; t += kSumSlices) acc += __ldg(partial + size_t(t) * n + q);
  sm[sl][lane] = acc;
  __syncthreads();
  if (sl != 0) return;
#pragma unroll
  for (int k = 1; k < kSumSlices; ++k) acc += sm[k][lane];
  const int e = blockIdx.x % S::NACC, d = blockIdx.x / S::NACC;
  const int h = e / (S::TN * S::TK), tn = e / S::TK % S::TN, tk = e % S::TK;
  const int np = lane % S::NG * S::TN + tn, col = lane / S::NG * S::TK + tk;
  const int o = 2 * (np >> 2) + (np & 1), part = (np >> 1) & 1;
  out[size_t(2 * o + part) * 18 * CIN + (2 * d + col / S::CH) * CIN + S::CH * h + col % S::CH] = float(acc);
}

// spinor field (FP32, full lattice) <-> 4-channel features [site][spin][colour]
__global__ void spinor_to_feat_kernel(int Vh, SpinorPtr e, SpinorPtr o, float2* feat, const int* skip) {
  if (skip && *skip) return;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < 2 * Vh; s += gridDim.x * blockDim.x) {
    const int p = s >= Vh ? 1 : 0;
    Cx<float> v[12];
    SpinorIO<PREC_SINGLE>::load(p ? o : e, s - p * Vh, v);
#pragma unroll
    for (int k = 0; k < 12; ++k) feat_set(feat, s, k / 3, k % 3, 2 * Vh, make_float2(v[k].re, v[k].im));
  }
}
template <int PO>
__global__ void feat_to_spinor_kernel(int Vh, const float2* feat, SpinorPtr e, SpinorPtr o, const int* skip) {
  if (skip && *skip) return;
  for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < 2 * Vh; s += gridDim.x * blockDim.x) {
    const int p = s >= Vh ? 1 : 0;
    Cx<float> v[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) {
      const float2 t = feat_get(feat, s, k / 3, k % 3, 2 * Vh);
      v[k] = {t.x, t.y};
    }
    SpinorIO<PO>::store(p ? o : e, s - p * Vh, v);
  }
}

// ---- warp-level layer ----------------------------------------------------------------------
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t r[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
// c (16x8, FP32) += a (16x8) b (8x8), BF16
__device__ __forceinline__ void mma_1688(float c[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(b0));
}

template <int CIN, int COUT>
struct PtcLayer {
  static constexpr int CH = CIN < 8 ? CIN : 8;    // channels transported at a time
  static constexpr int NH = CIN / CH;
  static constexpr int NB = CH == 8 ? 2 : 1;      // weight words per MMA (K = 16 or 8)
  static constexpr int NT = 2 * COUT / 8;         // 8-column output tiles
  static constexpr int AS = CH == 8 ? 48 : 16;    // bytes of a staged row (padded: conflict-free)
  static constexpr int A_BYTES = 96 * AS;         // the three colours of a warp's 32 sites
  static constexpr int WORDS = 9 * NH * NT * NB * 32;
  // the next direction's loads: in registers (few channels), or requested into
  // L1 (more); with 4 -> 16 channels the accumulators leave no registers for it
  static constexpr bool RAW = CIN == 4 && NT <= 2;
  static constexpr bool AHEAD = CIN >= 8;
  static constexpr int THREADS = NT == 1 && CIN < 16 ? 512 : NT == 4 && CIN >= 8 ? 256 : 384;
  static constexpr int SMEM = WORDS * 4 + (THREADS / 32) * A_BYTES;
  // four warps sharing a tile's displacements (a few tiles per SM): the tiles of
  // a CTA, and the bytes of each one's partial sums
  static constexpr int SLOTS = RAW ? 0 : THREADS / 128;
  static constexpr int RED_BYTES = 4 * 6 * NT * 32 * 16;
};

// The feature rows and links of the next direction, requested into L1 while the
// present one is multiplied: the loads of a direction wait ~7 issue slots per
// instruction on L2 otherwise (long scoreboard; 20 warps an SM).
template <int CIN, int KIND>
__device__ __forceinline__ void prefetch_dir(const PtcGeo& G, const float2* __restrict__ in, int p, int hs, int mu,
                                             int nb) {
  const float4* f4 = reinterpret_cast<const float4*>(in) + ((1 - p) * G.g.Vh + nb);
#pragma unroll
  for (int q = 0; q < 3 * CIN / 2; ++q) asm volatile("prefetch.global.L1 [%0];" ::"l"(f4 + size_t(q) * G.V));
  const float4* u = link_chunk0<3>(static_cast<const float4*>(G.gauge.a), G.g.Vh, KIND == 1 ? p : 1 - p, mu,
                                   KIND == 1 ? hs : nb);
#pragma unroll
  for (int k = 0; k < 3; ++k) asm volatile("prefetch.global.L1 [%0];" ::"l"(u + 32 * k));
}

// The loads of one direction (4 input channels), kept in registers while the
// direction before is multiplied
struct RawDir {
  float4 f[6], u[3];
};
template <int KIND>
__device__ __forceinline__ void load_dir4(const PtcGeo& G, const float2* __restrict__ in, int p, int hs, int mu, int nb,
                                          RawDir& r) {
  const float4* f4 = reinterpret_cast<const float4*>(in) + (KIND == 0 ? p * G.g.Vh + hs : (1 - p) * G.g.Vh + nb);
#pragma unroll
  for (int k = 0; k < 6; ++k) r.f[k] = __ldg(f4 + size_t(k) * G.V);
  if (KIND != 0) {
    const float4* u = link_chunk0<3>(static_cast<const float4*>(G.gauge.a), G.g.Vh, KIND == 1 ? p : 1 - p, mu,
                                     KIND == 1 ? hs : nb);
#pragma unroll
    for (int k = 0; k < 3; ++k) r.u[k] = __ldg(u + 32 * k);
  }
}
template <int COUT, int KIND>
__device__ __forceinline__ void mul_dir4(const RawDir& r, int D, const uint32_t* W, unsigned char* As, uint32_t a_addr,
                                         float acc[6][PtcLayer<4, COUT>::NT][4]) {
  using S = PtcLayer<4, COUT>;
  const int lane = threadIdx.x & 31;
  Su3<float> U;
  if (KIND != 0) {
    U.e[0][0] = {r.u[0].x, r.u[0].y};
    U.e[0][1] = {r.u[0].z, r.u[0].w};
    U.e[0][2] = {r.u[1].x, r.u[1].y};
    U.e[1][0] = {r.u[1].z, r.u[1].w};
    U.e[1][1] = {r.u[2].x, r.u[2].y};
    U.e[1][2] = {r.u[2].z, r.u[2].w};
    reconstruct_row2(U);
  }
  uint32_t wre[3][2], wim[3][2];
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float4 a = r.f[3 * q], b = r.f[3 * q + 1], e = r.f[3 * q + 2];
    const Cp h0 = {make_float2(a.x, a.y), make_float2(a.z, a.w)};
    const Cp h1 = {make_float2(b.x, b.y), make_float2(b.z, b.w)};
    const Cp h2 = {make_float2(e.x, e.y), make_float2(e.z, e.w)};
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      Cp w;
      if (KIND == 0) w = c == 0 ? h0 : (c == 1 ? h1 : h2);
      else w = su3_row<KIND == 2>(U, c, h0, h1, h2);
      const __nv_bfloat162 br = __floats2bfloat162_rn(w.re.x, w.re.y);
      const __nv_bfloat162 bi = __floats2bfloat162_rn(w.im.x, w.im.y);
      wre[c][q] = *reinterpret_cast<const uint32_t*>(&br);
      wim[c][q] = *reinterpret_cast<const uint32_t*>(&bi);
    }
  }
  __syncwarp();  // the staged rows of the previous product are read
#pragma unroll
  for (int c = 0; c < 3; ++c)
    *reinterpret_cast<uint4*>(As + (32 * c + lane) * S::AS) = make_uint4(wre[c][0], wre[c][1], wim[c][0], wim[c][1]);
  __syncwarp();
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    uint32_t a[4];
    ldsm4(a_addr + 32 * c * S::AS, a);
#pragma unroll
    for (int n = 0; n < S::NT; ++n) {
      const uint32_t b = W[(D * S::NT + n) * 32 + lane];
      mma_1688(acc[2 * c][n], a[0], a[1], b);
      mma_1688(acc[2 * c + 1][n], a[2], a[3], b);
    }
  }
}

// The channels of displacement D at one site, transported, as BF16 rows of the
// warp's staging tile: row 32 colour + lane holds the real parts of the
// channels, then the imaginary parts.  Then their product with the weights.
// KIND 0: the site itself; 1: forward, 2: backward along mu (a run-time index:
// one copy of the code per kind, and no direction's loads hoisted over
// another's, which spilled)
template <int CIN, int COUT, int KIND>
__device__ __forceinline__ void layer_dir(const PtcGeo& G, const float2* __restrict__ in, int p, int hs, int mu, int nb,
                                          const uint32_t* W, unsigned char* As, uint32_t a_addr,
                                          float acc[6][PtcLayer<CIN, COUT>::NT][4]) {
  using S = PtcLayer<CIN, COUT>;
  const int lane = threadIdx.x & 31;
  const int D = KIND == 0 ? 0 : 2 * mu + KIND;
  const size_t V = size_t(G.V);
  const float4* f4 = reinterpret_cast<const float4*>(in) + (KIND == 0 ? p * G.g.Vh + hs : (1 - p) * G.g.Vh + nb);
  Su3<float> U;
  if (KIND == 1) GaugeIO<PREC_SINGLE, 12>::load(G.gauge, p, mu, hs, U);
  if (KIND == 2) GaugeIO<PREC_SINGLE, 12>::load(G.gauge, 1 - p, mu, nb, U);
#pragma unroll
  for (int h = 0; h < S::NH; ++h) {
    uint32_t wre[3][S::CH / 2], wim[3][S::CH / 2];
#pragma unroll
    for (int q = 0; q < S::CH / 2; ++q) {
      const float4* f = f4 + size_t(3 * (q + 4 * h)) * V;
      const float4 a = __ldg(f), b = __ldg(f + V), e = __ldg(f + 2 * V);
      const Cp h0 = {make_float2(a.x, a.y), make_float2(a.z, a.w)};
      const Cp h1 = {make_float2(b.x, b.y), make_float2(b.z, b.w)};
      const Cp h2 = {make_float2(e.x, e.y), make_float2(e.z, e.w)};
#pragma unroll
      for (int r = 0; r < 3; ++r) {
        Cp w;
        if (KIND == 0) w = r == 0 ? h0 : (r == 1 ? h1 : h2);
        else w = su3_row<KIND == 2>(U, r, h0, h1, h2);
        const __nv_bfloat162 br = __floats2bfloat162_rn(w.re.x, w.re.y);
        const __nv_bfloat162 bi = __floats2bfloat162_rn(w.im.x, w.im.y);
        wre[r][q] = *reinterpret_cast<const uint32_t*>(&br);
        wim[r][q] = *reinterpret_cast<const uint32_t*>(&bi);
      }
    }
    __syncwarp();  // the staged rows of the previous product are read
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      unsigned char* row = As + (32 * r + lane) * S::AS;
      if constexpr (S::CH == 4) {
        *reinterpret_cast<uint4*>(row) = make_uint4(wre[r][0], wre[r][1], wim[r][0], wim[r][1]);
      } else {
        *reinterpret_cast<uint4*>(row) = make_uint4(wre[r][0], wre[r][1], wre[r][2], wre[r][3]);
        *reinterpret_cast<uint4*>(row + 16) = make_uint4(wim[r][0], wim[r][1], wim[r][2], wim[r][3]);
      }
    }
    __syncwarp();
    uint32_t b[S::NT][S::NB];
#pragma unroll
    for (int n = 0; n < S::NT; ++n)
#pragma unroll
      for (int k = 0; k < S::NB; ++k) b[n][k] = W[(((D * S::NH + h) * S::NT + n) * S::NB + k) * 32 + lane];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      if constexpr (S::CH == 4) {
        uint32_t a[4];
        ldsm4(a_addr + 32 * r * S::AS, a);
#pragma unroll
        for (int n = 0; n < S::NT; ++n) {
          mma_1688(acc[2 * r][n], a[0], a[1], b[n][0]);
          mma_1688(acc[2 * r + 1][n], a[2], a[3], b[n][0]);
        }
      } else {
#pragma unroll
        for (int m = 0; m < 2; ++m) {
          uint32_t a[4];
          ldsm4(a_addr + (32 * r + 16 * m) * S::AS, a);
#pragma unroll
          for (int n = 0; n < S::NT; ++n) mma_16816(acc[2 * r + m][n], a, b[n][0], b[n][S::NB - 1]);
        }
      }
    }
  }
}

// PARTS 4: four warps share a tile, one pair of directions each, the first also
// the site itself
template <int CIN, int COUT, int PARTS>
__global__ void __launch_bounds__(PtcLayer<CIN, COUT>::THREADS, 1)
    ptc_layer_kernel(PtcGeo G, const float2* __restrict__ in, float2* __restrict__ out,
                     const __nv_bfloat16* __restrict__ bop, int ntiles, int slots) {
  if (G.skip && *G.skip) return;
  using S = PtcLayer<CIN, COUT>;
  extern __shared__ __align__(1024) unsigned char smem[];
  uint32_t* W = reinterpret_cast<uint32_t*>(smem);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  unsigned char* As = smem + S::WORDS * 4 + warp * S::A_BYTES;
  // the weights in the order of the MMA's B fragments: lane l of word k of
  // (displacement d, channel block h, tile n) holds two consecutive k of
  // output row 8n + l/4
  constexpr int KP = Ptc<CIN, COUT>::KP;
#pragma unroll
  for (int j = 0; j < (S::WORDS + S::THREADS - 1) / S::THREADS; ++j) {
    const int i = threadIdx.x + j * S::THREADS;
    if (i >= S::WORDS) break;
    const int l = i & 31, k = (i >> 5) % S::NB, n = (i >> 5) / S::NB % S::NT;
    const int dh = (i >> 5) / (S::NB * S::NT), d = dh / S::NH, h = dh % S::NH;
    const int part = S::CH == 8 ? k : (l & 3) >> 1;
    const int ch = S::CH == 8 ? 8 * h + 2 * (l & 3) : 2 * (l & 1);
    W[i] = __ldg(reinterpret_cast<const uint32_t*>(bop + size_t(8 * n + (l >> 2)) * KP + (2 * d + part) * CIN + ch));
  }
  __syncthreads();
  const int lj = lane >> 3, lr = lane & 7;
  const uint32_t a_addr = smem_u32(As) + (S::CH == 4 ? uint32_t((8 * lj + lr) * S::AS)
                                                     : uint32_t((8 * (lj & 1) + lr) * S::AS + 16 * (lj >> 1)));
  const int slot = warp / PARTS, part = warp % PARTS;
  if (slot >= slots) return;
  for (int tile = blockIdx.x * slots + slot; tile < ntiles; tile += gridDim.x * slots) {
    const int p = tile & 1, hs = (tile >> 1) * kFwdSites + lane;
    const Coord c = coord_of(G.g, hs, p);
    int nb[8];
    neighbours(G.g, c, hs, nb);
    float acc[6][S::NT][4];
#pragma unroll
    for (int m = 0; m < 6; ++m)
#pragma unroll
      for (int n = 0; n < S::NT; ++n)
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[m][n][k] = 0.f;
    if constexpr (S::RAW) {
      RawDir ra, rb;
      load_dir4<0>(G, in, p, hs, 0, 0, ra);
      load_dir4<1>(G, in, p, hs, 0, nb[0], rb);
      mul_dir4<COUT, 0>(ra, 0, W, As, a_addr, acc);
#pragma unroll 1
      for (int mu = 0; mu < 4; ++mu) {
        load_dir4<2>(G, in, p, hs, mu, mu == 0 ? nb[1] : mu == 1 ? nb[3] : mu == 2 ? nb[5] : nb[7], ra);
        mul_dir4<COUT, 1>(rb, 2 * mu + 1, W, As, a_addr, acc);
        if (mu < 3) load_dir4<1>(G, in, p, hs, mu + 1, mu == 0 ? nb[2] : mu == 1 ? nb[4] : nb[6], rb);
        mul_dir4<COUT, 2>(ra, 2 * mu + 2, W, As, a_addr, acc);
      }
    } else {
      const int m0 = part, m1 = PARTS > 1 ? part + 1 : 4;
      if constexpr (S::AHEAD)
        prefetch_dir<CIN, 1>(G, in, p, hs, m0, m0 == 0 ? nb[0] : m0 == 1 ? nb[2] : m0 == 2 ? nb[4] : nb[6]);
      if (part == 0) layer_dir<CIN, COUT, 0>(G, in, p, hs, 0, 0, W, As, a_addr, acc);
#pragma unroll 1
      for (int mu = m0; mu < m1; ++mu) {
        const int nf = mu == 0 ? nb[0] : mu == 1 ? nb[2] : mu == 2 ? nb[4] : nb[6];
        const int nr = mu == 0 ? nb[1] : mu == 1 ? nb[3] : mu == 2 ? nb[5] : nb[7];
        if constexpr (S::AHEAD) prefetch_dir<CIN, 2>(G, in, p, hs, mu, nr);
        layer_dir<CIN, COUT, 1>(G, in, p, hs, mu, nf, W, As, a_addr, acc);
        if (S::AHEAD && mu + 1 < m1)
          prefetch_dir<CIN, 1>(G, in, p, hs, mu + 1, mu == 0 ? nb[2] : mu == 1 ? nb[4] : nb[6]);
        layer_dir<CIN, COUT, 2>(G, in, p, hs, mu, nr, W, As, a_addr, acc);
      }
      if constexpr (PARTS > 1) {
        // the four warps' sums, each warp adding one column tile in order
        float4* red = reinterpret_cast<float4*>(smem + S::SMEM + slot * S::RED_BYTES);
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int n = 0; n < S::NT; ++n)
            red[((part * 6 + m) * S::NT + n) * 32 + lane] =
                make_float4(acc[m][n][0], acc[m][n][1], acc[m][n][2], acc[m][n][3]);
        asm volatile("bar.sync %0, 128;" ::"r"(1 + slot) : "memory");
#pragma unroll
        for (int n = 0; n < S::NT; ++n)
          if (n == part)
#pragma unroll
            for (int m = 0; m < 6; ++m) {
              float4 v = red[(m * S::NT + n) * 32 + lane];
#pragma unroll
              for (int k = 1; k < 4; ++k) {
                const float4 w = red[((k * 6 + m) * S::NT + n) * 32 + lane];
                v = make_float4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
              }
              acc[m][n][0] = v.x;
              acc[m][n][1] = v.y;
              acc[m][n][2] = v.z;
              acc[m][n][3] = v.w;
            }
        asm volatile("bar.sync %0, 128;" ::"r"(1 + slot) : "memory");  // read before the next tile's
      }
    }
    // Lane (g, t) = (lane / 4, lane % 4) holds channel 4n + t of rows g and
    // g + 8; neighbouring lanes exchange one row each, so that every lane has
    // both channels of a pair for one row and stores them as one float4.
    const int t = lane & 3;
    const bool odd = t & 1;
    float4* o4 = reinterpret_cast<float4*>(out) + (p * G.g.Vh + (tile >> 1) * kFwdSites + (lane >> 2) + (odd ? 8 : 0));
#pragma unroll
    for (int m = 0; m < 6; ++m)
#pragma unroll
      for (int n = 0; n < S::NT; ++n) {
        if (PARTS > 1 && n != part) continue;
        const float* v = acc[m][n];
        const float r0 = __shfl_xor_sync(0xffffffffu, odd ? v[0] : v[2], 1);
        const float r1 = __shfl_xor_sync(0xffffffffu, odd ? v[1] : v[3], 1);
        const int q = 2 * n + (t >> 1);
        o4[size_t(3 * q + m / 2) * G.V + 16 * (m & 1)] =
            odd ? make_float4(r0, v[2], r1, v[3]) : make_float4(v[0], r0, v[1], r1);
      }
  }
}

// ---- host launchers ------------------------------------------------------------------
static int sm_count() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (n < 1) n = 1;
  }
  return n;
}

template <int CIN, int COUT, int PARTS>
static cudaError_t fwd_go(const PtcGeo& G, const float2* in, float2* out, const __nv_bfloat16* bop, int ntiles,
                          int slots, cudaStream_t st) {
  using S = PtcLayer<CIN, COUT>;
  constexpr int SMEM = S::SMEM + (PARTS > 1 ? S::SLOTS * S::RED_BYTES : 0);
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(ptc_layer_kernel<CIN, COUT, PARTS>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int grid = std::min((ntiles + slots - 1) / slots, sm_count());
  ptc_layer_kernel<CIN, COUT, PARTS><<<grid, S::THREADS, SMEM, st>>>(G, in, out, bop, ntiles, slots);
  return cudaGetLastError();
}

// One CTA per SM (its register budget), each warp looping over tiles;
// consecutive tiles in one CTA, which share the lines of their gathers.  A small
// lattice's tiles are spread over all SMs, and while four warps per tile fit,
// those share its displacements (not with 4 channels in and few out, where a
// lone warp is fast enough).  An application in full CTAs / spread / shared too,
// us: (4,4,4,4) 2^12 sites 53 / 41, (4,8,8,4) 2^11 64 / 48 / 38, (4,16,16,16,4)
// 2^12 107 / 82 / 54, 2^13 - / 83 / 59, 2^14 (two layers shared) 116 / 88 / 90.
template <int CIN, int COUT>
static cudaError_t fwd_t(const PtcGeo& G, const float2* in, float2* out, const __nv_bfloat16* bop, cudaStream_t st) {
  using S = PtcLayer<CIN, COUT>;
  const int ntiles = (G.V + kFwdSites - 1) / kFwdSites;
  const int per_sm = (ntiles + sm_count() - 1) / sm_count();
  if constexpr (S::SLOTS > 0)
    if (per_sm <= S::SLOTS) return fwd_go<CIN, COUT, 4>(G, in, out, bop, ntiles, per_sm, st);
  return fwd_go<CIN, COUT, 1>(G, in, out, bop, ntiles, std::min(per_sm, S::THREADS / 32), st);
}

// CTAs of the weight-gradient kernel (its buffer of sums holds as many blocks)
static int db_grid(int V) {
  const int ntiles = (V + kFwdSites - 1) / kFwdSites;
  return std::min(ntiles, 2 * sm_count());
}

template <int CIN, int COUT>
static cudaError_t db_t(const PtcGeo& G, const float2* in, const float2* dy, double* partial, float* db,
                        cudaStream_t st) {
  using S = PtcDb<CIN, COUT>;
  static bool attr = false;
  if (!attr) {
    cudaError_t e = cudaFuncSetAttribute(ptc_db_kernel<CIN, COUT>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM);
    if (e != cudaSuccess) return e;
    attr = true;
  }
  const int grid = db_grid(G.V);
  ptc_db_kernel<CIN, COUT><<<grid, kDbThreads, S::SMEM, st>>>(G, in, dy, partial,
                                                               (G.V + kFwdSites - 1) / kFwdSites);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  sum_partials_kernel<CIN, COUT><<<9 * S::NACC, dim3(32, kSumSlices), 0, st>>>(partial, grid, db);
  return cudaGetLastError();
}

int ptc_shape_ok(int cin, int cout) {
  return (cin == 4 || cin == 8 || cin == 16) && (cout == 4 || cout == 8 || cout == 16);
}

#define IRO_PTC_DISPATCH(CALL)                              \
  switch (cin * 100 + cout) {                               \
    case 404: return CALL(4, 4);                            \
    case 408: return CALL(4, 8);                            \
    case 416: return CALL(4, 16);                           \
    case 804: return CALL(8, 4);                            \
    case 808: return CALL(8, 8);                            \
    case 816: return CALL(8, 16);                           \
    case 1604: return CALL(16, 4);                          \
    case 1608: return CALL(16, 8);                          \
    case 1616: return CALL(16, 16);                         \
  }                                                         \
  return cudaErrorInvalidValue;

cudaError_t launch_ptc_fwd(int cin, int cout, const PtcGeo& G, const float2* in, float2* out,
                           const void* bop, cudaStream_t st) {
#define IRO_F(A, B) fwd_t<A, B>(G, in, out, static_cast<const __nv_bfloat16*>(bop), st)
  IRO_PTC_DISPATCH(IRO_F)
#undef IRO_F
}

cudaError_t launch_ptc_db(int cin, int cout, const PtcGeo& G, const float2* in, const float2* dy,
                          double* partial, float* db, cudaStream_t st) {
#define IRO_B(A, B) db_t<A, B>(G, in, dy, partial, db, st)
  IRO_PTC_DISPATCH(IRO_B)
#undef IRO_B
}

void ptc_dims(int cin, int cout, int* kf, int* kp, int* nf, int* np) {
  *kf = 18 * cin;
  *kp = (*kf + 15) / 16 * 16;
  *nf = 2 * cout;
  *np = *nf < 16 ? 16 : (*nf + 15) / 16 * 16;
}

cudaError_t launch_spinor_to_feat(int Vh, SpinorPtr e, SpinorPtr o, float2* feat, cudaStream_t st,
                                  const int* skip = nullptr) {
  spinor_to_feat_kernel<<<(2 * Vh + 255) / 256, 256, 0, st>>>(Vh, e, o, feat, skip);
  return cudaGetLastError();
}
// to an FP32 (or, prec = PREC_HALF, FP16) spinor field
cudaError_t launch_feat_to_spinor(int Vh, const float2* feat, SpinorPtr e, SpinorPtr o, cudaStream_t st,
                                  const int* skip = nullptr, int prec = PREC_SINGLE) {
  if (prec == PREC_HALF)
    feat_to_spinor_kernel<PREC_HALF><<<(2 * Vh + 255) / 256, 256, 0, st>>>(Vh, feat, e, o, skip);
  else
    feat_to_spinor_kernel<PREC_SINGLE><<<(2 * Vh + 255) / 256, 256, 0, st>>>(Vh, feat, e, o, skip);
  return cudaGetLastError();
}

// ---- loss of a training pair: |y - t|^2 and |t|^2, and dy = 2 (y - t) / |t|^2 ------------
constexpr int kRedBlocks = 296;

__global__ void loss_partials_kernel(int n, const float2* y, const float2* t, double* part) {
  __shared__ double sa[256], sb[256];
  double a = 0.0, b = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float2 yy = y[i], tt = t[i];
    const double dr = double(yy.x) - tt.x, di = double(yy.y) - tt.y;
    a += dr * dr + di * di;
    b += double(tt.x) * tt.x + double(tt.y) * tt.y;
  }
  sa[threadIdx.x] = a;
  sb[threadIdx.x] = b;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      sa[threadIdx.x] += sa[threadIdx.x + h];
      sb[threadIdx.x] += sb[threadIdx.x + h];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    part[2 * blockIdx.x] = sa[0];
    part[2 * blockIdx.x + 1] = sb[0];
  }
}

__global__ void loss_grad_kernel(int n, const float2* y, const float2* t, float scale, float2* dy) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float2 yy = y[i], tt = t[i];
    dy[i] = make_float2(scale * (yy.x - tt.x), scale * (yy.y - tt.y));
  }
}

cudaError_t launch_loss_partials(int n, const float2* y, const float2* t, double* part, cudaStream_t st) {
  loss_partials_kernel<<<kRedBlocks, 256, 0, st>>>(n, y, t, part);
  return cudaGetLastError();
}
cudaError_t launch_loss_grad(int n, const float2* y, const float2* t, float scale, float2* dy,
                             cudaStream_t st) {
  loss_grad_kernel<<<kRedBlocks, 256, 0, st>>>(n, y, t, scale, dy);
  return cudaGetLastError();
}
int loss_blocks() { return kRedBlocks; }

// ---- complex linear algebra for GCR on FP32 fields ---------------------------------------
// <w_q, t> = sum conj(w_q) t for q < m, per-block partials [block][2m]; the
// last listed field is FP32 (GCR's residual), the others and t of type PW
// M fields (a compile-time count: the loads of every field of a site can be
// issued together and only 2M accumulators are live), 128-thread blocks
constexpr int kCdotThreads = 128;
template <int PW, int M>
__global__ void __launch_bounds__(kCdotThreads) cdot_kernel(int64_t n, CFieldList w, SpinorPtr t,
                                                            double* part, const int* skip) {
  if (skip && *skip) return;  // the same value in every thread
  __shared__ double sm[2 * M][kCdotThreads / 32];
  double acc[2 * M];
#pragma unroll
  for (int q = 0; q < 2 * M; ++q) acc[q] = 0.0;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    Cx<float> tv[12];
    SpinorIO<PW>::load(t, i, tv);
#pragma unroll
    for (int q = 0; q < M; ++q) {
      Cx<float> wv[12];
      if (q == M - 1)
        SpinorIO<PREC_SINGLE>::load(w.f[q], i, wv);
      else
        SpinorIO<PW>::load(w.f[q], i, wv);
      double re = 0.0, im = 0.0;
#pragma unroll
      for (int k = 0; k < 12; ++k) {
        re += double(wv[k].re) * tv[k].re + double(wv[k].im) * tv[k].im;
        im += double(wv[k].re) * tv[k].im - double(wv[k].im) * tv[k].re;
      }
      acc[2 * q] += re;
      acc[2 * q + 1] += im;
    }
  }
#pragma unroll
  for (int q = 0; q < 2 * M; ++q) {
    double v = acc[q];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sm[q][threadIdx.x >> 5] = v;
  }
  __syncthreads();
  if (threadIdx.x < 2 * M) {
    double v = 0.0;
#pragma unroll
    for (int wv = 0; wv < kCdotThreads / 32; ++wv) v += sm[threadIdx.x][wv];
    part[size_t(blockIdx.x) * 2 * M + threadIdx.x] = v;
  }
}

// the block partials of cdot_kernel summed in a fixed order: one warp per
// real component (block q), lane l summing blocks l, l + 32, ..., then a
// shuffle tree over the lanes
__global__ void cdot_finish_kernel(int blocks, int m2, const double* part, double* out, const int* skip) {
  if (skip && *skip) return;
  const int q = blockIdx.x, l = threadIdx.x;
  if (q >= m2) return;
  double v = 0.0;
  for (int b = l; b < blocks; b += 32) v += part[size_t(b) * m2 + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (l == 0) out[q] = v;
}

// y += sign sum_q c_q x_q  (complex coefficients from the cycle state; the
// first *count of the m fields when count is given); x of type PX, y FP32
template <int PX>
__global__ void caxpy_dev_kernel(int64_t n, int m, CFieldList x, const GcrState* s, const int* count,
                                 float sign, SpinorPtr y, const int* skip) {
  if (skip && *skip) return;
  __shared__ float cre[kMaxList], cim[kMaxList];
  __shared__ int mm;
  if (threadIdx.x < kMaxList) {
    cre[threadIdx.x] = sign * s->cre[threadIdx.x];
    cim[threadIdx.x] = sign * s->cim[threadIdx.x];
  }
  if (threadIdx.x == 0) mm = count ? min(*count, m) : m;
  __syncthreads();
  const int k = mm;
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    Cx<float> yv[12], xv[12];
    SpinorIO<PREC_SINGLE>::load(y, i, yv);
    for (int q = 0; q < k; ++q) {
      SpinorIO<PX>::load(x.f[q], i, xv);
      const Cx<float> cq = {cre[q], cim[q]};
#pragma unroll
      for (int c = 0; c < 12; ++c) yv[c] = yv[c] + cq * xv[c];
    }
    SpinorIO<PREC_SINGLE>::store(y, i, yv);
  }
}

// iteration j (the w of type PW, r FP32): wj += sum_{q<m} c_q w_q; then, unless the coefficient kernel
// found w_j nearly in the span of the w_q (s->plain[j] = 0: a second pass
// forms |w'_j|^2 and <r, w'_j> first), r -= alpha wj with the updated wj,
// and, given feat, the network's input features of the new r
template <int PW>
__global__ void gcr_update_kernel(int64_t n, int m, CFieldList w, const GcrState* s, int j,
                                  SpinorPtr wj, SpinorPtr r, float2* feat) {
  if (s->skip[j]) return;
  __shared__ float cre[kMaxList], cim[kMaxList];
  if (threadIdx.x < kMaxList) {
    cre[threadIdx.x] = s->cre[threadIdx.x];
    cim[threadIdx.x] = s->cim[threadIdx.x];
  }
  __syncthreads();
  const bool plain = s->plain[j] != 0;
  const Cx<float> a = {s->ure, s->uim};
  for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    Cx<float> yv[12], xv[12];
    SpinorIO<PW>::load(wj, i, yv);
    for (int q = 0; q < m; ++q) {
      SpinorIO<PW>::load(w.f[q], i, xv);
      const Cx<float> cq = {cre[q], cim[q]};
#pragma unroll
      for (int k = 0; k < 12; ++k) yv[k] = yv[k] + cq * xv[k];
    }
    SpinorIO<PW>::store(wj, i, yv);
    if (plain) {
      SpinorIO<PREC_SINGLE>::load(r, i, xv);
#pragma unroll
      for (int k = 0; k < 12; ++k) xv[k] = xv[k] - a * yv[k];
      SpinorIO<PREC_SINGLE>::store(r, i, xv);
      if (feat) {
        // the network's input features of the new r (as spinor_to_feat: site
        // i of the full field, spin pair q and colour c in float4 row 3q + c)
        float4* f4 = reinterpret_cast<float4*>(feat);
#pragma unroll
        for (int q = 0; q < 2; ++q)
#pragma unroll
          for (int c = 0; c < 3; ++c) {
            const Cx<float> lo = xv[6 * q + c], hi = xv[6 * q + 3 + c];
            f4[size_t(3 * q + c) * size_t(n) + size_t(i)] = make_float4(lo.re, hi.re, lo.im, hi.im);
          }
      }
    }
  }
}

__global__ void gcr_init_kernel(GcrState* s, double rr, double target, double d2, int limit) {
  const int t = threadIdx.x;
  if (t < kMaxVec) {
    s->skip[t] = 0;
    s->plain[t] = 1;
  }
  for (int i = t; i < kMaxVec * kMaxVec; i += blockDim.x) s->tre[i] = s->tim[i] = 0.0;
  if (t == 0) {
    s->rr_it = s->rr_start = rr;
    s->target = target;
    s->d2 = d2;
    s->limit = limit;
    s->jdone = 0;
  }
}

// alpha_j, column j of T, the iterated |r|^2 and the restart test, from
// |w'_j|^2 and <r, w'_j> (r is orthogonal to every earlier w'_q, so
// <r, w'_j> = <r, w_j>); the beta_q of the iteration are in s->bre/bim
__device__ void gcr_finish_iteration(GcrState* s, int j, int m, double nwj, double rre, double rim) {
  constexpr int K = kMaxVec;
  s->nw[j] = nwj;
  const double ar = rre / nwj, ai = -rim / nwj;  // alpha = conj(<r, w'_j>) / |w'_j|^2
  s->are[j] = ar;
  s->aim[j] = ai;
  s->ure = float(ar);
  s->uim = float(ai);
  // z'_j = z_j + sum_q beta_q z'_q
  s->tre[j * K + j] = 1.0;
  for (int q = 0; q < j; ++q) {
    const double br = s->bre[q], bi = s->bim[q];
    for (int i = 0; i <= q; ++i) {
      const double tr = s->tre[i * K + q], ti = s->tim[i * K + q];
      s->tre[i * K + j] += br * tr - bi * ti;
      s->tim[i * K + j] += br * ti + bi * tr;
    }
  }
  // r minus its projection on w'_j; only the restart test reads it, the FP64
  // residual decides
  s->rr_it = s->rr_it - (rre * rre + rim * rim) / nwj;
  s->jdone = j + 1;
  if (s->rr_it < s->target || s->rr_it < s->d2 * s->rr_start || s->jdone >= s->limit)
    for (int k = j + 1; k < m; ++k) s->skip[k] = 1;
}

// One thread.  First pass (second = 0): g = <w_q, w_j> (q < j), |w_j|^2,
// <r, w_j> as (re, im) pairs.  The w_q are orthogonal, hence for w'_j = w_j +
// sum_q beta_q w_q with beta_q = -<w_q, w_j>/|w_q|^2, |w'_j|^2 = |w_j|^2 -
// sum_q |<w_q, w_j>|^2/|w_q|^2; when that falls below 1e-4 |w_j|^2 the
// orthogonalised vector is formed first and a second pass (second = 1, g =
// |w'_j|^2, <r, w'_j>) finishes the iteration.
__global__ void gcr_coef_kernel(GcrState* s, const double* g, int j, int m, int second) {
  if (s->skip[j]) return;
  if (!second) {
    double nwj = g[2 * j];
    for (int q = 0; q < j; ++q) {
      const double gr = g[2 * q], gi = g[2 * q + 1], nq = s->nw[q];
      const double br = -gr / nq, bi = -gi / nq;
      s->bre[q] = br;
      s->bim[q] = bi;
      s->cre[q] = float(br);
      s->cim[q] = float(bi);
      nwj -= (gr * gr + gi * gi) / nq;
    }
    if (nwj > 1e-4 * g[2 * j]) {
      gcr_finish_iteration(s, j, m, nwj, g[2 * j + 2], g[2 * j + 3]);
    } else {
      s->plain[j] = 0;
      s->ure = s->uim = 0.f;
    }
  } else {
    if (s->plain[j]) return;
    gcr_finish_iteration(s, j, m, g[0], g[2], g[3]);
    s->cre[0] = s->ure;  // r -= alpha w'_j (caxpy with sign -1)
    s->cim[0] = s->uim;
  }
}

// gamma_i = sum_{j >= i} T[i][j] alpha_j over the cycle's iterations, into
// s->cre/cim (zero beyond them)
__global__ void gcr_gamma_kernel(GcrState* s) {
  const int jd = s->jdone;
  for (int i = threadIdx.x; i < kMaxList; i += blockDim.x) {
    double gr = 0.0, gi = 0.0;
    for (int j = i; j < jd; ++j) {
      const double tr = s->tre[i * kMaxVec + j], ti = s->tim[i * kMaxVec + j];
      gr += tr * s->are[j] - ti * s->aim[j];
      gi += tr * s->aim[j] + ti * s->are[j];
    }
    s->cre[i] = float(gr);
    s->cim[i] = float(gi);
  }
}

template <int PW, int M>
static void cdot_go(int64_t n, const CFieldList& w, SpinorPtr t, double* part, int blocks,
                    const int* skip, cudaStream_t st) {
  cdot_kernel<PW, M><<<blocks, kCdotThreads, 0, st>>>(n, w, t, part, skip);
}
template <int PW>
static cudaError_t cdot_count(int64_t n, int m, const CFieldList& w, SpinorPtr t, double* part,
                              int blocks, const int* skip, cudaStream_t st) {
  static_assert(kMaxList == 18, "one case per field count");
  switch (m) {
#define IRO_CD(M) \
  case M: cdot_go<PW, M>(n, w, t, part, blocks, skip, st); break;
    IRO_CD(1) IRO_CD(2) IRO_CD(3) IRO_CD(4) IRO_CD(5) IRO_CD(6) IRO_CD(7) IRO_CD(8) IRO_CD(9)
    IRO_CD(10) IRO_CD(11) IRO_CD(12) IRO_CD(13) IRO_CD(14) IRO_CD(15) IRO_CD(16) IRO_CD(17)
    IRO_CD(18)
#undef IRO_CD
    default: return cudaErrorInvalidValue;
  }
  return cudaSuccess;
}
cudaError_t launch_cdot(int64_t n, int m, const CFieldList& w, SpinorPtr t, double* part, int blocks,
                        double* out, const int* skip, int pw, cudaStream_t st) {
  const cudaError_t e = pw == PREC_HALF ? cdot_count<PREC_HALF>(n, m, w, t, part, blocks, skip, st)
                                        : cdot_count<PREC_SINGLE>(n, m, w, t, part, blocks, skip, st);
  if (e != cudaSuccess) return e;
  cdot_finish_kernel<<<2 * m, 32, 0, st>>>(blocks, 2 * m, part, out, skip);
  return cudaGetLastError();
}
static int blas_grid(int64_t n) {
  int grid = int((n + 255) / 256);
  return grid > 148 * 16 ? 148 * 16 : grid;
}
cudaError_t launch_caxpy_dev(int64_t n, int m, const CFieldList& x, int px, const GcrState* s,
                             const int* count, float sign, SpinorPtr y, const int* skip,
                             cudaStream_t st) {
  if (px == PREC_HALF)
    caxpy_dev_kernel<PREC_HALF><<<blas_grid(n), 256, 0, st>>>(n, m, x, s, count, sign, y, skip);
  else
    caxpy_dev_kernel<PREC_SINGLE><<<blas_grid(n), 256, 0, st>>>(n, m, x, s, count, sign, y, skip);
  return cudaGetLastError();
}
cudaError_t launch_gcr_update(int64_t n, int m, const CFieldList& w, int pw, const GcrState* s, int j,
                              SpinorPtr wj, SpinorPtr r, float2* feat, cudaStream_t st) {
  if (pw == PREC_HALF)
    gcr_update_kernel<PREC_HALF><<<blas_grid(n), 256, 0, st>>>(n, m, w, s, j, wj, r, feat);
  else
    gcr_update_kernel<PREC_SINGLE><<<blas_grid(n), 256, 0, st>>>(n, m, w, s, j, wj, r, feat);
  return cudaGetLastError();
}
cudaError_t launch_gcr_init(GcrState* s, double rr, double target, double d2, int limit,
                            cudaStream_t st) {
  gcr_init_kernel<<<1, 64, 0, st>>>(s, rr, target, d2, limit);
  return cudaGetLastError();
}
cudaError_t launch_gcr_coef(GcrState* s, const double* g, int j, int m, int second,
                            cudaStream_t st) {
  gcr_coef_kernel<<<1, 1, 0, st>>>(s, g, j, m, second);
  return cudaGetLastError();
}
__global__ void fill_int_kernel(int* p, int v) { *p = v; }
cudaError_t launch_fill_int(int* p, int v, cudaStream_t st) {
  fill_int_kernel<<<1, 1, 0, st>>>(p, v);
  return cudaGetLastError();
}
cudaError_t launch_gcr_gamma(GcrState* s, cudaStream_t st) {
  gcr_gamma_kernel<<<1, 32, 0, st>>>(s);
  return cudaGetLastError();
}

}  // namespace iro

// =====================================================================================
// Host side: the network object, training gradients and flexible GCR.
// =====================================================================================
#include <algorithm>
#include <chrono>
#include <cmath>
#include <memory>
#include <string>

namespace iro {
namespace host {
int apply(iro_ctx* c, int op, double mass, double csw, bool dag, const DevField& in, DevField& out,
          const Reduce* red, int red_mask, const int* skip);
DevField* workspace(iro_ctx* c, int subset, int prec, int nrhs, int slot, int* rc);
void* pinned(iro_ctx* c);
void* scratch(iro_ctx* c, size_t bytes, int* rc);
int import_field(iro_ctx* c, const double* host, bool full, DevField& f);
int export_field(iro_ctx* c, const DevField& f, bool full, double* host);
int norms(iro_ctx* c, const DevField& v, const DevField* w, std::vector<double>& nv,
          std::vector<double>* nw);
int axpby(iro_ctx* c, double a, const DevField& x, double b, const DevField& y, DevField& v);
int convert(iro_ctx* c, const DevField& in, DevField& out);
int set_error(iro_ctx* c, int code, const std::string& msg);
int cuda_error(iro_ctx* c, cudaError_t e, const char* where);
cudaStream_t stream(iro_ctx* c);
int device(iro_ctx* c);
DevField* field_dev(iro_field* f);
const Geom& geom(iro_ctx* c);
GaugePtr gauge_single(iro_ctx* c);
bool gauge_su3(iro_ctx* c);
int64_t volume(iro_ctx* c);
}  // namespace host
}  // namespace iro

// CG on device fields (solvers.cu), the fallback of the preconditioned solve
int cg_any_dev(iro_ctx* c, int op, double mass, double csw, const iro_cg_params* prm,
               const iro::DevField* B, iro::DevField* X, int nrhs, iro_solver_out* out);

using namespace iro;
using namespace iro::host;

#define LCK(call)                                            \
  do {                                                       \
    cudaError_t e__ = (call);                                \
    if (e__ != cudaSuccess) return cuda_error(c, e__, #call); \
  } while (0)
#define LRC(call)                  \
  do {                             \
    int r__ = (call);              \
    if (r__ != IRO_OK) return r__; \
  } while (0)

struct iro_ptc {
  iro_ctx* ctx = nullptr;
  int dev = 0;  // device of the buffers (iro_ptc_destroy does not touch the context)
  int nl = 0;
  std::vector<int> w;                 // widths, nl+1 entries
  std::vector<std::vector<float>> W;  // host weights, complex [9][cout][cin] (re,im)
  std::vector<void*> bop, badj;       // device BF16 packed weights per layer, and its adjoint's
  std::vector<float2*> act;           // act[l]: input of layer l (act[nl]: output)
  float2* g0 = nullptr;               // gradient ping-pong buffers
  float2* g1 = nullptr;
  double* partial = nullptr;          // weight-gradient sums, one block per CTA
  float* db = nullptr;                // every layer's dL/dB, consecutive
  double* lpart = nullptr;
  size_t maxc = 0;
};

namespace {

void pack_bop(int cin, int cout, const std::vector<float>& W, std::vector<__nv_bfloat16>& bop) {
  int kf, kp, nf, np;
  ptc_dims(cin, cout, &kf, &kp, &nf, &np);
  std::vector<float> B(size_t(np) * kp, 0.f);
  for (int d = 0; d < 9; ++d)
    for (int o = 0; o < cout; ++o)
      for (int i = 0; i < cin; ++i) {
        const size_t w = ((size_t(d) * cout + o) * cin + i) * 2;
        const float wr = W[w], wi = W[w + 1];
        const int kre = (2 * d) * cin + i, kim = (2 * d + 1) * cin + i;
        B[size_t(2 * o) * kp + kre] = wr;
        B[size_t(2 * o) * kp + kim] = -wi;
        B[size_t(2 * o + 1) * kp + kre] = wi;
        B[size_t(2 * o + 1) * kp + kim] = wr;
      }
  bop.resize(B.size());
  for (size_t k = 0; k < B.size(); ++k) bop[k] = __float2bfloat16_rn(B[k]);
}

// The adjoint layer's weights [9][cin][cout]: with y = sum_d W_d T_d x the
// gradient of x is sum_d W_d^dag T_d^dag dy, and T_{+mu}^dag = T_{-mu}, so it is
// a layer on dy whose displacement d has the weights of the opposite one,
// conjugate transposed.
std::vector<float> adjoint_weights(int cin, int cout, const std::vector<float>& W) {
  std::vector<float> A(W.size());
  for (int d = 0; d < 9; ++d) {
    const int e = d == 0 ? 0 : ((d - 1) ^ 1) + 1;
    for (int o = 0; o < cout; ++o)
      for (int i = 0; i < cin; ++i) {
        const size_t w = ((size_t(e) * cout + o) * cin + i) * 2, a = ((size_t(d) * cin + i) * cout + o) * 2;
        A[a] = W[w];
        A[a + 1] = -W[w + 1];
      }
  }
  return A;
}

// dL/dB (NF x KF, real) -> dL/dW (complex [9][cout][cin])
void unpack_grad(int cin, int cout, const float* dB, float* g) {
  int kf, kp, nf, np;
  ptc_dims(cin, cout, &kf, &kp, &nf, &np);
  for (int d = 0; d < 9; ++d)
    for (int o = 0; o < cout; ++o)
      for (int i = 0; i < cin; ++i) {
        const int kre = (2 * d) * cin + i, kim = (2 * d + 1) * cin + i;
        const float rr = dB[size_t(2 * o) * kf + kre], ri = dB[size_t(2 * o) * kf + kim];
        const float ir = dB[size_t(2 * o + 1) * kf + kre], ii = dB[size_t(2 * o + 1) * kf + kim];
        const size_t w = ((size_t(d) * cout + o) * cin + i) * 2;
        g[w] = rr + ii;
        g[w + 1] = -ri + ir;
      }
}

PtcGeo make_geo(iro_ctx* c) {
  PtcGeo G;
  G.g = geom(c);
  G.gauge = gauge_single(c);
  G.V = int(volume(c));
  G.skip = nullptr;
  return G;
}

// features of a full-lattice spinor field (FP32 or FP64; converted to FP32);
// `skip` (FP32 fields only) as the forward pass's
int field_to_feat(iro_ctx* c, const DevField& f, float2* feat, const int* skip = nullptr) {
  const DevField* src = &f;
  int rc = IRO_OK;
  if (f.prec != PREC_SINGLE) {
    DevField* t = workspace(c, 2, PREC_SINGLE, 1, 70, &rc);
    if (!t) return rc;
    LRC(convert(c, f, *t));
    src = t;
  }
  LCK(launch_spinor_to_feat(int(src->Vh), src->half(0), src->half(1), feat, stream(c),
                            f.prec == PREC_SINGLE ? skip : nullptr));
  return IRO_OK;
}

int feat_to_field(iro_ctx* c, const float2* feat, DevField& f, const int* skip = nullptr) {
  if (f.prec == PREC_SINGLE || f.prec == PREC_HALF) {
    LCK(launch_feat_to_spinor(int(f.Vh), feat, f.half(0), f.half(1), stream(c), skip, f.prec));
    return IRO_OK;
  }
  int rc = IRO_OK;
  DevField* t = workspace(c, 2, PREC_SINGLE, 1, 71, &rc);
  if (!t) return rc;
  LCK(launch_feat_to_spinor(int(t->Vh), feat, t->half(0), t->half(1), stream(c)));
  return convert(c, *t, f);
}

int wait_done(iro_ctx* c) {
  LCK(cudaStreamSynchronize(stream(c)));
  return IRO_OK;
}

// act[0] must hold the input features; runs every layer
// the network's layers on n->act[0]; nothing when `skip` is set and nonzero
int forward(iro_ctx* c, iro_ptc* n, const int* skip = nullptr) {
  PtcGeo G = make_geo(c);
  G.skip = skip;
  for (int l = 0; l < n->nl; ++l)
    LCK(launch_ptc_fwd(n->w[l], n->w[l + 1], G, n->act[l], n->act[l + 1], n->bop[l], stream(c)));
  return IRO_OK;
}

}  // namespace

extern "C" {

int iro_ptc_create(iro_ctx* c, int nlayers, const int* widths, iro_ptc** out) {
  if (!c || !widths || !out || nlayers < 1 || nlayers > 8)
    return set_error(c, IRO_BAD_ARG, "bad network arguments");
  if (widths[0] != 4 || widths[nlayers] != 4)
    return set_error(c, IRO_BAD_ARG, "network input and output must be 4 channels (a spinor)");
  for (int l = 0; l < nlayers; ++l)
    if (!ptc_shape_ok(widths[l], widths[l + 1]))
      return set_error(c, IRO_BAD_ARG, "layer widths must be 4, 8 or 16 channels");
  LCK(cudaSetDevice(device(c)));
  std::unique_ptr<iro_ptc> n(new iro_ptc());
  n->ctx = c;
  n->dev = device(c);
  n->nl = nlayers;
  n->w.assign(widths, widths + nlayers + 1);
  const size_t V = size_t(volume(c));
  size_t maxc = 0;
  for (int w : n->w) maxc = std::max(maxc, size_t(w));
  n->maxc = maxc;
  n->W.resize(nlayers);
  n->bop.resize(nlayers);
  n->badj.resize(nlayers);
  n->act.resize(nlayers + 1);
  int maxnk = 0;
  size_t gradn = 0;
  for (int l = 0; l < nlayers; ++l) {
    int kf, kp, nf, np;
    ptc_dims(n->w[l], n->w[l + 1], &kf, &kp, &nf, &np);
    gradn += size_t(nf) * kf;
    maxnk = std::max(maxnk, nf * kf);
    n->W[l].assign(size_t(9) * n->w[l + 1] * n->w[l] * 2, 0.f);
    LCK(cudaMalloc(&n->bop[l], size_t(np) * kp * 2));
    int akf, akp, anf, anp;
    ptc_dims(n->w[l + 1], n->w[l], &akf, &akp, &anf, &anp);
    LCK(cudaMalloc(&n->badj[l], size_t(anp) * akp * 2));
    LCK(cudaMemset(n->bop[l], 0, size_t(np) * kp * 2));
    LCK(cudaMemset(n->badj[l], 0, size_t(anp) * akp * 2));
  }
  for (int l = 0; l <= nlayers; ++l) LCK(cudaMalloc(&n->act[l], V * n->w[l] * 3 * sizeof(float2)));
  LCK(cudaMalloc(&n->g0, V * maxc * 3 * sizeof(float2)));
  LCK(cudaMalloc(&n->g1, V * maxc * 3 * sizeof(float2)));
  LCK(cudaMalloc(&n->db, gradn * sizeof(float)));
  LCK(cudaMalloc(&n->partial, size_t(db_grid(int(V))) * maxnk * sizeof(double)));
  LCK(cudaMalloc(&n->lpart, sizeof(double) * 2 * loss_blocks()));
  *out = n.release();
  return IRO_OK;
}

int iro_ptc_destroy(iro_ptc* n) {
  if (!n) return IRO_BAD_ARG;
  // cudaFree waits for the device's work on these buffers; the context may be gone
  cudaSetDevice(n->dev);
  for (void* p : n->bop) cudaFree(p);
  for (void* p : n->badj) cudaFree(p);
  for (float2* p : n->act) cudaFree(p);
  void* ps[] = {n->g0, n->g1, n->db, n->partial, n->lpart};
  for (void* p : ps)
    if (p) cudaFree(p);
  delete n;
  return IRO_OK;
}

int iro_ptc_set_weights(iro_ptc* n, int layer, const float* w) {
  if (!n || !w || layer < 0 || layer >= n->nl) return IRO_BAD_ARG;
  iro_ctx* c = n->ctx;
  LCK(cudaSetDevice(device(c)));
  const int cin = n->w[layer], cout = n->w[layer + 1];
  n->W[layer].assign(w, w + size_t(9) * cout * cin * 2);
  std::vector<__nv_bfloat16> b, bt;
  pack_bop(cin, cout, n->W[layer], b);
  pack_bop(cout, cin, adjoint_weights(cin, cout, n->W[layer]), bt);
  LCK(cudaMemcpyAsync(n->bop[layer], b.data(), b.size() * 2, cudaMemcpyHostToDevice, stream(c)));
  LCK(cudaMemcpyAsync(n->badj[layer], bt.data(), bt.size() * 2, cudaMemcpyHostToDevice, stream(c)));
  LCK(cudaStreamSynchronize(stream(c)));
  return IRO_OK;
}

static bool same_lattice(iro_ctx* c, const iro_ptc* n) {
  return volume(c) == volume(n->ctx) && geom(c).L[0] == geom(n->ctx).L[0] &&
         geom(c).L[1] == geom(n->ctx).L[1] && geom(c).L[2] == geom(n->ctx).L[2];
}

int iro_ptc_apply_field(iro_ctx* c, iro_ptc* n, const iro_field* in, iro_field* out) {
  if (!c || !n || !in || !out) return IRO_BAD_ARG;
  if (!same_lattice(c, n)) return set_error(c, IRO_BAD_ARG, "network built for another lattice");
  const DevField* fi = field_dev(const_cast<iro_field*>(in));
  DevField* fo = field_dev(out);
  if (fi->subset != 2 || fo->subset != 2 || fi->nrhs != 1 || fo->nrhs != 1 || fi->prec == PREC_HALF ||
      fo->prec == PREC_HALF)
    return set_error(c, IRO_BAD_ARG, "network fields must be full-lattice FP32/FP64, one rhs");
  if (!gauge_su3(c)) return set_error(c, IRO_NO_GAUGE, "network needs an SU(3) gauge field");
  LCK(cudaSetDevice(device(c)));
  LRC(field_to_feat(c, *fi, n->act[0]));
  LRC(forward(c, n));
  LRC(feat_to_field(c, n->act[n->nl], *fo));
  return wait_done(c);
}

int iro_ptc_apply(iro_ctx* c, iro_ptc* n, const double* in, double* out) {
  if (!c || !n || !in || !out) return IRO_BAD_ARG;
  if (!same_lattice(c, n)) return set_error(c, IRO_BAD_ARG, "network built for another lattice");
  if (!gauge_su3(c)) return set_error(c, IRO_NO_GAUGE, "network needs an SU(3) gauge field");
  LCK(cudaSetDevice(device(c)));
  int rc = IRO_OK;
  DevField* a = workspace(c, 2, PREC_DOUBLE, 1, 72, &rc);
  if (!a) return rc;
  DevField* b = workspace(c, 2, PREC_DOUBLE, 1, 73, &rc);
  if (!b) return rc;
  LRC(import_field(c, in, true, *a));
  LRC(field_to_feat(c, *a, n->act[0]));
  LRC(forward(c, n));
  LRC(wait_done(c));
  LRC(feat_to_field(c, n->act[n->nl], *b));
  return export_field(c, *b, true, out);
}

int iro_ptc_loss_grad(iro_ctx* c, iro_ptc* n, const iro_field* in, const iro_field* target,
                      double* loss, float* grad) {
  if (!c || !n || !in || !target || !loss) return IRO_BAD_ARG;
  if (!same_lattice(c, n)) return set_error(c, IRO_BAD_ARG, "network built for another lattice");
  const DevField* fi = field_dev(const_cast<iro_field*>(in));
  const DevField* ft = field_dev(const_cast<iro_field*>(target));
  if (fi->subset != 2 || ft->subset != 2 || fi->nrhs != 1 || ft->nrhs != 1)
    return set_error(c, IRO_BAD_ARG, "training fields must be full-lattice, one rhs");
  if (!gauge_su3(c)) return set_error(c, IRO_NO_GAUGE, "network needs an SU(3) gauge field");
  LCK(cudaSetDevice(device(c)));
  cudaStream_t st = stream(c);
  const int V = int(volume(c));
  LRC(field_to_feat(c, *fi, n->act[0]));
  LRC(forward(c, n));
  // target features into g1, loss and dL/dy into g0
  LRC(field_to_feat(c, *ft, n->g1));
  const int nel = V * 12;
  LCK(launch_loss_partials(nel, n->act[n->nl], n->g1, n->lpart, st));
  std::vector<double> part(2 * loss_blocks());
  LCK(cudaMemcpyAsync(part.data(), n->lpart, sizeof(double) * part.size(), cudaMemcpyDeviceToHost, st));
  LCK(cudaStreamSynchronize(st));
  double dd = 0.0, tt = 0.0;
  for (int b = 0; b < loss_blocks(); ++b) {
    dd += part[2 * b];
    tt += part[2 * b + 1];
  }
  *loss = dd / tt;
  if (!grad) return wait_done(c);
  LCK(launch_loss_grad(nel, n->act[n->nl], n->g1, float(2.0 / tt), n->g0, st));
  PtcGeo G = make_geo(c);
  float2* dy = n->g0;
  float2* dx = n->g1;
  std::vector<size_t> goff(n->nl + 1, 0), boff(n->nl + 1, 0);
  for (int l = 0; l < n->nl; ++l) {
    goff[l + 1] = goff[l] + size_t(9) * n->w[l + 1] * n->w[l] * 2;
    boff[l + 1] = boff[l] + size_t(18) * n->w[l] * 2 * n->w[l + 1];
  }
  for (int l = n->nl - 1; l >= 0; --l) {
    const int cin = n->w[l], cout = n->w[l + 1];
    LCK(launch_ptc_db(cin, cout, G, n->act[l], dy, n->partial, n->db + boff[l], st));
    if (l > 0) LCK(launch_ptc_fwd(cout, cin, G, dy, dx, n->badj[l], st));
    std::swap(dy, dx);
  }
  std::vector<float> dB(boff[n->nl]);
  LCK(cudaMemcpyAsync(dB.data(), n->db, dB.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
  LCK(cudaStreamSynchronize(st));
  for (int l = 0; l < n->nl; ++l) unpack_grad(n->w[l], n->w[l + 1], dB.data() + boff[l], grad + goff[l]);
  return wait_done(c);
}

// ---- flexible GCR on A = D^dag D with the network as right preconditioner ---------------
int iro_gcr_solve_field(iro_ctx* c, int op, double mass, double csw, const iro_ptc* net,
                        const iro_gcr_params* prm, const iro_field* b, iro_field* x, iro_gcr_out* out) {
  const DevField* B = field_dev(const_cast<iro_field*>(b));
  DevField* X = field_dev(x);
  if (!c || !prm || !B || !X || !out || (op != IRO_OP_WILSON_FULL && op != IRO_OP_CLOVER_FULL) ||
      B->subset != 2 || X->subset != 2 || B->prec != PREC_DOUBLE || X->prec != PREC_DOUBLE ||
      B->nrhs != 1 || X->nrhs != 1 || prm->nkrylov < 1 || prm->nkrylov > kMaxVec ||
      !(prm->precision > 0.0))
    return set_error(c, IRO_BAD_ARG, "bad GCR arguments");
  if (net && !same_lattice(c, net)) return set_error(c, IRO_BAD_ARG, "network built for another lattice");
  LCK(cudaSetDevice(device(c)));
  auto t0 = std::chrono::steady_clock::now();
  cudaStream_t st = stream(c);
  const int m = prm->nkrylov;
  int rc = IRO_OK;
  DevField* R = workspace(c, 2, PREC_DOUBLE, 1, 80, &rc); if (!R) return rc;
  DevField* Q = workspace(c, 2, PREC_DOUBLE, 1, 81, &rc); if (!Q) return rc;
  DevField* S = workspace(c, 2, PREC_DOUBLE, 1, 82, &rc); if (!S) return rc;
  DevField* r32 = workspace(c, 2, PREC_SINGLE, 1, 83, &rc); if (!r32) return rc;
  DevField* e32 = workspace(c, 2, PREC_SINGLE, 1, 84, &rc); if (!e32) return rc;
  // the Krylov fields z_j, w_j (and D z_j) in FP32 or FP16
  const int kp = prm->krylov_half ? PREC_HALF : PREC_SINGLE;
  DevField* tk = workspace(c, 2, kp, 1, 85, &rc); if (!tk) return rc;
  std::vector<DevField*> Z(m), W(m);
  for (int j = 0; j < m; ++j) {
    Z[j] = workspace(c, 2, kp, 1, 90 + j, &rc); if (!Z[j]) return rc;
    W[j] = workspace(c, 2, kp, 1, 90 + kMaxVec + j, &rc); if (!W[j]) return rc;
  }
  const int64_t nel = R->sites();
  const int blocks = 148 * 8;  // inner-product partials: 8 blocks of 128 threads per SM
  // block partials, the first and second passes' sums, then the cycle state
  const size_t sum_off = size_t(blocks) * 2 * kMaxList;
  const size_t state_off = sum_off + 4 * kMaxList;
  // (the context's solver scratch: a solve allocates nothing)
  const size_t mask_off = sizeof(double) * state_off + (sizeof(GcrState) + 15) / 16 * 16;
  char* scr = static_cast<char*>(scratch(c, mask_off + 16, &rc));
  if (!scr) return rc;
  double* part = reinterpret_cast<double*>(scr);
  double* dsum = part + sum_off;
  double* dsum2 = dsum + 2 * kMaxList;
  GcrState* gs = reinterpret_cast<GcrState*>(part + state_off);
  int* dmask = reinterpret_cast<int*>(scr + mask_off);
  // the cycle's iteration count comes back through the context's pinned host
  // buffer (the solvers use its first bytes for their flags; GCR does not run
  // beside them)
  int* hjdone = reinterpret_cast<int*>(static_cast<char*>(pinned(c)) + 2048);
  // x = 0, r = b
  LRC(axpby(c, 0.0, *B, 0.0, *B, *X));
  LRC(axpby(c, 1.0, *B, 0.0, *B, *R));
  std::vector<double> bn;
  LRC(norms(c, *B, nullptr, bn, nullptr));
  const double target = prm->precision * bn[0];
  double rr = bn[0];
  const double delta = prm->delta > 0.0 ? prm->delta : 0.1;
  int iters = 0, restarts = 0, fallback = 0, pcapplies = 0, stalls = 0;
  bool converged = rr < target || rr == 0.0;  // b = 0: x = 0 is the solution
  LCK(launch_fill_int(dmask, 1, st));
  while (!converged && iters < prm->max_iter) {
    // One restart cycle, enqueued whole: the coefficients of every iteration
    // are formed on the device (gcr_coef_kernel), and the iterations after
    // the one that meets the restart test (|r|^2 below delta^2 of its value
    // at the cycle start, or the target) return at once.  The z_j are kept as
    // the network produced them; the orthogonalised directions are z'_j =
    // sum_i T[i][j] z_i (T unit upper triangular, from the Gram-Schmidt
    // coefficients of the w_j), and the correction of the cycle e = sum_j
    // alpha_j z'_j = sum_i gamma_i z_i is formed once at its end.
    const int cyc = std::min(m, prm->max_iter - iters);
    LRC(convert(c, *R, *r32));
    LRC(axpby(c, 0.0, *r32, 0.0, *r32, *e32));
    LCK(launch_gcr_init(gs, rr, target, delta * delta, cyc, st));
    for (int j = 0; j < cyc; ++j) {
      const int* skip = &gs->skip[j];
      // z_j = N(r) (or r without a network), w_j = A z_j
      if (net) {
        // the features of r: the previous iteration's update wrote them
        // unless it took the second pass (plain[j - 1] = 0)
        LRC(field_to_feat(c, *r32, net->act[0], j == 0 ? skip : &gs->plain[j - 1]));
        LRC(forward(c, const_cast<iro_ptc*>(net), skip));
        LRC(feat_to_field(c, net->act[net->nl], *Z[j], skip));
      } else if (kp == PREC_SINGLE) {
        LRC(axpby(c, 1.0, *r32, 0.0, *r32, *Z[j]));
      } else {
        LRC(convert(c, *r32, *Z[j]));
      }
      LRC(apply(c, op, mass, csw, false, *Z[j], *tk, nullptr, 0, skip));
      LRC(apply(c, op, mass, csw, true, *tk, *W[j], nullptr, 0, skip));
      // one pass forms <w_q, w_j> (q < j), |w_j|^2 and <r, w_j>; the
      // coefficient kernel turns them into beta_q, |w'_j|^2 and alpha, and a
      // second pass orthogonalises w_j and updates r -= alpha w'_j
      CFieldList L{};
      for (int q = 0; q <= j; ++q) L.f[q] = W[q]->all();
      L.f[j + 1] = r32->all();
      LCK(launch_cdot(nel, j + 2, L, W[j]->all(), part, blocks, dsum, skip, kp, st));
      LCK(launch_gcr_coef(gs, dsum, j, m, 0, st));
      LCK(launch_gcr_update(nel, j, L, kp, gs, j, W[j]->all(), r32->all(),
                            net ? net->act[0] : nullptr, st));
      // w_j nearly in the span of the w_q (plain[j] = 0): |w'_j|^2 and
      // <r, w'_j> from the orthogonalised vector, then r -= alpha w'_j
      const int* single = &gs->plain[j];
      CFieldList L2{};
      L2.f[0] = W[j]->all();
      L2.f[1] = r32->all();
      LCK(launch_cdot(nel, 2, L2, W[j]->all(), part, blocks, dsum2, single, kp, st));
      LCK(launch_gcr_coef(gs, dsum2, j, m, 1, st));
      LCK(launch_caxpy_dev(nel, 1, L2, kp, gs, nullptr, -1.f, r32->all(), single, st));
    }
    // e = sum_i gamma_i z_i, gamma = T alpha over the iterations done
    {
      LCK(launch_gcr_gamma(gs, st));
      CFieldList L{};
      for (int i = 0; i < cyc; ++i) L.f[i] = Z[i]->all();
      LCK(launch_caxpy_dev(nel, cyc, L, kp, gs, &gs->jdone, 1.f, e32->all(), nullptr, st));
      LCK(cudaMemcpyAsync(hjdone, &gs->jdone, sizeof(int), cudaMemcpyDeviceToHost, st));
    }
    // x += e, r = b - A x in FP64
    LCK(launch_mx_merge(PREC_SINGLE, X->sites(), 1, X->all(), e32->all(), dmask, st));
    LRC(apply(c, op, mass, csw, false, *X, *Q, nullptr, 0, nullptr));
    LRC(apply(c, op, mass, csw, true, *Q, *S, nullptr, 0, nullptr));
    LRC(axpby(c, 1.0, *B, -1.0, *S, *R));
    std::vector<double> rnorm;
    LRC(norms(c, *R, nullptr, rnorm, nullptr));
    const int jd = *hjdone;  // copied before the norms, which synchronise the stream
    iters += jd;
    if (net) pcapplies += jd;
    ++restarts;
    stalls = (rnorm[0] > 0.25 * rr) ? stalls + 1 : 0;
    rr = rnorm[0];
    converged = rr < target;
    if (!std::isfinite(rr)) break;
    if (!converged && stalls >= 2) {
      // the preconditioned iteration stalls: finish with mixed-precision CG on
      // the correction A e = r, then x += e
      iro_cg_params cp{prm->precision * bn[0] / rr, prm->max_iter, IRO_PREC_SINGLE, 0.1, 1};
      DevField* E = workspace(c, 2, PREC_DOUBLE, 1, 86, &rc); if (!E) return rc;
      iro_solver_out co;
      const int crc = cg_any_dev(c, op, mass, csw, &cp, R, E, 1, &co);
      if (crc != IRO_OK && crc != IRO_NOT_CONVERGED) return crc;
      LRC(axpby(c, 1.0, *X, 1.0, *E, *X));
      LRC(apply(c, op, mass, csw, false, *X, *Q, nullptr, 0, nullptr));
      LRC(apply(c, op, mass, csw, true, *Q, *S, nullptr, 0, nullptr));
      LRC(axpby(c, 1.0, *B, -1.0, *S, *R));
      LRC(norms(c, *R, nullptr, rnorm, nullptr));
      rr = rnorm[0];
      converged = rr < target;
      iters += co.iterations > 0 ? co.iterations : 0;
      fallback = 1;
      break;
    }
  }
  auto t1 = std::chrono::steady_clock::now();
  out->diff = bn[0] > 0.0 ? std::sqrt(rr / bn[0]) : 0.0;
  out->iterations = converged ? iters : -1;
  out->timing_ms = std::chrono::duration<double, std::milli>(t1 - t0).count();
  out->restarts = restarts;
  out->fallback = fallback;
  out->precond_applies = pcapplies;
  if (net) {
    int e = wait_done(c);
    if (e) return e;
  }
  if (!converged) return set_error(c, IRO_NOT_CONVERGED, "GCR not converged");
  return IRO_OK;
}

}  // extern "C"
