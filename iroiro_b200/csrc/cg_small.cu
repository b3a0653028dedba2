// CG iterations of small lattices in one cooperative launch.
//
// On a small lattice an iteration of Solver_CG on D^dag D is all latency: its
// stencil and update launches each wait for the one before, a thread walks
// the eight neighbours of its site one load after another, and the two
// reductions end in a chain of tickets.  Here one grid that fits the device
// runs whole iterations: the phases (the operator's stencils, the x and p
// update) are separated by a grid barrier, the eight neighbour terms of a site
// are formed by eight warps and summed through shared memory, and every block
// sums the block partials itself after the barrier and carries its own copy of
// the solver's scalars (the stages of solver_scalars.cuh), so that no block
// waits for another's update.  The recurrences, flags and reductions are those
// of the launched iteration, in another (fixed) order of summation.
//
// What bounds it is the chain of a phase: ~1.5 us for a barrier, ~1 us for the
// scalars, ~2.5 us for a stencil (its loads ~1500 cycles, the index arithmetic
// of a first group kept from the launch's start, the sums).  FP64 CG on the
// full 8^3x16 lattice, host arrays included: 31 us an iteration launched, 16 us
// here.
#include "dslash_split.cuh"
#include "internal.h"

namespace iro {

namespace {

using namespace split;

// The barrier of a cooperative grid: the arrivals counted in `bar`, `blocks` of
// them (the grid's) awaited each time, for at most limit_ns
struct GridBarrier {
  unsigned* bar;
  int* err;
  unsigned blocks;
  uint64_t limit_ns;
};

struct CgSmallParams {
  Geom g;
  int nrhs, full, clover;
  GaugePtr gauge;
  CloverPtr A[2], Ainv;  // Ainv: the odd sites' inverse
  double kappa;
  SpinorPtr p[2], q[2], r[2];  // by parity ([0] only for a Schur operator)
  SpinorPtr t;                 // the Schur operator's odd field
  SpinorPtr pall, rall, xall;  // the same p and r, and x, over all elements
  int64_t nelem;
  CGState* state;
  int* done;
  int max_iter, iters;
  double* partials;
  GridBarrier wait;
};

template <typename R>
struct SmallShared : Shared<R> {
  double red[kThreads];
  double tot[16];
  CGState st[16];
  int done[16];
  int ok;
};

// What a thread keeps over a launch: its right-hand side and site in a group,
// and the neighbour of its warp's direction at its block's first group's site
// for the output parity of stencil k (the index arithmetic with its divisions
// took as long as the loads)
struct SmallSite {
  int sl, r, S, per, nb[2];
};
__device__ __forceinline__ SmallSite small_site(const CgSmallParams& P) {
  SmallSite s;
  const int lane = threadIdx.x & 31;
  s.S = 32 / P.nrhs;
  s.sl = lane / P.nrhs;
  s.r = lane - s.sl * P.nrhs;
  s.per = (P.g.Vh + s.S - 1) / s.S;
  const int y = P.full && int(blockIdx.x) >= s.per ? 1 : 0;
  const int hs = (int(blockIdx.x) - y * s.per) * s.S + s.sl;
  s.nb[0] = s.nb[1] = 0;
  if (s.sl < s.S && hs < P.g.Vh) {
    s.nb[0] = neighbour(P.g, coord_of(P.g, hs, 1), hs, threadIdx.x >> 5);
    s.nb[1] = neighbour(P.g, coord_of(P.g, hs, y), hs, threadIdx.x >> 5);
  }
  return s;
}

// One stencil of the operator over this block's groups, and the sum that its
// reduction takes.  k 0: Schur's first stencil, into the odd t; k 1: its second,
// or the full operator's both parities.  dag 0: D p into q; 1: D^dag q
// subtracted, times alpha, from the residual.
template <int SP>
__device__ __forceinline__ double hop_phase(const CgSmallParams& P, SmallShared<typename SpinorIO<SP>::Real>& sm,
                                            const SmallSite& site, int k, int dag) {
  using R = typename SpinorIO<SP>::Real;
  const int p0 = k == 0 ? 1 : 0, npar = k != 0 && P.full ? 2 : 1;
  const int epi = k == 0 ? (P.clover ? EPI_SCALE_CLOV : EPI_SCALE) : (P.clover ? EPI_XPAY_CLOV : EPI_XPAY);
  const bool res = dag != 0 && k != 0;
  const R scale = R(k != 0 && !P.full ? P.kappa : -P.kappa);
  const R alpha = R(sm.st[site.r].alpha);
  const int nrhs = P.nrhs, r = site.r;
  const bool mine = site.sl < site.S && !sm.done[r];
  double sum = 0.0;
#pragma unroll 1
  for (int grp = blockIdx.x; grp < npar * site.per; grp += gridDim.x) {
    const int y = grp >= site.per ? 1 : 0;
    const int p = p0 ^ y;
    const int hs = (grp - y * site.per) * site.S + site.sl;
    const bool act = mine && hs < P.g.Vh;
    // the operator's input at the output parity, its other parity (or t), and
    // where the result goes
    const SpinorPtr own = dag ? (y ? P.q[1] : P.q[0]) : (y ? P.p[1] : P.p[0]);
    const SpinorPtr in = k == 0 ? own : !P.full ? P.t : dag ? (y ? P.q[0] : P.q[1]) : (y ? P.p[0] : P.p[1]);
    const SpinorPtr out = k == 0 ? P.t : res ? (y ? P.r[1] : P.r[0]) : (y ? P.q[1] : P.q[0]);
    const CloverPtr cl = k == 0 ? P.Ainv : y ? P.A[1] : P.A[0];
    int nb = k == 0 ? site.nb[0] : site.nb[1];
    if (act && grp != int(blockIdx.x)) nb = neighbour(P.g, coord_of(P.g, hs, p), hs, threadIdx.x >> 5);
    sum += group<SP>(P.gauge, uint32_t(P.g.Vh), sm, in, own, out, cl, epi, dag, scale, res, alpha, act, p, hs,
                     hs * nrhs + r, nb, nrhs, r);
  }
  return sum;
}

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// Waits until every block has arrived `gen` times (the counter only grows
// within a launch).  The grid is resident as a whole (cooperative launch); the
// wait is bounded all the same: after limit_ns of global time the block sets
// the error flag and leaves, and so do the others.
__device__ __noinline__ bool grid_barrier(const GridBarrier& B, int& shared_ok, unsigned& gen) {
  ++gen;
  __syncthreads();
  if (threadIdx.x == 0) {
    // the block's writes (ordered before this by the barrier above) are
    // released with the arrival, the others' acquired with the last poll
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(B.bar) : "memory");
    const unsigned want = gen * B.blocks;
    const uint64_t t0 = global_ns();
    int ok = 1;
    for (unsigned it = 0; ld_acquire(B.bar) < want; ++it)
      if ((it & 255u) == 255u && global_ns() - t0 > B.limit_ns) {
        ok = 0;
        atomicExch(B.err, 1);
        break;
      }
    shared_ok = ok;
  }
  __syncthreads();
  return shared_ok != 0;
}

// This block's partials of a sum per right-hand side (fixed order): one right-hand
// side, one per warp that holds terms; otherwise one per right-hand side
template <typename SM>
__device__ __forceinline__ void put_partial(const CgSmallParams& P, SM& sm, double* part, double v) {
  const int t = threadIdx.x, nrhs = P.nrhs;
  if (nrhs == 1) {
    v = warp_sum(v);
    if ((t & 31) == 0 && t < 128) part[4 * blockIdx.x + (t >> 5)] = v;
  } else {
    sm.red[t] = v;
    __syncthreads();
    const int S = 32 / nrhs;
    if (t < nrhs) {
      double s = 0.0;
      for (int w = 0; w < 4; ++w)
        for (int k = 0; k < S; ++k) s += sm.red[32 * w + k * nrhs + t];
      part[int64_t(blockIdx.x) * nrhs + t] = s;
    }
  }
}
// Sums every block's partials, the same way in every block, and runs the stage
template <typename SM>
__device__ __forceinline__ void take_totals(const CgSmallParams& P, SM& sm, const double* part, int stage) {
  const int t = threadIdx.x, nrhs = P.nrhs, nb = gridDim.x;
  if (nrhs == 1) {
    double s = 0.0;
#pragma unroll 4
    for (int b = t; b < 4 * nb; b += kThreads) s += __ldcg(part + b);
    s = warp_sum(s);
    if ((t & 31) == 0) sm.red[t >> 5] = s;
    __syncthreads();
    if (t == 0) {
      s = 0.0;
#pragma unroll
      for (int w = 0; w < kThreads / 32; ++w) s += sm.red[w];
      sm.tot[0] = s;
    }
  } else {
    const int ns = kThreads / nrhs, sl = t / nrhs, r = t - sl * nrhs;
    double s = 0.0;
    if (sl < ns)
      for (int b = sl; b < nb; b += ns) s += __ldcg(part + int64_t(b) * nrhs + r);
    sm.red[t] = s;
    __syncthreads();
    double s8 = 0.0;
    if (t < 8 * nrhs)
      for (int k = t / nrhs; k < ns; k += 8) s8 += sm.red[k * nrhs + t % nrhs];
    __syncthreads();
    if (t < 8 * nrhs) sm.red[t] = s8;
    __syncthreads();
    if (t < nrhs) {
      double u = 0.0;
#pragma unroll
      for (int k = 0; k < 8; ++k) u += sm.red[k * nrhs + t];
      sm.tot[t] = u;
    }
  }
  __syncthreads();
  if (t == 0) {
    Reduce R{};
    R.stage = stage;
    R.state = sm.st;
    R.done = sm.done;
    R.max_iter = P.max_iter;
    stage_update(R, sm.tot, 1, nrhs);
  }
  __syncthreads();
}

// x += alpha p, p = r + beta p (as cg_p_kernel), by 16-byte chunks (FP64, FP32)
// or by elements (FP16, which renormalises)
template <int SP, typename SM>
__device__ __forceinline__ void update_phase(const CgSmallParams& P, SM& sm) {
  using R = typename SpinorIO<SP>::Real;
  const int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, step = int64_t(gridDim.x) * blockDim.x;
  if constexpr (SP == PREC_HALF) {
    for (int64_t e = t0; e < P.nelem; e += step) {
      const int r = int(e % P.nrhs);
      const bool ux = sm.st[r].xpend != 0, up = sm.done[r] == RUNNING;
      if (!ux && !up) continue;
      const float a = float(sm.st[r].alpha), b = float(sm.st[r].beta);
      uint32_t w[12];
      Cx<float> pv[12], v[12];
      auto get = [&](const SpinorPtr& s, Cx<float> d[12]) {
        const float n = load_co_w(s, int(e), w);
#pragma unroll
        for (int k = 0; k < 12; ++k) {
          const float2 f = unpack_h2(w[k]);
          d[k] = {n * f.x, n * f.y};
        }
      };
      get(P.pall, pv);
      if (ux) {
        get(P.xall, v);
#pragma unroll
        for (int k = 0; k < 12; ++k) v[k] = v[k] + a * pv[k];
        SpinorIO<SP>::store(P.xall, e, v);
      }
      if (up) {
        get(P.rall, v);
#pragma unroll
        for (int k = 0; k < 12; ++k) pv[k] = b * pv[k] + v[k];
        SpinorIO<SP>::store(P.pall, e, pv);
      }
    }
  } else {
    constexpr int NC = SpinorIO<SP>::NCHUNK;
    constexpr int W = 16 / sizeof(R);
    struct alignas(16) Chunk {
      R v[W];
    };
    const int64_t n = P.nelem * NC;
    for (int64_t j = t0; j < n; j += step) {
      const int64_t e = j / (32 * NC) * 32 + (j & 31);
      const int r = int(e % P.nrhs);
      const bool ux = sm.st[r].xpend != 0, up = sm.done[r] == RUNNING;
      if (!ux && !up) continue;
      const R a = R(sm.st[r].alpha), b = R(sm.st[r].beta);
      auto get = [&](const SpinorPtr& s) {
        const uint4 u = __ldcg(static_cast<const uint4*>(s.data) + j);
        return *reinterpret_cast<const Chunk*>(&u);
      };
      Chunk p = get(P.pall), x = get(P.xall);
      const Chunk q = get(P.rall);
      if (ux) {
#pragma unroll
        for (int k = 0; k < W; ++k) x.v[k] += a * p.v[k];
        static_cast<Chunk*>(P.xall.data)[j] = x;
      }
      if (up) {
#pragma unroll
        for (int k = 0; k < W; ++k) p.v[k] = b * p.v[k] + q.v[k];
        static_cast<Chunk*>(P.pall.data)[j] = p;
      }
    }
  }
}

template <int SP>
__global__ void __launch_bounds__(kThreads, 2) cg_small_kernel(const __grid_constant__ CgSmallParams P) {
  using R = typename SpinorIO<SP>::Real;
  __shared__ SmallShared<R> sm;
  const int t = threadIdx.x;
  if (t < P.nrhs) {
    sm.st[t] = P.state[t];
    sm.done[t] = P.done[t];
  }
  fill_tables(sm.dir, sm.spin);
  __syncthreads();
  unsigned gen = 0;
  const SmallSite site = small_site(P);
  // two sets of partials: a block may write the next sum's while another still
  // reads this one's
  const int64_t set = int64_t(gridDim.x) * (P.nrhs == 1 ? 4 : P.nrhs);
  const int first = P.full ? 1 : 0;
  for (int it = 0; it < P.iters; ++it) {
    // q = D p and (p, A p) = |q|^2; then r -= alpha D^dag q and |r|^2.  One copy
    // of the code for both: what an iteration executes is mostly latency, the
    // instructions' too.
#pragma unroll 1
    for (int dag = 0; dag < 2; ++dag) {
      double v = 0.0;
#pragma unroll 1
      for (int k = first; k < 2; ++k) {
        if (k > first && !grid_barrier(P.wait, sm.ok, gen)) return;
        v = hop_phase<SP>(P, sm, site, k, dag);
      }
      double* part = P.partials + dag * set;
      put_partial(P, sm, part, v);
      if (!grid_barrier(P.wait, sm.ok, gen)) return;
      take_totals(P, sm, part, dag == 0 ? ST_CG_ALPHA : ST_CG_BETA);
    }
    update_phase<SP>(P, sm);
    bool left = true;
    for (int r = 0; r < P.nrhs; ++r) left = left && sm.done[r] != RUNNING;
    if (left) break;  // the same in every block
    if (!grid_barrier(P.wait, sm.ok, gen)) return;
  }
  __syncthreads();
  if (blockIdx.x == 0 && t < P.nrhs) {
    P.state[t] = sm.st[t];
    P.done[t] = sm.done[t];
  }
}

// Self-test of the barrier (iro_selftest_bounded_wait): the time of one wait
__global__ void __launch_bounds__(kThreads) barrier_probe_kernel(GridBarrier B, unsigned long long* waited_ns) {
  __shared__ int ok;
  unsigned gen = 0;
  const uint64_t t0 = global_ns();
  grid_barrier(B, ok, gen);
  if (blockIdx.x == 0 && threadIdx.x == 0) *waited_ns = global_ns() - t0;
}

template <int SP>
cudaError_t go(CgSmallParams P, int sms, cudaStream_t st) {
  int per_sm = 0;
  cudaError_t e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cg_small_kernel<SP>, kThreads, 0);
  if (e != cudaSuccess) return e;
  const int S = 32 / P.nrhs;
  const int groups = (P.full ? 2 : 1) * ((P.g.Vh + S - 1) / S);
  int grid = sms * per_sm;
  if (grid > groups) grid = groups;
  P.wait.blocks += grid;
  void* args[] = {&P};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(cg_small_kernel<SP>), dim3(grid),
                                     dim3(kThreads), args, 0, st);
}

}  // namespace

cudaError_t launch_cg_small(const CgSmallLaunch& L, cudaStream_t st) {
  CgSmallParams P{};
  P.g = L.g;
  P.nrhs = L.p->nrhs;
  P.full = L.full;
  P.clover = L.clover;
  P.gauge = L.gauge;
  for (int y = 0; y < 2; ++y) {
    P.A[y] = L.A[y];
    const int h = L.full ? y : 0;
    P.p[y] = L.p->half(h);
    P.q[y] = L.q->half(h);
    P.r[y] = L.r->half(h);
  }
  P.Ainv = L.Ainv;
  P.kappa = L.kappa;
  if (!L.full) P.t = L.t->half(1);
  P.pall = L.p->all();
  P.rall = L.r->all();
  P.xall = L.x->all();
  P.nelem = L.p->sites() * L.p->nrhs;
  P.state = L.state;
  P.done = L.done;
  P.max_iter = L.max_iter;
  P.iters = L.iters;
  P.partials = L.partials;
  P.wait = GridBarrier{L.bar, L.err, unsigned(L.missing), L.limit_ns};
  cudaError_t e = cudaMemsetAsync(L.bar, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  switch (L.p->prec) {
    case PREC_DOUBLE: return go<PREC_DOUBLE>(P, L.sms, st);
    case PREC_SINGLE: return go<PREC_SINGLE>(P, L.sms, st);
    default: return go<PREC_HALF>(P, L.sms, st);
  }
}

cudaError_t launch_barrier_probe(int blocks, int missing, uint64_t limit_ns, unsigned* bar, int* err,
                                 unsigned long long* waited_ns, cudaStream_t st) {
  cudaError_t e = cudaMemsetAsync(bar, 0, sizeof(unsigned), st);
  if (e != cudaSuccess) return e;
  GridBarrier B{bar, err, unsigned(blocks + missing), limit_ns};
  void* args[] = {&B, &waited_ns};
  return cudaLaunchCooperativeKernel(reinterpret_cast<void*>(barrier_probe_kernel), dim3(blocks), dim3(kThreads), args,
                                     0, st);
}

}  // namespace iro
