// Launch dispatch of the stencil over (dagger, epilogue); included once per
// storage precision so the instantiations compile in parallel.
#pragma once

#include <atomic>

#include "dslash.cuh"
#include "dslash_pair.cuh"
#include "internal.h"

namespace iro {

// A capped grid is no larger than the blocks that are resident at once: a
// thread loops over the sites anyway, and what is left over would run as a
// further wave that fills the device only in part (the cap of 8 blocks per SM
// was 1.3 to 4 times what the kernels' registers let in).  Operator
// applications, cap / resident: full Wilson 12x20x28x44 FP64 0.0668 / 0.0508 ms,
// 12 right-hand sides 0.586 / 0.486, FP16 0.199 / 0.167; e/o 32^3x64 FP16 with
// 5 right-hand sides 0.641 / 0.576.
template <auto Kernel>
static int resident_grid(const LaunchCfg& c, const HopLaunch& L) {
  if (L.grid_cap() != L.max_blocks) return c.grid;
  static std::atomic<int> per_sm[9];  // of this kernel, by warps per block
  const int w = (c.block + 31) / 32;
  int n = per_sm[w].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, Kernel, c.block, 0) != cudaSuccess || n < 1) {
      cudaGetLastError();
      n = 8;
    }
    per_sm[w].store(n, std::memory_order_relaxed);
  }
  // max_blocks is 8 per SM
  const int fit = L.max_blocks / 8 * n / L.nparity;
  return c.grid > fit ? (fit > 0 ? fit : 1) : c.grid;
}

// The same as one block per SM.  Blocks of another stream's launch take an SM's
// slots one by one as this launch's blocks leave them; with several per SM the
// two launches then run half and half through all of their length, and from
// kSweepBytes of spinors on the slices that neighbours share no longer fit L2
// for both.  Applications, us, one context / contexts in turn, small blocks and
// one per SM: FP32 clover 28x20x26x66, 16 right-hand sides, 1520 / 1763, 1482 /
// 1703; FP64 clover 32x26x30x34, 2: 364 / 429, 359 / 359; FP16 e/o 32^3x64, 5:
// 596 / 633, 580 / 587.  Launches that reduce keep the small blocks
// (block_reduce_finish takes 256 threads), and a shape's variant is tuned with
// them: one block per SM levels the variants (FP16 e/o 32^3x64, 12 right-hand
// sides, variants 10 / 12: 1345 / 1346 us, small blocks 1370 / 1540), and 12
// picked on that made the solve with its reductions 5 % slower.
constexpr int64_t kSweepBytes = int64_t(200) << 20;
static void block_per_sm(LaunchCfg& c, const HopLaunch& L, int full, int nthreads) {
  if (L.red_mask || L.cg || L.tuning || full <= c.block || int64_t(c.grid) * c.block >= nthreads) return;
  const int site = L.prec == PREC_DOUBLE ? 192 : L.prec == PREC_SINGLE ? 96 : 52;
  if (int64_t(L.nparity) * L.g.Vh * L.nrhs * site < kSweepBytes) return;
  c.block = full / L.nrhs * L.nrhs;
  c.grid = L.max_blocks / 8 / L.nparity;
}

template <int SP, int GP, int RECON, bool DAG, int EPI, int VAR>
static cudaError_t hop_go(const HopLaunch& L, cudaStream_t st) {
  HopParams P;
  P.g = L.g;
  P.p0 = L.p0;
  P.nrhs = L.nrhs;
  P.dn = make_fastdiv(uint32_t(L.nrhs));
  for (int i = 0; i < 2; ++i) {
    P.in[i] = L.in[i];
    P.out[i] = L.out[i];
    P.xin[i] = L.xin[i];
    P.clov[i] = L.clov[i];
  }
  P.gauge = L.gauge;
  P.scale = L.scale;
  P.red_mask = L.red_mask;
  P.red = L.red;
  P.skip = L.skip;
  P.cg = L.cg;
  P.cst = L.cst;
  for (int i = 0; i < 2; ++i) {
    P.cr[i] = L.cr[i];
  }
  P.hs0 = L.hs0;
  P.nhs = L.nhs < 0 ? L.g.Vh - L.hs0 : L.nhs;
  LaunchCfg c = launch_cfg(P.nhs, L.nrhs, L.grid_cap(),
                           L.block_cap < HopBounds<VAR>::threads ? L.block_cap
                                                                 : HopBounds<VAR>::threads);
  c.grid = resident_grid<hop_kernel<SP, GP, RECON, DAG, EPI, SP, VAR>>(c, L);
  block_per_sm(c, L, HopBounds<VAR>::full, P.nhs * L.nrhs);
  // programmatic dependent launch: the blocks of this grid may be scheduled
  // while the previous kernel's last blocks retire (hop_kernel waits for
  // that kernel's completion before it reads anything), hiding the launch
  // gap between the dependent stencil launches of an operator
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(c.grid, L.nparity);
  cfg.blockDim = dim3(c.block);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, hop_kernel<SP, GP, RECON, DAG, EPI, SP, VAR>, P);
}

// two right-hand sides per thread (FP32/FP16, reconstruct-12, even nrhs)
template <int SP, int RECON, bool DAG, int EPI, int VAR>
static cudaError_t hop_go_pair(const HopLaunch& L, cudaStream_t st) {
  if constexpr (SP == PREC_DOUBLE || RECON != 12) {
    return cudaErrorInvalidValue;
  } else {
    if (L.nrhs % 2 != 0 || L.hs0 != 0 || (L.nhs >= 0 && L.nhs != L.g.Vh)) return cudaErrorInvalidValue;
    HopParams P;
    P.g = L.g;
    P.p0 = L.p0;
    P.nrhs = L.nrhs;
    for (int i = 0; i < 2; ++i) {
      P.in[i] = L.in[i];
      P.out[i] = L.out[i];
      P.xin[i] = L.xin[i];
      P.clov[i] = L.clov[i];
    }
    P.gauge = L.gauge;
    P.scale = L.scale;
    P.red_mask = L.red_mask;
    P.red = L.red;
    P.skip = L.skip;
    P.cg = L.cg;
    P.cst = L.cst;
    for (int i = 0; i < 2; ++i) {
      P.cr[i] = L.cr[i];
    }
    LaunchCfg c = launch_cfg(L.g.Vh, L.nrhs / 2, L.grid_cap(), L.block_cap);
    c.grid = resident_grid<hop_pair_kernel<SP, DAG, EPI, VAR>>(c, L);
    dim3 grid(c.grid, L.nparity);
    hop_pair_kernel<SP, DAG, EPI, VAR><<<grid, c.block, 0, st>>>(P);
    return cudaGetLastError();
  }
}

// Variants 0-3: hop_kernel (bits: see there).  FP32/FP16 with even nrhs:
// 4-7 two right-hand sides per thread with the register cap none / 128 /
// 152 / 168.
// FP64: 4/5 the 168-register 128-thread hop_kernel (5 with the rolled loop).
// FP32, any nrhs: 15 the 80-register hop_kernel.
// FP16 on links with three stored rows (RECON 18): only 10/11/12, the
// mixed-precision hop_kernel (VAR 8 / 9 / 10: 3 / 4 / 2 blocks per SM).
// FP16 on the 12-real links: also 13/14, the mixed-precision hop_kernel with
// row 2 rebuilt (VAR 8 / 9).
template <int SP, int GP, int RECON, bool DAG, int EPI>
static cudaError_t hop_var_more(const HopLaunch& L, cudaStream_t st);

template <int SP, int GP, int RECON, bool DAG, int EPI>
static cudaError_t hop_var(const HopLaunch& L, cudaStream_t st) {
  if constexpr (SP == PREC_HALF && RECON == 18) {
    switch (L.variant) {
      case 10: return hop_go<SP, GP, RECON, DAG, EPI, 8>(L, st);
      case 11: return hop_go<SP, GP, RECON, DAG, EPI, 9>(L, st);
      case 12: return hop_go<SP, GP, RECON, DAG, EPI, 10>(L, st);
      default: return cudaErrorInvalidValue;
    }
  } else {
    switch (L.variant) {
      case 0: return hop_go<SP, GP, RECON, DAG, EPI, 0>(L, st);
      case 1: return hop_go<SP, GP, RECON, DAG, EPI, 1>(L, st);
      case 2: return hop_go<SP, GP, RECON, DAG, EPI, 2>(L, st);
      case 3: return hop_go<SP, GP, RECON, DAG, EPI, 3>(L, st);
      default: break;
    }
    return hop_var_more<SP, GP, RECON, DAG, EPI>(L, st);
  }
}

template <int SP, int GP, int RECON, bool DAG, int EPI>
static cudaError_t hop_var_more(const HopLaunch& L, cudaStream_t st) {
  if constexpr (SP == PREC_DOUBLE) {
    switch (L.variant) {
      case 4: return hop_go<SP, GP, RECON, DAG, EPI, 4>(L, st);
      case 5: return hop_go<SP, GP, RECON, DAG, EPI, 6>(L, st);
      default: return cudaErrorInvalidValue;
    }
  } else {
    switch (L.variant) {
      case 4: return hop_go_pair<SP, RECON, DAG, EPI, 0>(L, st);
      case 5: return hop_go_pair<SP, RECON, DAG, EPI, 1>(L, st);
      case 6: return hop_go_pair<SP, RECON, DAG, EPI, 2>(L, st);
      case 7: return hop_go_pair<SP, RECON, DAG, EPI, 3>(L, st);
      default: break;
    }
    if constexpr (SP == PREC_SINGLE)
      if (L.variant == 15) return hop_go<SP, GP, RECON, DAG, EPI, 16>(L, st);
    if constexpr (SP == PREC_HALF && RECON == 12) {
      switch (L.variant) {
        case 13: return hop_go<SP, GP, RECON, DAG, EPI, 8>(L, st);
        case 14: return hop_go<SP, GP, RECON, DAG, EPI, 9>(L, st);
        default: break;
      }
    }
    return cudaErrorInvalidValue;
  }
}

template <int SP, int RECON, bool DAG>
static cudaError_t hop_epi(const HopLaunch& L, cudaStream_t st) {
  switch (L.epi) {
    case EPI_SCALE: return hop_var<SP, SP, RECON, DAG, EPI_SCALE>(L, st);
    case EPI_SCALE_CLOV: return hop_var<SP, SP, RECON, DAG, EPI_SCALE_CLOV>(L, st);
    case EPI_XPAY: return hop_var<SP, SP, RECON, DAG, EPI_XPAY>(L, st);
    case EPI_XPAY_CLOV: return hop_var<SP, SP, RECON, DAG, EPI_XPAY_CLOV>(L, st);
  }
  return cudaErrorInvalidValue;
}

template <int SP, int RECON>
static cudaError_t hop_dag(const HopLaunch& L, cudaStream_t st) {
  return L.dag ? hop_epi<SP, RECON, true>(L, st) : hop_epi<SP, RECON, false>(L, st);
}

}  // namespace iro
