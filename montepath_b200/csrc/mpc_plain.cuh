// mpc_plain.cuh -- the FP64 plain path: one request per launch, every sample
// generated where it is used, stepped, paid and reduced in one kernel.
//
// One unit per thread (up to four for short units), one tile per block; the
// hardware's block scheduler balances the tiles, so blocks of 128 threads keep the
// last wave full.  Blocks of 64 and 32 are no faster for requests that leave SMs
// without a block either, since every block stages its own tables: Heston x 64 on
// Sobol 1,000 paths 41 / 43 / 45 us with 128 / 64 / 32 threads, 20,000 paths
// 47 / 48 / 55; Asian x 64 on Halton 1,000 paths 58 / 62 / 70.  The descriptor travels as a kernel
// parameter and the last tile writes the moments straight into the host's
// pinned buffer: a request is one launch with no copies.  Before, samples
// were written to HBM, read back by a second kernel, payoffs reduced by a
// third, and four small copies and fills went with them: the Heston and Merton
// pair of 131,072 paths x 256 steps on scrambled Sobol took 2,890 us
// (generation 1,185 + 1,303, most of it the inverse normal's tail run by whole
// warps for single lanes and the Merton dimensions drawn but not used) against
// 552 us here.  Bound by issue and FP64 latency together (issue slots 0.69, FP64
// pipe 0.45 of peak in the Heston kernel at 27 warps an SM).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mpc_launch.h"
#include "mpc_models.cuh"

namespace mpc {

template <int SMP>
struct PlainSource {
  using type = Source<SMP>;
};
template <>
struct PlainSource<SMP_SOBOL> {
  using type = SobolPlain;
};
template <>
struct PlainSource<SMP_XORSHIFT> {
  using type = XorshiftPairs<double>;
};

// Resident blocks the register allocation must allow.  A basket keeps the FP64
// sums of up to 8 assets beside a sample in the making: 64 registers (8 blocks)
// spill, 2,000 x 252 of 8 assets 397 -> 419 us pseudorandom and 601 -> 642 on the
// counter hash, where larger requests gain 2 to 8%.
constexpr int plain_min_blocks(int fam) { return fam == FAM_BASKET ? 3 : 8; }

// The block's moment sums as its tile partial; the request's last tile to
// finish sums the partials (finalize_request).
__device__ __forceinline__ void plain_finish(const DevReq& q, uint64_t units, double v[5], double (*red)[5], int* s_last) {
  block_reduce5(v, red);
  if (threadIdx.x == 0) {
    double* pt = q.partials + (size_t)blockIdx.x * MPC_MOMENTS;
    pt[0] = (double)units;
    for (int i = 0; i < 5; ++i) pt[1 + i] = v[i];
    __threadfence();
    *s_last = (atomicAdd(q.tiles_done, 1u) == q.n_tiles - 1) ? 1 : 0;
  }
  __syncthreads();
  if (*s_last) {
    __threadfence();
    finalize_request(q, red);
  }
}

template <int FAM, int SMP>
__global__ void __launch_bounds__(kPlainBlock, plain_min_blocks(FAM)) plain_kernel(const __grid_constant__ DevReq q, SrcCtx ctx) {
  __shared__ double red[kPlainBlock / 32][5];
  __shared__ int s_last;
  if constexpr (SMP == SMP_SOBOL) {
    __shared__ __align__(16) uint32_t s_window[kSobolWindowWords];
    ctx.win = s_window;
  }
  const uint64_t first = (uint64_t)blockIdx.x * q.tile_units;
  const uint64_t last = min(first + (uint64_t)q.tile_units, q.n_units);
  double v[5] = {0, 0, 0, 0, 0};
  for (uint64_t base = first; base < last; base += kPlainBlock) {
    // a thread past the end repeats the last unit and discards it (block- and
    // warp-synchronous sources need every thread)
    const bool valid = base + threadIdx.x < last;
    const uint64_t u = valid ? base + threadIdx.x : last - 1;
    typename PlainSource<SMP>::type src;
    src.template begin<true>(q, ctx, u);
    double p, c;
    run_family<double, FAM>(q, src, p, c);
    if (!valid) continue;
    v[0] += p;
    v[1] += p * p;
    if (q.cv) {
      v[2] += c;
      v[3] += c * c;
      v[4] += p * c;
    }
    if (q.per_unit) q.per_unit[u] = p;
  }
  plain_finish(q, last - first, v, red, &s_last);
}

template <int SMP>
cudaError_t launch_plain_s(const DevReq& q, const DeviceTables& tabs, cudaStream_t stream) {
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr, nullptr, tabs.icdf_tail};
  const uint32_t grid = q.n_tiles;
  switch (q.family) {
    case FAM_GBM_STEP:
      plain_kernel<FAM_GBM_STEP, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_GBM_TERMINAL:
      plain_kernel<FAM_GBM_TERMINAL, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_HESTON:
      plain_kernel<FAM_HESTON, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_BASKET:
      plain_kernel<FAM_BASKET, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_MLMC_LEVEL:
      plain_kernel<FAM_MLMC_LEVEL, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_GBM_BRIDGE:
      if constexpr (SMP != SMP_SOBOL) return cudaErrorInvalidValue;
      else plain_kernel<FAM_GBM_BRIDGE, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_MERTON_STEP:  // the pseudorandom Merton is the stream replay (mpc_merton.cu)
      if constexpr (SMP == SMP_XORSHIFT) return cudaErrorInvalidValue;
      else plain_kernel<FAM_MERTON_STEP, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    case FAM_MERTON_TERMINAL:
      if constexpr (SMP == SMP_XORSHIFT) return cudaErrorInvalidValue;
      else plain_kernel<FAM_MERTON_TERMINAL, SMP><<<grid, kPlainBlock, 0, stream>>>(q, ctx);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  count_graph_launches(1);  // adds to the launch count
  return cudaGetLastError();
}

}  // namespace mpc
