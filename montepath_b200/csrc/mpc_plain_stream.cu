// FP64 plain path, instances by sampler (one translation unit each compiles in parallel).
#include "mpc_plain.cuh"

namespace mpc {

// Pseudorandom GBM paths, `lanes` threads per path (a power of two up to 32,
// plain_lanes in mpc_runtime.cu): a few thousand paths leave most of the FP64
// pipes idle with one thread each, since a path is one chain of dependent
// FP64 operations of several hundred cycles a pair.  Lane j draws the j-th
// share of the path's Box-Muller pairs (its own stream seek), the lanes'
// sums give every lane its starting log price, and path-dependent payoffs walk
// the shares from there.  20,000 paths x 64 steps, 4
// lanes: 22 us, 30 us with one thread per path.
template <int W>
__device__ __forceinline__ void split_walk(const DevReq& q, double ls, double sign, uint32_t count, const double* z,
                                           double& acc, bool& ko) {
  for (uint32_t i = 0; i < count; ++i) {
    ls += q.drift_dt + q.vol_dt * (sign * z[i * kPlainBlock]);
    if constexpr (W == W_ASIAN) acc += exp(ls);
    if constexpr (W == W_LOOKBACK) {
      const double s = exp(ls);
      acc = acc > s ? acc : s;
    }
    if constexpr (W == W_DAO) ko |= exp(ls) <= q.barrier;
    if constexpr (W == W_UAO) ko |= exp(ls) >= q.barrier;
  }
}

template <int W>
__global__ void __launch_bounds__(kPlainBlock, 4) plain_split_kernel(const __grid_constant__ DevReq q,
                                                                    const uint64_t* __restrict__ jump, uint32_t lanes) {
  __shared__ double s_z[kPlainSplitNormals * kPlainBlock];  // [normal][thread]
  __shared__ double red[kPlainBlock / 32][5];
  __shared__ int s_last;
  const uint64_t first = (uint64_t)blockIdx.x * q.tile_units;
  const uint64_t last = min(first + (uint64_t)q.tile_units, q.n_units);
  const uint32_t lane = threadIdx.x & (lanes - 1u);
  const uint64_t at = first + threadIdx.x / lanes;
  const bool valid = at < last;
  const uint64_t u = valid ? at : last - 1;  // a path past the end repeats the last one and is discarded
  uint64_t seed, local;
  chunk_of(q, u, &seed, &local);
  const uint32_t n = q.n_steps;
  const uint64_t idx = local * n;            // the path's first normal in its stream
  const uint32_t odd = (uint32_t)(idx & 1u);  // it is the second of a pair
  const uint32_t pairs = (odd + n + 1u) / 2u;  // pairs the path touches
  const uint32_t p0 = (uint32_t)((uint64_t)pairs * lane / lanes), p1 = (uint32_t)((uint64_t)pairs * (lane + 1u) / lanes);
  XorshiftStream st;
  st.state = xorshift_seek_warp(jump, seed, 2 * ((idx >> 1) + p0));
  st.has_cached = false;
  double* z = s_z + threadIdx.x;
  uint32_t count = 0;
  double sum = 0.0;
  for (uint32_t p = p0; p < p1; ++p) {
    const double a = st.normal_f64(), b = st.normal_f64();
    const uint32_t e = 2u * p - odd;  // step of the pair's first normal (wraps below 0 for an odd start)
    if (e < n && count < kPlainSplitNormals) {
      z[count++ * kPlainBlock] = a;
      sum += a;
    }
    if (e + 1u < n && count < kPlainSplitNormals) {
      z[count++ * kPlainBlock] = b;
      sum += b;
    }
  }
  double before = sum;
  for (uint32_t o = 1; o < lanes; o <<= 1) {
    const double prev = __shfl_up_sync(0xFFFFFFFFu, before, o, (int)lanes);
    if (lane >= o) before += prev;
  }
  const double total = __shfl_sync(0xFFFFFFFFu, before, (int)lanes - 1, (int)lanes);
  before -= sum;
  const uint32_t s0 = 2u * p0 < odd ? 0u : 2u * p0 - odd;  // the share's first step
  double pay = 0.0, ctl = 0.0;
  for (int side = 0; side < (q.anti ? 2 : 1); ++side) {
    const double sign = side ? -1.0 : 1.0;
    double acc = W == W_LOOKBACK ? q.s0 : 0.0;
    bool ko = (W == W_DAO && q.s0 <= q.barrier) || (W == W_UAO && q.s0 >= q.barrier);
    if constexpr (W != W_EURO) {
      split_walk<W>(q, q.log_s0 + (double)s0 * q.drift_dt + q.vol_dt * (sign * before), sign, count, z, acc, ko);
      for (uint32_t o = lanes >> 1; o > 0; o >>= 1) {
        const double other = __shfl_xor_sync(0xFFFFFFFFu, acc, (int)o, (int)lanes);
        acc = W == W_ASIAN ? acc + other : acc > other ? acc : other;
        ko |= __shfl_xor_sync(0xFFFFFFFFu, (int)ko, (int)o, (int)lanes) != 0;
      }
    }
    const double st_end = exp(q.log_s0 + (double)n * q.drift_dt + q.vol_dt * (sign * total));
    double v = W == W_ASIAN ? acc / (double)n - q.k : W == W_LOOKBACK ? acc - q.k : st_end - q.k;
    if (ko) v = 0.0;
    pay += (v > 0.0 ? v : 0.0) * q.discount;
    if (side == 0) ctl = q.discount * st_end;
  }
  if (q.anti) pay *= 0.5;
  double v[5] = {0, 0, 0, 0, 0};
  if (valid && lane == 0) {
    v[0] = pay;
    v[1] = pay * pay;
    if (q.cv) {
      v[2] = ctl;
      v[3] = ctl * ctl;
      v[4] = pay * ctl;
    }
    if (q.per_unit) q.per_unit[u] = pay;
  }
  plain_finish(q, last - first, v, red, &s_last);
}

cudaError_t launch_plain_split(const DevReq& q, const DeviceTables& tabs, uint32_t lanes, cudaStream_t stream) {
  if (lanes < 2 || lanes > 32 || (lanes & (lanes - 1)) || q.tile_units * lanes != kPlainBlock ||
      (q.n_steps / 2 + 1) / lanes + 1 > kPlainSplitNormals / 2)
    return cudaErrorInvalidValue;
  switch (q.workload) {
    case W_ASIAN:
      plain_split_kernel<W_ASIAN><<<q.n_tiles, kPlainBlock, 0, stream>>>(q, tabs.jump, lanes);
      break;
    case W_DAO:
      plain_split_kernel<W_DAO><<<q.n_tiles, kPlainBlock, 0, stream>>>(q, tabs.jump, lanes);
      break;
    case W_UAO:
      plain_split_kernel<W_UAO><<<q.n_tiles, kPlainBlock, 0, stream>>>(q, tabs.jump, lanes);
      break;
    case W_LOOKBACK:
      plain_split_kernel<W_LOOKBACK><<<q.n_tiles, kPlainBlock, 0, stream>>>(q, tabs.jump, lanes);
      break;
    default:
      plain_split_kernel<W_EURO><<<q.n_tiles, kPlainBlock, 0, stream>>>(q, tabs.jump, lanes);
      break;
  }
  count_graph_launches(1);  // adds to the launch count
  return cudaGetLastError();
}

template cudaError_t launch_plain_s<SMP_XORSHIFT>(const DevReq&, const DeviceTables&, cudaStream_t);
template cudaError_t launch_plain_s<SMP_COUNTER>(const DevReq&, const DeviceTables&, cudaStream_t);
}  // namespace mpc
