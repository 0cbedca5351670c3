// FP64 plain path, instances by sampler (one translation unit each compiles in parallel).
#include "mpc_plain.cuh"

namespace mpc {
extern template cudaError_t launch_plain_s<SMP_XORSHIFT>(const DevReq&, const DeviceTables&, cudaStream_t);
extern template cudaError_t launch_plain_s<SMP_COUNTER>(const DevReq&, const DeviceTables&, cudaStream_t);
extern template cudaError_t launch_plain_s<SMP_HALTON>(const DevReq&, const DeviceTables&, cudaStream_t);
extern template cudaError_t launch_plain_s<SMP_LHS>(const DevReq&, const DeviceTables&, cudaStream_t);
template cudaError_t launch_plain_s<SMP_SOBOL>(const DevReq&, const DeviceTables&, cudaStream_t);

// The lower tail of the FP64 inverse normal at the 23-bit midpoint uniforms.
static __global__ void __launch_bounds__(256) icdf_tail_kernel(double* __restrict__ out) {
  const uint32_t m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m < MPC_ICDF_TAIL) out[m] = icdf_f64(((double)m + 0.5) * 1.1920928955078125e-07);
}
cudaError_t launch_icdf_tail(double* d_out, cudaStream_t stream) {
  icdf_tail_kernel<<<(MPC_ICDF_TAIL + 255) / 256, 256, 0, stream>>>(d_out);
  count_graph_launches(1);  // adds to the launch count
  return cudaGetLastError();
}

cudaError_t launch_plain(const DevReq& q, int sampler, const DeviceTables& tabs, cudaStream_t stream) {
  switch (sampler) {
    case SMP_XORSHIFT:
      return launch_plain_s<SMP_XORSHIFT>(q, tabs, stream);
    case SMP_HALTON:
      return launch_plain_s<SMP_HALTON>(q, tabs, stream);
    case SMP_LHS:
      return launch_plain_s<SMP_LHS>(q, tabs, stream);
    case SMP_SOBOL:
      return launch_plain_s<SMP_SOBOL>(q, tabs, stream);
    case SMP_COUNTER:
      return launch_plain_s<SMP_COUNTER>(q, tabs, stream);
    default:
      return cudaErrorInvalidValue;
  }
}
}  // namespace mpc
