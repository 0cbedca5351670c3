// FP64 plain path, instances by sampler (one translation unit each compiles in parallel).
#include "mpc_plain.cuh"

namespace mpc {
template cudaError_t launch_plain_s<SMP_HALTON>(const DevReq&, const DeviceTables&, cudaStream_t);
template cudaError_t launch_plain_s<SMP_LHS>(const DevReq&, const DeviceTables&, cudaStream_t);
}  // namespace mpc
