// Divisions of the device code beside CUDA's own, for tests/test_gpu_arithmetic.py.
#include <cuda_runtime.h>
#include <stdint.h>

#include "mpc_device.cuh"

using namespace mpc;

namespace {

struct Buffer {
  void* p = nullptr;
  explicit Buffer(size_t bytes) { cudaMalloc(&p, bytes); }
  ~Buffer() { cudaFree(p); }
  template <class T>
  T* as() const {
    return static_cast<T*>(p);
  }
};

unsigned blocks(uint64_t n) { return (unsigned)((n + 255) / 256); }
__device__ uint64_t thread_index() { return (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; }

__global__ void quotient_kernel(const double* num, const double* den, uint64_t n, double* ours, double* plain,
                                double* ours_inv, double* plain_inv) {
  const uint64_t i = thread_index();
  if (i >= n) return;
  ours[i] = quotient(num[i], den[i]);
  plain[i] = __ddiv_rn(num[i], den[i]);
  ours_inv[i] = newton_reciprocal(den[i]);
  plain_inv[i] = __drcp_rn(den[i]);
}

__global__ void sixth_f32_kernel(uint32_t first, uint32_t n, unsigned long long* differing) {
  const uint64_t i = thread_index();
  if (i >= n) return;
  const float x = __uint_as_float(first + (uint32_t)i);
  if (__float_as_uint(sixth(x)) != __float_as_uint(__fdiv_rn(x, 6.0f))) atomicAdd(differing, 1ull);
}

__global__ void sixth_f64_kernel(const double* x, uint64_t n, double* ours, double* plain) {
  const uint64_t i = thread_index();
  if (i >= n) return;
  ours[i] = sixth(x[i]);
  plain[i] = __ddiv_rn(x[i], 6.0);
}

// solve_lsm_normal_equations with every division CUDA's.
template <int DIM>
__device__ bool solve_plain(double a[4][4], double rhs[4]) {
  for (int piv = 0; piv < DIM; ++piv) {
    int best = piv;
    for (int row = piv + 1; row < DIM; ++row)
      if (fabs(a[row][piv]) > fabs(a[best][piv])) best = row;
    if (fabs(a[best][piv]) <= 1e-12) return false;
    for (int c = 0; c < DIM; ++c) {
      const double t = a[piv][c];
      a[piv][c] = a[best][c];
      a[best][c] = t;
    }
    const double t = rhs[piv];
    rhs[piv] = rhs[best];
    rhs[best] = t;
    const double pv = a[piv][piv];
    for (int c = piv + 1; c < DIM; ++c) a[piv][c] = __ddiv_rn(a[piv][c], pv);
    rhs[piv] = __ddiv_rn(rhs[piv], pv);
    for (int row = 0; row < DIM; ++row) {
      if (row == piv) continue;
      const double f = a[row][piv];
      for (int c = piv + 1; c < DIM; ++c) a[row][c] = fma(-f, a[piv][c], a[row][c]);
      rhs[row] = fma(-f, rhs[piv], rhs[row]);
    }
  }
  return true;
}

template <int DIM>
__global__ void solve_kernel(const double* systems, uint64_t n, double* ours, double* plain) {
  const uint64_t i = thread_index();
  if (i >= n) return;
  double a[4][4], b[4], pa[4][4], pb[4];
  for (int r = 0; r < 4; ++r) {
    for (int c = 0; c < 4; ++c) pa[r][c] = a[r][c] = systems[i * 20 + r * 4 + c];
    pb[r] = b[r] = systems[i * 20 + 16 + r];
  }
  const bool ok = solve_fixed<DIM, false>(a, b), pok = solve_plain<DIM>(pa, pb);
  ours[i * 5] = ok;
  plain[i * 5] = pok;
  for (int r = 0; r < 4; ++r) {
    ours[i * 5 + 1 + r] = ok && r < DIM ? b[r] : 0.0;
    plain[i * 5 + 1 + r] = pok && r < DIM ? pb[r] : 0.0;
  }
}

int finish() {
  const cudaError_t e = cudaDeviceSynchronize();
  return (int)(e != cudaSuccess ? e : cudaGetLastError());
}

}  // namespace

extern "C" int quotients(const double* num, const double* den, uint64_t n, double* ours, double* plain,
                         double* ours_inv, double* plain_inv) {
  Buffer bn(n * 8), bd(n * 8), bo(n * 8), bp(n * 8), boi(n * 8), bpi(n * 8);
  cudaMemcpy(bn.p, num, n * 8, cudaMemcpyHostToDevice);
  cudaMemcpy(bd.p, den, n * 8, cudaMemcpyHostToDevice);
  quotient_kernel<<<blocks(n), 256>>>(bn.as<double>(), bd.as<double>(), n, bo.as<double>(), bp.as<double>(),
                                      boi.as<double>(), bpi.as<double>());
  cudaMemcpy(ours, bo.p, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(plain, bp.p, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(ours_inv, boi.p, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(plain_inv, bpi.p, n * 8, cudaMemcpyDeviceToHost);
  return finish();
}

// Floats with the bit patterns first .. first + n - 1: how many differ.
extern "C" int sixths_f32(uint32_t first, uint32_t n, unsigned long long* differing) {
  Buffer count(8);
  cudaMemset(count.p, 0, 8);
  sixth_f32_kernel<<<blocks(n), 256>>>(first, n, count.as<unsigned long long>());
  cudaMemcpy(differing, count.p, 8, cudaMemcpyDeviceToHost);
  return finish();
}

extern "C" int sixths_f64(const double* x, uint64_t n, double* ours, double* plain) {
  Buffer bx(n * 8), bo(n * 8), bp(n * 8);
  cudaMemcpy(bx.p, x, n * 8, cudaMemcpyHostToDevice);
  sixth_f64_kernel<<<blocks(n), 256>>>(bx.as<double>(), n, bo.as<double>(), bp.as<double>());
  cudaMemcpy(ours, bo.p, n * 8, cudaMemcpyDeviceToHost);
  cudaMemcpy(plain, bp.p, n * 8, cudaMemcpyDeviceToHost);
  return finish();
}

// systems: [n][20], the matrix by rows, then the right side; results [n][5]: solved, coefficients.
extern "C" int solves(int dim, const double* systems, uint64_t n, double* ours, double* plain) {
  Buffer bs(n * 160), bo(n * 40), bp(n * 40);
  cudaMemcpy(bs.p, systems, n * 160, cudaMemcpyHostToDevice);
  if (dim == 2) solve_kernel<2><<<blocks(n), 256>>>(bs.as<double>(), n, bo.as<double>(), bp.as<double>());
  if (dim == 3) solve_kernel<3><<<blocks(n), 256>>>(bs.as<double>(), n, bo.as<double>(), bp.as<double>());
  if (dim == 4) solve_kernel<4><<<blocks(n), 256>>>(bs.as<double>(), n, bo.as<double>(), bp.as<double>());
  cudaMemcpy(ours, bo.p, n * 40, cudaMemcpyDeviceToHost);
  cudaMemcpy(plain, bp.p, n * 40, cudaMemcpyDeviceToHost);
  return finish();
}
