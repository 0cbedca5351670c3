// mpc_models.cuh -- sample sources, models and block reductions shared by the
// pricing kernels: a Source yields the samples of one unit, a unit_* function
// runs one unit of a model family through it, and finalize_request sums a
// request's tile partials.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/montepath_cuda.h"
#include "mpc_device.cuh"
#include "mpc_types.h"

namespace mpc {

enum Workload : int32_t {
  W_EURO = 0,
  W_ASIAN = 1,
  W_DAO = 2,
  W_UAO = 3,
  W_LOOKBACK = 4,
};

struct SrcCtx {
  const uint32_t* sobol;  // device lookup table (MPC_SOBOL_TABLE_WORDS words)
  const uint64_t* jump;
  uint32_t* win;          // shared-memory window of Sobol table rows (fused kernel), null elsewhere
  const float4* icdf;     // shared-memory copy of the inverse-normal segments (fused kernel)
  const double* tail;     // lower tail of the FP64 inverse normal (plain kernel)
};

// Dimensions of the Sobol table rows staged in shared memory at a time, and
// the row stride in words: kSobolWindow + 4 is 4 mod 32, so the 16 rows one
// warp touches with a 128-bit load fall into two wavefronts.  The window
// holds the 48 rows of the index's three low nibbles and one constant row:
// a bit of the Owen-shuffled index depends only on the point's bits at and
// above it (and the seed), so bits 12..31 of the shuffled index are the same
// for every point of one aligned 4,096-point group, and the XOR of their five
// nibble rows is one word per dimension.  The points a block runs together
// (one iteration of a tile: at most 512 consecutive aligned units, the tile's
// idle threads repeating its last unit) lie in one such group.
// The output scramble's seed of a dimension, hash_combine(seed_g, dim),
// depends on the block's seed and the dimension alone, so a last row holds
// it for the window's dimensions: a quad reads its four seeds with one load.
constexpr uint32_t kSobolWindow = 64;
constexpr uint32_t kSobolRowStride = kSobolWindow + 4;
constexpr uint32_t kSobolLowNibbles = 3;                        // nibble positions 0..2 staged per point
constexpr uint32_t kSobolLowRows = 16 * kSobolLowNibbles;       // 48 rows
constexpr uint32_t kSobolConstRow = kSobolLowRows;              // XOR of the upper nibble rows
constexpr uint32_t kSobolSeedRow = kSobolLowRows + 1;           // output-scramble seed per dimension
constexpr uint32_t kSobolWindowWords = (kSobolLowRows + 2) * kSobolRowStride;  // 13,600 bytes

// Phi^-1(u) for the 23-bit midpoint uniform u of a Sobol sample x, from the
// segment table.  With m = x >> 9 the uniform is u = (m + 0.5) 2^-23, and its
// mirror 1 - u is the same expression of the 23-bit complement of m, so
// v = min(u, 1 - u) is built from x ^ (x >> 31, arithmetic): the complement
// exactly when bit 31 (u > 1/2) is set, which also gives the result's sign, with
// no compare or select.  v selects binade and one of 32 segments from its
// exponent and top mantissa bits, the remaining 18 mantissa bits give the
// position t in [0, 1/32) in the segment (they sit below 1.0's exponent as they
// are, so no shift is needed), and the segment's cubic gives Phi^-1(v).
// Defined for v in [2^-24, 1/2), which every 23-bit midpoint uniform meets.
__device__ __forceinline__ float icdf_sobol_bits(const float4* __restrict__ seg, uint32_t x) {
  const uint32_t xm = x ^ (uint32_t)((int32_t)x >> 31);
  const float v = __fsub_rn(__uint_as_float((xm >> 9) + 0x3F800000u), 0.99999994f);
  const uint32_t bits = __float_as_uint(v);
  const uint32_t idx = (bits >> 18) - (103u << 5);
  const float t = __int_as_float((bits & 0x3FFFFu) | 0x3F800000u) - 1.0f;
  const float4 c = seg[idx];
  const float p = fmaf(fmaf(fmaf(c.w, t, c.z), t, c.y), t, c.x);
  return __uint_as_float(__float_as_uint(p) ^ (x & 0x80000000u));
}
// Two samples at once: the floating-point steps as packed FP32 pairs
// (FADD2 / FFMA2, each lane rounded exactly as the scalar operation), so the
// pair equals two icdf_sobol_bits calls bit for bit.
__device__ __forceinline__ float2 icdf_sobol_bits2(const float4* __restrict__ seg, uint32_t xa, uint32_t xb) {
  const uint32_t ma = xa ^ (uint32_t)((int32_t)xa >> 31), mb = xb ^ (uint32_t)((int32_t)xb >> 31);
  const float2 v = __fadd2_rn(make_float2(__uint_as_float((ma >> 9) + 0x3F800000u), __uint_as_float((mb >> 9) + 0x3F800000u)),
                              make_float2(-0.99999994f, -0.99999994f));
  const uint32_t ba = __float_as_uint(v.x), bb = __float_as_uint(v.y);
  const float4 ca = seg[(ba >> 18) - (103u << 5)], cb = seg[(bb >> 18) - (103u << 5)];
  const float2 t = __fadd2_rn(make_float2(__int_as_float((ba & 0x3FFFFu) | 0x3F800000u),
                                          __int_as_float((bb & 0x3FFFFu) | 0x3F800000u)),
                              make_float2(-1.0f, -1.0f));
  float2 p = __ffma2_rn(make_float2(ca.w, cb.w), t, make_float2(ca.z, cb.z));
  p = __ffma2_rn(p, t, make_float2(ca.y, cb.y));
  p = __ffma2_rn(p, t, make_float2(ca.x, cb.x));
  return make_float2(__uint_as_float(__float_as_uint(p.x) ^ (xa & 0x80000000u)),
                     __uint_as_float(__float_as_uint(p.y) ^ (xb & 0x80000000u)));
}

// ------------------------------------------------------------- sources ----
// A Source yields the samples of one unit (path or antithetic pair) by
// dimension index.  n32/n64: standard normal in FP32 / FP64; u64: the raw
// uniform (Merton's Poisson dimension).  Models announce each step's
// dimensions with at_step(first, count) before sampling them; every thread
// of a block makes the same at_step calls, which lets the Sobol source stage
// its tables block-synchronously.
template <int S>
struct Source;

template <>
struct Source<SMP_COUNTER> {
  uint32_t seed, unit;
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx&, uint64_t u) {
    seed = q.seed32;
    unit = (uint32_t)u;
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  __device__ __forceinline__ float n32(uint32_t d) { return counter_normal_f32(seed, unit, d); }
  __device__ __forceinline__ double n64(uint32_t d) { return (double)counter_normal_f32(seed, unit, d); }
  __device__ __forceinline__ double u64(uint32_t d) {
    return (double)counter_open01(hash_u32(counter_mix(seed, unit, d, 0u)));
  }
  __device__ __forceinline__ float u32(uint32_t d) { return counter_open01(hash_u32(counter_mix(seed, unit, d, 0u))); }
};

// Scrambled Sobol with the per-point work hoisted: the Owen-shuffled index
// and its nibble offsets depend only on (point, dimension group of 256), so
// they are recomputed when a path crosses into the next group; per
// dimension only the 8 table lookups and the output scramble remain.  Blocks of
// 2^16 points and the dimension wrap are seeded as ScrambledSobol::
// standard_normal does (cpu.rs:5665-5677).  Reads the [dim][q][v] layout from
// global memory (the sample generator).
template <>
struct Source<SMP_SOBOL> {
  const uint32_t* table;
  uint32_t local, block_seed, group, seed_g, combine_g;
  uint32_t off[8];
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx& c, uint64_t u) {
    table = c.sobol;
    local = (uint32_t)(u & 0xFFFFu);
    block_seed = q.seed32 + (uint32_t)(u >> 16) * 0x9E3779B9u;
    group = 0xFFFFFFFFu;
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  __device__ __forceinline__ uint32_t sample(uint32_t d) {
    const uint32_t g = d / MPC_SOBOL_TABLE_DIMS;
    if (g != group) {
      group = g;
      seed_g = block_seed + g;
      const uint32_t shuffled = nested_uniform_scramble(local, seed_g);
#pragma unroll
      for (int q = 0; q < 8; ++q) off[q] = q * 16 + ((shuffled >> (4 * q)) & 0xFu);
      combine_g = 0x9e3779b9u + (seed_g << 6) + (seed_g >> 2);
    }
    const uint32_t dim = d & (MPC_SOBOL_TABLE_DIMS - 1);
    const uint32_t* td = table + dim * 128;
    uint32_t x = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) x ^= __ldg(td + off[q]);
    return nested_uniform_scramble(x, seed_g ^ (dim + combine_g));  // hash_combine(seed_g, dim)
  }
  __device__ __forceinline__ float n32(uint32_t d) { return normcdfinvf(sobol_unit_f32(sample(d))); }
  __device__ __forceinline__ float u32(uint32_t d) { return sobol_unit_f32(sample(d)); }
  __device__ __forceinline__ double n64(uint32_t d) { return icdf_f64(sobol_unit_f64(sample(d))); }
  __device__ __forceinline__ double u64(uint32_t d) { return sobol_unit_f64(sample(d)); }
};

template <>
struct Source<SMP_HALTON> {
  uint64_t index;
  const HaltonDim* dims;
  const double* weights;
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx&, uint64_t u) {
    index = u + 1;
    dims = q.halton;
    weights = q.halton_weights;
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  __device__ __forceinline__ double u64(uint32_t d) { return halton_f64(index, dims + d, weights); }
  __device__ __forceinline__ double n64(uint32_t d) { return icdf_f64(u64(d)); }
  __device__ __forceinline__ float u32(uint32_t d) { return (float)halton_f32(index, dims + d); }
  __device__ __forceinline__ float n32(uint32_t d) {
    float u = fminf(fmaxf(u32(d), 5.9604645e-08f), 0.99999994f);
    return normcdfinvf(u);
  }
};

template <>
struct Source<SMP_LHS> {
  uint64_t point, mixed, n_paths;
  double inv_n;  // FP32 samples scale by it; FP64 ones divide, as the reference does
  const LhsDim* dims;
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx&, uint64_t u) {
    point = u;
    mixed = u * 0xBF58476D1CE4E5B9ull;
    n_paths = q.n_paths;
    inv_n = 1.0 / (double)n_paths;
    dims = q.lhs;
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  __device__ __forceinline__ double u64(uint32_t d) {
    const double u = lhs_place(dims + d, point, mixed, n_paths) / (double)n_paths;
    return fmin(fmax(u, 2.2250738585072014e-308), 1.0 - 2.220446049250313e-16);
  }
  __device__ __forceinline__ double n64(uint32_t d) { return icdf_f64(u64(d)); }
  __device__ __forceinline__ float u32(uint32_t d) { return (float)(lhs_place(dims + d, point, mixed, n_paths) * inv_n); }
  __device__ __forceinline__ float n32(uint32_t d) {
    float u = fminf(fmaxf(u32(d), 5.9604645e-08f), 0.99999994f);
    return normcdfinvf(u);
  }
};

template <>
struct Source<SMP_XORSHIFT> {
  XorshiftStream st;
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx& c, uint64_t u) {
    uint64_t seed, local;
    chunk_of(q, u, &seed, &local);
    st.seek(c.jump, seed, local * q.normals_per_unit, !FP64);
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  // Sequential stream: dimensions must be requested in increasing order.
  __device__ __forceinline__ float n32(uint32_t) { return st.normal_f32(); }
  __device__ __forceinline__ double n64(uint32_t) { return st.normal_f64(); }
  __device__ __forceinline__ double u64(uint32_t) { return st.next_open01(); }
  __device__ __forceinline__ float u32(uint32_t) { return st.next_open01_f32(); }
};

// ------------------------------------------------ fused FP32 sources ---
// The fused kernels draw their samples through FusedUnitSource<FAM, SMP>::type:
// the generic sources except for scrambled Sobol, the counter hash and the
// pseudorandom stream.

// Scrambled Sobol for the fused kernels, bit-identical to Source<SMP_SOBOL>.
// A block-synchronous window in shared memory holds, for each table row
// r = 16 q + v of the three low nibble positions, the bit-reversed nibble
// products of kSobolWindow consecutive dimensions, the constant row of the
// upper positions and the output-scramble seeds, so one 128-bit load per row
// serves four dimensions: a quad of dimensions costs 5 shared loads and 12
// XORs instead of 32 loads.  XOR commutes with bit reversal, so the quad
// holds brev(x) and the output scramble skips its first reversal.
struct SobolQuad {
  const uint32_t* rows_global;  // [128][256] bit-reversed rows
  uint32_t* win;                // [kSobolLowRows + 2][kSobolRowStride] shared-memory window
  const float4* icdf;           // inverse-normal segments in shared memory
  uint32_t win_first;           // first dimension in the window (multiple of 4)
  uint32_t dims;                // dimensions the request reads
  uint32_t local, block_seed, group, quad;
  uint32_t rows[kSobolLowNibbles];  // window word offset of this point's row per low nibble position
  uint32_t x0, x1, x2, x3;      // reversed products of the dimensions of `quad`
  uint32_t s0, s1, s2, s3;      // their output-scramble seeds
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx& c, uint64_t u) {
    rows_global = c.sobol + MPC_SOBOL_NIBBLE_WORDS;
    win = c.win;
    icdf = c.icdf;
    win_first = 0xFFFFFFFFu;
    dims = (uint32_t)q.normals_per_unit;
    local = (uint32_t)(u & 0xFFFFu);
    block_seed = q.seed32 + (uint32_t)(u >> 16) * 0x9E3779B9u;
    group = 0xFFFFFFFFu;
    quad = 0xFFFFFFFFu;
  }
  // Block-synchronous: restages the window at d0 rounded down to a multiple
  // of 4 when [d0, d0 + count) is not inside it.  Requires
  // count <= kSobolWindow - 3 so that the step fits the aligned window, and
  // every point the block runs together in one aligned 4,096-point group, so
  // that the constant row is theirs.  The low
  // rows are 16-byte asynchronous global-to-shared transfers (four dimensions
  // of one row each; an aligned quad never crosses the 256-dimension wrap),
  // all in flight at once while the constant row is computed, then one wait.
  // Only the quads the request still reads are staged, rounded up to a power
  // of two of them: a terminal request stages 1 of 16 (1,048,576 paths:
  // 70 -> 61 us of device time).
  __device__ __forceinline__ void at_step(uint32_t d0, uint32_t count) {
    if (win_first != 0xFFFFFFFFu && d0 >= win_first && d0 + count <= win_first + kSobolWindow) return;
    __syncthreads();
    const uint32_t w0 = d0 & ~3u;
    const uint32_t left = dims - w0;
    const uint32_t shift = left > 32u ? 4u : left > 16u ? 3u : left > 8u ? 2u : left > 4u ? 1u : 0u;  // log2(quads per row)
    const uint32_t win_s = (uint32_t)__cvta_generic_to_shared(win);
    for (uint32_t i = threadIdx.x; i < (kSobolLowRows << shift); i += blockDim.x) {
      const uint32_t row = i >> shift, j = 4 * (i & ((1u << shift) - 1u));
      const uint32_t* src = rows_global + row * MPC_SOBOL_TABLE_DIMS + ((w0 + j) & (MPC_SOBOL_TABLE_DIMS - 1));
      const uint32_t dst = win_s + 4u * (row * kSobolRowStride + j);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
    }
    for (uint32_t j = threadIdx.x; j < (4u << shift); j += blockDim.x) {
      const uint32_t d = w0 + j;
      const uint32_t sg = block_seed + d / MPC_SOBOL_TABLE_DIMS;
      // bits 12..31 of the shuffled index of this block's points (its bits
      // below 12 do not reach them)
      const uint32_t hi = nested_uniform_scramble(local & 0xF000u, sg);
      const uint32_t dm = d & (MPC_SOBOL_TABLE_DIMS - 1);
      uint32_t c = 0;
#pragma unroll
      for (int k = kSobolLowNibbles; k < 8; ++k)
        c ^= __ldg(rows_global + (16u * k + ((hi >> (4 * k)) & 0xFu)) * MPC_SOBOL_TABLE_DIMS + dm);
      win[kSobolConstRow * kSobolRowStride + j] = c;
      win[kSobolSeedRow * kSobolRowStride + j] = hash_combine(sg, dm);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    win_first = w0;
  }
  // Loads the quad of dimensions [d0, d0 + 4), d0 a multiple of 4 inside
  // the window (the chunked model loops call it directly).
  __device__ __forceinline__ void quad_load(uint32_t d0) {
    const uint32_t g = d0 / MPC_SOBOL_TABLE_DIMS;
    if (g != group) {
      group = g;
      const uint32_t shuffled = nested_uniform_scramble(local, block_seed + g);
#pragma unroll
      for (int k = 0; k < (int)kSobolLowNibbles; ++k) rows[k] = (16u * k + ((shuffled >> (4 * k)) & 0xFu)) * kSobolRowStride;
    }
    quad = d0 >> 2;
    const uint32_t* base = win + (d0 - win_first);
    const uint4 sd = *reinterpret_cast<const uint4*>(base + kSobolSeedRow * kSobolRowStride);
    s0 = sd.x;
    s1 = sd.y;
    s2 = sd.z;
    s3 = sd.w;
    uint4 a = *reinterpret_cast<const uint4*>(base + kSobolConstRow * kSobolRowStride);
#pragma unroll
    for (int k = 0; k < (int)kSobolLowNibbles; ++k) {
      const uint4 b = *reinterpret_cast<const uint4*>(base + rows[k]);
      a.x ^= b.x;
      a.y ^= b.y;
      a.z ^= b.z;
      a.w ^= b.w;
    }
    x0 = a.x;
    x1 = a.y;
    x2 = a.z;
    x3 = a.w;
  }
  // Scrambled value of dimension d0 + K of the quad loaded at d0.
  template <int K>
  __device__ __forceinline__ uint32_t take(uint32_t) const {
    return __brev(lk_permute(K == 0 ? x0 : K == 1 ? x1 : K == 2 ? x2 : x3, K == 0 ? s0 : K == 1 ? s1 : K == 2 ? s2 : s3));
  }
  template <int K>
  __device__ __forceinline__ float take_n(uint32_t d0) const {
    return icdf_sobol_bits(icdf, take<K>(d0));
  }
  template <int K0, int K1>
  __device__ __forceinline__ float2 take_n2(uint32_t d0) const {
    return icdf_sobol_bits2(icdf, take<K0>(d0), take<K1>(d0));
  }
  __device__ __forceinline__ uint32_t sample(uint32_t d) {
    if ((d >> 2) != quad) quad_load(d & ~3u);
    const uint32_t k = d & 3u;
    return __brev(lk_permute((k & 2u) ? ((k & 1u) ? x3 : x2) : ((k & 1u) ? x1 : x0),
                             (k & 2u) ? ((k & 1u) ? s3 : s2) : ((k & 1u) ? s1 : s0)));
  }
  __device__ __forceinline__ float u32(uint32_t d) { return sobol_unit_f32_bits(sample(d)); }
  __device__ __forceinline__ float n32(uint32_t d) { return icdf_sobol_bits(icdf, sample(d)); }
};

// The FP64 plain path's Sobol samples: the staged window, FP64 inverse normal.
struct SobolPlain {
  SobolQuad s;
  const double* tail;
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx& c, uint64_t u) {
    s.template begin<true>(q, c, u);
    tail = c.tail;
  }
  __device__ __forceinline__ void at_step(uint32_t d0, uint32_t count) { s.at_step(d0, count); }
  __device__ __forceinline__ double n64(uint32_t d) { return icdf_sobol_f64(tail, s.sample(d)); }
  __device__ __forceinline__ double u64(uint32_t d) { return sobol_unit_f64(s.sample(d)); }
  __device__ __forceinline__ void quad_load(uint32_t d0) { s.quad_load(d0); }
  template <int K>
  __device__ __forceinline__ uint32_t take(uint32_t d0) const {
    return s.template take<K>(d0);
  }
  template <int K>
  __device__ __forceinline__ double take_n(uint32_t d0) const {
    return icdf_sobol_f64(tail, take<K>(d0));
  }
  template <int K0, int K1>
  __device__ __forceinline__ double2 take_n2(uint32_t d0) const {
    return make_double2(take_n<K0>(d0), take_n<K1>(d0));
  }
};

// Counter-hash normals for the fused kernels: the reference's u32 hashes with
// the short FP32 transform, two dimensions at a time where the model can.
template <bool HWCOS>
struct CounterFastT {
  uint32_t seed, unit, base;
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx&, uint64_t u) {
    seed = q.seed32;
    unit = (uint32_t)u;
    base = counter_mix(seed, unit, 0u, 0u);
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  __device__ __forceinline__ float n32(uint32_t d) { return counter_normal_fast<HWCOS>(seed, unit, d); }
  __device__ __forceinline__ float2 n2(uint32_t d) {
    return counter_normal_pair<HWCOS>(base ^ (d * 2891336453u), base ^ ((d + 1u) * 2891336453u));
  }
  __device__ __forceinline__ float u32(uint32_t d) {
    return counter_open01_fast(hash_u32(counter_mix(seed, unit, d, 0u)));
  }
  __device__ __forceinline__ double n64(uint32_t d) { return (double)counter_normal_f32(seed, unit, d); }
  __device__ __forceinline__ double u64(uint32_t d) {
    return (double)counter_open01(hash_u32(counter_mix(seed, unit, d, 0u)));
  }
};

// The MonteCarloRng stream a Box-Muller pair at a time: no cached-normal branch
// per sample, and the sine branch a unit with an odd start carries over stays
// in the path's precision.  Dimensions in increasing order.
__device__ __forceinline__ float2 make_pair2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ double2 make_pair2(double a, double b) { return make_double2(a, b); }
template <class Real>
struct XorshiftPairs {
  XorshiftStream st;
  Real carry;
  bool odd;  // the next normal is `carry`
  __device__ __forceinline__ auto pair() {
    if constexpr (sizeof(Real) == 4) {
      const float u1 = st.next_open01_f32(), u2 = st.next_open01_f32();
      const float r = sqrt_ftz(neg2_log_fast(u1));
      float s, c;
      // hardware sine and cosine of 2 pi (u2 - 1/2) in [-pi, pi], where their
      // documented error is 2^-21.4 absolute
      __sincosf(6.28318548f * (u2 - 0.5f), &s, &c);
      return make_float2(r * -c, r * -s);
    } else {
      st.has_cached = false;
      const double z = st.normal_f64();
      return make_double2(z, st.cached);
    }
  }
  // Starts from `aligned`, the state after 2 * (idx / 2) draws.
  __device__ __forceinline__ void start(uint64_t aligned, uint64_t idx) {
    st.state = aligned;
    odd = (idx & 1) != 0;
    carry = (Real)0;
    if (odd) carry = pair().y;
  }
  // All 32 lanes of the warp together.
  template <bool FP64>
  __device__ __forceinline__ void begin(const DevReq& q, const SrcCtx& c, uint64_t u) {
    uint64_t seed, local;
    chunk_of(q, u, &seed, &local);
    const uint64_t idx = local * q.normals_per_unit;
    start(xorshift_seek_warp(c.jump, seed, 2 * (idx >> 1)), idx);
  }
  __device__ __forceinline__ void at_step(uint32_t, uint32_t) {}
  __device__ __forceinline__ Real next() {
    if (odd) {
      odd = false;
      return carry;
    }
    const auto z = pair();
    odd = true;
    carry = z.y;
    return z.x;
  }
  __device__ __forceinline__ float n32(uint32_t) { return (float)next(); }
  __device__ __forceinline__ double n64(uint32_t) { return (double)next(); }
  __device__ __forceinline__ auto n2(uint32_t) {
    const auto z = pair();
    const auto out = odd ? make_pair2(carry, z.x) : z;
    carry = z.y;
    return out;
  }
};

// Sources with the explicit-quad interface (quad_load / take_n).
template <class S>
constexpr bool kQuadSource = false;
template <>
constexpr bool kQuadSource<SobolQuad> = true;
template <>
constexpr bool kQuadSource<SobolPlain> = true;

template <class S>
constexpr bool kCounterSource = false;
template <bool HWCOS>
constexpr bool kCounterSource<CounterFastT<HWCOS>> = true;

// Sources that give the normals of two consecutive dimensions at once (n2).
template <class S>
constexpr bool kPairSource = false;
template <int SMP>
struct LatticePairs;
template <int SMP>
constexpr bool kPairSource<LatticePairs<SMP>> = true;
template <bool HWCOS>
constexpr bool kPairSource<CounterFastT<HWCOS>> = true;
template <class Real>
constexpr bool kPairSource<XorshiftPairs<Real>> = true;

// Halton and Latin hypercube FP32 normals of two dimensions at once: the same
// values, with both samples' loads and chains in flight together (100,000 paths
// are 5 warps per scheduler, which waited on one sample's chain at 0.55 of the
// issue slots; 100,000 x 64 by device events 42.6 -> 37.0 us Halton, 44.7 ->
// 39.9 Latin hypercube).
template <int SMP>
struct LatticePairs : Source<SMP> {
  __device__ __forceinline__ float2 n2(uint32_t d) {
    float a, b;
    if constexpr (SMP == SMP_HALTON) {
      const double2 u = halton_f32_pair(this->index, this->dims + d);
      a = (float)u.x;
      b = (float)u.y;
    } else {
      a = this->u32(d);
      b = this->u32(d + 1);
    }
    a = fminf(fmaxf(a, 5.9604645e-08f), 0.99999994f);
    b = fminf(fmaxf(b, 5.9604645e-08f), 0.99999994f);
    return make_float2(normcdfinvf(a), normcdfinvf(b));
  }
};

template <int FAM, int SMP>
struct FusedUnitSource {
  using type = LatticePairs<SMP>;
};
template <int FAM>
struct FusedUnitSource<FAM, SMP_SOBOL> {
  using type = SobolQuad;
};
// The single-asset GBM families (one normal per step, the MUFU pipe about a
// third busy) take the hardware cosine; the others keep the polynomial.
template <int FAM>
struct FusedUnitSource<FAM, SMP_COUNTER> {
  using type = CounterFastT<FAM == FAM_GBM_STEP || FAM == FAM_GBM_TERMINAL>;
};
template <int FAM>
struct FusedUnitSource<FAM, SMP_XORSHIFT> {
  using type = XorshiftPairs<float>;
};

template <class Real, class Src>
__device__ __forceinline__ Real normal(Src& s, uint32_t d) {
  if constexpr (sizeof(Real) == 4)
    return s.n32(d);
  else
    return s.n64(d);
}

template <class Real>
__device__ __forceinline__ Real ex(Real x) {
  if constexpr (sizeof(Real) == 4)
    return __expf(x);
  else
    return exp(x);
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <class Real>
__device__ __forceinline__ Real sq_root(Real x) {
  if constexpr (sizeof(Real) == 4)
    return sqrt_approx(x);
  else
    return sqrt(x);
}

// sample_poisson by inversion with the uniform supplied (cpu.rs:932-953),
// entered only when u > exp(-mean) (at least one jump); p0 = exp(-mean) is
// precomputed on the host.
__device__ __forceinline__ uint32_t poisson_tail(double u, double mean, double p0) {
  double prob = p0, cum = p0;
  uint32_t k = 0;
  while (u > cum && k < 4095u) {
    ++k;
    prob *= mean / (double)k;
    cum += prob;
  }
  return k;
}

// ------------------------------------------------------- Brownian bridge ---
// fill_step_normals_from_inputs (cpu.rs:5964-5981) as a streaming walk: the
// reference fills w[0..n] op by op and then differences it; here the same
// ops run in the same (depth-first) order, but only the right endpoints still
// needed stay on a small stack (the nearest one in a register), and each step
// yields its increment (w[s] - w[s-1]) / sqrt(dt) at once.  Input dimensions are
// drawn in increasing order (0 = W(T), then one per op), a quad of them at a
// time; every thread of a request runs the same sequence, so the staged Sobol
// source stays in lockstep.  FP64 keeps the reference's two-rounding products
// and left-to-right sums.  The weights come in the path's precision (one
// 16-byte load an op) with the number of steps after the op in the fourth word,
// and the samples by quads.  Bound by latency (stack, weights and table loads at
// 5 warps per scheduler: 100,000 x 64 in FP32 62.2 us with the op counts in a
// table by step, a second load before each op, 57.8 so; the weights loaded one op
// ahead spilled at 64 registers: 76).
template <class Real, class Src>
struct BridgeWalk {
  static_assert(kQuadSource<Src>, "bridge paths are drawn from scrambled Sobol");
  Real stack[kBridgeDepth];
  Real w_left, top;
  Real z0, z1, z2, z3;  // the current quad's normals
  uint32_t sp, op, dim;

  __device__ __forceinline__ Real draw(Src& src) {
    const uint32_t k = dim & 3u;
    if (k == 0) {
      src.at_step(dim, 4);
      src.quad_load(dim);
      const auto a = src.template take_n2<0, 1>(dim), b = src.template take_n2<2, 3>(dim);
      z0 = a.x;
      z1 = a.y;
      z2 = b.x;
      z3 = b.y;
    }
    ++dim;
    return k & 2u ? (k & 1u ? z3 : z2) : (k & 1u ? z1 : z0);
  }
  __device__ __forceinline__ void begin(const DevReq& q, Src& src) {
    dim = 0;
    const Real z = draw(src);
    if constexpr (sizeof(Real) == 8)
      top = __dmul_rn(q.bridge_sqrt_t, z);
    else
      top = (Real)q.bridge_sqrt_t * z;
    sp = 0;
    w_left = (Real)0;
    op = 0;
  }
  // The next op; returns the steps after it (the host checked the program: it
  // never needs more than kBridgeDepth values).
  __device__ __forceinline__ uint32_t midpoint(const DevReq& q, Src& src) {
    uint32_t steps;
    if constexpr (sizeof(Real) == 8) {
      const double2* o = static_cast<const double2*>(q.bridge_ops) + 2 * op;
      const double2 w = __ldg(o), d = __ldg(o + 1);
      const Real z = draw(src);
      stack[sp++] = top;
      top = __dadd_rn(__dadd_rn(__dmul_rn(w.x, w_left), __dmul_rn(w.y, top)), __dmul_rn(d.x, z));
      steps = (uint32_t)d.y;
    } else {
      const float4 o = __ldg(static_cast<const float4*>(q.bridge_ops) + op);
      const Real z = draw(src);
      stack[sp++] = top;
      top = o.x * w_left + o.y * top + o.z * z;
      steps = (uint32_t)o.w;
    }
    ++op;
    return steps;
  }
  // The next step's increment.
  __device__ __forceinline__ Real step(const DevReq& q) {
    Real inc;
    if constexpr (sizeof(Real) == 8)
      inc = __dmul_rn(__dsub_rn(top, w_left), q.bridge_inv_sqrt_dt);
    else
      inc = (top - w_left) * (Real)q.bridge_inv_sqrt_dt;
    w_left = top;
    if (sp > 0) top = stack[--sp];
    return inc;
  }
};

// ------------------------------------------------------------- models -----
// GBM stepwise with the payoff observer of workload W (cpu.rs:6443-6591,
// 7973-8009, 8324-8354; up-and-out mirrors down-and-out).  FP32 compares the
// barrier in log space; FP64 compares exp(log S) with the barrier as the
// reference does.
template <class Real, int W, class Src, bool BRIDGE = false>
__device__ __forceinline__ void unit_gbm_step(const DevReq& q, Src& src, double& pay, double& ctl) {
  const Real drift = (Real)q.drift_dt, vol = (Real)q.vol_dt, kk = (Real)q.k, disc = (Real)q.discount;
  const Real lbar = (Real)q.log_barrier, bar = (Real)q.barrier;
  const bool anti = q.anti != 0;
  Real ls0 = (Real)q.log_s0, ls1 = ls0;
  Real acc0 = (W == W_LOOKBACK) ? (Real)q.s0 : (Real)0, acc1 = acc0;
  bool ko0 = (W == W_DAO && q.s0 <= q.barrier) || (W == W_UAO && q.s0 >= q.barrier), ko1 = ko0;
  const uint32_t n = q.n_steps;
  auto advance = [&](const Real z) {
    ls0 += drift + vol * z;
    if (anti) ls1 += drift - vol * z;
    if constexpr (W == W_ASIAN) {
      acc0 += ex<Real>(ls0);
      if (anti) acc1 += ex<Real>(ls1);
    } else if constexpr (W == W_LOOKBACK) {
      acc0 = acc0 > ex<Real>(ls0) ? acc0 : ex<Real>(ls0);
      if (anti) acc1 = acc1 > ex<Real>(ls1) ? acc1 : ex<Real>(ls1);
    } else if constexpr (W == W_DAO) {
      if constexpr (sizeof(Real) == 4) {
        ko0 |= ls0 <= lbar;
        if (anti) ko1 |= ls1 <= lbar;
      } else {
        ko0 |= ex<Real>(ls0) <= bar;
        if (anti) ko1 |= ex<Real>(ls1) <= bar;
      }
    } else if constexpr (W == W_UAO) {
      if constexpr (sizeof(Real) == 4) {
        ko0 |= ls0 >= lbar;
        if (anti) ko1 |= ls1 >= lbar;
      } else {
        ko0 |= ex<Real>(ls0) >= bar;
        if (anti) ko1 |= ex<Real>(ls1) >= bar;
      }
    }
  };
  uint32_t s = 0;
  if constexpr (BRIDGE) {  // increments from the Brownian bridge over the inputs
    BridgeWalk<Real, Src> bw;
    bw.begin(q, src);
    uint32_t steps = n == 1 ? 1u : 0u;  // a longer path starts with an op
    for (;;) {
      for (; steps > 0; --steps) advance(bw.step(q));
      if (++s >= n) break;  // n - 1 ops in all
      steps = bw.midpoint(q, src);
    }
    s = n;
  } else if constexpr (kQuadSource<Src>) {
    for (; s + 4 <= n; s += 4) {  // four steps per quad of dimensions
      src.at_step(s, 4);
      src.quad_load(s);
      const auto z01 = src.template take_n2<0, 1>(s), z23 = src.template take_n2<2, 3>(s);
      advance(z01.x);
      advance(z01.y);
      advance(z23.x);
      advance(z23.y);
    }
  } else if constexpr (kPairSource<Src>) {
    for (; s + 2 <= n; s += 2) {
      const auto z = src.n2(s);
      advance(z.x);
      advance(z.y);
    }
  }
  for (; s < n; ++s) {
    src.at_step(s, 1);
    advance(normal<Real>(src, s));
  }
  auto payoff = [&](Real ls, Real acc, bool ko) -> Real {
    Real v;
    if constexpr (W == W_ASIAN) {
      if constexpr (sizeof(Real) == 4)
        v = acc * (Real)(1.0 / (double)n) - kk;
      else
        v = acc / (Real)n - kk;
    } else if constexpr (W == W_LOOKBACK) {
      v = acc - kk;
    } else {
      v = ex<Real>(ls) - kk;
      if (ko) v = 0;
    }
    return (v > (Real)0 ? v : (Real)0) * disc;
  };
  Real p0 = payoff(ls0, acc0, ko0);
  if (anti) {
    Real p1 = payoff(ls1, acc1, ko1);
    pay = 0.5 * ((double)p0 + (double)p1);
  } else {
    pay = (double)p0;
  }
  ctl = (double)(disc * ex<Real>(ls0));
}

// GBM terminal European (european_call_payoff_from_shock, cpu.rs:7773-7783).
template <class Real, class Src>
__device__ __forceinline__ void unit_gbm_terminal(const DevReq& q, Src& src, double& pay, double& ctl) {
  src.at_step(0, 1);
  const Real z = normal<Real>(src, 0);
  const Real s0 = (Real)q.s0, drift = (Real)q.drift_dt, vol = (Real)q.vol_dt, kk = (Real)q.k,
             disc = (Real)q.discount;
  Real st = s0 * ex<Real>(drift + vol * z);
  Real p = (st - kk > (Real)0 ? st - kk : (Real)0) * disc;
  if (q.anti) {
    Real sb = s0 * ex<Real>(drift + vol * (-z));
    Real pb = (sb - kk > (Real)0 ? sb - kk : (Real)0) * disc;
    pay = 0.5 * ((double)p + (double)pb);
  } else {
    pay = (double)p;
  }
  ctl = (double)(disc * st);
}

// Heston Euler with the variance floored after every step (heston_path_terminal, cpu.rs:8667-8686).
template <class Real, class Src>
__device__ __forceinline__ void unit_heston(const DevReq& q, Src& src, double& pay, double& ctl) {
  const Real kappa = (Real)q.kappa, theta = (Real)q.theta, xi = (Real)q.xi, rho = (Real)q.rho,
             rho_perp = (Real)q.rho_perp, dt = (Real)q.dt, sqdt = (Real)q.sqrt_dt, rate = (Real)q.rate;
  const bool anti = q.anti != 0;
  Real ls0 = (Real)q.log_s0, ls1 = ls0, v0 = (Real)q.v0, v1 = v0;
  const uint32_t n = q.n_steps;
  // FP32 path: the same update with the step constants folded on the host
  // (rate dt, dt / 2, kappa dt, kappa theta dt, xi sqrt(dt)) and FMAs; the
  // variance is floored after every step and starts >= 0 (validated), so it
  // needs no floor before use.  The FP64 path keeps the reference's form.
  // (Rearranged into fewer instructions -- the drift of all steps folded into
  // the start, 1 - kappa dt, rho sqrt(dt) -- it measured 2.5% slower: two
  // dependent FMAs on the log-price per step instead of one add.)
  const float c_rdt = (float)(q.rate * q.dt), c_hdt = (float)(0.5 * q.dt), c_kdt = (float)(q.kappa * q.dt),
              c_ktdt = (float)(q.kappa * q.theta * q.dt), c_xsq = (float)(q.xi * q.sqrt_dt);
  auto step_f32 = [&](float& ls, float& v, const float zv, const float zi) {
    const float sv = sqrt_approx(v);
    const float zp = fmaf(rho, zv, rho_perp * zi);
    ls += fmaf(sv * sqdt, zp, fmaf(-c_hdt, v, c_rdt));
    const float vn = fmaf(c_xsq * sv, zv, v + fmaf(-c_kdt, v, c_ktdt));
    v = vn > 0.0f ? vn : 0.0f;
  };
  auto step = [&](const Real zv, const Real zi) {
    if constexpr (sizeof(Real) == 4) {
      step_f32(ls0, v0, zv, zi);
      if (anti) step_f32(ls1, v1, -zv, -zi);
      return;
    }
    {
      Real vp = v0 > (Real)0 ? v0 : (Real)0;
      Real sv = sq_root<Real>(vp);
      Real zp = rho * zv + rho_perp * zi;
      ls0 += (rate - (Real)0.5 * vp) * dt + sv * sqdt * zp;
      v0 = v0 + kappa * (theta - vp) * dt + xi * sv * sqdt * zv;
      v0 = v0 > (Real)0 ? v0 : (Real)0;
    }
    if (anti) {
      Real vp = v1 > (Real)0 ? v1 : (Real)0;
      Real sv = sq_root<Real>(vp);
      Real zp = rho * (-zv) + rho_perp * (-zi);
      ls1 += (rate - (Real)0.5 * vp) * dt + sv * sqdt * zp;
      v1 = v1 + kappa * (theta - vp) * dt + xi * sv * sqdt * (-zv);
      v1 = v1 > (Real)0 ? v1 : (Real)0;
    }
  };
  uint32_t s = 0;
  if constexpr (kQuadSource<Src>) {
    for (; s + 2 <= n; s += 2) {  // two steps per quad: dimensions 2s .. 2s + 3
      const uint32_t d0 = 2 * s;
      src.at_step(d0, 4);
      src.quad_load(d0);
      const auto z01 = src.template take_n2<0, 1>(d0), z23 = src.template take_n2<2, 3>(d0);
      step(z01.x, z01.y);
      step(z23.x, z23.y);
    }
  } else if constexpr (kPairSource<Src>) {
    // four steps a turn, so that the next samples are under way beside a step's
    // chain: 5,000 x 365 on the counter hash 114 -> 82 us (rolled by the compiler
    // otherwise; 89 with single samples), 1,048,576 x 64 320 -> 286, pseudorandom
    // and Halton within 2%; eight steps a turn give no more
#pragma unroll 4
    for (; s < n; ++s) {
      const auto z = src.n2(2 * s);
      step(z.x, z.y);
    }
  }
  for (; s < n; ++s) {
    src.at_step(2 * s, 2);
    const Real zv = normal<Real>(src, 2 * s);
    const Real zi = normal<Real>(src, 2 * s + 1);
    step(zv, zi);
  }
  const Real kk = (Real)q.k, disc = (Real)q.discount;
  Real st = ex<Real>(ls0);
  Real p = (st - kk > (Real)0 ? st - kk : (Real)0) * disc;
  if (anti) {
    Real sb = ex<Real>(ls1);
    Real pb = (sb - kk > (Real)0 ? sb - kk : (Real)0) * disc;
    pay = 0.5 * ((double)p + (double)pb);
  } else {
    pay = (double)p;
  }
  ctl = (double)(st * disc);
}

// Merton: stepwise extension (z, u, z_J per step) and the reference terminal
// form (cpu.rs:6408-6441) with dims (z, u, z_J).
template <class Real, bool STEP, class Src>
__device__ __forceinline__ void unit_merton(const DevReq& q, Src& src, double& pay, double& ctl) {
  const Real drift = (Real)q.drift_dt, vol = (Real)q.vol_dt, jm = (Real)q.jump_mean, jv = (Real)q.jump_vol;
  Real ls = (Real)q.log_s0;
  const uint32_t n = STEP ? q.n_steps : 1;
  uint32_t s0 = 0;
  // The FP32 Sobol path adds the deterministic drift of all n steps to the
  // start (only the terminal log-price is read), so a step is one FMA.
  constexpr bool kFold = kQuadSource<Src> && sizeof(Real) == 4;
  if constexpr (kFold) ls = (float)(q.log_s0 + q.drift_dt * (double)n);
  if constexpr (kQuadSource<Src>) {
    // four steps per three quads: step k of the chunk uses dimensions
    // d0 + 3k (z), d0 + 3k + 1 (Poisson uniform), d0 + 3k + 2 (jump normal)
    // xu: the scrambled 32-bit Poisson sample; its top 23 bits against the
    // integer thresholds give the jump count of sample_poisson exactly (the
    // FP64 inversion only from four jumps on)
    // (xu >> 9) >= m0 exactly when xu >= m0 << 9 (m0 < 2^23): the shift
    // leaves the common no-jump case.  m0 = 2^23 (no sample jumps) lets at
    // most the largest sample in, which then counts no jump.
    const uint32_t pois_x0 = q.pois_m[0] >= 0x800000u ? 0xFFFFFFFFu : q.pois_m[0] << 9;
    auto step = [&](const Real z, const uint32_t xu, auto&& jump_normal) {
      if constexpr (kFold)
        ls = fmaf(vol, z, ls);
      else
        ls += drift + vol * z;
      if (xu >= pois_x0) {
        const uint32_t mu = xu >> 9;
        uint32_t jumps = (mu >= q.pois_m[0] ? 1u : 0u) + (mu >= q.pois_m[1] ? 1u : 0u) + (mu >= q.pois_m[2] ? 1u : 0u) + (mu >= q.pois_m[3] ? 1u : 0u);
        if (jumps == 4u) jumps = poisson_tail(sobol_unit_f64(xu), q.lam_dt, q.lam_p0);
        ls += (Real)jumps * jm + jv * sq_root<Real>((Real)jumps) * jump_normal();
      }
    };
    for (; s0 + 4 <= n; s0 += 4) {
      const uint32_t d0 = 3 * s0;
      src.at_step(d0, 12);
      src.quad_load(d0);
      const Real z0 = src.template take_n<0>(d0);
      const uint32_t u0 = src.template take<1>(d0);
      step(z0, u0, [&] { return src.template take_n<2>(d0); });
      const Real z1 = src.template take_n<3>(d0);
      src.quad_load(d0 + 4);
      const uint32_t u1 = src.template take<0>(d0 + 4);
      step(z1, u1, [&] { return src.template take_n<1>(d0 + 4); });
      const Real z2 = src.template take_n<2>(d0 + 4);
      const uint32_t u2 = src.template take<3>(d0 + 4);
      src.quad_load(d0 + 8);
      step(z2, u2, [&] { return src.template take_n<0>(d0 + 8); });
      step(src.template take_n<1>(d0 + 8), src.template take<2>(d0 + 8),
           [&] { return src.template take_n<3>(d0 + 8); });
    }
  }
  for (uint32_t s = s0; s < n; ++s) {
    src.at_step(3 * s, 3);
    const Real z = normal<Real>(src, 3 * s);
    uint32_t jumps;
    if constexpr (sizeof(Real) == 4) {
      const float u = src.u32(3 * s + 1);
      jumps = u <= q.lam_p0_f ? 0u : poisson_tail((double)u, q.lam_dt, q.lam_p0);
    } else {
      const double u = src.u64(3 * s + 1);
      jumps = u <= q.lam_p0 ? 0u : poisson_tail(u, q.lam_dt, q.lam_p0);
    }
    if constexpr (kFold)
      ls = fmaf(vol, z, ls);
    else
      ls += drift + vol * z;
    if (jumps > 0) {
      const Real zj = normal<Real>(src, 3 * s + 2);
      ls += (Real)jumps * jm + jv * sq_root<Real>((Real)jumps) * zj;
    }
  }
  const Real kk = (Real)q.k, disc = (Real)q.discount;
  Real st = ex<Real>(ls);
  pay = (double)((st - kk > (Real)0 ? st - kk : (Real)0) * disc);
  ctl = (double)(st * disc);
}

// FP64 Halton and Latin hypercube normals are long (a digit loop or a hash, a
// division, the inverse normal with its tail): the normals of a step are one copy
// of that code in a loop, since a copy per asset passes the instruction cache.
// Copies -> loop: 8 assets, 4,000,000 x 3 Halton 6,734 -> 1,539 us and 300,000 x 64
// Latin hypercube 3,450 -> 1,987; 5 assets, 1,000,000 x 20 Halton 2,103 -> 957;
// 3 assets, 4,000,000 x 3 885 -> 720; 2 assets 511 -> 502 there but 183 -> 191 at
// 100,000 x 64.  Called out of line instead of a loop: 10 to 25% slower.
template <class S>
constexpr bool kLongSample = false;
template <>
constexpr bool kLongSample<Source<SMP_HALTON>> = true;
template <>
constexpr bool kLongSample<Source<SMP_LHS>> = true;

// Sums over n steps of a path's D normals per step.  FP32 samples are summed
// in FP32 over four steps at a time and in FP64 from there on: a sum of
// hundreds of normals grows to 10 or 20, where FP32 adds lose 5e-7 each (a
// 154,595 x 290 basket of small price: 2.7e-6 off with FP32 sums).
template <class Real, int D, class Src>
__device__ __forceinline__ void sum_step_normals(Src& src, uint32_t n, Real zs[D]) {
  double total[D];
#pragma unroll
  for (int a = 0; a < D; ++a) total[a] = 0.0;
  uint32_t dim = 0, s = 0;
  if constexpr (sizeof(Real) == 4) {
    for (; s + 4 <= n; s += 4) {
      float part[D];
#pragma unroll
      for (int a = 0; a < D; ++a) part[a] = 0.0f;
      if constexpr (kPairSource<Src>) {
#pragma unroll 1
        for (int h = 0; h < 2; ++h) {  // two steps are D pairs whatever D's parity
#pragma unroll
          for (int p = 0; p < D; ++p) {
            const auto z = src.n2(dim + 2 * p);
            part[(2 * p) % D] += z.x;
            part[(2 * p + 1) % D] += z.y;
          }
          dim += 2 * D;
        }
      } else {
#pragma unroll 1
        for (int h = 0; h < 4; ++h) {
          src.at_step(dim, D);
#pragma unroll
          for (int a = 0; a < D; ++a) part[a] += normal<Real>(src, dim + a);
          dim += D;
        }
      }
#pragma unroll
      for (int a = 0; a < D; ++a) total[a] += (double)part[a];
    }
  }
  for (; s < n; ++s) {
    src.at_step(dim, D);
    if constexpr (sizeof(Real) == 8 && D > 1 && kLongSample<Src>) {
      double z[D];
#pragma unroll 1
      for (int a = 0; a < D; ++a) z[a] = normal<Real>(src, dim + a);
#pragma unroll
      for (int a = 0; a < D; ++a) total[a] += z[a];
    } else {
#pragma unroll
      for (int a = 0; a < D; ++a) total[a] += (double)normal<Real>(src, dim + a);
    }
    dim += D;
  }
#pragma unroll
  for (int a = 0; a < D; ++a) zs[a] = (Real)total[a];
}

// d-asset basket, terminal or stepwise (basket_terminal_payoff, cpu.rs:7616-7635),
// for a compile-time asset count D.  The payoff reads terminal values only and
// the log returns are linear in the normals, so a path keeps the D sums of its
// normals over the steps and correlates them once at the end:
// sum_steps (drift + vol (L z)_a) = n drift + vol (L sum_steps z)_a.  A step is
// then D normals and D adds; correlating every step cost D (D + 1) / 2 + 2 D
// more and held the Cholesky factor in registers through the whole path (64
// registers a thread: 356 bytes spilled with D up to 8).  1.6e9 normals of
// 5-asset baskets: 3,829 us, 3,211 us so, 2,434 us with the normals in pairs.
// On the counter hash the final loop takes two assets a turn: whole, it spilled
// 100 bytes inside the path (2,534 us); on the pseudorandom stream whole is up
// to 9% faster.
template <class Real, int D, class Src>
__device__ __forceinline__ void unit_basket_d(const DevReq& q, Src& src, double& pay, double& ctl) {
  const uint32_t n = q.n_steps;
  Real zs[D];
  sum_step_normals<Real, D>(src, n, zs);
  Real b0 = 0, b1 = 0;
  constexpr int kTurn = kCounterSource<Src> ? 2 : D;  // assets a turn
#pragma unroll kTurn
  for (int a = 0; a < D; ++a) {
    Real w = (Real)0;
#pragma unroll
    for (int b = 0; b <= a; ++b) w += (Real)q.chol[a * D + b] * zs[b];
    const Real drift = (Real)(q.b_drift[a] * (double)n), vol = (Real)q.b_vol[a];
    b0 += (Real)q.weights[a] * ((Real)q.spots[a] * ex<Real>(drift + vol * w));
    if (q.anti) b1 += (Real)q.weights[a] * ((Real)q.spots[a] * ex<Real>(drift - vol * w));
  }
  const Real kk = (Real)q.k, disc = (Real)q.discount;
  Real p = (b0 - kk > (Real)0 ? b0 - kk : (Real)0) * disc;
  if (q.anti) {
    Real pb = (b1 - kk > (Real)0 ? b1 - kk : (Real)0) * disc;
    pay = 0.5 * ((double)p + (double)pb);
  } else {
    pay = (double)p;
  }
  ctl = (double)(b0 * disc);
}

template <class Real, class Src>
__device__ __forceinline__ void unit_basket(const DevReq& q, Src& src, double& pay, double& ctl) {
  switch (q.n_assets) {
    case 1:
      unit_basket_d<Real, 1>(q, src, pay, ctl);
      break;
    case 2:
      unit_basket_d<Real, 2>(q, src, pay, ctl);
      break;
    case 3:
      unit_basket_d<Real, 3>(q, src, pay, ctl);
      break;
    case 4:
      unit_basket_d<Real, 4>(q, src, pay, ctl);
      break;
    case 5:
      unit_basket_d<Real, 5>(q, src, pay, ctl);
      break;
    case 6:
      unit_basket_d<Real, 6>(q, src, pay, ctl);
      break;
    case 7:
      unit_basket_d<Real, 7>(q, src, pay, ctl);
      break;
    default:
      unit_basket_d<Real, 8>(q, src, pay, ctl);
      break;
  }
}

// Coupled MLMC level of the arithmetic Asian (cpu.rs:6641-6894): level 0 is
// the plain Asian with the base steps; level l couples M fine normals per
// coarse step with a coarse path driven by sum(z)/sqrt(M).
template <class Real, class Src>
__device__ __forceinline__ void unit_mlmc(const DevReq& q, Src& src, double& pay, double& ctl) {
  const Real kk = (Real)q.k, disc = (Real)q.discount;
  ctl = 0.0;
  if (q.level == 0) {
    const Real drift = (Real)q.f_drift, vol = (Real)q.f_vol;
    Real ls = (Real)q.log_s0, acc = 0;
    auto advance = [&](const Real z) {
      ls += drift + vol * z;
      acc += ex<Real>(ls);
    };
    uint32_t s = 0;
    if constexpr (kPairSource<Src>) {
      for (; s + 2 <= q.n_steps; s += 2) {
        const auto z = src.n2(s);
        advance(z.x);
        advance(z.y);
      }
    }
    for (; s < q.n_steps; ++s) {
      src.at_step(s, 1);
      advance(normal<Real>(src, s));
    }
    Real avg;
    if constexpr (sizeof(Real) == 4)
      avg = acc * (Real)q.inv_fine;
    else
      avg = acc / (Real)q.n_steps;
    pay = (double)((avg - kk > (Real)0 ? avg - kk : (Real)0) * disc);
    return;
  }
  const Real fd = (Real)q.f_drift, fv = (Real)q.f_vol, cd = (Real)q.c_drift, cv = (Real)q.c_vol;
  const uint32_t M = q.refinement;
  Real fl = (Real)q.log_s0, cl = fl, fs = 0, cs = 0;
  uint32_t j = 0;
  for (uint64_t c = 0; c < q.coarse_steps; ++c) {
    Real zsum = 0;
    auto fine = [&](const Real z) {
      zsum += z;
      fl += fd + fv * z;
      fs += ex<Real>(fl);
    };
    uint32_t m = 0;
    if constexpr (kPairSource<Src>) {
      for (; m + 2 <= M; m += 2, j += 2) {
        const auto z = src.n2(j);
        fine(z.x);
        fine(z.y);
      }
    }
    for (; m < M; ++m) {
      src.at_step(j, 1);  // one dimension at a time: M may exceed what a window step holds
      fine(normal<Real>(src, j++));
    }
    Real zc;
    if constexpr (sizeof(Real) == 4)
      zc = zsum * (Real)q.inv_sqrt_m;
    else
      zc = zsum / sqrt((double)M);
    cl += cd + cv * zc;
    cs += ex<Real>(cl);
  }
  Real fa, ca;
  if constexpr (sizeof(Real) == 4) {
    fa = fs * (Real)q.inv_fine;
    ca = cs * (Real)q.inv_coarse;
  } else {
    fa = fs / (Real)q.n_steps;
    ca = cs / (Real)q.coarse_steps;
  }
  Real pf = (fa - kk > (Real)0 ? fa - kk : (Real)0) * disc;
  Real pc = (ca - kk > (Real)0 ? ca - kk : (Real)0) * disc;
  pay = (double)pf - (double)pc;
}

template <class Real, int FAM, class Src>
__device__ __forceinline__ void run_family(const DevReq& q, Src& src, double& p, double& c) {
  if constexpr (FAM == FAM_GBM_BRIDGE) {
    switch (q.workload) {
      case W_ASIAN:
        unit_gbm_step<Real, W_ASIAN, Src, true>(q, src, p, c);
        break;
      case W_DAO:
        unit_gbm_step<Real, W_DAO, Src, true>(q, src, p, c);
        break;
      case W_UAO:
        unit_gbm_step<Real, W_UAO, Src, true>(q, src, p, c);
        break;
      case W_LOOKBACK:
        unit_gbm_step<Real, W_LOOKBACK, Src, true>(q, src, p, c);
        break;
      default:
        unit_gbm_step<Real, W_EURO, Src, true>(q, src, p, c);
        break;
    }
  } else if constexpr (FAM == FAM_GBM_STEP) {
    switch (q.workload) {
      case W_ASIAN:
        unit_gbm_step<Real, W_ASIAN>(q, src, p, c);
        break;
      case W_DAO:
        unit_gbm_step<Real, W_DAO>(q, src, p, c);
        break;
      case W_UAO:
        unit_gbm_step<Real, W_UAO>(q, src, p, c);
        break;
      case W_LOOKBACK:
        unit_gbm_step<Real, W_LOOKBACK>(q, src, p, c);
        break;
      default:
        unit_gbm_step<Real, W_EURO>(q, src, p, c);
        break;
    }
  } else if constexpr (FAM == FAM_GBM_TERMINAL) {
    unit_gbm_terminal<Real>(q, src, p, c);
  } else if constexpr (FAM == FAM_HESTON) {
    unit_heston<Real>(q, src, p, c);
  } else if constexpr (FAM == FAM_MERTON_STEP) {
    unit_merton<Real, true>(q, src, p, c);
  } else if constexpr (FAM == FAM_MERTON_TERMINAL) {
    unit_merton<Real, false>(q, src, p, c);
  } else if constexpr (FAM == FAM_BASKET) {
    unit_basket<Real>(q, src, p, c);
  } else {
    unit_mlmc<Real>(q, src, p, c);
  }
}

// ----------------------------------------------------- block reduction ----
constexpr int kFusedBlock = 256;
constexpr int kWarps = kFusedBlock / 32;
// The fused pricing kernel runs 128-, 256- or 512-thread blocks (the
// autotuner's choice); its launch bounds are written for 512 threads.
constexpr int kMaxFusedBlock = 512;
constexpr int kMaxWarps = kMaxFusedBlock / 32;

// Reduces v[0..4] over the block in a fixed order; result valid in thread 0.
// The leading barrier keeps a previous call's reader of `red` safe, so calls
// may follow each other directly.
__device__ __forceinline__ void block_reduce5(double v[5], double (*red)[5]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
  for (int i = 0; i < 5; ++i) v[i] = warp_sum(v[i]);
  __syncthreads();
  if (lane == 0) {
#pragma unroll
    for (int i = 0; i < 5; ++i) red[warp][i] = v[i];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    const int warps = (blockDim.x + 31) >> 5;
    for (int i = 0; i < 5; ++i) {
      double s = 0.0;
      for (int w = 0; w < warps; ++w) s += red[w][i];
      v[i] = s;
    }
  }
}

// Sums the request's tile partials in tile order (strided per thread, then a
// fixed block tree) into q.moments.  Called by the block that finished the
// request's last tile.
static __device__ void finalize_request(const DevReq& q, double (*red)[5]) {
  double v[5] = {0, 0, 0, 0, 0};
#pragma unroll 4
  for (uint32_t t = threadIdx.x; t < q.n_tiles; t += blockDim.x) {
    const double* pt = q.partials + (size_t)t * MPC_MOMENTS;
#pragma unroll
    for (int i = 0; i < 5; ++i) v[i] += __ldcg(pt + 1 + i);
  }
  block_reduce5(v, red);
  if (threadIdx.x == 0) {
    q.moments[0] = (double)q.n_units;  // the tiles cover every unit once
    for (int i = 0; i < 5; ++i) q.moments[1 + i] = v[i];
    q.moments[6] = 0.0;
    q.moments[7] = 0.0;
    *q.tiles_done = 0u;  // reusable without a memset
  }
}

}  // namespace mpc
