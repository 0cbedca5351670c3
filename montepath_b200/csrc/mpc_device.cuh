// mpc_device.cuh -- device-side generators, inverse CDF and reductions of the
// B200 Monte Carlo backend.  Everything here is evaluated in registers inside
// the pricing kernels; no sample is written to memory.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mpc_types.h"

namespace mpc {

// ----------------------------------------------------------- xorshift64* --
// MonteCarloRng (crates/mc-core/src/runtime/cpu.rs:2955-3007) replayed on the
// device.  The state transition x -> x^(x>>12), ^(x<<25), ^(x>>27) is linear
// over GF(2), so T^k is a 64x64 bit matrix.  The host tabulates
// T^(2^b) for b = 0..63 in nibble form: jump[b][q][v] = T^(2^b) applied to
// the nibble value v placed at bit position 4q.  Jumping k draws ahead costs
// popcount(k) * 16 table lookups.
__device__ __forceinline__ uint64_t gf2_apply(const uint64_t* __restrict__ table, uint64_t x) {
  uint64_t y = 0;
#pragma unroll
  for (int q = 0; q < 16; ++q) y ^= __ldg(table + q * 16 + ((x >> (4 * q)) & 0xF));
  return y;
}

__device__ __forceinline__ uint64_t xorshift_jump(const uint64_t* __restrict__ nibble, uint64_t state,
                                                  uint64_t k) {
  while (k) {
    int b = __ffsll((long long)k) - 1;
    state = gf2_apply(nibble + (size_t)b * 256, state);
    k &= k - 1;
  }
  return state;
}

// xorshift_jump by a count that is the same for the whole warp, all 32 lanes
// calling together: lane q looks up nibble q and two warp reductions combine
// the 16 images, about 12 instructions per set bit instead of about 100.
__device__ __forceinline__ uint64_t xorshift_jump_uniform(const uint64_t* __restrict__ nibble, uint64_t state,
                                                          uint64_t k) {
  const uint32_t lane = threadIdx.x & 31u, q = lane & 15u;
  while (k) {
    const int b = __ffsll((long long)k) - 1;
    uint64_t y = __ldg(nibble + (size_t)b * 256 + q * 16 + ((state >> (4 * q)) & 0xF));
    if (lane >= 16) y = 0;
    state = ((uint64_t)__reduce_xor_sync(0xFFFFFFFFu, (uint32_t)(y >> 32)) << 32) |
            __reduce_xor_sync(0xFFFFFFFFu, (uint32_t)y);
    k &= k - 1;
  }
  return state;
}

// xorshift_jump for a whole warp (all 32 lanes call it together) whose lanes
// start from one state and jump k = k0 + d draws, k0 lane 0's and d >= 0
// small: the common k0 by the uniform jump, then every set bit of any d with
// all lanes on the same table, whose 16-entry rows are one 128-byte line each.
// Jumping lane by lane, one iteration touches a table per distinct bit.
__device__ __forceinline__ uint64_t xorshift_jump_warp(const uint64_t* __restrict__ nibble, uint64_t state, uint64_t k) {
  const uint64_t k0 = __shfl_sync(0xFFFFFFFFu, k, 0);
  state = xorshift_jump_uniform(nibble, state, k0);
  const uint64_t d = k - k0;
  uint64_t any = ((uint64_t)__reduce_or_sync(0xFFFFFFFFu, (uint32_t)(d >> 32)) << 32) |
                 __reduce_or_sync(0xFFFFFFFFu, (uint32_t)d);
  while (any) {
    const int b = __ffsll((long long)any) - 1;
    const uint64_t y = gf2_apply(nibble + (size_t)b * 256, state);
    if ((d >> b) & 1u) state = y;
    any &= any - 1;
  }
  return state;
}
// The state `k` draws into the stream of `seed`, for all lanes of a warp at
// once: by the shared jump when the lanes follow one stream forward, else
// (a chunk edge inside the warp) lane by lane.
__device__ __forceinline__ uint64_t xorshift_seek_warp(const uint64_t* __restrict__ nibble, uint64_t seed, uint64_t k) {
  const uint64_t first = seed == 0 ? 0x9E3779B97F4A7C15ull : seed;  // MonteCarloRng replaces seed 0
  // both shuffles before any test: every lane takes part in each
  const uint64_t first0 = __shfl_sync(0xFFFFFFFFu, first, 0), k0 = __shfl_sync(0xFFFFFFFFu, k, 0);
  return __all_sync(0xFFFFFFFFu, first == first0 && k >= k0) ? xorshift_jump_warp(nibble, first, k) : xorshift_jump(nibble, first, k);
}

// Sequential MonteCarloRng positioned at an arbitrary normal index.
__device__ __forceinline__ float neg2_log_fast(float u);

struct XorshiftStream {
  uint64_t state;
  double cached;
  bool has_cached;

  __device__ __forceinline__ uint64_t next_u64() {
    uint64_t x = state;
    x ^= x >> 12;
    x ^= x << 25;
    x ^= x >> 27;
    state = x;
    return x * 0x2545F4914F6CDD1Dull;
  }
  __device__ __forceinline__ double next_open01() {
    uint64_t raw = next_u64() >> 11;
    double v = (double)raw * (1.0 / 9007199254740992.0);
    return fmax(v, 2.2250738585072014e-308);
  }
  // The same uniform rounded to FP32: (float)((double)(raw >> 11) * 2^-53)
  // is one rounding of the 53-bit integer, which the direct conversion does
  // too (the scale is an exact power of two; raw = 0 gives 0 either way).
  __device__ __forceinline__ float next_open01_f32() {
    return __ull2float_rn(next_u64() >> 11) * 1.1102230246251565e-16f;
  }
  // Box-Muller in FP64 (cpu.rs:2992-3006): returns cos branch, caches sin branch.
  __device__ __forceinline__ double normal_f64() {
    if (has_cached) {
      has_cached = false;
      return cached;
    }
    double u1 = next_open01();
    double u2 = next_open01();
    double radius = sqrt(-2.0 * log(u1));
    double s, c;
    sincospi(2.0 * u2, &s, &c);  // exact argument reduction (the reference rounds 2 pi u2 first)
    cached = radius * s;
    has_cached = true;
    return radius * c;
  }
  // Same draw with the Box-Muller transform evaluated in FP32: the integer
  // stream and the uniforms (rounded to f32) are the reference's.
  __device__ __forceinline__ float normal_f32() {
    if (has_cached) {
      has_cached = false;
      return (float)cached;
    }
    // FP32 path: the stream's uniforms with the short Box-Muller of the
    // counter-hash normals (atanh series near 1 / hardware log2, approximate
    // square root) and the hardware sine and cosine of 2 pi (u2 - 1/2) in
    // [-pi, pi], where their documented error is 2^-21.4 absolute:
    // sin / cos (2 pi u2) = -sin / -cos (2 pi (u2 - 1/2)).
    const float u1 = next_open01_f32();
    const float u2 = next_open01_f32();
    float radius;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(radius) : "f"(neg2_log_fast(u1)));
    float s, c;
    __sincosf(6.28318548f * (u2 - 0.5f), &s, &c);
    cached = (double)(radius * -s);
    has_cached = true;
    return radius * -c;
  }
  // First state of the stream of `seed` (MonteCarloRng replaces seed 0).
  __device__ __forceinline__ static uint64_t first_state(uint64_t seed) { return seed == 0 ? 0x9E3779B97F4A7C15ull : seed; }
  // Starts from `aligned`, the state after 2 * (normal_index / 2) draws, so
  // that the next normal is normal number `normal_index` (an odd index first
  // draws the pair and keeps its second normal).
  __device__ __forceinline__ void seek_aligned(uint64_t aligned, uint64_t normal_index, bool fp32) {
    state = aligned;
    has_cached = false;
    if (normal_index & 1) {
      if (fp32)
        (void)normal_f32();
      else
        (void)normal_f64();
    }
  }
  // Position the stream of `seed` so that the next normal is normal number
  // `normal_index` of the sequential stream.
  __device__ __forceinline__ void seek(const uint64_t* __restrict__ nibble, uint64_t seed,
                                       uint64_t normal_index, bool fp32) {
    seek_aligned(xorshift_jump(nibble, first_state(seed), 2 * (normal_index >> 1)), normal_index, fp32);
  }
};

__host__ __device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
  x += 0x9E3779B97F4A7C15ull;
  uint64_t z = x;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// derive_chunk_seed (cpu.rs:8922-8924)
__host__ __device__ __forceinline__ uint64_t derive_chunk_seed(uint64_t base, uint64_t idx) {
  return splitmix64(base + idx * 0x9E3779B97F4A7C15ull);
}

// The reference's CPU thread split (cpu.rs:6232-6276): `chunks` streams of
// base or base+1 units, the first `rem` chunks one larger.  Maps a global
// unit index to (chunk seed, index inside the chunk).
__device__ __forceinline__ void chunk_of(const DevReq& q, uint64_t unit, uint64_t* seed, uint64_t* local) {
  if (q.n_chunks <= 1) {
    *seed = q.seed;
    *local = unit;
    return;
  }
  uint64_t big = q.chunk_rem * (q.chunk_base + 1);
  uint64_t c;
  if (unit < big) {
    c = unit / (q.chunk_base + 1);
    *local = unit - c * (q.chunk_base + 1);
  } else {
    c = q.chunk_rem + (unit - big) / q.chunk_base;
    *local = unit - big - (c - q.chunk_rem) * q.chunk_base;
  }
  *seed = derive_chunk_seed(q.seed, c);
}

// --------------------------------------------------------- counter hash ---
// hash_u32 / stateless_open01_f32 / stateless_standard_normal_f32
// (cpu.rs:5626-5652, european_call_stepwise_v1.metal:6-28).
__host__ __device__ __forceinline__ uint32_t hash_u32(uint32_t x) {
  x += 0x9E3779B9u;
  x ^= x >> 16;
  x *= 0x85EBCA6Bu;
  x ^= x >> 13;
  x *= 0xC2B2AE35u;
  return x ^ (x >> 16);
}
__host__ __device__ __forceinline__ uint32_t counter_mix(uint32_t seed, uint32_t path, uint32_t step,
                                                         uint32_t lane) {
  return seed ^ (path * 747796405u) ^ (step * 2891336453u) ^ (lane * 277803737u);
}
// f32((h + 1) / 4294967297.0): the quotient lies within one unit of 2^-32
// below (h+1)/2^32, so the correctly rounded f64 quotient rounds to the same
// f32 as (h+1)/2^32 rounded to nearest with ties toward zero.  Evaluated
// exactly in integer arithmetic, no FP64 division.
__device__ __forceinline__ float counter_open01(uint32_t h) {
  if (h == 0xFFFFFFFFu) return 1.0f;
  uint32_t m = h + 1u;
  int bits = 32 - __clz(m);
  if (bits <= 24) return (float)m * 2.3283064365386963e-10f;  // exact
  int s = bits - 24;
  uint32_t q = m >> s;
  uint32_t rem = m & ((1u << s) - 1u);
  uint32_t half = 1u << (s - 1);
  if (rem > half) q += 1u;  // ties go down
  return __uint2float_rn(q) * __int_as_float((127 + s - 32) << 23);
}
__device__ __forceinline__ float counter_normal_f32(uint32_t seed, uint32_t path, uint32_t step) {
  float u1 = counter_open01(hash_u32(counter_mix(seed, path, step, 0u)));
  float u2 = counter_open01(hash_u32(counter_mix(seed, path, step, 1u)));
  float radius = sqrtf(-2.0f * logf(u1));
  float theta = 2.0f * 3.14159265358979323846f * u2;
  return radius * cosf(theta);
}

// --- fused FP32 form of the counter-hash normal --------------------------
// Same u32 hashes as counter_normal_f32; the transform is evaluated with
// short instruction sequences and stays within about 1e-5 absolute of it.
//
// (h + 1) / 2^32 rounded to nearest-even in one conversion.  counter_open01
// rounds ties toward zero; the two differ by one ulp at exact ties only.
__device__ __forceinline__ float counter_open01_fast(uint32_t h) {
  return h == 0xFFFFFFFFu ? 1.0f : __uint2float_rn(h + 1u) * 2.3283064365386963e-10f;
}
// PTX's approximate base-2 logarithm, reciprocal and square root, flushing
// denormals: the operands here are uniforms above 2^-54 and values of order one.
__device__ __forceinline__ float log2_ftz(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rcp_ftz(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_ftz(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// -2 ln(u), u in (0, 1].  Above 15/16, 4 atanh(s) with s = e / (2 - e) and
// e = 1 - u (exact there), three series terms (truncation < 2e-10 relative);
// below, the hardware log2, whose absolute error is small against |ln u|.
__device__ __forceinline__ float neg2_log_fast(float u) {
  const float e = 1.0f - u;
  const float s = e * rcp_ftz(2.0f - e), s2 = s * s;
  const float near1 = 4.0f * s * fmaf(s2, fmaf(s2, 0.2f, 0.33333334f), 1.0f);
  const float far = -1.3862943611198906f * log2_ftz(u);
  return u > 0.9375f ? near1 : far;
}
// cos(2 pi u) for u in [0, 1] as -cos(2 pi t), t = u - 1/2, by a degree-8
// polynomial in t^2 (Chebyshev least-squares fit rounded to float32,
// reproduced by fit_cos2pi.py; max error 3.3e-7).
__device__ __forceinline__ float cos_2pi_fast(float u) {
  const float t = u - 0.5f, x = t * t;
  float p = 2.437560558e-01f;
  p = fmaf(p, x, -1.696802378e+00f);
  p = fmaf(p, x, 7.899099350e+00f);
  p = fmaf(p, x, -2.642559624e+01f);
  p = fmaf(p, x, 6.024458313e+01f);
  p = fmaf(p, x, -8.545681763e+01f);
  p = fmaf(p, x, 6.493939209e+01f);
  p = fmaf(p, x, -1.973920822e+01f);
  p = fmaf(p, x, 1.0f);
  return -p;
}
// The same as -cos(2 pi t) with CUDA's fast cosine on t in [-1/2, 1/2]: its
// documented absolute error bound on [-pi, pi] (2^-21.41) matches the fit
// above, for one multiply and one MUFU operation instead of nine FMAs.
__device__ __forceinline__ float cos_2pi_hw(float u) {
  return -__cosf(6.28318548f * (u - 0.5f));
}
// Box-Muller cosine branch of the counter-hash uniforms; HWCOS picks the
// hardware cosine (for kernels with room on the MUFU pipe) over the
// polynomial (for kernels already bound by it, such as multi-asset baskets).
template <bool HWCOS = false>
__device__ __forceinline__ float counter_normal_fast(uint32_t seed, uint32_t path, uint32_t step) {
  const float u1 = counter_open01_fast(hash_u32(counter_mix(seed, path, step, 0u)));
  const float u2 = counter_open01_fast(hash_u32(counter_mix(seed, path, step, 1u)));
  float radius;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(radius) : "f"(neg2_log_fast(u1)));
  return radius * (HWCOS ? cos_2pi_hw(u2) : cos_2pi_fast(u2));
}

// Two of them at once, bit for bit the same values, from their counter_mix
// words (lane 0).  Everything that has a packed form runs as FP32 pairs (FFMA2,
// each lane rounded as the scalar operation), h + 1 is kept from wrapping by a
// minimum instead of a test, and the angle needs neither (u = 0 and u = 1 have
// the same cosine).  The kernels on counter-hash samples are bound by issue
// (0.81 to 0.85 of the slots): 24 contracts of a book, single-asset part
// (2.1e8 path-steps) 647 -> 396 us, 5-asset baskets (1.6e9 normals) 3,211 ->
// 2,434 us (one normal at a time took 63 instructions there).
__device__ __forceinline__ float2 splat2(float x) { return make_float2(x, x); }
template <bool HWCOS>
__device__ __forceinline__ float2 counter_normal_pair(uint32_t a, uint32_t b) {
  const uint32_t a1 = hash_u32(a), b1 = hash_u32(b);
  const uint32_t a2 = hash_u32(a ^ 277803737u), b2 = hash_u32(b ^ 277803737u);
  const float2 f = make_float2(__uint2float_rn(min(a1, 0xFFFFFFFEu) + 1u), __uint2float_rn(min(b1, 0xFFFFFFFEu) + 1u));
  const float2 u = __fmul2_rn(f, splat2(2.3283064365386963e-10f));
  const float2 e = __ffma2_rn(f, splat2(-2.3283064365386963e-10f), splat2(1.0f));
  const float2 d = __ffma2_rn(f, splat2(2.3283064365386963e-10f), splat2(1.0f));  // 2 - e
  const float2 s = __fmul2_rn(e, make_float2(rcp_ftz(d.x), rcp_ftz(d.y)));
  const float2 s2 = __fmul2_rn(s, s);
  const float2 near1 = __fmul2_rn(__fmul2_rn(splat2(4.0f), s),
                                  __ffma2_rn(s2, __ffma2_rn(s2, splat2(0.2f), splat2(0.33333334f)), splat2(1.0f)));
  const float2 far = __fmul2_rn(splat2(-1.3862943611198906f), make_float2(log2_ftz(u.x), log2_ftz(u.y)));
  const float2 r = make_float2(sqrt_ftz(u.x > 0.9375f ? near1.x : far.x), sqrt_ftz(u.y > 0.9375f ? near1.y : far.y));
  const float2 t = __ffma2_rn(make_float2(__uint2float_rn(a2 + 1u), __uint2float_rn(b2 + 1u)),
                              splat2(2.3283064365386963e-10f), splat2(-0.5f));
  if constexpr (HWCOS) {
    const float2 w = __fmul2_rn(splat2(6.28318548f), t);
    return __fmul2_rn(r, make_float2(-__cosf(w.x), -__cosf(w.y)));
  } else {
    const float2 x = __fmul2_rn(t, t);
    float2 p = __ffma2_rn(splat2(2.437560558e-01f), x, splat2(-1.696802378e+00f));
    p = __ffma2_rn(p, x, splat2(7.899099350e+00f));
    p = __ffma2_rn(p, x, splat2(-2.642559624e+01f));
    p = __ffma2_rn(p, x, splat2(6.024458313e+01f));
    p = __ffma2_rn(p, x, splat2(-8.545681763e+01f));
    p = __ffma2_rn(p, x, splat2(6.493939209e+01f));
    p = __ffma2_rn(p, x, splat2(-1.973920822e+01f));
    p = __ffma2_rn(p, x, splat2(1.0f));
    return __fmul2_rn(r, make_float2(-p.x, -p.y));
  }
}

// ---------------------------------------------------------------- Sobol ---
// Burley 2020 hash-based Owen scrambling (the algorithm of the `sobol_burley`
// crate called at cpu.rs:5399-5431): Owen-shuffled index, Sobol matrix
// product, Owen-scrambled output.  The matrix product uses per-dimension
// nibble tables sob[dim][q][v] = XOR of V[dim][4q + j] over the bits j of v,
// 8 lookups per sample instead of 32 conditional XORs.
__host__ __device__ __forceinline__ uint32_t lk_permute(uint32_t x, uint32_t seed) {
  x += seed;
  x ^= x * 0x6c50b47cu;
  x ^= x * 0xb82f1e52u;
  x ^= x * 0xc7afe638u;
  x ^= x * 0x8d22f6e6u;
  return x;
}
__device__ __forceinline__ uint32_t nested_uniform_scramble(uint32_t x, uint32_t seed) {
  return __brev(lk_permute(__brev(x), seed));
}
__host__ __device__ __forceinline__ uint32_t hash_combine(uint32_t seed, uint32_t v) {
  return seed ^ (v + 0x9e3779b9u + (seed << 6) + (seed >> 2));
}
// 23-bit midpoint uniform: exact in both precisions, never 0 or 1.
__device__ __forceinline__ float sobol_unit_f32(uint32_t x) {
  return ((float)(x >> 9) + 0.5f) * 1.1920928955078125e-07f;
}
// The same value assembled from bits: 1 + (x >> 9) 2^-23 in [1, 2) minus
// (1 - 2^-24); the difference is exact (Sterbenz), so no conversion is needed.
// (x >> 9) has no bit in common with the exponent, so + equals | here and
// lets the shift and the add issue as one instruction.
__device__ __forceinline__ float sobol_unit_f32_bits(uint32_t x) {
  return __fsub_rn(__int_as_float((x >> 9) + 0x3F800000u), 0.99999994f);
}
__device__ __forceinline__ double sobol_unit_f64(uint32_t x) {
  return ((double)(x >> 9) + 0.5) * 1.1920928955078125e-07;
}

// 1 / x by Newton's iteration from the hardware's 20-bit approximation, for
// normal x away from the range's ends: the first step leaves 2^-40, the second
// squares that and rounds once, within 2^-27 units of half a unit in the last
// place.
__device__ __forceinline__ double newton_reciprocal(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(y, fma(-x, y, 1.0), y);
  return fma(y, fma(-x, y, 1.0), y);
}
// num / den by the reciprocal y = newton_reciprocal(den) and one correction with
// the exact remainder (Markstein 1990), without the tests and the branch a
// general quotient needs, for quotients and remainders in the normal range.  It
// differs from the correctly rounded quotient only where the exact one lies
// within about 2^-50 units of a rounding boundary (tests/test_gpu_arithmetic.py
// finds none in 2^23 arguments of the inverse normal and 10^6 normal equations).
__device__ __forceinline__ double quotient(double num, double den, double y) {
  const double q = num * y;
  return fma(fma(-den, q, num), y, q);
}
__device__ __forceinline__ double quotient(double num, double den) { return quotient(num, den, newton_reciprocal(den)); }

// ------------------------------------------------------- Acklam inverse ---
// inverse_standard_normal (cpu.rs:6012-6061): the reference rational in FP64.
// The FP32 path calls CUDA's normcdfinvf: the rational's 1.15e-9 relative
// error is far below what FP32 resolves, so only the exact inverse matters there.
__device__ __forceinline__ double icdf_f64(double p) {
  const double a0 = -3.969683028665376e1, a1 = 2.209460984245205e2, a2 = -2.759285104469687e2,
               a3 = 1.38357751867269e2, a4 = -3.066479806614716e1, a5 = 2.506628277459239;
  const double b0 = -5.447609879822406e1, b1 = 1.615858368580409e2, b2 = -1.556989798598866e2,
               b3 = 6.680131188771972e1, b4 = -1.328068155288572e1;
  const double c0 = -7.784894002430293e-3, c1 = -3.223964580411365e-1, c2 = -2.400758277161838,
               c3 = -2.549732539343734, c4 = 4.374664141464968, c5 = 2.938163982698783;
  const double d0 = 7.784695709041462e-3, d1 = 3.224671290700398e-1, d2 = 2.445134137142996,
               d3 = 3.754408661907416;
  // Every product and sum is rounded separately (no FMA contraction), as the
  // CPU reference evaluates it, so both give the same bits up to log().
  p = fmin(fmax(p, 2.2250738585072014e-308), 1.0 - 2.220446049250313e-16);
  auto mad = [](double acc, double x, double c) { return __dadd_rn(__dmul_rn(acc, x), c); };
  if (p < 0.02425) {
    double q = sqrt(__dmul_rn(-2.0, log(p)));
    double num = mad(mad(mad(mad(mad(c0, q, c1), q, c2), q, c3), q, c4), q, c5);
    double den = mad(mad(mad(mad(d0, q, d1), q, d2), q, d3), q, 1.0);
    return num / den;
  }
  if (p <= 1.0 - 0.02425) {
    double q = __dadd_rn(p, -0.5);
    double r = __dmul_rn(q, q);
    double num = __dmul_rn(mad(mad(mad(mad(mad(a0, r, a1), r, a2), r, a3), r, a4), r, a5), q);
    double den = mad(mad(mad(mad(mad(b0, r, b1), r, b2), r, b3), r, b4), r, 1.0);
    return quotient(num, den);
  }
  double q = sqrt(__dmul_rn(-2.0, log(__dadd_rn(1.0, -p))));
  double num = mad(mad(mad(mad(mad(c0, q, c1), q, c2), q, c3), q, c4), q, c5);
  double den = mad(mad(mad(mad(d0, q, d1), q, d2), q, d3), q, 1.0);
  return -num / den;
}

// icdf_f64(sobol_unit_f64(x)) from the Sobol sample's bits.  The uniform and
// its mirror 1 - u are the same expression of m = x >> 9 and of its 23-bit
// complement, the rational is odd about 1/2 bit for bit, and the two tails
// mirror each other, so the lower half serves both with the sign of bit 31.
// `tail` holds the MPC_ICDF_TAIL values of the lower tail (icdf_f64 itself,
// tabulated): evaluated in place, one lane of a warp in the tail (4.85% of the
// samples, so four warps in five) makes all 32 wait for log, sqrt and a second
// rational.  The centre's argument comes from the bits exactly: 2 m + 1 below
// 2^52's exponent, less 2^52 + 2^23, times 2^-24.
__device__ __forceinline__ double icdf_sobol_f64(const double* __restrict__ tail, uint32_t x) {
  const double a0 = -3.969683028665376e1, a1 = 2.209460984245205e2, a2 = -2.759285104469687e2,
               a3 = 1.38357751867269e2, a4 = -3.066479806614716e1, a5 = 2.506628277459239;
  const double b0 = -5.447609879822406e1, b1 = 1.615858368580409e2, b2 = -1.556989798598866e2,
               b3 = 6.680131188771972e1, b4 = -1.328068155288572e1;
  const uint32_t xm = x ^ (uint32_t)((int32_t)x >> 31);
  const uint32_t m = xm >> 9;
  const double q = (__hiloint2double(0x43300000, (int)((xm >> 8) | 1u)) - 4503599635759104.0) * 5.9604644775390625e-08;
  const double r = __dmul_rn(q, q);
  auto mad = [](double acc, double y, double c) { return __dadd_rn(__dmul_rn(acc, y), c); };
  const double num = __dmul_rn(mad(mad(mad(mad(mad(a0, r, a1), r, a2), r, a3), r, a4), r, a5), q);
  const double den = mad(mad(mad(mad(mad(b0, r, b1), r, b2), r, b3), r, b4), r, 1.0);
  double z = quotient(num, den);  // den in [0.0026, 1] over the centre
  if (m < MPC_ICDF_TAIL) z = __ldg(tail + m);
  return __hiloint2double(__double2hiint(z) ^ (int)(x & 0x80000000u), __double2loint(z));
}

// --------------------------------------------------------------- Halton ---
// halton / halton_with_shift (cpu.rs:6063-6077): the sum of digit times
// 1 / base^k, plus a shift, modulo 1.  halton_f64 adds the reference's own terms
// in its order with the quotients tabulated (FP64 normals answer to the
// reference's bits: near the ends of the inverse normal's centre an ulp of the
// uniform is 3e-13 of the normal); halton_f32 reverses the digits in integers
// and scales once, within an ulp of the exact value, which FP32 cannot see.  A
// digit takes about 8 and 5 instructions instead of a 64-bit division and an
// FP64 division: 100,000 x 64 in FP32 92 -> 38 us.
static __device__ __noinline__ double halton_general(uint64_t index, uint32_t base, double shift) {
  double f = 1.0 / (double)base;
  double value = 0.0;
  while (index > 0) {
    uint64_t next = index / base;
    value += f * (double)(index - next * base);
    index = next;
    f /= (double)base;
  }
  value = fmax(value, 2.2250738585072014e-308);
  double shifted = value + shift;
  return shifted - floor(shifted);
}
__device__ __forceinline__ double halton_f64(uint64_t index, const HaltonDim* __restrict__ dim,
                                             const double* __restrict__ weights) {
  const uint4 head = __ldg(reinterpret_cast<const uint4*>(dim));
  const double offset = __ldg(&dim->offset);
  const uint32_t base = head.x, magic = head.y, shift = head.z & 0xFFu, digits = (head.z >> 8) & 0xFFu;
  if (digits == 0) return halton_general(index, base, offset);
  uint32_t n = (uint32_t)index;
  double value = 0.0;
  for (uint32_t k = 0; k < digits; ++k) {
    const uint32_t q = __umulhi(n, magic) >> shift;
    const double digit = __hiloint2double(0x43300000, (int)(n - q * base)) - 4503599627370496.0;  // exact
    value = __dadd_rn(value, __dmul_rn(__ldg(weights + head.w + k), digit));
    n = q;
  }
  const double shifted = value + offset;
  return shifted >= 1.0 ? shifted - 1.0 : shifted;
}
__device__ __forceinline__ double halton_f32(uint64_t index, const HaltonDim* __restrict__ dim) {
  const uint4 head = __ldg(reinterpret_cast<const uint4*>(dim));
  const double2 tail = __ldg(reinterpret_cast<const double2*>(dim) + 1);  // inv, offset
  const uint32_t base = head.x, magic = head.y, shift = head.z & 0xFFu, digits = (head.z >> 8) & 0xFFu;
  if (digits == 0) return halton_general(index, base, tail.y);
  uint32_t n = (uint32_t)index;
  double reversed;
  if ((head.z >> 16) & 0xFFu) {
    uint64_t r = 0;
    for (uint32_t k = 0; k < digits; ++k) {
      const uint32_t q = __umulhi(n, magic) >> shift;
      r = r * base + (n - q * base);
      n = q;
    }
    reversed = (double)r;
  } else {
    uint32_t r = 0;
    for (uint32_t k = 0; k < digits; ++k) {
      const uint32_t q = __umulhi(n, magic) >> shift;
      r = r * base + (n - q * base);
      n = q;
    }
    reversed = __hiloint2double(0x43300000, (int)r) - 4503599627370496.0;  // exact: 2^52 + r
  }
  const double shifted = fma(reversed, tail.x, tail.y);
  return shifted >= 1.0 ? shifted - 1.0 : shifted;
}
// Two consecutive dimensions: the same values, both digit chains in one loop
// (bases rise with the dimension, so the second has no more digits).
__device__ __forceinline__ double2 halton_f32_pair(uint64_t index, const HaltonDim* __restrict__ dim) {
  const uint4 ha = __ldg(reinterpret_cast<const uint4*>(dim)), hb = __ldg(reinterpret_cast<const uint4*>(dim + 1));
  if (((ha.z | hb.z) & 0xFF0000u) || !(ha.z & 0xFF00u) || !(hb.z & 0xFF00u))
    return make_double2(halton_f32(index, dim), halton_f32(index, dim + 1));
  const double2 ta = __ldg(reinterpret_cast<const double2*>(dim) + 1);
  const double2 tb = __ldg(reinterpret_cast<const double2*>(dim + 1) + 1);
  const uint32_t sa = ha.z & 0xFFu, sb = hb.z & 0xFFu, da = (ha.z >> 8) & 0xFFu, db = (hb.z >> 8) & 0xFFu;
  uint32_t na = (uint32_t)index, nb = na, ra = 0, rb = 0, k = 0;
  for (; k < db; ++k) {
    const uint32_t qa = __umulhi(na, ha.y) >> sa, qb = __umulhi(nb, hb.y) >> sb;
    ra = ra * ha.x + (na - qa * ha.x);
    rb = rb * hb.x + (nb - qb * hb.x);
    na = qa;
    nb = qb;
  }
  for (; k < da; ++k) {
    const uint32_t qa = __umulhi(na, ha.y) >> sa;
    ra = ra * ha.x + (na - qa * ha.x);
    na = qa;
  }
  const double a = fma(__hiloint2double(0x43300000, (int)ra) - 4503599627370496.0, ta.x, ta.y);
  const double b = fma(__hiloint2double(0x43300000, (int)rb) - 4503599627370496.0, tb.x, tb.y);
  return make_double2(a >= 1.0 ? a - 1.0 : a, b >= 1.0 ? b - 1.0 : b);
}

__device__ __forceinline__ double open01_from_u64(uint64_t v) {
  return fmax((double)(v >> 11) * (1.0 / 9007199254740992.0), 2.2250738585072014e-308);
}
// LatinHypercube::standard_normal's uniform (cpu.rs:5764-5780) of a point:
// stratum plus jitter over n.  `mixed` = point * 0xBF58476D1CE4E5B9, the same
// for all dimensions.
__device__ __forceinline__ double lhs_place(const LhsDim* __restrict__ dim, uint64_t point, uint64_t mixed, uint64_t n_paths) {
  const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2*>(dim));  // multiplier, offset
  const ulonglong2 b = __ldg(reinterpret_cast<const ulonglong2*>(dim) + 1);  // jitter seed, shoup | small << 32
  double stratum;
  if (b.y >> 32) {
    // m p mod n by the quotient estimate floor(shoup p / 2^32), at most one
    // below the true one: the remainder is below 2 n < 2^32
    const uint32_t p = (uint32_t)point, n = (uint32_t)n_paths;
    uint32_t r = (uint32_t)a.x * p - __umulhi((uint32_t)b.y, p) * n;
    r = min(r, r - n);
    r += (uint32_t)a.y;
    r = min(r, r - n);
    stratum = (double)r;
  } else {
    stratum = (double)((a.x * point + a.y) % n_paths);
  }
  return stratum + open01_from_u64(splitmix64(b.x ^ mixed));
}

// ----------------------------------------- Longstaff-Schwartz arithmetic ---
// x / 6.  FP32: x C + x c with C = 1/6 rounded and c the rest of it, one
// multiplication and one FMA (division by a constant known in advance,
// Brisebarre, Muller and Raina 2004).  FP64: x C, less than one unit in the last
// place off, corrected by its exact remainder (Markstein 1990).  Both are the
// correctly rounded quotient (tests/test_gpu_arithmetic.py: every FP32 mantissa).
__device__ __forceinline__ float sixth(float x) { return fmaf(x, 0.16666667f, x * -4.967053731882189e-09f); }
__device__ __forceinline__ double sixth(double x) {
  const double c = 0.16666666666666666, q = x * c;
  return fma(fma(-6.0, q, x), c, q);
}

template <class Real>
__device__ __forceinline__ void laguerre4(Real x, Real b[4]) {
  // laguerre_lsm_basis (cpu.rs:7667-7682); degrees above `degree` are unused
  const Real x2 = x * x, x3 = x2 * x;
  b[0] = (Real)1;
  b[1] = (Real)1 - x;
  b[2] = (Real)1 - (Real)2 * x + (Real)0.5 * x2;
  b[3] = (Real)1 - (Real)3 * x + (Real)1.5 * x2 - sixth(x3);
}

// solve_lsm_normal_equations (cpu.rs:7684-7736) for a compile-time size:
// Gauss-Jordan with partial pivoting in FP64, the reference's operations in
// its order, every index static (the pivot row swap is a predicated exchange),
// so the system stays in registers.  FP64 paths divide each entry of a pivot row
// by the pivot (|pivot| > 1e-12), all from one reciprocal; RECIP (FP32 paths)
// multiplies by the reciprocal.
template <int DIM, bool RECIP>
__device__ __forceinline__ bool solve_fixed(double a[4][4], double rhs[4]) {
#pragma unroll
  for (int piv = 0; piv < DIM; ++piv) {
    int best = piv;
    double best_abs = fabs(a[piv][piv]);
#pragma unroll
    for (int row = piv + 1; row < DIM; ++row) {
      const double c = fabs(a[row][piv]);
      if (c > best_abs) {
        best = row;
        best_abs = c;
      }
    }
    if (best_abs <= 1e-12) return false;
#pragma unroll
    for (int row = piv + 1; row < DIM; ++row) {
      if (row == best) {
#pragma unroll
        for (int c = piv; c < DIM; ++c) {
          const double t = a[piv][c];
          a[piv][c] = a[row][c];
          a[row][c] = t;
        }
        const double t = rhs[piv];
        rhs[piv] = rhs[row];
        rhs[row] = t;
      }
    }
    const double pv = a[piv][piv], ip = newton_reciprocal(pv);
#pragma unroll
    for (int c = piv + 1; c < DIM; ++c) a[piv][c] = RECIP ? a[piv][c] * ip : quotient(a[piv][c], pv, ip);
    rhs[piv] = RECIP ? rhs[piv] * ip : quotient(rhs[piv], pv, ip);
#pragma unroll
    for (int row = 0; row < DIM; ++row) {
      if (row == piv) continue;
      const double f = a[row][piv];
#pragma unroll
      for (int c = piv + 1; c < DIM; ++c) a[row][c] -= f * a[piv][c];
      rhs[row] -= f * rhs[piv];
    }
  }
  return true;
}

// ------------------------------------------------------------- reductions -
__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
  return v;
}

}  // namespace mpc
