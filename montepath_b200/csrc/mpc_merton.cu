// mpc_merton.cu -- the reference's Merton jump-diffusion estimator on the
// device: terminal sampling from one sequential MonteCarloRng stream per
// chunk (simulate_merton_jump_diffusion_chunk, crates/mc-core/src/runtime/
// cpu.rs:6408-6441; chunk split cpu.rs:6154-6199).
//
// Each path draws a Box-Muller normal (two stream outputs, or none when the
// stream holds a cached normal), one uniform for the Poisson jump count
// (sample_poisson, cpu.rs:932-953) and, only when the count is positive, a
// second normal.  Where a path starts in the stream therefore depends on the
// jump counts of every earlier path of its chunk.  With the stream position p
// of a path start and the cache state c (NONE, or a cached sine branch of the
// pair drawn 2 or 3 positions back), a path starting at (p, NONE) reads its
// Poisson uniform at p + 2 and moves to (p + 3, NONE) after a jump or
// (p + 3, CACHE3) without one; a path starting at (p, CACHE) reads it at p
// and moves to (p + 3, CACHE2) or (p + 1, NONE).  Path starts advance by one
// or three positions and depend only on one "jump" bit per position
// J[q] = (open01(x[q]) > exp(-lambda T)), i.e. "sample_poisson would return
// k > 0 from this uniform", so the chain of path starts is found in parallel.
// Two kernels, each block owning kBlockPos consecutive positions of a chunk
// and each thread a run of kRun of them:
//
//   1. maps:   every thread generates its run (GF(2) jump-ahead, then
//              sequential xorshift64*), and for each of the 6 ways a path can
//              first start in the run (offset 0, 1 or 2, with or without a
//              cached normal) walks the jump bits to the state in which the
//              next run is entered and the number of starts.  The maps are
//              composed over the block (a scan of byte permutations), and the
//              chunk's last block to finish composes the block maps from the
//              chunk's first path (position 0, no cache): every block's true
//              entry state and the number of paths before it.
//   2. paths:  every block generates its positions again into shared memory,
//              walks each run from its true entry, replaces each Box-Muller
//              pair it meets by its two normals in place (once per pair,
//              although the two normals may belong to two paths), and prices
//              its paths from there, all in FP64 with every product and sum
//              rounded separately as the reference does (no FMA contraction).
//              The payoff moments are reduced in the same launch.
//
// Nothing but the maps goes through memory.  1,000,003 paths on a B200: 66 us
// a call (20 us maps, 31 us paths), 411 us with the outputs, path starts and
// payoffs in HBM, six launches and the segment chain walked by one 512-thread
// block (301 us of it); 100 us with each lane jumping to its run by its own
// bits and the six walks as loops.  The second kernel is bound by FP64 issue
// (log, sqrt, sincos per pair, exp per path), the first by its integer
// instructions and the latency of the last block's chain.
//
// With lambda T == 0, sample_poisson draws no uniform, so paths alternate
// between the cosine and sine branch of consecutive pairs and need no chain.

#include <cuda_runtime.h>
#include <stdint.h>

#include "mpc_device.cuh"
#include "mpc_launch.h"

namespace mpc {

namespace {

constexpr uint32_t kRun = kMertonRun;           // positions per thread
constexpr uint32_t kThreads = kMertonThreads;
constexpr uint32_t kWarpsPerBlock = kThreads / 32;
constexpr uint32_t kBlockPos = kMertonBlockPos;  // positions per block
constexpr uint32_t kHalo = 4;                    // positions kept before and after a block's own
// Any two consecutive path starts advance by at least 4 positions (a start
// that advances by one leaves no cached normal, and the next one advances by
// three), so a block holds at most kBlockPos / 2 + 1 starts, and one pair more
// (the entry's cached one).
constexpr uint32_t kMaxStarts = kBlockPos / 2 + 8;
static_assert(kRun + 2 <= 32 && kBlockPos == kThreads * kRun, "a run's jump bits fit one word");
static_assert(((kBlockPos + 2 * kHalo) << 2) < 65536, "positions and cache states fit 16 bits");

enum : uint32_t { CS_NONE = 0, CS_CACHE2 = 1, CS_CACHE3 = 2 };

__device__ __forceinline__ uint64_t chunk_seed(const MertonStreamArgs& a, uint32_t c) {
  uint64_t s = a.n_chunks <= 1 ? a.seed : derive_chunk_seed(a.seed, c);
  return s == 0 ? 0x9E3779B97F4A7C15ull : s;  // MonteCarloRng::new (cpu.rs:2961-2970)
}

__device__ __forceinline__ uint64_t chunk_paths(const MertonStreamArgs& a, uint32_t c) {
  if (a.n_chunks <= 1) return a.n_paths;
  return a.chunk_base + (c < a.chunk_rem ? 1 : 0);
}

__device__ __forceinline__ uint64_t chunk_first_path(const MertonStreamArgs& a, uint32_t c) {
  if (a.n_chunks <= 1) return 0;
  return uint64_t(c) * a.chunk_base + (c < a.chunk_rem ? c : a.chunk_rem);
}

__device__ __forceinline__ double open01(uint64_t x) {  // next_f64_open01 (cpu.rs:2985-2990)
  double v = (double)(x >> 11) * (1.0 / 9007199254740992.0);
  return fmax(v, 2.2250738585072014e-308);
}

// The stream state at this thread's run: the warp's first run by a jump all
// lanes share, then T^(kRun lane) of that common state as 16 rows of the lane
// table, each a coalesced 256-byte load (lane table: images of the 16 values of
// every nibble under T^(kRun lane), mpc_launch.h).  Jumping each lane by its
// own bits took 1,000 instructions a lane, more than generating the run; this
// takes about 200.
__device__ __forceinline__ uint64_t run_state(const MertonStreamArgs& a, const DeviceTables& tabs, uint32_t c, uint32_t b) {
  const uint64_t run = uint64_t(b) * kThreads + (threadIdx.x & ~31u);
  const uint64_t s = xorshift_jump_uniform(tabs.jump, chunk_seed(a, c), run * kRun);
  const uint64_t* lane = tabs.lane_jump + (threadIdx.x & 31u);
  uint64_t y = 0;
#pragma unroll
  for (int q = 0; q < 16; ++q) y ^= __ldg(lane + (q * 16 + ((s >> (4 * q)) & 0xF)) * 32);
  return y;
}

// One path-start transition from relative position p with jump bits w.
__device__ __forceinline__ void advance(uint32_t& p, uint32_t& cs, uint32_t w) {
  if (cs == CS_NONE) {
    const bool j = (w >> (p + 2)) & 1u;
    p += 3;
    cs = j ? CS_NONE : CS_CACHE3;
  } else {
    const bool j = (w >> p) & 1u;
    p += j ? 3u : 1u;
    cs = j ? CS_CACHE2 : CS_NONE;
  }
}

// A run's exit state, (offset into the next run) * 3 + cache state, and its
// class, offset * 2 + (a normal is cached): the class alone decides the walk.
__device__ __forceinline__ uint32_t class_of(uint32_t label) {
  const uint32_t off = (label * 11u) >> 5;  // label / 3 for labels 0..8
  return off * 2u + (label != off * 3u ? 1u : 0u);
}

// A map of the 6 classes as bytes (entries 0..3 and 4..5).
struct ClassMap {
  uint32_t lo, hi;
};
__device__ __forceinline__ uint32_t byte_at(uint32_t lo, uint32_t hi, uint32_t i) {
  return __byte_perm(lo, hi, i) & 0xFFu;
}
__device__ __forceinline__ uint32_t nibbles(uint32_t bytes) {  // four bytes below 16 -> a byte_perm selector
  const uint32_t t = bytes | (bytes >> 4);
  return __byte_perm(t, 0u, 0x4420u);
}
// First a, then b.
__device__ __forceinline__ ClassMap compose(ClassMap a, ClassMap b) {
  return ClassMap{__byte_perm(b.lo, b.hi, nibbles(a.lo)), __byte_perm(b.lo, b.hi, nibbles(a.hi))};
}
__device__ __forceinline__ ClassMap identity_map() { return ClassMap{0x03020100u, 0x00000504u}; }

// Exclusive scan of the block's maps in thread order; *total: all of them.
__device__ __forceinline__ ClassMap scan_maps(ClassMap m, ClassMap* s_warp, ClassMap* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const ClassMap prev{__shfl_up_sync(0xFFFFFFFFu, m.lo, o), __shfl_up_sync(0xFFFFFFFFu, m.hi, o)};
    if (lane >= o) m = compose(prev, m);
  }
  __syncthreads();  // an earlier scan's readers of s_warp
  if (lane == 31) s_warp[warp] = m;
  __syncthreads();
  ClassMap before = identity_map(), all = identity_map();
  for (uint32_t w = 0; w < kWarpsPerBlock; ++w) {
    if (w == warp) before = all;
    all = compose(all, s_warp[w]);
  }
  *total = all;
  const ClassMap prev{__shfl_up_sync(0xFFFFFFFFu, m.lo, 1), __shfl_up_sync(0xFFFFFFFFu, m.hi, 1)};
  return lane == 0 ? before : compose(before, prev);
}

// Exclusive sum over the block in thread order; *total: the block's sum.
__device__ __forceinline__ uint32_t scan_sums(uint32_t v, uint32_t* s_warp, uint32_t* total) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  uint32_t inc = v;
#pragma unroll
  for (uint32_t o = 1; o < 32; o <<= 1) {
    const uint32_t prev = __shfl_up_sync(0xFFFFFFFFu, inc, o);
    if (lane >= o) inc += prev;
  }
  __syncthreads();
  if (lane == 31) s_warp[warp] = inc;
  __syncthreads();
  uint32_t before = 0, all = 0;
  for (uint32_t w = 0; w < kWarpsPerBlock; ++w) {
    if (w == warp) before = all;
    all += s_warp[w];
  }
  *total = all;
  return before + inc - v;
}

// 1. Run maps, block maps, and (in the chunk's last block) the chain of blocks.
__global__ void __launch_bounds__(kThreads) merton_maps_kernel(MertonStreamArgs a, DeviceTables tabs) {
  __shared__ ClassMap s_maps[kWarpsPerBlock];
  __shared__ uint32_t s_sum[kWarpsPerBlock];
  __shared__ uint32_t s_count[kWarpsPerBlock][6];
  __shared__ uint32_t s_label[kThreads];
  __shared__ uint32_t s_exit, s_last;
  const uint32_t c = blockIdx.x / a.blocks_per_chunk, b = blockIdx.x - c * a.blocks_per_chunk;
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  XorshiftStream st;
  st.state = run_state(a, tabs, c, b);
  uint32_t w = 0;
#pragma unroll
  for (uint32_t i = 0; i < kRun + 2; ++i) {
    const uint64_t x = st.next_u64();
    w |= ((int64_t)(x >> 11) > a.jump_above ? 1u : 0u) << i;
    if (i >= kRun - kHalo && i < kRun && t == kThreads - 1) a.halo[size_t(blockIdx.x) * kHalo + (i - (kRun - kHalo))] = x;
  }
  // Exit label and number of starts (bits 4 and up) per entry class, by
  // position from the run's end: n[p], k[p] for a path starting at p without
  // and with a cached normal.  Two selects a position, no branches.
  uint32_t n[kRun + 3], k[kRun + 3];
#pragma unroll
  for (uint32_t o = 0; o < 3; ++o) {
    n[kRun + o] = o * 3u + CS_NONE;
    k[kRun + o] = o * 3u + CS_CACHE3;
  }
#pragma unroll
  for (int p = int(kRun) - 1; p >= 0; --p) {
    // the pair of a normal cached on leaving the run: 3 positions back, or 2 when the cached start jumped
    const uint32_t jumped = p + 3 >= int(kRun) ? (p + 3 - kRun) * 3u + CS_CACHE2 : k[p + 3];
    n[p] = ((w >> (p + 2)) & 1u ? n[p + 3] : k[p + 3]) + 16u;
    k[p] = ((w >> p) & 1u ? jumped : n[p + 1]) + 16u;
  }
  uint32_t label_lo = 0, label_hi = 0, count_lo = 0, count_hi = 0;
  ClassMap m{0u, 0u};
#pragma unroll
  for (uint32_t e = 0; e < 6; ++e) {
    const uint32_t r = (e & 1u) ? k[e >> 1] : n[e >> 1], label = r & 15u, shift = 8u * (e & 3u);
    if (e < 4) {
      label_lo |= label << shift;
      count_lo |= (r >> 4) << shift;
      m.lo |= class_of(label) << shift;
    } else {
      label_hi |= label << shift;
      count_hi |= (r >> 4) << shift;
      m.hi |= class_of(label) << shift;
    }
  }
  ClassMap total;
  const ClassMap ex = scan_maps(m, s_maps, &total);
  a.run_entry[size_t(blockIdx.x) * kThreads + t] = nibbles(ex.lo) | (nibbles(ex.hi) << 16);
#pragma unroll
  for (uint32_t e = 0; e < 6; ++e) {
    const uint32_t n = __reduce_add_sync(0xFFFFFFFFu, byte_at(count_lo, count_hi, byte_at(ex.lo, ex.hi, e)));
    if (lane == 0) s_count[warp][e] = n;
  }
  if (t == kThreads - 1) {
    uint32_t row = 0;
#pragma unroll
    for (uint32_t e = 0; e < 6; ++e) row |= byte_at(label_lo, label_hi, byte_at(ex.lo, ex.hi, e)) << (4u * e);
    s_exit = row;
  }
  __syncthreads();
  if (t < 6) {
    uint32_t n = 0;
    for (uint32_t k = 0; k < kWarpsPerBlock; ++k) n += s_count[k][t];
    a.block_map[size_t(blockIdx.x) * 8 + 1 + t] = n;
  }
  if (t == 0) a.block_map[size_t(blockIdx.x) * 8] = s_exit;
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(a.chunk_done + c, 1u) == a.blocks_per_chunk - 1 ? 1u : 0u;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  const uint32_t first = c * a.blocks_per_chunk;
  uint32_t carry = 0;  // entry label of the next block: position 0, no cached normal
  unsigned long long before = 0;
  for (uint32_t base = 0; base < a.blocks_per_chunk; base += kThreads) {
    const uint32_t i = base + t;
    const bool valid = i < a.blocks_per_chunk;
    const uint32_t* rec = a.block_map + size_t(first + (valid ? i : 0)) * 8;
    const uint32_t row = valid ? __ldcg(rec) : 0u;
    ClassMap bm = identity_map();
    if (valid) {
      bm = ClassMap{0u, 0u};
#pragma unroll
      for (uint32_t e = 0; e < 6; ++e) {
        const uint32_t cl = class_of((row >> (4u * e)) & 15u);
        if (e < 4)
          bm.lo |= cl << (8u * e);
        else
          bm.hi |= cl << (8u * (e - 4));
      }
    }
    ClassMap unused;
    const ClassMap bex = scan_maps(bm, s_maps, &unused);
    const uint32_t entry = byte_at(bex.lo, bex.hi, class_of(carry));
    const uint32_t n = valid ? __ldcg(rec + 1 + entry) : 0u;
    uint32_t sum;
    const uint32_t ahead = scan_sums(n, s_sum, &sum);
    s_label[t] = (row >> (4u * entry)) & 15u;
    __syncthreads();
    if (valid) {
      a.block_state[first + i] = t == 0 ? carry : s_label[t - 1];
      a.block_before[first + i] = before + ahead;
    }
    const uint32_t last = min(a.blocks_per_chunk - base, kThreads) - 1;
    carry = s_label[last];
    before += sum;
    __syncthreads();
  }
  if (t == 0) a.chunk_done[c] = 0u;  // ready for the next call
}

// Box-Muller of one pair of stream outputs (cpu.rs:2992-3006), in place.
__device__ __forceinline__ void box_muller(unsigned long long* x) {
  const double u1 = open01(x[0]);
  const double u2 = open01(x[1]);
  const double radius = sqrt(__dmul_rn(-2.0, log(u1)));
  double s, c;
  sincospi(__dmul_rn(2.0, u2), &s, &c);  // exact argument reduction; the reference rounds 2 pi u2 first
  x[0] = (unsigned long long)__double_as_longlong(__dmul_rn(radius, c));
  x[1] = (unsigned long long)__double_as_longlong(__dmul_rn(radius, s));
}

// sample_poisson (cpu.rs:932-953) from its uniform, with exp(-mean) from the host.
__device__ __forceinline__ uint32_t poisson_count(double u, double mean, double p0) {
  double prob = p0, cum = p0;
  uint32_t k = 0;
  while (u > cum && k < 4095) {
    ++k;
    prob = __dmul_rn(prob, __ddiv_rn(mean, (double)k));
    cum = __dadd_rn(cum, prob);
  }
  return k;
}

constexpr size_t kPathsSmem = (kBlockPos + 2 * kHalo) * 8 + 2 * kMaxStarts * 2;

// 2. Payoffs (cpu.rs:6420-6437) and their moments.  CHAIN: paths follow the
// block's entry state; without (lambda T == 0), path i reads the normal at
// position i.
template <bool CHAIN>
__global__ void __launch_bounds__(kThreads, 4) merton_paths_kernel(MertonStreamArgs a, DeviceTables tabs) {
  extern __shared__ __align__(16) unsigned long long s_x[];  // kHalo positions, the block's, kHalo positions
  uint16_t* s_starts = reinterpret_cast<uint16_t*>(s_x + kBlockPos + 2 * kHalo);  // (position + kHalo) << 2 | cache state
  uint16_t* s_pairs = s_starts + kMaxStarts;                                      // position + kHalo
  __shared__ uint32_t s_sum[kWarpsPerBlock];
  __shared__ uint8_t s_label[kThreads];
  __shared__ double s_red[kWarpsPerBlock][2];
  __shared__ uint32_t s_last;
  const uint32_t c = blockIdx.x / a.blocks_per_chunk, b = blockIdx.x - c * a.blocks_per_chunk;
  const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  const uint64_t n_c = chunk_paths(a, c);
  const uint64_t before = CHAIN ? a.block_before[blockIdx.x] : uint64_t(b) * kBlockPos;
  double sum = 0.0, sq = 0.0;
  if (before < n_c) {  // blocks past the chunk's last path have nothing to price
    XorshiftStream st;
    st.state = run_state(a, tabs, c, b);
    uint32_t w = 0;
#pragma unroll
    for (uint32_t i = 0; i < kRun + 2; ++i) {
      const uint64_t x = st.next_u64();
      if (i < kRun || t == kThreads - 1) s_x[kHalo + t * kRun + i] = x;
      if (CHAIN) w |= ((int64_t)(x >> 11) > a.jump_above ? 1u : 0u) << i;
    }
    uint32_t n_pairs, n_starts;
    if constexpr (CHAIN) {
      if (t == kThreads - 1) {
        s_x[kHalo + kBlockPos + 2] = st.next_u64();
        s_x[kHalo + kBlockPos + 3] = st.next_u64();
      }
      if (t < kHalo) s_x[t] = b > 0 ? a.halo[size_t(blockIdx.x - 1) * kHalo + t] : 0ull;
      const uint32_t block_entry = a.block_state[blockIdx.x];
      const uint32_t entry =
          (a.run_entry[size_t(blockIdx.x) * kThreads + t] >> (4u * class_of(block_entry))) & 15u;
      // count the run's starts (low half) and new pairs (high half)
      uint32_t p = entry >> 1, cs = (entry & 1u) ? CS_CACHE3 : CS_NONE, count = 0;
      while (p < kRun) {
        const bool pair = cs == CS_NONE || ((w >> p) & 1u);
        count += pair ? 0x10001u : 1u;
        advance(p, cs, w);
      }
      s_label[t] = uint8_t((p - kRun) * 3u + cs);
      if (t == 0 && block_entry % 3u != CS_NONE) count += 0x10000u;  // the pair of the entry's cached normal
      uint32_t total;
      uint32_t at = scan_sums(count, s_sum, &total);
      const uint32_t label = t == 0 ? block_entry : s_label[t - 1];
      p = entry >> 1;
      cs = label - 3u * (label / 3u);
      uint32_t si = at & 0xFFFFu, pi = at >> 16;
      const uint32_t origin = kHalo + t * kRun;
      if (t == 0 && cs != CS_NONE) s_pairs[pi++] = uint16_t(origin + p - (cs == CS_CACHE2 ? 2u : 3u));
      while (p < kRun) {
        const bool cached = cs != CS_NONE;
        if (si < kMaxStarts) s_starts[si] = uint16_t(((origin + p) << 2) | cs);
        ++si;
        if (!cached || ((w >> p) & 1u)) {
          if (pi < kMaxStarts) s_pairs[pi] = uint16_t(origin + p + (cached ? 1u : 0u));
          ++pi;
        }
        advance(p, cs, w);
      }
      n_starts = min(total & 0xFFFFu, kMaxStarts);
      n_pairs = min(total >> 16, kMaxStarts);
    } else {
      n_starts = kBlockPos;
      n_pairs = kBlockPos / 2;
    }
    n_starts = uint32_t(min(uint64_t(n_starts), n_c - before));
    __syncthreads();
    for (uint32_t i = t; i < n_pairs; i += kThreads) box_muller(s_x + (CHAIN ? s_pairs[i] : kHalo + 2 * i));
    __syncthreads();
    const double* s_z = reinterpret_cast<const double*>(s_x);
    for (uint32_t i = t; i < n_starts; i += kThreads) {
      double z, zj = 0.0;
      uint32_t jumps = 0;
      if constexpr (CHAIN) {
        const uint32_t e = s_starts[i], p = e >> 2, cs = e & 3u;
        z = s_z[cs == CS_NONE ? p : (cs == CS_CACHE2 ? p - 1 : p - 2)];
        jumps = poisson_count(open01(s_x[cs == CS_NONE ? p + 2 : p]), a.mean, a.p0);
        if (jumps > 0) zj = s_z[p + 1];  // the pair's sine after a cosine, the new pair's cosine after a cached sine
      } else {
        z = s_z[kHalo + i];
      }
      const double diffusion = __dmul_rn(a.vol_t, z);
      double jump = 0.0;
      if (jumps > 0) {
        const double n = (double)jumps;
        jump = __dadd_rn(__dmul_rn(n, a.jump_mean), __dmul_rn(__dmul_rn(a.jump_vol, sqrt(n)), zj));
      }
      const double log_st = __dadd_rn(__dadd_rn(__dadd_rn(a.log_s0, a.drift_t), diffusion), jump);
      const double s_t = exp(log_st);
      const double pay = __dmul_rn(fmax(__dsub_rn(s_t, a.k), 0.0), a.discount);
      sum += pay;
      sq += pay * pay;
      if (a.payoff) a.payoff[chunk_first_path(a, c) + before + i] = pay;
    }
  }
  // block sums, then (in the last block) the sum of the blocks' in block order per thread
  auto reduce = [&]() {
    sum = warp_sum(sum);
    sq = warp_sum(sq);
    __syncthreads();
    if (lane == 0) {
      s_red[warp][0] = sum;
      s_red[warp][1] = sq;
    }
    __syncthreads();
    sum = sq = 0.0;
    for (uint32_t k = 0; k < kWarpsPerBlock; ++k) {
      sum += s_red[k][0];
      sq += s_red[k][1];
    }
  };
  reduce();
  if (t == 0) {
    a.partials[2 * size_t(blockIdx.x)] = sum;
    a.partials[2 * size_t(blockIdx.x) + 1] = sq;
    __threadfence();
    s_last = atomicAdd(a.done, 1u) == gridDim.x - 1 ? 1u : 0u;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  sum = sq = 0.0;
  for (uint32_t i = t; i < gridDim.x; i += kThreads) {
    sum += __ldcg(a.partials + 2 * size_t(i));
    sq += __ldcg(a.partials + 2 * size_t(i) + 1);
  }
  reduce();
  if (t == 0) {
    a.out[0] = (double)a.n_paths;
    a.out[1] = sum;
    a.out[2] = sq;
    *a.done = 0u;
  }
}

}  // namespace

cudaError_t launch_merton_stream(const MertonStreamArgs& a, const DeviceTables& tabs, cudaStream_t stream) {
  static_assert(kPathsSmem <= 48 * 1024, "default dynamic shared memory limit");
  const uint32_t grid = a.blocks_per_chunk * a.n_chunks;
  uint32_t launches = 1;
  if (a.mean != 0.0) {
    merton_maps_kernel<<<grid, kThreads, 0, stream>>>(a, tabs);
    merton_paths_kernel<true><<<grid, kThreads, kPathsSmem, stream>>>(a, tabs);
    ++launches;
  } else {
    merton_paths_kernel<false><<<grid, kThreads, kPathsSmem, stream>>>(a, tabs);
  }
  count_graph_launches(launches);  // adds to the launch count
  return cudaGetLastError();
}

}  // namespace mpc
