// mpc_kernels.cu -- sm_100a kernels of the B200 Monte Carlo pricing backend.
//
// Fused path (FP32 path arithmetic, FP64 accumulation): samples are generated
// in registers, stepped through the model, turned into a payoff and reduced
// warp -> block -> tile partial; the block that completes a request's last
// tile sums the tile partials in tile order (deterministic, independent of
// which requests share the launch).  One persistent kernel walks a tile work
// list, so a single request, a heterogeneous book and a serving wave all use
// the same launch.
//
// Longstaff-Schwartz: one cooperative launch.  Paths are written date-major,
// each date's ITM basis moments are reduced block -> grid (FP64), every block
// solves the 4x4 normal equations redundantly after a bounded grid barrier,
// and exercise decisions are applied in registers.

#include <atomic>
#include <mutex>
#include <set>
#include <utility>
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/montepath_cuda.h"
#include "mpc_device.cuh"
#include "mpc_launch.h"
#include "mpc_models.cuh"
#include "mpc_types.h"

namespace mpc {

static std::atomic<uint64_t> g_launches{0};
uint64_t kernel_launch_count() { return g_launches.load(); }
void count_graph_launches(uint64_t kernels) { g_launches.fetch_add(kernels); }
void discount_captured_launches(uint64_t kernels) { g_launches.fetch_sub(kernels); }
static inline void count_launch() { g_launches.fetch_add(1); }

template <int FAM, int SMP>
__device__ __forceinline__ void fused_unit(const DevReq& q, const SrcCtx& ctx, uint64_t u, double& p, double& c) {
  typename FusedUnitSource<FAM, SMP>::type src;
  src.template begin<false>(q, ctx, u);
  run_family<float, FAM>(q, src, p, c);
}

template <int SMP>
__device__ __forceinline__ void fused_unit_any(const DevReq& q, const SrcCtx& ctx, uint64_t u, double& p,
                                               double& c) {
  switch (q.family) {
    case FAM_GBM_STEP:
      fused_unit<FAM_GBM_STEP, SMP>(q, ctx, u, p, c);
      break;
    case FAM_GBM_TERMINAL:
      fused_unit<FAM_GBM_TERMINAL, SMP>(q, ctx, u, p, c);
      break;
    case FAM_HESTON:
      fused_unit<FAM_HESTON, SMP>(q, ctx, u, p, c);
      break;
    case FAM_BASKET:
      fused_unit<FAM_BASKET, SMP>(q, ctx, u, p, c);
      break;
    case FAM_MLMC_LEVEL:
      fused_unit<FAM_MLMC_LEVEL, SMP>(q, ctx, u, p, c);
      break;
    case FAM_GBM_BRIDGE:
      if constexpr (SMP == SMP_SOBOL)
        fused_unit<FAM_GBM_BRIDGE, SMP>(q, ctx, u, p, c);
      else
        p = c = 0.0;
      break;
    default:
      if constexpr (SMP != SMP_XORSHIFT) {
        if (q.family == FAM_MERTON_STEP)
          fused_unit<FAM_MERTON_STEP, SMP>(q, ctx, u, p, c);
        else
          fused_unit<FAM_MERTON_TERMINAL, SMP>(q, ctx, u, p, c);
      } else {
        p = c = 0.0;
      }
      break;
  }
}

// --------------------------------------------------------- fused kernel ---
// Resident blocks per SM the register allocation must allow: the
// family-switching instance is the widest; terminal paths on the counter hash
// are one short chain that wants more warps (stepwise ones draw two normals at
// a time and want the registers: 439 us with 40 of them, 375 us with 64 and 396
// with __expf's range check, the book's single-asset part).
constexpr int fused_min_blocks(int fam, int smp) {
  return fam < 0 ? 2 : (fam == FAM_GBM_TERMINAL && smp == SMP_COUNTER ? 6 : 4);
}
// The same resident threads per SM (hence the same register budget per
// thread) expressed in 512-thread blocks, for the launch bounds.
constexpr int fused_min_blocks512(int fam, int smp) { return fused_min_blocks(fam, smp) * kFusedBlock / kMaxFusedBlock; }

// One tile of request `sq`: its units through the model, the block's moment
// sums written as the tile's partial, and *s_last (shared) set when this was
// the request's last tile to finish.  Ends with the block synchronised.
// gf2_apply with the nibble table in shared memory.
__device__ __forceinline__ uint64_t gf2_apply_shared(const uint64_t* table, uint64_t x) {
  uint64_t y = 0;
#pragma unroll
  for (int q = 0; q < 16; ++q) y ^= table[q * 16 + ((x >> (4 * q)) & 0xF)];
  return y;
}

// A unit of a single-family fused kernel whose pseudorandom stream is
// already positioned: `aligned` is the chunk stream's state after
// 2 * (idx / 2) draws, idx the unit's first normal in its chunk.
template <int FAM>
__device__ __forceinline__ void fused_unit_stream(const DevReq& q, uint64_t aligned, uint64_t idx, double& p, double& c) {
  XorshiftPairs<float> src;
  src.start(aligned, idx);
  run_family<float, FAM>(q, src, p, c);
}

template <int FAM, int SMP>
__device__ __forceinline__ void fused_tile(const DevReq& sq, const SrcCtx& ctx, uint32_t tile, double (*red)[5],
                                           int* s_last) {
  const uint64_t first = (uint64_t)tile * sq.tile_units;
  const uint64_t last = min(first + (uint64_t)sq.tile_units, sq.n_units);
  double v[5] = {0, 0, 0, 0, 0};
  const bool cv = sq.cv != 0;
  double* per_unit = sq.per_unit;
  // Every thread runs the same number of units so that block- and
  // warp-synchronous sources stay in lockstep; a thread past the tile end
  // repeats the tile's last unit and discards it.
  const uint32_t iters = (uint32_t)((last - first + blockDim.x - 1) / blockDim.x);
  // Pseudorandom streams in a single-family kernel: a thread's units of one
  // tile lie blockDim units apart, so inside one chunk the next unit's
  // stream starts one jump of T^(blockDim x normals per unit) draws later
  // (blockDim is even, so the pair alignment carries over).  The block
  // tabulates that jump in shared memory for the tile (the images of the 64
  // basis vectors, then the nibble table), and each unit after a thread's
  // first in the tile takes 16 lookups instead of a full seek.
  constexpr bool kStride = SMP == SMP_XORSHIFT && FAM >= 0;
  uint64_t* stride_tab = nullptr;
  if constexpr (kStride) {
    __shared__ uint64_t s_cols[64];
    __shared__ uint64_t s_stride[256];
    stride_tab = s_stride;
    if (iters > 1) {
      const uint64_t delta = (uint64_t)blockDim.x * sq.normals_per_unit;
      for (uint32_t i = threadIdx.x; i < 64; i += blockDim.x) s_cols[i] = xorshift_jump(ctx.jump, 1ull << i, delta);
      __syncthreads();
      for (uint32_t e = threadIdx.x; e < 256; e += blockDim.x) {
        uint64_t y = 0;
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j)
          if ((e >> j) & 1u) y ^= s_cols[4 * (e >> 4) + j];
        s_stride[e] = y;
      }
      __syncthreads();
    }
  }
  uint64_t aligned = 0, prev_seed = 0;
  bool chained = false;  // `aligned` holds this thread's previous unit's start in the same tile
  for (uint32_t it = 0; it < iters; ++it) {
    uint64_t u = first + threadIdx.x + (uint64_t)it * blockDim.x;
    const bool valid = u < last;
    if (!valid) u = last - 1;  // a unit of the same iteration: same Sobol index bits 12..31, and not behind the warp's first
    double p, c;
    if constexpr (kStride) {
      uint64_t seed, local;
      chunk_of(sq, u, &seed, &local);
      const uint64_t idx = local * sq.normals_per_unit;
      const bool jump = chained && valid && seed == prev_seed;
      if (__all_sync(0xFFFFFFFFu, jump)) {
        aligned = gf2_apply_shared(stride_tab, aligned);
      } else {
        const uint64_t sought = xorshift_seek_warp(ctx.jump, seed, 2 * (idx >> 1));
        aligned = jump ? gf2_apply_shared(stride_tab, aligned) : sought;
      }
      chained = valid;
      prev_seed = seed;
      fused_unit_stream<FAM>(sq, aligned, idx, p, c);
    } else if constexpr (FAM >= 0)
      fused_unit<FAM, SMP>(sq, ctx, u, p, c);
    else
      fused_unit_any<SMP>(sq, ctx, u, p, c);
    if (!valid) continue;
    v[0] += p;
    v[1] += p * p;
    if (cv) {
      v[2] += c;
      v[3] += c * c;
      v[4] += p * c;
    }
    if (per_unit) per_unit[u] = p;
  }
  block_reduce5(v, red);
  if (threadIdx.x == 0) {
    double* pt = sq.partials + (size_t)tile * MPC_MOMENTS;
    pt[0] = (double)(last - first);
    for (int i = 0; i < 5; ++i) pt[1 + i] = v[i];
    __threadfence();
    *s_last = (atomicAdd(sq.tiles_done, 1u) == sq.n_tiles - 1) ? 1 : 0;
  }
  __syncthreads();
}

// FAM >= 0: every request of the launch has that family; FAM < 0: switch per tile.
// A block's first tile is its own index and later ones come off the cursor, so
// a launch of at most one tile per block touches no counter.
template <int FAM, int SMP>
__global__ void __launch_bounds__(kMaxFusedBlock, fused_min_blocks512(FAM, SMP)) fused_kernel(
    const __grid_constant__ FusedWork work, SrcCtx ctx) {
  extern __shared__ __align__(16) uint32_t sobol_window[];
  if constexpr (SMP == SMP_SOBOL) {
    // window rows, then the inverse-normal segments (staged once per launch)
    float4* seg = reinterpret_cast<float4*>(sobol_window + kSobolWindowWords);
    const float4* src = reinterpret_cast<const float4*>(ctx.sobol + MPC_ICDF_OFFSET);
    for (uint32_t i = threadIdx.x; i < MPC_ICDF_SEGMENTS; i += blockDim.x) seg[i] = src[i];
    ctx.win = sobol_window;
    ctx.icdf = seg;
  } else {
    ctx.win = nullptr;
    ctx.icdf = nullptr;
  }
  __shared__ DevReq sq;
  __shared__ double red[kMaxWarps][5];
  __shared__ uint32_t s_tile;
  __shared__ int s_last;
  const bool cursor = work.n_tiles > gridDim.x;
  for (uint32_t t = blockIdx.x; t < work.n_tiles;) {
    uint32_t tile;
    const DevReq* req;
    if (work.n_inline) {
      uint32_t r = 0;
      while (r + 1 < work.n_inline && t >= work.first[r + 1]) ++r;
      tile = t - work.first[r];
      req = &work.inl[r];
    } else {
      const Tile tl = work.tiles[t];
      tile = tl.tile;
      req = work.reqs + tl.req;
    }
    {  // stage the request descriptor in shared memory
      const uint4* src = reinterpret_cast<const uint4*>(req);
      uint4* dst = reinterpret_cast<uint4*>(&sq);
      for (uint32_t i = threadIdx.x; i < sizeof(DevReq) / sizeof(uint4); i += blockDim.x) dst[i] = src[i];
    }
    __syncthreads();
    fused_tile<FAM, SMP>(sq, ctx, tile, red, &s_last);
    if (s_last) {
      __threadfence();
      finalize_request(sq, red);
    }
    if (!cursor) break;
    if (threadIdx.x == 0) s_tile = gridDim.x + atomicAdd(work.counter, 1u);
    __syncthreads();
    t = s_tile;
  }
  // an inline launch leaves its cursor as it found it: the last block to go resets it
  if (cursor && work.n_inline && threadIdx.x == 0 && atomicAdd(work.counter + 1, 1u) == gridDim.x - 1) {
    work.counter[0] = 0u;
    work.counter[1] = 0u;
  }
}

template <int SMP>
constexpr size_t fused_dynamic_smem() {
  return SMP == SMP_SOBOL ? kSobolWindowWords * sizeof(uint32_t) + MPC_ICDF_SEGMENTS * sizeof(float4) : 0;
}

template <int FAM, int SMP>
static cudaError_t launch_fused_t(const FusedWork& work, const SrcCtx& ctx, int grid, int block, cudaStream_t stream) {
  fused_kernel<FAM, SMP><<<grid, block, fused_dynamic_smem<SMP>(), stream>>>(work, ctx);
  count_launch();
  return cudaGetLastError();
}

template <int SMP>
static cudaError_t launch_fused_s(int family, const FusedWork& work, const SrcCtx& ctx, int grid, int block,
                                  cudaStream_t stream) {
  switch (family) {
    case FAM_GBM_STEP:
      return launch_fused_t<FAM_GBM_STEP, SMP>(work, ctx, grid, block, stream);
    case FAM_GBM_TERMINAL:
      return launch_fused_t<FAM_GBM_TERMINAL, SMP>(work, ctx, grid, block, stream);
    case FAM_HESTON:
      return launch_fused_t<FAM_HESTON, SMP>(work, ctx, grid, block, stream);
    case FAM_BASKET:
      return launch_fused_t<FAM_BASKET, SMP>(work, ctx, grid, block, stream);
    case FAM_MLMC_LEVEL:
      return launch_fused_t<FAM_MLMC_LEVEL, SMP>(work, ctx, grid, block, stream);
    case FAM_GBM_BRIDGE:
      if constexpr (SMP == SMP_SOBOL)
        return launch_fused_t<FAM_GBM_BRIDGE, SMP>(work, ctx, grid, block, stream);
      return cudaErrorInvalidValue;
    case FAM_MERTON_STEP:
      if constexpr (SMP != SMP_XORSHIFT)
        return launch_fused_t<FAM_MERTON_STEP, SMP>(work, ctx, grid, block, stream);
      return cudaErrorInvalidValue;
    case FAM_MERTON_TERMINAL:
      if constexpr (SMP != SMP_XORSHIFT)
        return launch_fused_t<FAM_MERTON_TERMINAL, SMP>(work, ctx, grid, block, stream);
      return cudaErrorInvalidValue;
    default:
      return launch_fused_t<-1, SMP>(work, ctx, grid, block, stream);
  }
}

cudaError_t launch_fused(const FusedWork& work, int family, int sampler, const DeviceTables& tabs, int grid, int block,
                         cudaStream_t stream) {
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr};
  if (block != 128 && block != 256 && block != kMaxFusedBlock) return cudaErrorInvalidValue;
  switch (sampler) {
    case SMP_XORSHIFT:
      return launch_fused_s<SMP_XORSHIFT>(family, work, ctx, grid, block, stream);
    case SMP_HALTON:
      return launch_fused_s<SMP_HALTON>(family, work, ctx, grid, block, stream);
    case SMP_LHS:
      return launch_fused_s<SMP_LHS>(family, work, ctx, grid, block, stream);
    case SMP_SOBOL:
      return launch_fused_s<SMP_SOBOL>(family, work, ctx, grid, block, stream);
    case SMP_COUNTER:
      return launch_fused_s<SMP_COUNTER>(family, work, ctx, grid, block, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

// ---------------------------------------------------- resident serving loop ---
__device__ __forceinline__ void st_release_sys(uint32_t* p, uint32_t v) {
  asm volatile("st.release.sys.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint64_t loop_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ LoopEntry loop_entry(const LoopArgs& a, uint32_t pos) {
  const LoopEntry* ep = a.ring + (pos % a.ring_cap);
  LoopEntry e;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(e.slot), "=r"(e.gen), "=r"(e.n_tiles), "=r"(e.pos)
               : "l"(ep)
               : "memory");
  return e;
}

// 0: the entry at `pos` has no tile left to claim (its claim word has moved
// past its last tile or on to a later request of the slot, or the ring entry
// was reused by a later request, which happens only after it finished);
// otherwise its claim word.
__device__ __forceinline__ unsigned long long loop_open(const LoopArgs& a, const LoopEntry& e, uint32_t pos) {
  if (e.pos != pos || e.slot >= a.max_slots) return 0ull;
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(a.claim + e.slot) : "memory");
  if ((uint32_t)(v >> 32) != e.gen || (uint32_t)v >= e.n_tiles) return 0ull;
  return v;
}

// Thread 0: the next tile to run, or 0 when the block should leave (stop,
// pause, or idle_ns without claimable work).  The live entries are the ring
// positions [cursor, tail) after the exhausted front ones are skipped; each
// claim starts its scan at a position that rotates per block and per claim,
// so concurrent requests share the blocks tile by tile (a large request does
// not hold back the small ones behind it).  The doorbell, ring and claim
// words are device memory read through L2; an idle poll is followed by a
// sleep that doubles up to 4 us.
__device__ __forceinline__ int loop_claim(const LoopArgs& a, uint32_t& cursor, uint32_t& turn, uint32_t* slot,
                                          uint32_t* tile, uint32_t* gen) {
  uint64_t idle_since = 0;
  uint32_t nap = 500;
  for (;;) {
    uint32_t db[4];  // tail, stop, pause and a padding word, read in one load
    asm volatile("ld.acquire.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(db[0]), "=r"(db[1]), "=r"(db[2]), "=r"(db[3])
                 : "l"(a.doorbell)
                 : "memory");
    const uint32_t tail = db[0];
    if (db[1] | db[2]) return 0;  // stop or pause
    while (cursor != tail && loop_open(a, loop_entry(a, cursor), cursor) == 0ull) ++cursor;
    const uint32_t live = tail - cursor;
    const uint32_t first = live ? turn++ % live : 0u;
    for (uint32_t k = 0; k < live; ++k) {
      const uint32_t pos = cursor + (first + k) % live;
      const LoopEntry e = loop_entry(a, pos);
      unsigned long long v = loop_open(a, e, pos);
      for (int tries = 0; v != 0ull && tries < 64; ++tries) {  // bounded: contention leaves the entry for the next pass
        const unsigned long long w = atomicCAS(a.claim + e.slot, v, v + 1ull);
        if (w == v) {
          *slot = e.slot;
          *tile = (uint32_t)v;
          *gen = e.gen;
          return 1;
        }
        v = ((uint32_t)(w >> 32) == e.gen && (uint32_t)w < e.n_tiles) ? w : 0ull;
      }
    }
    const uint64_t now = loop_ns();
    if (idle_since == 0)
      idle_since = now;
    else if (now - idle_since > a.idle_ns)
      return 0;
    __nanosleep(nap);
    nap = nap < 4000u ? 2u * nap : 4000u;
  }
}

// The loop's tile body per sampler, kept out of line so that each sampler's
// register allocation stands on its own.
template <int SMP>
__device__ __noinline__ void loop_tile(const DevReq& sq, const SrcCtx& ctx, uint32_t tile, double (*red)[5],
                                       int* s_last) {
  fused_tile<-1, SMP>(sq, ctx, tile, red, s_last);
}

__global__ void __launch_bounds__(kFusedBlock, 2) serve_loop_kernel(LoopArgs a, SrcCtx ctx) {
  extern __shared__ __align__(16) uint32_t sobol_window[];
  {  // SMs kept free for the host-batched launches
    uint32_t smid;
    asm volatile("mov.u32 %0, %%smid;" : "=r"(smid));
    if (smid < a.reserve_sms) return;
  }
  {  // Sobol window rows, then the inverse-normal segments (staged once per launch)
    float4* seg = reinterpret_cast<float4*>(sobol_window + kSobolWindowWords);
    const float4* src = reinterpret_cast<const float4*>(ctx.sobol + MPC_ICDF_OFFSET);
    for (uint32_t i = threadIdx.x; i < MPC_ICDF_SEGMENTS; i += blockDim.x) seg[i] = src[i];
    ctx.win = sobol_window;
    ctx.icdf = seg;
  }
  __shared__ DevReq sq;
  __shared__ double red[kWarps][5];
  __shared__ uint32_t s_slot, s_tile, s_gen, s_go;
  __shared__ int s_last;
  uint32_t cursor = 0;            // thread 0: ring entries before it have no tile left to claim
  uint32_t turn = blockIdx.x;     // thread 0: rotation of the scan start
  for (;;) {
    if (threadIdx.x == 0) s_go = loop_claim(a, cursor, turn, &s_slot, &s_tile, &s_gen);
    __syncthreads();
    if (!s_go) break;
    {  // the slot's descriptor, through L2 (the host rewrites slots between requests)
      const uint4* src = reinterpret_cast<const uint4*>(a.slots + s_slot);
      uint4* dst = reinterpret_cast<uint4*>(&sq);
      for (uint32_t i = threadIdx.x; i < sizeof(DevReq) / sizeof(uint4); i += blockDim.x) dst[i] = __ldcg(src + i);
    }
    __syncthreads();
    switch (sq.sampling) {
      case MPC_SAMPLING_PSEUDORANDOM:
        loop_tile<SMP_XORSHIFT>(sq, ctx, s_tile, red, &s_last);
        break;
      case MPC_SAMPLING_COUNTER_HASH:
        loop_tile<SMP_COUNTER>(sq, ctx, s_tile, red, &s_last);
        break;
      default:  // scrambled Sobol (the host publishes no other sampler)
        loop_tile<SMP_SOBOL>(sq, ctx, s_tile, red, &s_last);
        break;
    }
    if (s_last) {
      __threadfence();
      finalize_request(sq, red);  // moments go to mapped host memory
      if (threadIdx.x == 0) {
        __threadfence_system();
        st_release_sys(a.done + s_slot, s_gen);
      }
    }
    __syncthreads();
  }
}

constexpr size_t kLoopSmem = kSobolWindowWords * sizeof(uint32_t) + MPC_ICDF_SEGMENTS * sizeof(float4);

cudaError_t launch_serve_loop(const LoopArgs& a, const DeviceTables& tabs, int grid, cudaStream_t stream) {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(serve_loop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kLoopSmem));
  });
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr, nullptr};
  serve_loop_kernel<<<grid, kFusedBlock, kLoopSmem, stream>>>(a, ctx);
  count_launch();
  return cudaGetLastError();
}

int serve_loop_blocks_per_sm() {
  static std::once_flag once;
  std::call_once(once, [] {
    cudaFuncSetAttribute(serve_loop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kLoopSmem));
  });
  int n = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, serve_loop_kernel, kFusedBlock, kLoopSmem);
  return n;
}

template <int FAM, int SMP>
static int occ_t(int block) {
  static std::atomic<int> known[3];  // 128, 256, 512 threads; as lsm_capacity_t's
  const int at = block == 128 ? 0 : block == 256 ? 1 : 2;
  int n = known[at].load(std::memory_order_relaxed);
  if (n <= 0) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fused_kernel<FAM, SMP>, block, fused_dynamic_smem<SMP>());
    known[at].store(n, std::memory_order_relaxed);
  }
  return n;
}
template <int SMP>
static int occ_s(int family, int block) {
  switch (family) {
    case FAM_GBM_STEP:
      return occ_t<FAM_GBM_STEP, SMP>(block);
    case FAM_GBM_TERMINAL:
      return occ_t<FAM_GBM_TERMINAL, SMP>(block);
    case FAM_HESTON:
      return occ_t<FAM_HESTON, SMP>(block);
    case FAM_BASKET:
      return occ_t<FAM_BASKET, SMP>(block);
    case FAM_MLMC_LEVEL:
      return occ_t<FAM_MLMC_LEVEL, SMP>(block);
    case FAM_GBM_BRIDGE:
      if constexpr (SMP == SMP_SOBOL) return occ_t<FAM_GBM_BRIDGE, SMP>(block);
      return 1;
    case FAM_MERTON_STEP:
      if constexpr (SMP != SMP_XORSHIFT) return occ_t<FAM_MERTON_STEP, SMP>(block);
      return 1;
    case FAM_MERTON_TERMINAL:
      if constexpr (SMP != SMP_XORSHIFT) return occ_t<FAM_MERTON_TERMINAL, SMP>(block);
      return 1;
    default:
      return occ_t<-1, SMP>(block);
  }
}
int fused_max_blocks_per_sm(int family, int sampler, int block) {
  switch (sampler) {
    case SMP_XORSHIFT:
      return occ_s<SMP_XORSHIFT>(family, block);
    case SMP_HALTON:
      return occ_s<SMP_HALTON>(family, block);
    case SMP_LHS:
      return occ_s<SMP_LHS>(family, block);
    case SMP_SOBOL:
      return occ_s<SMP_SOBOL>(family, block);
    default:
      return occ_s<SMP_COUNTER>(family, block);
  }
}

// Raises a kernel's dynamic shared memory limit to `bytes` once per device
// (the attribute is per device).  Kernels whose Sobol window and
// inverse-normal table (46,592 bytes) plus their static shared memory pass
// the 48 KB default need it before their first launch and occupancy query.
static cudaError_t allow_dynamic_smem(const void* fn, size_t bytes) {
  static std::mutex mu;
  static std::set<std::pair<const void*, int>> done;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  std::lock_guard<std::mutex> lock(mu);
  if (done.count({fn, dev})) return cudaSuccess;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done.insert({fn, dev});
  return e;
}

// ------------------------------------------------ scenario (bump) kernel ---
// Bump-and-revalue Greeks with common random numbers: every leg of the
// recipe (base, then up and down per Greek) has the same seed, so every leg
// sees the same normals.  Here one thread draws each normal once and advances
// all legs' paths with it; each leg keeps its own FP32 state and payoff, with
// the same arithmetic as the single-request unit of its family.  Per unit the
// legs' payoffs are warp-summed (FP64 sum and sum of squares) into per-warp
// shared slots; per tile the slots are summed in warp order into tile
// partials [tile][leg][NM], and the last tile sums those in tile order.
// TECH follows the request's technique: antithetic legs also run the mirrored
// path (-z) and record the pair average, as unit_* does; control-variate legs
// also record the discounted terminal price c with sum c, sum c^2 and sum p c
// (NM = 5 moments per leg instead of 2).
// Scenario parameters, struct of arrays [field][kMaxScen] (float):
//   GBM:    log_s0, s0, drift_dt, vol_dt, discount, knocked-out-at-start (0/1)
//   Heston: log_s0, v0, rate, dt, sqrt_dt, discount
constexpr int kScenStd = MPC_TECHNIQUE_STANDARD, kScenAnti = MPC_TECHNIQUE_ANTITHETIC,
              kScenCv = MPC_TECHNIQUE_CONTROL_VARIATE;

template <int W, int TECH, class Src>
__device__ __forceinline__ void scen_gbm_step(const DevReq& q, Src& src, const float* __restrict__ sp, int n_scen,
                                              float pay[kMaxScen], float pay2[kMaxScen], float ctl[kMaxScen]) {
  constexpr bool ANTI = TECH == kScenAnti;
  float ls[kMaxScen], acc[kMaxScen], drift[kMaxScen], vol[kMaxScen];
  float ls2[kMaxScen], acc2[kMaxScen];  // mirrored paths (antithetic)
  bool ko[kMaxScen], ko2[kMaxScen];
#pragma unroll
  for (int s = 0; s < kMaxScen; ++s) {
    ls[s] = sp[0 * kMaxScen + s];
    acc[s] = (W == W_LOOKBACK) ? sp[1 * kMaxScen + s] : 0.0f;
    drift[s] = sp[2 * kMaxScen + s];
    vol[s] = sp[3 * kMaxScen + s];
    ko[s] = sp[5 * kMaxScen + s] != 0.0f;
    if constexpr (ANTI) {
      ls2[s] = ls[s];
      acc2[s] = acc[s];
      ko2[s] = ko[s];
    }
  }
  const float lbar = (float)q.log_barrier;
  const uint32_t n = q.n_steps;
  auto advance = [&](const float z) {
#pragma unroll
    for (int s = 0; s < kMaxScen; ++s) {
      if (s >= n_scen) break;
      ls[s] += drift[s] + vol[s] * z;
      if constexpr (W == W_ASIAN) acc[s] += ex<float>(ls[s]);
      else if constexpr (W == W_LOOKBACK) acc[s] = acc[s] > ex<float>(ls[s]) ? acc[s] : ex<float>(ls[s]);
      else if constexpr (W == W_DAO) ko[s] |= ls[s] <= lbar;
      else if constexpr (W == W_UAO) ko[s] |= ls[s] >= lbar;
      if constexpr (ANTI) {
        ls2[s] += drift[s] - vol[s] * z;
        if constexpr (W == W_ASIAN) acc2[s] += ex<float>(ls2[s]);
        else if constexpr (W == W_LOOKBACK) acc2[s] = acc2[s] > ex<float>(ls2[s]) ? acc2[s] : ex<float>(ls2[s]);
        else if constexpr (W == W_DAO) ko2[s] |= ls2[s] <= lbar;
        else if constexpr (W == W_UAO) ko2[s] |= ls2[s] >= lbar;
      }
    }
  };
  uint32_t st = 0;
  if constexpr (kQuadSource<Src>) {
    for (; st + 4 <= n; st += 4) {
      src.at_step(st, 4);
      src.quad_load(st);
      const float2 z01 = src.template take_n2<0, 1>(st), z23 = src.template take_n2<2, 3>(st);
#pragma unroll 2
      for (int k = 0; k < 4; ++k) advance(k == 0 ? z01.x : k == 1 ? z01.y : k == 2 ? z23.x : z23.y);
    }
  } else if constexpr (kPairSource<Src>) {
    for (; st + 2 <= n; st += 2) {
      const auto z = src.n2(st);
      advance(z.x);
      advance(z.y);
    }
  }
  for (; st < n; ++st) {
    src.at_step(st, 1);
    advance(normal<float>(src, st));
  }
  const float kk = (float)q.k, inv_n = (float)(1.0 / (double)n);
  auto payoff = [&](float l, float a, bool out, float disc) {
    float v;
    if constexpr (W == W_ASIAN) v = a * inv_n - kk;
    else if constexpr (W == W_LOOKBACK) v = a - kk;
    else {
      v = ex<float>(l) - kk;
      if (out) v = 0.0f;
    }
    return (v > 0.0f ? v : 0.0f) * disc;
  };
#pragma unroll
  for (int s = 0; s < kMaxScen; ++s) {
    const float disc = sp[4 * kMaxScen + s];
    pay[s] = payoff(ls[s], acc[s], ko[s], disc);
    if constexpr (ANTI) pay2[s] = payoff(ls2[s], acc2[s], ko2[s], disc);
    if constexpr (TECH == kScenCv) ctl[s] = disc * ex<float>(ls[s]);
  }
}

template <int TECH, class Src>
__device__ __forceinline__ void scen_gbm_terminal(const DevReq& q, Src& src, const float* __restrict__ sp, int n_scen,
                                                  float pay[kMaxScen], float pay2[kMaxScen], float ctl[kMaxScen]) {
  src.at_step(0, 1);
  const float z = normal<float>(src, 0);
  const float kk = (float)q.k;
#pragma unroll
  for (int s = 0; s < kMaxScen; ++s) {
    const float s0 = sp[1 * kMaxScen + s], drift = sp[2 * kMaxScen + s],
                vol = sp[3 * kMaxScen + s], disc = sp[4 * kMaxScen + s];
    const float st = s0 * ex<float>(drift + vol * z);
    pay[s] = (st - kk > 0.0f ? st - kk : 0.0f) * disc;
    if constexpr (TECH == kScenAnti) {
      const float sb = s0 * ex<float>(drift + vol * (-z));
      pay2[s] = (sb - kk > 0.0f ? sb - kk : 0.0f) * disc;
    }
    if constexpr (TECH == kScenCv) ctl[s] = disc * st;
  }
  (void)n_scen;
}

template <int TECH, class Src>
__device__ __forceinline__ void scen_heston(const DevReq& q, Src& src, const float* __restrict__ sp, int n_scen,
                                            float pay[kMaxScen], float pay2[kMaxScen], float ctl[kMaxScen]) {
  constexpr bool ANTI = TECH == kScenAnti;
  const float kappa = (float)q.kappa, theta = (float)q.theta, xi = (float)q.xi, rho = (float)q.rho,
              rho_perp = (float)q.rho_perp;
  float ls[kMaxScen], v[kMaxScen], rate[kMaxScen], dt[kMaxScen], sqdt[kMaxScen];
  float ls2[kMaxScen], v2[kMaxScen];  // mirrored paths (antithetic)
#pragma unroll
  for (int s = 0; s < kMaxScen; ++s) {
    ls[s] = sp[0 * kMaxScen + s];
    v[s] = sp[1 * kMaxScen + s];
    rate[s] = sp[2 * kMaxScen + s];
    dt[s] = sp[3 * kMaxScen + s];
    sqdt[s] = sp[4 * kMaxScen + s];
    if constexpr (ANTI) {
      ls2[s] = ls[s];
      v2[s] = v[s];
    }
  }
  auto step = [&](float& l, float& var, int s, float zp, float zv) {
    const float vp = var > 0.0f ? var : 0.0f;
    const float sv = sqrt_approx(vp);
    l += (rate[s] - 0.5f * vp) * dt[s] + sv * sqdt[s] * zp;
    var = var + kappa * (theta - vp) * dt[s] + xi * sv * sqdt[s] * zv;
    var = var > 0.0f ? var : 0.0f;
  };
  const uint32_t n = q.n_steps;
  for (uint32_t st = 0; st < n; ++st) {
    float zv, zi;
    if constexpr (kPairSource<Src>) {
      const auto z = src.n2(2 * st);
      zv = z.x;
      zi = z.y;
    } else {
      src.at_step(2 * st, 2);
      zv = normal<float>(src, 2 * st);
      zi = normal<float>(src, 2 * st + 1);
    }
    const float zp = rho * zv + rho_perp * zi;
#pragma unroll
    for (int s = 0; s < kMaxScen; ++s) {
      if (s >= n_scen) break;
      step(ls[s], v[s], s, zp, zv);
      if constexpr (ANTI) step(ls2[s], v2[s], s, rho * (-zv) + rho_perp * (-zi), -zv);
    }
  }
  const float kk = (float)q.k;
#pragma unroll
  for (int s = 0; s < kMaxScen; ++s) {
    const float disc = sp[5 * kMaxScen + s];
    const float stv = ex<float>(ls[s]);
    pay[s] = (stv - kk > 0.0f ? stv - kk : 0.0f) * disc;
    if constexpr (ANTI) {
      const float sb = ex<float>(ls2[s]);
      pay2[s] = (sb - kk > 0.0f ? sb - kk : 0.0f) * disc;
    }
    if constexpr (TECH == kScenCv) ctl[s] = stv * disc;
  }
}

template <int FAM, int TECH, class Src>
__device__ __forceinline__ void scen_unit(const DevReq& q, Src& src, const float* sp, int n_scen, float pay[kMaxScen],
                                          float pay2[kMaxScen], float ctl[kMaxScen]) {
  if constexpr (FAM == FAM_HESTON) {
    scen_heston<TECH>(q, src, sp, n_scen, pay, pay2, ctl);
  } else if constexpr (FAM == FAM_GBM_TERMINAL) {
    scen_gbm_terminal<TECH>(q, src, sp, n_scen, pay, pay2, ctl);
  } else {
    switch (q.workload) {
      case W_ASIAN:
        scen_gbm_step<W_ASIAN, TECH>(q, src, sp, n_scen, pay, pay2, ctl);
        break;
      case W_DAO:
        scen_gbm_step<W_DAO, TECH>(q, src, sp, n_scen, pay, pay2, ctl);
        break;
      case W_UAO:
        scen_gbm_step<W_UAO, TECH>(q, src, sp, n_scen, pay, pay2, ctl);
        break;
      case W_LOOKBACK:
        scen_gbm_step<W_LOOKBACK, TECH>(q, src, sp, n_scen, pay, pay2, ctl);
        break;
      default:
        scen_gbm_step<W_EURO, TECH>(q, src, sp, n_scen, pay, pay2, ctl);
        break;
    }
  }
}

// Sums `n_rows` rows of `cols` doubles (row stride `stride`) into out[cols]:
// warp w takes rows w, w + 8, ..., a lane per column (a row is one or two
// coalesced loads), then the warps' sums in warp order.  acc: [kWarps * cols]
// shared.  With one thread per column walking all rows the 512 tiles of a
// 262,144-path report ended 6 us later (98 -> 92 us).
__device__ __forceinline__ void sum_rows(const double* rows, uint32_t n_rows, uint32_t stride, uint32_t cols,
                                         double* acc, double* out) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  for (uint32_t c = lane; c < cols; c += 32) {
    double sum = 0.0;
#pragma unroll 8
    for (uint32_t r = warp; r < n_rows; r += kWarps) sum += __ldcg(rows + (size_t)r * stride + c);
    acc[warp * cols + c] = sum;
  }
  __syncthreads();
  if (threadIdx.x < cols) {
    double sum = 0.0;
    for (int w = 0; w < kWarps; ++w) sum += acc[w * cols + threadIdx.x];
    out[threadIdx.x] = sum;
  }
}

// Next tile of a scenario launch, first the block's own index; the cursor is
// q.tiles_done[1], and the last block to go leaves all three words zero.
__device__ __forceinline__ uint32_t next_scenario_tile(const DevReq& q, uint32_t* s_tile) {
  if (threadIdx.x == 0) *s_tile = gridDim.x + atomicAdd(q.tiles_done + 1, 1u);
  __syncthreads();
  return *s_tile;
}

// One request split into q.n_tiles tiles of q.tile_units units.  262,144
// antithetic Asian paths x 64 steps on Sobol, 9 legs: 98 -> 92 us with the
// normals by quads (two steps a turn of the inner loop: one takes 100), the legs in
// the parameter bank and the rows summed by all warps.  Bound by the 18
// exponentials a normal and the chains around them (MUFU 45%, issue 65%).  Three
// blocks per SM where a leg has one path (9 states in 80 registers: Asian x 64 on
// the counter hash, 262,144 paths a report, 145 -> 122 us; 5,000 paths 52 and 52),
// two for antithetic legs, whose 18 would spill (30,000 x 128 on Sobol 99 -> 105).
template <int FAM, int SMP, int TECH>
__global__ void __launch_bounds__(kFusedBlock, TECH == kScenAnti ? 2 : 3) scenario_kernel(const __grid_constant__ DevReq sq,
                                                                 const __grid_constant__ ScenarioLegs legs, SrcCtx ctx) {
  constexpr int NM = TECH == kScenCv ? 5 : 2;  // moments per leg
  extern __shared__ __align__(16) uint32_t sobol_window[];
  if constexpr (SMP == SMP_SOBOL) {
    float4* seg = reinterpret_cast<float4*>(sobol_window + kSobolWindowWords);
    const float4* src = reinterpret_cast<const float4*>(ctx.sobol + MPC_ICDF_OFFSET);
    for (uint32_t i = threadIdx.x; i < MPC_ICDF_SEGMENTS; i += blockDim.x) seg[i] = src[i];
    ctx.win = sobol_window;
    ctx.icdf = seg;
  } else {
    ctx.win = nullptr;
    ctx.icdf = nullptr;
  }
  __shared__ double slots[kWarps][kMaxScen][NM];
  __shared__ uint32_t s_tile;
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n_tiles = sq.n_tiles;
  const int n_scen = (int)sq.n_scen;
  for (uint32_t t = blockIdx.x; t < n_tiles; t = next_scenario_tile(sq, &s_tile)) {
    for (uint32_t i = threadIdx.x; i < kWarps * kMaxScen * NM; i += blockDim.x) (&slots[0][0][0])[i] = 0.0;
    __syncthreads();
    const uint64_t first = (uint64_t)t * sq.tile_units;
    const uint64_t last = min(first + (uint64_t)sq.tile_units, sq.n_units);
    const uint32_t iters = (uint32_t)((last - first + blockDim.x - 1) / blockDim.x);
    for (uint32_t it = 0; it < iters; ++it) {
      uint64_t u = first + threadIdx.x + (uint64_t)it * blockDim.x;
      const bool valid = u < last;
      if (!valid) u = last - 1;  // lockstep for block- and warp-synchronous sources; discarded below
      typename FusedUnitSource<FAM, SMP>::type src;  // the samples fused_unit<FAM, SMP> draws
      src.template begin<false>(sq, ctx, u);
      float pay[kMaxScen], pay2[kMaxScen], ctl[kMaxScen];
      scen_unit<FAM, TECH>(sq, src, legs.f, n_scen, pay, pay2, ctl);
#pragma unroll
      for (int s = 0; s < kMaxScen; ++s) {
        if (s >= n_scen) break;
        double p = (double)pay[s];
        if constexpr (TECH == kScenAnti) p = 0.5 * ((double)pay[s] + (double)pay2[s]);
        if (!valid) p = 0.0;
        const double a = warp_sum(p), b = warp_sum(p * p);
        if constexpr (TECH == kScenCv) {
          const double c = valid ? (double)ctl[s] : 0.0;
          const double cs = warp_sum(c), cc = warp_sum(c * c), pc = warp_sum(p * c);
          if (lane == 0) {
            slots[warp][s][2] += cs;
            slots[warp][s][3] += cc;
            slots[warp][s][4] += pc;
          }
        }
        if (lane == 0) {
          slots[warp][s][0] += a;
          slots[warp][s][1] += b;
        }
      }
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)(NM * n_scen)) {
      const int s = threadIdx.x / NM, k = threadIdx.x % NM;
      double sum = 0.0;
      for (int w = 0; w < kWarps; ++w) sum += slots[w][s][k];
      sq.partials[((size_t)t * kMaxScen + s) * NM + k] = sum;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(sq.tiles_done, 1u) == n_tiles - 1) ? 1 : 0;
    __syncthreads();
    if (s_last) {
      __threadfence();
      sum_rows(sq.partials, n_tiles, kMaxScen * NM, NM * n_scen, &slots[0][0][0], sq.moments);
    }
  }
  // the last block to go leaves the counters zero for the next report
  if (threadIdx.x == 0 && atomicAdd(sq.tiles_done + 2, 1u) == gridDim.x - 1)
    sq.tiles_done[0] = sq.tiles_done[1] = sq.tiles_done[2] = 0u;
}

using ScenarioKernel = void (*)(const DevReq, const ScenarioLegs, SrcCtx);
template <int SMP, int TECH>
static ScenarioKernel scenario_kernel_of(int family) {
  switch (family) {
    case FAM_GBM_STEP:
      return scenario_kernel<FAM_GBM_STEP, SMP, TECH>;
    case FAM_GBM_TERMINAL:
      return scenario_kernel<FAM_GBM_TERMINAL, SMP, TECH>;
    case FAM_HESTON:
      return scenario_kernel<FAM_HESTON, SMP, TECH>;
    default:
      return nullptr;
  }
}

template <int SMP, int TECH>
static cudaError_t launch_scen_t(int family, const DevReq& q, const ScenarioLegs& legs, const SrcCtx& ctx, int grid,
                                 cudaStream_t stream) {
  const size_t smem = fused_dynamic_smem<SMP>();
  const ScenarioKernel kernel = scenario_kernel_of<SMP, TECH>(family);
  if (!kernel) return cudaErrorInvalidValue;
  const cudaError_t e = allow_dynamic_smem((const void*)kernel, smem);
  if (e != cudaSuccess) return e;
  kernel<<<grid, kFusedBlock, smem, stream>>>(q, legs, ctx);
  count_launch();
  return cudaGetLastError();
}

template <int SMP>
static cudaError_t launch_scen_s(int family, int technique, const DevReq& q, const ScenarioLegs& legs,
                                 const SrcCtx& ctx, int grid, cudaStream_t stream) {
  switch (technique) {
    case kScenStd:
      return launch_scen_t<SMP, kScenStd>(family, q, legs, ctx, grid, stream);
    case kScenAnti:
      return launch_scen_t<SMP, kScenAnti>(family, q, legs, ctx, grid, stream);
    case kScenCv:
      return launch_scen_t<SMP, kScenCv>(family, q, legs, ctx, grid, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

template <int SMP, int TECH>
static int scen_occ_t(int family) {
  int n = 0;
  const size_t smem = fused_dynamic_smem<SMP>();
  const ScenarioKernel kernel = scenario_kernel_of<SMP, TECH>(family);
  if (!kernel || allow_dynamic_smem((const void*)kernel, smem) != cudaSuccess) return 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kFusedBlock, smem);
  return n;
}

template <int SMP>
static int scen_occ_s(int family, int technique) {
  if (technique == kScenAnti) return scen_occ_t<SMP, kScenAnti>(family);
  if (technique == kScenCv) return scen_occ_t<SMP, kScenCv>(family);
  return scen_occ_t<SMP, kScenStd>(family);
}

int scenario_max_blocks_per_sm(int family, int sampler, int technique) {
  if (sampler == SMP_XORSHIFT) return scen_occ_s<SMP_XORSHIFT>(family, technique);
  if (sampler == SMP_SOBOL) return scen_occ_s<SMP_SOBOL>(family, technique);
  if (sampler == SMP_COUNTER) return scen_occ_s<SMP_COUNTER>(family, technique);
  return 0;
}

cudaError_t launch_scenarios(const DevReq& q, const ScenarioLegs& legs, int family, int sampler, int technique,
                             const DeviceTables& tabs, int grid, cudaStream_t stream) {
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr};
  switch (sampler) {
    case SMP_XORSHIFT:
      return launch_scen_s<SMP_XORSHIFT>(family, technique, q, legs, ctx, grid, stream);
    case SMP_SOBOL:
      return launch_scen_s<SMP_SOBOL>(family, technique, q, legs, ctx, grid, stream);
    case SMP_COUNTER:
      return launch_scen_s<SMP_COUNTER>(family, technique, q, legs, ctx, grid, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

// ------------------------------------------- basket scenario (bump) kernel ---
// Bump legs of a d-asset basket with common random numbers.  A path draws
// its n_steps x D normals once and keeps only the per-asset sums Z_a; the
// correlated sums are W = L Z (L the Cholesky factor), and leg s prices
//   basket_s = sum_a wspot[s][a] exp(log_drift[s][a] + step_vol[s][a] W_a)
// (basket_terminal_payoff, cpu.rs:7616-7635, with the stepwise log return
// sum_steps (drift_dt + vol_dt zc) regrouped as T drift + vol_dt W).  The
// moment reduction is that of scenario_kernel: per-warp FP64 slots, tile
// partials in warp order, the last tile sums the partials in tile order.
template <int D, class Src>
__device__ __forceinline__ void scen_basket_d(const DevReq& q, Src& src, const BasketScen& legs,
                                              float pay[kBasketScen]) {
  float zs[D];
  sum_step_normals<float, D>(src, q.n_steps, zs);
  float w[D];
#pragma unroll
  for (int a = 0; a < D; ++a) {
    float acc = 0.0f;
#pragma unroll
    for (int b = 0; b <= a; ++b) acc += (float)q.chol[a * D + b] * zs[b];
    w[a] = acc;
  }
  const float kk = (float)q.k;
#pragma unroll
  for (int s = 0; s < kBasketScen; ++s) {
    float basket = 0.0f;
#pragma unroll
    for (int a = 0; a < D; ++a) basket += legs.wspot[s][a] * ex<float>(legs.log_drift[s][a] + legs.step_vol[s][a] * w[a]);
    pay[s] = (basket - kk > 0.0f ? basket - kk : 0.0f) * legs.discount[s];
  }
}

template <class Src>
__device__ __forceinline__ void scen_basket(const DevReq& q, Src& src, const BasketScen& legs,
                                            float pay[kBasketScen]) {
  switch (q.n_assets) {
    case 1:
      scen_basket_d<1>(q, src, legs, pay);
      break;
    case 2:
      scen_basket_d<2>(q, src, legs, pay);
      break;
    case 3:
      scen_basket_d<3>(q, src, legs, pay);
      break;
    case 4:
      scen_basket_d<4>(q, src, legs, pay);
      break;
    case 5:
      scen_basket_d<5>(q, src, legs, pay);
      break;
    case 6:
      scen_basket_d<6>(q, src, legs, pay);
      break;
    case 7:
      scen_basket_d<7>(q, src, legs, pay);
      break;
    default:
      scen_basket_d<8>(q, src, legs, pay);
      break;
  }
}

// One basket request split into q.n_tiles tiles of q.tile_units units.
template <int SMP>
__global__ void __launch_bounds__(kFusedBlock, 2) basket_scenario_kernel(const __grid_constant__ DevReq sq, SrcCtx ctx,
                                                                        const __grid_constant__ BasketScen legs) {
  extern __shared__ __align__(16) uint32_t sobol_window[];
  if constexpr (SMP == SMP_SOBOL) {
    float4* seg = reinterpret_cast<float4*>(sobol_window + kSobolWindowWords);
    const float4* src = reinterpret_cast<const float4*>(ctx.sobol + MPC_ICDF_OFFSET);
    for (uint32_t i = threadIdx.x; i < MPC_ICDF_SEGMENTS; i += blockDim.x) seg[i] = src[i];
    ctx.win = sobol_window;
    ctx.icdf = seg;
  } else {
    ctx.win = nullptr;
    ctx.icdf = nullptr;
  }
  __shared__ double slots[kWarps][kBasketScen][2];
  __shared__ uint32_t s_tile;
  __shared__ int s_last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t n_tiles = sq.n_tiles;
  for (uint32_t t = blockIdx.x; t < n_tiles; t = next_scenario_tile(sq, &s_tile)) {
    for (uint32_t i = threadIdx.x; i < kWarps * kBasketScen * 2; i += blockDim.x) (&slots[0][0][0])[i] = 0.0;
    __syncthreads();
    const uint64_t first = (uint64_t)t * sq.tile_units;
    const uint64_t last = min(first + (uint64_t)sq.tile_units, sq.n_units);
    const uint32_t iters = (uint32_t)((last - first + blockDim.x - 1) / blockDim.x);
    for (uint32_t it = 0; it < iters; ++it) {
      uint64_t u = first + threadIdx.x + (uint64_t)it * blockDim.x;
      const bool valid = u < last;
      if (!valid) u = last - 1;  // lockstep for block- and warp-synchronous sources; discarded below
      typename FusedUnitSource<FAM_BASKET, SMP>::type src;  // the samples fused_unit<FAM_BASKET, SMP> draws
      src.template begin<false>(sq, ctx, u);
      float pay[kBasketScen];
      scen_basket(sq, src, legs, pay);
#pragma unroll
      for (int s = 0; s < kBasketScen; ++s) {
        const double p = valid ? (double)pay[s] : 0.0;
        const double a = warp_sum(p), b = warp_sum(p * p);
        if (lane == 0) {
          slots[warp][s][0] += a;
          slots[warp][s][1] += b;
        }
      }
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)(2 * kBasketScen)) {
      const int s = threadIdx.x >> 1, k = threadIdx.x & 1;
      double sum = 0.0;
      for (int w = 0; w < kWarps; ++w) sum += slots[w][s][k];
      sq.partials[((size_t)t * kBasketScen + s) * 2 + k] = sum;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = (atomicAdd(sq.tiles_done, 1u) == n_tiles - 1) ? 1 : 0;
    __syncthreads();
    if (s_last) {
      __threadfence();
      sum_rows(sq.partials, n_tiles, kBasketScen * 2, kBasketScen * 2, &slots[0][0][0], sq.moments);
    }
  }
  if (threadIdx.x == 0 && atomicAdd(sq.tiles_done + 2, 1u) == gridDim.x - 1)
    sq.tiles_done[0] = sq.tiles_done[1] = sq.tiles_done[2] = 0u;
}

template <int SMP>
static cudaError_t launch_basket_scen_s(const DevReq& q, const SrcCtx& ctx, const BasketScen& legs, int grid,
                                        cudaStream_t stream) {
  const cudaError_t e = allow_dynamic_smem((const void*)basket_scenario_kernel<SMP>, fused_dynamic_smem<SMP>());
  if (e != cudaSuccess) return e;
  basket_scenario_kernel<SMP><<<grid, kFusedBlock, fused_dynamic_smem<SMP>(), stream>>>(q, ctx, legs);
  count_launch();
  return cudaGetLastError();
}

template <int SMP>
static int basket_scen_occ() {
  int n = 0;
  if (allow_dynamic_smem((const void*)basket_scenario_kernel<SMP>, fused_dynamic_smem<SMP>()) != cudaSuccess)
    return 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, basket_scenario_kernel<SMP>, kFusedBlock, fused_dynamic_smem<SMP>());
  return n;
}

int basket_scenario_max_blocks_per_sm(int sampler) {
  if (sampler == SMP_XORSHIFT) return basket_scen_occ<SMP_XORSHIFT>();
  if (sampler == SMP_SOBOL) return basket_scen_occ<SMP_SOBOL>();
  if (sampler == SMP_COUNTER) return basket_scen_occ<SMP_COUNTER>();
  return 0;
}

cudaError_t launch_basket_scenarios(const DevReq& q, int sampler, const BasketScen& legs, const DeviceTables& tabs,
                                    int grid, cudaStream_t stream) {
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr};
  switch (sampler) {
    case SMP_XORSHIFT:
      return launch_basket_scen_s<SMP_XORSHIFT>(q, ctx, legs, grid, stream);
    case SMP_SOBOL:
      return launch_basket_scen_s<SMP_SOBOL>(q, ctx, legs, grid, stream);
    case SMP_COUNTER:
      return launch_basket_scen_s<SMP_COUNTER>(q, ctx, legs, grid, stream);
    default:
      return cudaErrorInvalidValue;
  }
}

// ---------------------------------------- reference v1 kernel contract ----
// Same buffers and scalars as mc_cuda_european_call_stepwise_v1
// (european_call_stepwise_v1.cu:1-28): path-major FP64 normals, one path per
// thread, per-path discounted payoff.  Index arithmetic in 64 bits.
__global__ void __launch_bounds__(256) european_call_stepwise_v1_kernel(const double* __restrict__ normals,
                                                                       double* __restrict__ payoffs,
                                                                       int32_t n_paths, int32_t n_steps,
                                                                       double log_s0, double strike,
                                                                       double drift_dt, double vol_dt,
                                                                       double discount) {
  const int64_t path = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (path >= n_paths) return;
  double ls = log_s0;
  const double* z = normals + path * (int64_t)n_steps;
  for (int32_t s = 0; s < n_steps; ++s) ls += drift_dt + vol_dt * z[s];
  const double st = exp(ls);
  payoffs[path] = st > strike ? (st - strike) * discount : 0.0;
}

cudaError_t launch_european_call_stepwise_v1(const double* normals, double* payoffs, int32_t n_paths,
                                             int32_t n_steps, double log_s0, double strike, double drift_dt,
                                             double vol_dt, double discount, cudaStream_t stream) {
  if (n_paths <= 0) return cudaSuccess;
  int grid = (int)((n_paths + 255) / 256);
  european_call_stepwise_v1_kernel<<<grid, 256, 0, stream>>>(normals, payoffs, n_paths, n_steps, log_s0, strike,
                                                              drift_dt, vol_dt, discount);
  count_launch();
  return cudaGetLastError();
}

// ------------------------------------------------------------------ LSM ---
__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

constexpr int kLsmBlock = (int)kLsmThreads;

constexpr int kLsmMaxP = (int)kLsmPathsPerThreadMax;
constexpr int kLsmMom = 15;  // 10 unique A^T A, 4 A^T b, ITM count

// Records the first failed self-check of an LSM job (code and index).
__device__ __noinline__ void lsm_report(const LsmArgs& a, int code, uint64_t index) {
  if (atomicCAS(a.error, 0, code) == 0) {
    *(volatile unsigned long long*)a.diag = (unsigned long long)index;  // status and diag: mapped host memory
    *(volatile int*)a.status = code;
  }
}
__device__ __forceinline__ bool lsm_ok(const LsmArgs& a, uint64_t index, uint64_t len, int code) {
  if (index < len) return true;
  lsm_report(a, code, index);
  return false;
}

// Warp sums of 16 values per lane by reduce-scatter: in each of four rounds a
// lane keeps half of its values and adds the partner's copy of that half
// (partner lane ^ 16, ^ 8, ^ 4, ^ 2), then lanes l and l ^ 1 add their last
// value.  Lane l ends with the warp sum of value brev4(l >> 1) (lanes l and
// l ^ 1 hold the same bits): 16 double shuffles instead of 80 for 16 separate
// butterflies, in a fixed order.
template <class T>
__device__ __forceinline__ T warp_reduce_scatter16(T (&v)[16]) {
  const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int o = 16 >> r, c = 8 >> r;
    const bool up = (lane & (uint32_t)o) != 0;
#pragma unroll
    for (int i = 0; i < c; ++i) {
      const T send = up ? v[i] : v[i + c];
      const T keep = up ? v[i + c] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}
__device__ __forceinline__ uint32_t reduce_scatter16_index(uint32_t lane) {
  return (((lane >> 4) & 1u) << 3) | (((lane >> 3) & 1u) << 2) | (((lane >> 2) & 1u) << 1) | ((lane >> 1) & 1u);
}

// One exercise date's regression across the job's blocks (round = the date's
// position in the backward pass).  Every block writes its 15 moments to its
// own slot row partials[round][lb] with relaxed stores; the host marks every
// slot empty (all bits set) before the launch and no slot is written twice,
// so the data is its own arrival flag: each block reads every block's slots
// of the round at once and re-reads (bounded) only those still empty, with no
// fence, counter or separate poll between the write and the read.  Then every
// block sums the partials itself in the same fixed order (thread t: moment
// t % 16 over blocks t / 16, t / 16 + 32, ...; the lane groups' sums by a
// shuffle, then lane m of warp 0 over the 16 warps) and solves the normal
// equations in thread 0: the same operations on the same data, so
// every block holds the same coefficients, with no publication round trip
// after the solve.  The FP32 path scales each pivot row by the pivot's
// reciprocal instead of dividing every entry (the FP64 path divides, as the
// reference does).  The wait is bounded: after timeout_ns the block records
// kLsmErrTimeout and every block of the job leaves at its next check.
// Returns false when the job's error flag is set.
// Empty marker of a date's partial slot (all bits set); the host fills the
// partials with it before the launch, and a written value never equals it.
constexpr unsigned long long kLsmEmpty = 0xFFFFFFFFFFFFFFFFull;
__device__ __forceinline__ unsigned long long ld_relaxed_u64(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_f64(double* p, double x) {
  unsigned long long v = (unsigned long long)__double_as_longlong(x);
  if (v == kLsmEmpty) v = 0x7FF8000000000001ull;  // a NaN with the marker's bits: keep it a NaN
  asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}
// Sums of the 16 warps' values of moment `mom` (0..15), in two fixed chains.
__device__ __forceinline__ double sum_warps16(const double* rows, uint32_t mom) {
  double e = rows[mom], o = rows[17 + mom];
#pragma unroll
  for (int w = 2; w < 16; w += 2) {
    e += rows[w * 17 + mom];
    o += rows[(w + 1) * 17 + mom];
  }
  return e + o;
}
// s_bad: shared flag, 0 until a wait fails (then the job's blocks all leave).
template <bool RECIP>
__device__ __forceinline__ bool lsm_gather_solve(const LsmArgs& a, uint32_t nb, uint32_t round, int coeffs,
                                                 double* fold, double* s_mom, double* s_beta, int* s_ok, int* s_bad) {
  const uint64_t base_at = (uint64_t)round * nb * 16;
  const uint32_t mom = threadIdx.x & 15u, lane_grp = threadIdx.x >> 4, n_grp = blockDim.x >> 4;
  double acc = 0.0;
  if (mom < (uint32_t)kLsmMom && lsm_ok(a, base_at + (uint64_t)nb * 16 - 1, a.partials_len, kLsmErrPartials)) {
    // every load of the thread's blocks issued at once; the slots still empty
    // are read again (bounded) until their blocks have written them; then
    // the values are summed in block order
    constexpr int kBatch = 8;
    const uint64_t start = global_ns();
    for (uint32_t blk0 = lane_grp; blk0 < nb; blk0 += kBatch * n_grp) {
      unsigned long long v[kBatch];
#pragma unroll
      for (int i = 0; i < kBatch; ++i) {
        const uint32_t blk = blk0 + (uint32_t)i * n_grp;
        v[i] = blk < nb ? ld_relaxed_u64(a.partials + base_at + (size_t)blk * 16 + mom) : 0ull;
      }
      for (;;) {
        bool pending = false;
#pragma unroll
        for (int i = 0; i < kBatch; ++i) {
          if (v[i] != kLsmEmpty) continue;
          pending = true;
          v[i] = ld_relaxed_u64(a.partials + base_at + (size_t)(blk0 + (uint32_t)i * n_grp) * 16 + mom);
        }
        if (!pending) break;
        if (*((volatile int*)a.error) != 0) {
          *s_bad = 1;
          break;
        }
        if (global_ns() - start > a.timeout_ns) {
          lsm_report(a, kLsmErrTimeout, round);
          *s_bad = 1;
          break;
        }
      }
#pragma unroll
      for (int i = 0; i < kBatch; ++i) acc += __longlong_as_double((long long)v[i]);
    }
  }
  __syncwarp();
  acc += __shfl_xor_sync(0xffffffffu, acc, 16);  // the warp's two lane groups
  if ((threadIdx.x & 31u) < 16u) fold[(threadIdx.x >> 5) * 17 + mom] = acc;
  __syncthreads();
  if (*s_bad) return false;
  if (threadIdx.x < 32u) {
    if (threadIdx.x < (uint32_t)kLsmMom) s_mom[threadIdx.x] = sum_warps16(fold, threadIdx.x);
    __syncwarp();
  }
  if (threadIdx.x == 0) {
    double ata[4][4], atb[4];
    int idx = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = r; c < 4; ++c) {
        ata[r][c] = s_mom[idx];
        ata[c][r] = s_mom[idx];
        ++idx;
      }
#pragma unroll
    for (int r = 0; r < 4; ++r) atb[r] = s_mom[10 + r];
    // rows and columns past the basis degree are never read
    int ok = s_mom[14] >= (double)coeffs ? 1 : 0;
    if (ok)
      ok = (coeffs == 2   ? solve_fixed<2, RECIP>(ata, atb)
            : coeffs == 3 ? solve_fixed<3, RECIP>(ata, atb)
                          : solve_fixed<4, RECIP>(ata, atb))
               ? 1
               : 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) s_beta[r] = (ok && r < coeffs) ? atb[r] : 0.0;
    *s_ok = ok;
  }
  __syncthreads();
  return true;
}

// One 512-thread block per SM: the same warps per SM as two 256-thread
// blocks, but half the block partials to fold per date (the per-date
// cross-block round is this kernel's critical path).
// Bound by the latency of the date rounds (moments, one exchange through L2,
// the solve, the exercise pass, at 16 warps an SM) and by the path generation
// before them.  524,288 paths x 50 dates on a B200, before -> now: generation 96
// -> 76 us (pairs of normals), a round 4.84 -> 4.22 us in FP32 and 7.86 -> 5.86
// in FP64 (x^3 / 6 without a division, Newton reciprocals in the solve, three
// block barriers a round instead of five, and the generation loop not unrolled:
// with eight copies of the sampling code a round took 5.8 us).
template <class Real, int SMP>
__global__ void __launch_bounds__(kLsmBlock, 1) lsm_kernel(const LsmArgs* __restrict__ jobs, uint32_t n_jobs, SrcCtx ctx) {
  __shared__ double red[kLsmBlock / 32][5];
  __shared__ double s_mom[16];
  __shared__ double s_beta[4];
  __shared__ int s_ok;
  __shared__ uint32_t s_job;
  __shared__ double s_red15[kLsmBlock / 32][17];
  __shared__ double s_fold[kLsmBlock / 32 * 17];  // [warp][moment] of the fold over the blocks
  __shared__ int s_bad;
  __shared__ Real s_disc[512];
  if (threadIdx.x == 0) {
    uint32_t j = 0;
    while (j + 1 < n_jobs && blockIdx.x >= jobs[j + 1].block_first) ++j;
    s_job = j;
    s_bad = 0;
  }
  __syncthreads();
  const LsmArgs a = jobs[s_job];
  const uint32_t nb = a.n_blocks;             // blocks of this job
  const uint32_t lb = blockIdx.x - a.block_first;  // block index within the job
  const uint64_t n = a.n_paths;
  const uint32_t steps = a.n_steps;
  // launch-shape invariants: this block belongs to the job, the job's blocks
  // cover every path with <= kLsmMaxP paths per thread, the dates fit s_disc
  if (blockIdx.x < a.block_first || lb >= nb) {
    if (threadIdx.x == 0) lsm_report(a, kLsmErrJob, blockIdx.x);
    return;
  }
  if ((uint64_t)nb * blockDim.x * kLsmMaxP < n || steps >= 512 || a.n_sched == 0 || a.n_sched > steps) {
    if (threadIdx.x == 0) lsm_report(a, kLsmErrCoverage, n);
    return;
  }
  for (uint32_t j = threadIdx.x; j <= steps; j += blockDim.x) s_disc[j] = (Real)a.disc_pow[j];
  __syncthreads();
  const uint64_t nthreads = (uint64_t)nb * blockDim.x;
  const uint64_t gtid = (uint64_t)lb * blockDim.x + threadIdx.x;
  Real* paths = reinterpret_cast<Real*>(a.paths);
  const Real k = (Real)a.k, drift = (Real)a.drift, vol = (Real)a.vol, inv_k = (Real)(1.0 / fmax(a.k, 2.2250738585072014e-308));
  const int coeffs = (int)a.degree + 1;
  Real cash[kLsmMaxP];
  uint32_t exd[kLsmMaxP];
  DevReq q;  // sampler view of the request
  q.seed = a.seed;
  q.seed32 = a.seed32;
  q.n_chunks = 1;
  q.normals_per_unit = steps;
  // Pseudorandom sampler: a thread's paths lie nthreads paths apart, so the
  // stream state at each path start after the first is one jump of
  // T^(nthreads x steps) draws (nthreads is even, so the pair alignment of
  // the start carries over), 16 table lookups instead of a full seek.
  uint64_t aligned = 0;
#pragma unroll 1  // one copy of the sampling code: unrolled, it pushes the date loop out of the instruction cache
  for (int j = 0; j < kLsmMaxP; ++j) {
    const uint64_t path = gtid + (uint64_t)j * nthreads;
    if (path >= n) continue;
    // the path's last element bounds all of them
    if (!lsm_ok(a, (uint64_t)(steps - 1) * n + path, a.paths_len, kLsmErrPaths)) continue;
    Real* out = paths + path;
    Real s = (Real)a.s0;
    auto advance = [&](const Real z) {
      s *= ex<Real>(drift + vol * z);  // multiplicative update as cpu.rs:3829-3830
      *out = s;
      out += n;
    };
    if constexpr (SMP == SMP_XORSHIFT) {
      const uint64_t idx = path * steps;
      aligned = (j == 0 || a.stride_jump == nullptr)
                    ? xorshift_jump(ctx.jump, XorshiftStream::first_state(a.seed), 2 * (idx >> 1))
                    : gf2_apply(a.stride_jump, aligned);
      XorshiftPairs<Real> src;
      src.start(aligned, idx);
      uint32_t st = 0;
      for (; st + 2 <= steps; st += 2) {
        const auto z = src.n2(st);
        advance(z.x);
        advance(z.y);
      }
      if (st < steps) advance(src.next());
    } else {
      Source<SMP> src;
      src.template begin<sizeof(Real) == 8>(q, ctx, path);
      for (uint32_t st = 0; st < steps; ++st) advance(normal<Real>(src, st));
    }
  }
#pragma unroll
  for (int j = 0; j < kLsmMaxP; ++j) {  // maturity cashflows, from the thread's own stores
    const uint64_t path = gtid + (uint64_t)j * nthreads;
    cash[j] = (Real)0;
    exd[j] = steps;
    if (path >= n) continue;
    const uint64_t at = (uint64_t)(steps - 1) * n + path;
    if (!lsm_ok(a, at, a.paths_len, kLsmErrPaths)) continue;
    const Real s = paths[at];
    cash[j] = k - s > (Real)0 ? k - s : (Real)0;
  }
  uint32_t regressions = 0, round = 0;
  // The path values of a date are loaded one date ahead, before the
  // cross-block wait of the current date, so their latency hides behind it.
  Real sv_next[kLsmMaxP];
  auto load_date = [&](int si_load) {
    const uint32_t step_load = a.sched[si_load];
#pragma unroll
    for (int j = 0; j < kLsmMaxP; ++j) {
      const uint64_t path = gtid + (uint64_t)j * nthreads;
      sv_next[j] = (Real)0;
      if (path >= n || step_load == 0 || step_load > steps) continue;
      const uint64_t at = (uint64_t)(step_load - 1) * n + path;
      if (lsm_ok(a, at, a.paths_len, kLsmErrPaths)) sv_next[j] = __ldcg(paths + at);
    }
  };
  if (a.n_sched >= 2) load_date((int)a.n_sched - 2);
  for (int si = (int)a.n_sched - 2; si >= 0; --si) {
    const uint32_t step = a.sched[si];
    if (step == 0 || step > steps) {
      if (threadIdx.x == 0) lsm_report(a, kLsmErrSched, step);
    }
    // Each thread sums the 15 moments of its own <= kLsmMaxP paths, the FP32
    // path in FP32 (the warps too; FP64 takes over from the warp sums): 10 of
    // A^T A (the first is the count, as the basis starts with 1), 4 of A^T b.
    Real m[14];
#pragma unroll
    for (int i = 0; i < 14; ++i) m[i] = (Real)0;
    Real sv[kLsmMaxP];
#pragma unroll
    for (int j = 0; j < kLsmMaxP; ++j) sv[j] = sv_next[j];
#pragma unroll
    for (int j = 0; j < kLsmMaxP; ++j) {
      const uint64_t path = gtid + (uint64_t)j * nthreads;
      if (path >= n || step == 0 || step > steps) continue;
      const Real s = sv[j];
      if (!(k - s > (Real)0)) continue;
      if (exd[j] < step || exd[j] > steps) {
        lsm_report(a, kLsmErrDisc, exd[j]);
        continue;
      }
      const Real c = cash[j] * s_disc[exd[j] - step];
      Real b[4];
      laguerre4<Real>(s * inv_k, b);
      int idx = 0;
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int t = r; t < 4; ++t) {
          m[idx] = fma(b[r], b[t], m[idx]);
          ++idx;
        }
#pragma unroll
      for (int r = 0; r < 4; ++r) m[10 + r] = fma(b[r], c, m[10 + r]);
    }
    // block reduction: warp sums by reduce-scatter, then lane m of warp 0 over
    // the 16 warps; the slot's own value marks its arrival (lsm_gather_solve)
    const uint64_t part_at = ((uint64_t)round * nb + lb) * 16;
    {
      Real mv[16];
#pragma unroll
      for (int i = 0; i < 16; ++i) mv[i] = i < 14 ? m[i] : i == 14 ? m[0] : (Real)0;
      const double w = (double)warp_reduce_scatter16(mv);
      const uint32_t lane = threadIdx.x & 31u;
      if ((lane & 1u) == 0) s_red15[threadIdx.x >> 5][reduce_scatter16_index(lane)] = w;
    }
    __syncthreads();
    if (threadIdx.x < (uint32_t)kLsmMom && lsm_ok(a, part_at + threadIdx.x, a.partials_len, kLsmErrPartials))
      st_relaxed_f64(a.partials + part_at + threadIdx.x, sum_warps16(&s_red15[0][0], threadIdx.x));
    if (si > 0) load_date(si - 1);  // next date's values, in flight during the wait
    // Every block waits (bounded) for all blocks' partials of this date, then
    // sums them in block order and solves the normal equations itself.
    if (!lsm_gather_solve<sizeof(Real) == 4>(a, nb, round++, coeffs, s_fold, s_mom, s_beta, &s_ok, &s_bad)) return;
    if (s_ok) {
      ++regressions;
      const Real b0 = (Real)s_beta[0], b1 = (Real)s_beta[1], b2 = (Real)s_beta[2], b3 = (Real)s_beta[3];
#pragma unroll
      for (int j = 0; j < kLsmMaxP; ++j) {
        const uint64_t path = gtid + (uint64_t)j * nthreads;
        if (path >= n) continue;
        const Real imm = k - sv[j];
        if (!(imm > (Real)0)) continue;
        Real b[4];
        laguerre4<Real>(sv[j] * inv_k, b);
        Real cont = b0 * b[0] + b1 * b[1];
        if (coeffs > 2) cont += b2 * b[2];
        if (coeffs > 3) cont += b3 * b[3];
        if (imm > (cont > (Real)0 ? cont : (Real)0)) {
          cash[j] = imm;
          exd[j] = step;
        }
      }
    }
  }
  // estimator: discounted cashflows, exercise counts
  double v[5] = {0, 0, 0, 0, 0};
#pragma unroll
  for (int j = 0; j < kLsmMaxP; ++j) {
    const uint64_t path = gtid + (uint64_t)j * nthreads;
    if (path >= n) continue;
    if (exd[j] > steps) {
      lsm_report(a, kLsmErrDisc, exd[j]);
      continue;
    }
    const double d = (double)cash[j] * a.disc_pow[exd[j]];
    v[0] += d;
    v[1] += d * d;
    if (exd[j] < steps)
      v[2] += 1.0;
    else if (cash[j] > (Real)0)
      v[3] += 1.0;
  }
  block_reduce5(v, red);
  if (threadIdx.x == 0) {
    double* fp = a.final_partials + (size_t)lb * 4;
    if (lsm_ok(a, (uint64_t)lb * 4 + 3, a.final_len, kLsmErrFinal))
      for (int i = 0; i < 4; ++i) fp[i] = v[i];
    __threadfence();
    s_ok = atomicAdd(a.done, 1u) == nb - 1;
  }
  __syncthreads();
  if (s_ok) {
    __threadfence();
    double acc[5] = {0, 0, 0, 0, 0};
    for (uint32_t blk = threadIdx.x; blk < nb; blk += blockDim.x) {
      if (!lsm_ok(a, (uint64_t)blk * 4 + 3, a.final_len, kLsmErrFinal)) break;
      for (int i = 0; i < 4; ++i) acc[i] += __ldcg(a.final_partials + (size_t)blk * 4 + i);
    }
    block_reduce5(acc, red);
    if (threadIdx.x != 0) return;
    a.out[0] = (double)n;
    a.out[1] = acc[0];
    a.out[2] = acc[1];
    a.out[3] = acc[2];
    a.out[4] = acc[3];
    a.out[5] = (double)regressions;
    *a.done = 0u;
  }
}

template <class Real, int SMP>
static uint32_t lsm_capacity_t() {
  // blocks per SM follow from the kernel's registers and shared memory (one
  // architecture), so the first answer above zero stands
  static std::atomic<int> known{0};
  int dev = 0, sms = 148, per_sm = known.load(std::memory_order_relaxed);
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (per_sm <= 0) {
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lsm_kernel<Real, SMP>, kLsmBlock, 0);
    known.store(per_sm, std::memory_order_relaxed);
  }
  return per_sm > 0 ? (uint32_t)(sms * per_sm) : 0u;
}

uint32_t lsm_capacity(int fp64, int sampler) {
  if (fp64) return sampler == SMP_COUNTER ? lsm_capacity_t<double, SMP_COUNTER>() : lsm_capacity_t<double, SMP_XORSHIFT>();
  return sampler == SMP_COUNTER ? lsm_capacity_t<float, SMP_COUNTER>() : lsm_capacity_t<float, SMP_XORSHIFT>();
}

template <class Real, int SMP>
static cudaError_t launch_lsm_t(const LsmArgs* jobs, uint32_t n_jobs, uint32_t total_blocks, const SrcCtx& ctx,
                                cudaStream_t stream) {
  if (total_blocks == 0 || total_blocks > lsm_capacity_t<Real, SMP>()) return cudaErrorInvalidValue;
  const LsmArgs* j = jobs;
  uint32_t nj = n_jobs;
  SrcCtx c = ctx;
  void* params[] = {&j, &nj, &c};
  cudaError_t err = cudaLaunchCooperativeKernel((const void*)lsm_kernel<Real, SMP>, dim3(total_blocks),
                                                dim3(kLsmBlock), params, 0, stream);
  count_launch();
  return err;
}

cudaError_t launch_lsm_batch(const LsmArgs* d_jobs, uint32_t n_jobs, uint32_t total_blocks, int fp64, int sampler,
                             const DeviceTables& tabs, cudaStream_t stream) {
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr};
  if (fp64) {
    if (sampler == SMP_COUNTER) return launch_lsm_t<double, SMP_COUNTER>(d_jobs, n_jobs, total_blocks, ctx, stream);
    return launch_lsm_t<double, SMP_XORSHIFT>(d_jobs, n_jobs, total_blocks, ctx, stream);
  }
  if (sampler == SMP_COUNTER) return launch_lsm_t<float, SMP_COUNTER>(d_jobs, n_jobs, total_blocks, ctx, stream);
  return launch_lsm_t<float, SMP_XORSHIFT>(d_jobs, n_jobs, total_blocks, ctx, stream);
}

// ------------------------------------------------------ single-pass Greeks ---
// european_call_pathwise_greeks_cpu / european_call_likelihood_ratio_greeks_cpu
// (cpu.rs:4670-4869): path i draws normal i of MonteCarloRng(seed) (one
// sequential stream, replayed by jump-ahead), prices the terminal GBM state
// and records the per-path estimators; sums and sums of squares in FP64,
// combined in block order by the last block.
template <class Real>
__global__ void __launch_bounds__(256) greeks_single_pass_kernel(GreekArgs a, const uint64_t* __restrict__ jump) {
  __shared__ double red[kWarps][5];
  __shared__ int s_last;
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  const Real s0 = (Real)a.s0, k = (Real)a.k, r = (Real)a.r, sigma = (Real)a.sigma, t = (Real)a.t;
  const Real sqrt_t = (Real)a.sqrt_t, drift_t = (Real)a.drift_t, vol_t = (Real)a.vol_t, disc = (Real)a.discount;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.n_paths; i += stride) {
    XorshiftStream st;
    st.seek(jump, a.seed, i, sizeof(Real) == 4);
    const Real z = sizeof(Real) == 4 ? (Real)st.normal_f32() : (Real)st.normal_f64();
    const Real s = s0 * ex<Real>(drift_t + vol_t * z);
    Real g[4];
    if (a.estimator == MPC_GREEKS_PATHWISE) {
      const Real intrinsic = s - k;
      const bool active = intrinsic > (Real)0;
      const Real payoff = intrinsic > (Real)0 ? intrinsic : (Real)0;
      const Real dpay = disc * payoff;
      g[0] = active ? disc * s / s0 : (Real)0;
      g[1] = active ? disc * s * (-sigma * t + sqrt_t * z) : (Real)0;
      g[2] = active ? disc * (t * s - t * payoff) : -t * dpay;
      const Real dst_dt = s * (r - (Real)0.5 * sigma * sigma + sigma * z / ((Real)2 * sqrt_t));
      g[3] = -(active ? disc * (dst_dt - r * payoff) : -r * dpay);
    } else {
      const Real dpay = disc * (s - k > (Real)0 ? s - k : (Real)0);
      g[0] = dpay * z / (s0 * sigma * sqrt_t);
      g[1] = dpay * ((z * z - (Real)1) / sigma - sqrt_t * z);
      g[2] = dpay * (z / (sigma * sqrt_t) - t);
      g[3] = (Real)0;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const double v = (double)g[j];
      acc[2 * j] += v;
      acc[2 * j + 1] += v * v;
    }
  }
  double v0[5] = {acc[0], acc[1], acc[2], acc[3], acc[4]};
  double v1[5] = {acc[5], acc[6], acc[7], 0.0, 0.0};
  block_reduce5(v0, red);
  block_reduce5(v1, red);
  if (threadIdx.x == 0) {
    double* pt = a.partials + (size_t)blockIdx.x * 8;
    for (int j = 0; j < 5; ++j) pt[j] = v0[j];
    for (int j = 0; j < 3; ++j) pt[5 + j] = v1[j];
    __threadfence();
    s_last = atomicAdd(a.done, 1u) == gridDim.x - 1 ? 1 : 0;
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  {  // 32 rows at a time (a row per 8 lanes), then the lanes' and warps' sums in a fixed order
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, col = lane & 7u;
    double sum = 0.0;
#pragma unroll 4
    for (uint32_t b = warp * 4 + (lane >> 3); b < gridDim.x; b += kWarps * 4) sum += __ldcg(a.partials + (size_t)b * 8 + col);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 8);
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, 16);
    __shared__ double s_cols[kWarps][8];
    if (lane < 8) s_cols[warp][col] = sum;
    __syncthreads();
    if (threadIdx.x < 8) {
      double total = 0.0;
      for (int w = 0; w < kWarps; ++w) total += s_cols[w][threadIdx.x];
      a.out[threadIdx.x] = total;
    }
  }
  if (threadIdx.x == 0) *a.done = 0u;
}

cudaError_t launch_greeks_single_pass(const GreekArgs& a, uint32_t grid, const DeviceTables& tabs,
                                      cudaStream_t stream) {
  if (a.fp64)
    greeks_single_pass_kernel<double><<<grid, 256, 0, stream>>>(a, tabs.jump);
  else
    greeks_single_pass_kernel<float><<<grid, 256, 0, stream>>>(a, tabs.jump);
  count_launch();
  return cudaGetLastError();
}

// ------------------------------------------------------------ generators ---
template <int SMP>
__global__ void __launch_bounds__(256) generate_kernel(DevReq q, int fp32, void* out, uint64_t n_points,
                                                       uint32_t dims, SrcCtx ctx) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t p = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; p < n_points; p += stride) {
    Source<SMP> src;
    if (fp32) {
      src.template begin<false>(q, ctx, p);
      float* o = reinterpret_cast<float*>(out) + p * dims;
      for (uint32_t d = 0; d < dims; ++d) o[d] = src.n32(d);
    } else {
      src.template begin<true>(q, ctx, p);
      double* o = reinterpret_cast<double*>(out) + p * dims;
      for (uint32_t d = 0; d < dims; ++d) o[d] = src.n64(d);
    }
  }
}

cudaError_t launch_generate_normals(const DevReq& q, int sampler, int fp32, void* d_out, uint64_t n_points,
                                    uint32_t dims, const DeviceTables& tabs, cudaStream_t stream) {
  SrcCtx ctx{tabs.sobol, tabs.jump, nullptr};
  uint64_t want = (n_points + 255) / 256;
  int grid = (int)(want < 4096 ? want : 4096);
  if (grid < 1) grid = 1;
  switch (sampler) {
    case SMP_XORSHIFT:
      generate_kernel<SMP_XORSHIFT><<<grid, 256, 0, stream>>>(q, fp32, d_out, n_points, dims, ctx);
      break;
    case SMP_HALTON:
      generate_kernel<SMP_HALTON><<<grid, 256, 0, stream>>>(q, fp32, d_out, n_points, dims, ctx);
      break;
    case SMP_LHS:
      generate_kernel<SMP_LHS><<<grid, 256, 0, stream>>>(q, fp32, d_out, n_points, dims, ctx);
      break;
    case SMP_SOBOL:
      generate_kernel<SMP_SOBOL><<<grid, 256, 0, stream>>>(q, fp32, d_out, n_points, dims, ctx);
      break;
    case SMP_COUNTER:
      generate_kernel<SMP_COUNTER><<<grid, 256, 0, stream>>>(q, fp32, d_out, n_points, dims, ctx);
      break;
    default:
      return cudaErrorInvalidValue;
  }
  count_launch();
  return cudaGetLastError();
}

__global__ void counter_hash_kernel(uint32_t seed, uint32_t n_paths, uint32_t n_steps, uint32_t* out) {
  const uint64_t total = (uint64_t)n_paths * n_steps;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint32_t path = (uint32_t)(i / n_steps), step = (uint32_t)(i % n_steps);
    out[2 * i] = hash_u32(counter_mix(seed, path, step, 0u));
    out[2 * i + 1] = hash_u32(counter_mix(seed, path, step, 1u));
  }
}

cudaError_t launch_counter_hash(uint32_t seed, uint32_t n_paths, uint32_t n_steps, uint32_t* d_out,
                                cudaStream_t stream) {
  uint64_t total = (uint64_t)n_paths * n_steps;
  int grid = (int)((total + 255) / 256 < 4096 ? (total + 255) / 256 : 4096);
  if (grid < 1) grid = 1;
  counter_hash_kernel<<<grid, 256, 0, stream>>>(seed, n_paths, n_steps, d_out);
  count_launch();
  return cudaGetLastError();
}

// Each thread emits 64 consecutive draws after one jump.
__global__ void xorshift_kernel(uint64_t seed, uint64_t offset, uint64_t count, uint64_t* out, const uint64_t* jump) {
  const uint64_t chunk = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const uint64_t first = chunk * 64;
  if (first >= count) return;
  XorshiftStream st;
  uint64_t s0 = seed == 0 ? 0x9E3779B97F4A7C15ull : seed;
  st.state = xorshift_jump(jump, s0, offset + first);
  st.has_cached = false;
  const uint64_t last = first + 64 < count ? first + 64 : count;
  for (uint64_t i = first; i < last; ++i) out[i] = st.next_u64();
}

cudaError_t launch_xorshift(uint64_t seed, uint64_t offset, uint64_t count, uint64_t* d_out,
                            const DeviceTables& tabs, cudaStream_t stream) {
  uint64_t chunks = (count + 63) / 64;
  int grid = (int)((chunks + 255) / 256);
  if (grid < 1) grid = 1;
  xorshift_kernel<<<grid, 256, 0, stream>>>(seed, offset, count, d_out, tabs.jump);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_flush(void* d_buf, size_t bytes, cudaStream_t stream) {
  count_launch();
  return cudaMemsetAsync(d_buf, (int)(g_launches.load() & 0xFF), bytes, stream);
}

}  // namespace mpc
