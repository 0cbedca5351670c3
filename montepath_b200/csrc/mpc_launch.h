// mpc_launch.h -- host-side launch wrappers of the kernels in mpc_kernels.cu.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/montepath_cuda.h"
#include "mpc_types.h"

namespace mpc {

struct DeviceTables {
  const uint32_t* sobol;  // [256][8][16] nibble tables
  const uint64_t* jump;   // [64][16][16] xorshift jump nibble tables
  const uint64_t* lane_jump;  // [16][16][32] (q, v, lane): v << 4q jumped kMertonRun * lane draws; contexts only
  const double* icdf_tail;    // [MPC_ICDF_TAIL] lower tail of the FP64 inverse normal; contexts only
};

// Work of one fused launch (a kernel parameter): up to kFusedInline requests
// held in the parameter itself, or a tile list over descriptors in device
// memory.  Tile t of an inline launch belongs to the request r with
// first[r] <= t < first[r + 1].  `counter` is the work list's cursor, zero at
// launch; an inline launch has two words there and leaves them zero.
constexpr uint32_t kFusedInline = 4;
struct FusedWork {
  uint32_t n_tiles, n_inline;   // n_inline 0: reqs and tiles
  uint32_t* counter;
  const DevReq* reqs;
  const Tile* tiles;
  uint32_t first[kFusedInline + 4];
  DevReq inl[kFusedInline];
};

// Fused FP32 path: one persistent launch over a tile work list.  All
// requests of the launch must share `sampler`; `family` < 0 lets each tile
// switch on its request's family (mixed batches).
cudaError_t launch_fused(const FusedWork& work, int family, int sampler, const DeviceTables& tabs, int grid, int block,
                         cudaStream_t stream);
int fused_max_blocks_per_sm(int family, int sampler, int block);

// Resident serving loop (mpc_server mode 2): one persistent launch that
// takes pricing work as the host publishes it.  The host copies entries into
// a ring in device memory and then advances `tail` (the doorbell, also in
// device memory, copied after the entries on the same stream, so the loop's
// polls stay in L2 and never cross PCIe); every block claims tiles
// of the oldest entry that still has some (a 64-bit compare-and-swap on the
// slot's claim word, generation << 32 | next tile, so a claim can never land
// on a slot's later request), runs them through the fused tile body of the
// entry's sampler (xorshift, counter hash or Sobol; any family), and the
// block that finishes a request's last tile writes its moments into mapped
// host memory and then the request's generation into done[slot].  Blocks
// leave when the host sets stop or pause, or after idle_ns without work;
// every wait is a bounded poll.
struct LoopEntry {
  uint32_t slot, gen, n_tiles, pos;  // pos: absolute ring position (detects a reused ring entry)
};
struct LoopArgs {
  const DevReq* slots;           // device [max_slots]: slot descriptors
  unsigned long long* claim;     // device [max_slots]: gen << 32 | next tile
  const LoopEntry* ring;         // device [ring_cap]
  const uint32_t* doorbell;      // device, 16-byte aligned: [0] tail (entries published), [1] stop, [2] pause
  uint32_t* done;                // mapped host [max_slots]: generation finished last
  uint32_t ring_cap, max_slots;
  uint64_t idle_ns;
  uint32_t reserve_sms;          // blocks that start on an SM with %smid below this leave at once
  uint32_t _pad;
};
cudaError_t launch_serve_loop(const LoopArgs& a, const DeviceTables& tabs, int grid, cudaStream_t stream);
int serve_loop_blocks_per_sm();

// FP64 plain path: one launch per request (q.n_tiles blocks of kPlainBlock
// threads), moments written to q.moments by the last block; *q.tiles_done is
// zero before and after.
constexpr uint32_t kPlainBlock = 128;
cudaError_t launch_plain(const DevReq& q, int sampler, const DeviceTables& tabs, cudaStream_t stream);
// The same for pseudorandom stepwise GBM with `lanes` (2 to 32, a power of two)
// threads per path, q.tile_units * lanes = kPlainBlock; each lane holds at most
// kPlainSplitNormals normals.
constexpr uint32_t kPlainSplitNormals = 32;
cudaError_t launch_plain_split(const DevReq& q, const DeviceTables& tabs, uint32_t lanes, cudaStream_t stream);
// Fills the MPC_ICDF_TAIL values of DeviceTables::icdf_tail.
cudaError_t launch_icdf_tail(double* d_out, cudaStream_t stream);

// Reference kernel contract mc_cuda_european_call_stepwise_v1.
cudaError_t launch_european_call_stepwise_v1(const double* normals, double* payoffs, int32_t n_paths,
                                             int32_t n_steps, double log_s0, double strike, double drift_dt,
                                             double vol_dt, double discount, cudaStream_t stream);

// Longstaff-Schwartz: one cooperative launch (paths, backward induction, estimator).
struct LsmArgs {
  uint64_t n_paths;
  uint32_t n_steps, n_sched, degree, sampler;
  uint64_t seed;
  uint32_t seed32, fp64;
  double s0, k, drift, vol, disc_step;
  const uint32_t* sched;     // exercise dates (ascending, ends with n_steps)
  const double* disc_pow;    // disc_step^j, j = 0..n_steps
  const uint64_t* stride_jump;  // pseudorandom sampler: nibble table [16][16] of T^(grid threads x n_steps),
                                // the stream jump between a thread's successive paths
  void* paths;               // [n_steps][n_paths] float or double
  double* partials;          // [rounds][grid][16], every slot empty (all bits set) at launch
  double* final_partials;    // [grid][4]
  double* out;               // [8] in mapped host memory: n, sum, sumsq, early, maturity, regressions, -, -
  unsigned* done;            // last-block counter (zero before and after)
  int* error;                // first failure: kLsmErr* code (0 = none), device memory
  int* status;               // the same code, mapped host memory
  unsigned long long* diag;  // offending index of a failed self-check, mapped host memory
  uint64_t timeout_ns;
  uint32_t block_first;      // this job's blocks in the batched launch
  uint32_t n_blocks;
  uint64_t paths_len;        // elements allocated for `paths`
  uint32_t partials_len;     // elements allocated for `partials`
  uint32_t final_len;        // elements allocated for `final_partials`
};
// Failure codes written to LsmArgs::error.  Every indexed global or shared
// access of the kernel is checked against its allocation; a failed check
// records its code and index, skips the access and makes every block of the
// job leave at the next barrier.
enum : int {
  kLsmErrTimeout = 1,
  kLsmErrPaths = 2,
  kLsmErrPartials = 3,
  kLsmErrFinal = 4,
  kLsmErrSched = 5,
  kLsmErrDisc = 6,
  kLsmErrJob = 7,
  kLsmErrCoverage = 8,
};
// Several LSM requests in one cooperative launch: job j owns blocks
// [block_first, block_first + n_blocks) and synchronises only them.  All jobs
// of a launch share precision (fp64) and sampler.
cudaError_t launch_lsm_batch(const LsmArgs* d_jobs, uint32_t n_jobs, uint32_t total_blocks, int fp64, int sampler,
                             const DeviceTables& tabs, cudaStream_t stream);
// Co-resident LSM blocks on the device for (fp64, sampler); 0 if the kernel cannot launch.
uint32_t lsm_capacity(int fp64, int sampler);
constexpr uint32_t kLsmPathsPerThreadMax = 8;
constexpr uint32_t kLsmThreads = 512;

// Bump-and-revalue legs sharing every normal: one request q (GBM step,
// GBM terminal or Heston; xorshift, Sobol or counter-hash samples; any
// technique) and its legs' parameters; q.tiles_done holds three words, zero
// before and after (tiles done, cursor, blocks gone); with NM =
// scenario_moments(technique), q.partials must hold [n_tiles][kMaxScen][NM]
// doubles and q.moments [kMaxScen][NM]: sum p, sum p^2 (pair averages for
// antithetic requests), then for control variates sum c, sum c^2, sum p c.
constexpr int scenario_moments(int technique) { return technique == MPC_TECHNIQUE_CONTROL_VARIATE ? 5 : 2; }
struct ScenarioLegs {
  float f[kScenFields * kMaxScen];  // [field][leg]
};
cudaError_t launch_scenarios(const DevReq& q, const ScenarioLegs& legs, int family, int sampler, int technique,
                             const DeviceTables& tabs, int grid, cudaStream_t stream);
int scenario_max_blocks_per_sm(int family, int sampler, int technique);

// Basket bump legs sharing every normal: one basket request q
// (xorshift, Sobol or counter-hash samples); q.partials must hold
// [n_tiles][kBasketScen][2] doubles and q.moments [kBasketScen][2].
cudaError_t launch_basket_scenarios(const DevReq& q, int sampler, const BasketScen& legs, const DeviceTables& tabs,
                                    int grid, cudaStream_t stream);
int basket_scenario_max_blocks_per_sm(int sampler);

// Single-pass Greek estimators of the terminal-GBM European call
// (pathwise: delta, vega, rho, theta; likelihood ratio: delta, vega, rho)
// over the pseudorandom terminal shocks of one MonteCarloRng stream.
struct GreekArgs {
  uint64_t seed, n_paths;
  double s0, k, r, sigma, t;
  double sqrt_t, drift_t, vol_t, discount;
  int32_t estimator;  // mpc_greek_estimator_t (PATHWISE or LIKELIHOOD_RATIO)
  int32_t fp64;       // 1: FP64 shocks and arithmetic; 0: FP32 path arithmetic
  double* partials;   // [grid][8]: sum and sum of squares of 4 estimators
  double* out;        // [8] totals in block order
  unsigned* done;     // last-block counter (zero before the launch, zero after)
};
cudaError_t launch_greeks_single_pass(const GreekArgs& a, uint32_t grid, const DeviceTables& tabs,
                                      cudaStream_t stream);

// The reference's Merton estimator (terminal, pseudorandom): each chunk's
// sequential MonteCarloRng stream is replayed and the variable number of
// draws per path resolved by a parallel chain (mpc_merton.cu).  A block owns
// kMertonBlockPos stream positions of one chunk; a chunk of n paths takes at
// most 3 n positions.
constexpr uint32_t kMertonRun = 16;       // positions per thread
constexpr uint32_t kMertonThreads = 256;
constexpr uint32_t kMertonBlockPos = kMertonRun * kMertonThreads;
struct MertonStreamArgs {
  uint64_t n_paths;             // all chunks
  uint32_t n_chunks;            // chunk count (1 = one stream)
  uint32_t blocks_per_chunk;    // blocks of the launch are chunk-major
  uint64_t chunk_base, chunk_rem;  // the reference's split of n_paths
  uint64_t seed;                // request seed (chunk seeds derived from it)
  double mean, p0;              // lambda T and exp(-lambda T)
  int64_t jump_above;           // a path jumps when its 53-bit uniform exceeds this
  double log_s0, drift_t, vol_t, jump_mean, jump_vol, k, discount;
  uint64_t* halo;               // [blocks][4] last stream outputs of a block
  uint32_t* run_entry;          // [blocks][kMertonThreads] entry class of a run per entry class of its block (nibbles)
  uint32_t* block_map;          // [blocks][8]: exit state per entry class (nibbles), starts per entry class
  uint32_t* block_state;        // [blocks] entry state
  unsigned long long* block_before;  // [blocks] paths of the chunk before the block
  uint32_t* chunk_done;         // [n_chunks] finished blocks (zero before and after)
  uint32_t* done;               // finished blocks of the second kernel (zero before and after)
  double* partials;             // [blocks][2]: sum p, sum p^2
  double* out;                  // count, sum p, sum p^2
  double* payoff;               // [n_paths] or null
};
cudaError_t launch_merton_stream(const MertonStreamArgs& a, const DeviceTables& tabs, cudaStream_t stream);

// Device generators for the ABI's sampler entry points.
cudaError_t launch_generate_normals(const DevReq& q, int sampler, int fp32, void* d_out, uint64_t n_points,
                                    uint32_t dims, const DeviceTables& tabs, cudaStream_t stream);
cudaError_t launch_counter_hash(uint32_t seed, uint32_t n_paths, uint32_t n_steps, uint32_t* d_out,
                                cudaStream_t stream);
cudaError_t launch_xorshift(uint64_t seed, uint64_t offset, uint64_t count, uint64_t* d_out,
                            const DeviceTables& tabs, cudaStream_t stream);
cudaError_t launch_flush(void* d_buf, size_t bytes, cudaStream_t stream);

// Kernel launches issued by the wrappers above since process start.
uint64_t kernel_launch_count();
// Adds the kernels of a replayed CUDA graph to the count.
void count_graph_launches(uint64_t kernels);
// Takes back the counts of launches that were only captured into a graph.
void discount_captured_launches(uint64_t kernels);

}  // namespace mpc
