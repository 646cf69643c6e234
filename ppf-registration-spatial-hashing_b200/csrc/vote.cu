// The vote pass: the work of Scene::Scene + Model::ComputeUniqueVotes
// (src/cuda/scene.cu:24-55, src/cuda/model.cu:95-171) without materialising
// scene pair features or individual votes.
//
// One work item = (scene reference point s_r, a range of chunks of model
// reference points).  A persistent block (1024 threads, one per SM, or two of
// 512 for small models) takes items from an atomic counter.  For its s_r it
//  1. walks the scene points, two per lane: one pair feature and run lookup
//     each; matched pairs ("events") go to a list in shared memory and are
//     counted per model run in a small hash table,
//  2. groups the list by run (counting sort) and cuts each group into pieces
//     of at most kPieceEvents events,
//  3. per chunk, lets warps take units (a piece x a segment of the run's
//     entries whose m_r lies in the chunk) and adds their votes to a
//     shared-memory accumulator of (m_r, alpha bin) counters,
//  4. folds its largest count into a global running maximum and emits every
//     cell whose count exceeds threshold x running maximum: a superset of the
//     cells the final threshold (threshold x global maximum) keeps.
//
// Why the grouping: the scene pairs of one s_r fall into few distinct keys
// (the bench's first model: 2049 matched pairs of 154 keys per s_r, 7.2e7
// votes but 3.2e6 distinct run entries), so streaming a run once per scene
// pair reads and counts every entry G times.  A piece of G events adds a
// whole 30-bin histogram per entry instead (sweep_unit).  Vote pass at
// ref_point_df 50, a shared atomic per vote against this: 47.1 / 17.7 / 19.5 /
// 72.8 ms against 20.6 / 10.9 / 12.1 / 15.9 ms for the bench's four models,
// and 6.4 against 5.3 ms for the 2000-point model and 10000-point scene.  What
// bounds it now: shared-memory wavefronts of the swept entries (about 53 per
// 32 entries, two thirds of the time at long sub-runs) and issue slots of the
// events between them (short sub-runs).
#include <algorithm>
#include <cstring>
#include <mutex>
#include <string>

#include "engine.h"
#include "ppf_math.cuh"

namespace ppf {
namespace {

constexpr uint32_t kNoRun = 0xffffffffu;
constexpr uint32_t kExactGroup = 1u << 31;  // group key flag: every vote of its events takes the exact path

// Fixed-point angles: alpha + pi = beta_s - beta_m + 2^20 in 2^-21 turns.
// With A = 30 x = Q 2^21 + R for x = beta_s + 2^20 (events) and x = beta_m
// (entries), the bin is Q_s - Q_m - [R_s < R_m] modulo 30, and R_s - R_m
// modulo 2^21 is the position inside the bin; a vote is ambiguous within
// kMargin of an edge.
constexpr uint32_t kTurn = 1u << PPF_ANGLE_BITS;
constexpr uint32_t kMargin = PPF_BIN_MARGIN_UNITS * PPF_N_ANGLE;

constexpr int kBlock = 128;  // entries of one sub-run that a warp takes at a time
constexpr int kPerLane = kBlock / 32;
// A piece of at least kSweepMin events is sorted by R so that it can be swept;
// it is, where that is cheaper than counting its votes one by one.  Fitted to
// phase timings of the bench's models, in SM cycles x 32: a counted vote 6.8, a
// swept entry 40 and an event among its entries 1700, so that sub-runs below
// 250 entries are always counted and long ones swept from 7 events on.
constexpr uint32_t kSweepMin = 7;
__device__ __forceinline__ bool sweep_pays(uint32_t events, uint32_t entries) {
  return events >= kSweepMin && 7.f * (float)events * (float)entries > 40.f * (float)entries + 1700.f * (float)events;
}
struct VoteArgs {
  // model
  const uint32_t* entries;
  const uint32_t* epairs;
  const uint32_t* split;
  const uint32_t* run_count;
  const uint8_t* run_flags;
  const uint32_t* ht_keys;
  const uint32_t* ht_runs;
  uint32_t ht_mask;
  const uint32_t* lut;        // ModelTables::lut, or null: every scene pair is hashed
  const uint32_t* row_flags;
  const float4* m_r1;
  const float4* m_r2;
  const float4* m_pts;
  uint32_t n_m, chunk, n_chunks;
  const uint32_t* run_maxl;  // per run: most entries that share one m_r
  uint32_t unit_shift;  // log2 of the entries per unit
  uint32_t r_shift;     // entries of a sub-run are in ascending order of R >> r_shift
  uint32_t cpi, n_cg;   // chunks per work item, work items per scene reference point
  uint2* spill;         // per block: 32-bit counts of a chunk's cells (see spill_acc)
  // scene
  const float4* s_pts;
  const float4* s_nrm;
  uint32_t n_s, ref_df, n_ref, perm_mul;
  float d_dist, thr, floor;
  int emit_all;
  // control / outputs
  uint32_t n_items;
  uint32_t* work_counter;
  uint32_t* global_max;
  unsigned long long* stats;  // [0] votes, [1] matched pairs, [2] exact bins
  unsigned long long* cand_code;
  uint32_t* cand_count;
  uint32_t* n_cand;
  uint32_t cand_cap;
  unsigned long long* n_needed;  // cells all items of the launch asked to emit
  uint32_t cand_base;            // cells already in the buffer when the launch began
  uint32_t* redo_items;          // items that did not fit the buffer
  uint32_t* n_redo;
  uint32_t n_items_total;        // capacity of redo_items
  const uint32_t* item_list;     // second launch: the items to redo (else all items)
  uint32_t* flags;
  // bounds for the self-checking build (PPF_B200_CHECKS=1)
  size_t P, K;
  unsigned long long* bad;  // first out-of-range access: site, value, bound
};

// Self-checking build: every index the kernel derives is compared with its
// bound; the first violation is recorded (site, value, bound) in bad[0..2],
// kFlagBadIndex is raised and the access is skipped.
template <bool kCheck>
__device__ __forceinline__ bool in_range(const VoteArgs& a, uint32_t site, unsigned long long v,
                                         unsigned long long bound) {
  if (!kCheck) return true;
  if (v < bound) return true;
  if (atomicCAS(&a.bad[0], 0ull, (unsigned long long)site) == 0ull) {
    a.bad[1] = v;
    a.bad[2] = bound;
  }
  atomicOr(a.flags, (uint32_t)kFlagBadIndex);
  return false;
}

__device__ __forceinline__ uint32_t ht_lookup(const uint32_t* __restrict__ keys,
                                              const uint32_t* __restrict__ runs, uint32_t mask,
                                              uint32_t key) {
  uint32_t s = (key * 0x9E3779B1u) & mask;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    uint32_t k = __ldg(keys + s);
    if (k == key) return __ldg(runs + s);
    if (k == 0u) return kNoRun;
    s = (s + 1) & mask;
  }
  return kNoRun;
}

// Block barrier of the vote kernel.  __syncthreads() is an .aligned barrier:
// every lane of a warp must reach it together.  Each barrier here follows
// lane-conditional code (lane 31 stores a warp total before the scan
// barriers, lane 0 stores sh.item, sh.base and the counters), and with
// independent thread scheduling an optimised build may bring a warp to the
// barrier in two groups, so that the barrier releases on the first and the
// rest of the warp runs one barrier phase behind.  That is what a -O3 build
// without the __syncwarp() did on one 60000-point scene (the other warps
// read the segment scan before warp 0 had written it; -O1 and -O0 builds
// did not).
// __syncwarp() reconverges the warp first; the fences around the barrier
// order the shared-memory stores and loads on both sides.
__device__ __forceinline__ void block_sync() {
  __syncwarp();
  __threadfence_block();
  __syncthreads();
  __threadfence_block();
}

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t x) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  return x;
}

// Exact bin of one vote: the reference's own arithmetic for it.  The model
// pair comes from the entry's pair index, so every index is in range by
// construction.
template <bool kCheck>
__device__ __forceinline__ uint32_t exact_bin(const VoteArgs& a, uint32_t pos, float2 v) {
  if (!in_range<kCheck>(a, 20, pos, a.P)) return 0;
  const uint32_t pr = __ldg(a.epairs + pos);
  const uint32_t mr = pr / a.n_m, mi = pr - mr * a.n_m;
  if (!in_range<kCheck>(a, 21, mr, a.n_m) || !in_range<kCheck>(a, 22, mi, a.n_m)) return 0;
  FrameYZ fm;
  fm.r1 = __ldg(a.m_r1 + mr);
  fm.r2 = __ldg(a.m_r2 + mr);
  float4 q4 = __ldg(a.m_pts + mi);
  float2 u = frame_point_yz(fm, make_float3(q4.x, q4.y, q4.z));
  return alpha_bin_exact(u, v);
}

constexpr uint32_t kPieceEvents = 255;  // a histogram counter fits a byte
// pc_inf: first event (13 bits) | events (8) | exact (1) | largest histogram
// window (8, see sort_piece)
__device__ __forceinline__ uint32_t piece_info(uint32_t off, uint32_t cnt, bool exact, uint32_t win) {
  return off | cnt << 13 | (exact ? 1u << 21 : 0u) | win << 22;
}

// Per-thread vote statistics, folded into a request's counters when the
// block leaves the request.
struct VoteStats {
  unsigned long long votes = 0, matched = 0, exact = 0;
};

extern __shared__ __align__(16) uint32_t smem[];

// Several requests (model, scene) in one persistent launch: work items of
// all requests are numbered consecutively (request r owns items
// [item_off[r], item_off[r+1])) and fetched from one counter.  A block copies
// the arguments of an item's request into shared memory when the request
// changes; each request keeps its own running maximum, counters, candidate
// region and list of items that did not fit.
struct BatchArgs {
  const VoteArgs* reqs;
  const uint32_t* item_off;  // n_reqs + 1
  uint32_t n_reqs, n_items;
  uint32_t* work_counter;
};

constexpr uint32_t kCounterMax = 65535;  // of a 16-bit counter

// Two block shapes.  A wide block has an SM to itself: the longest lists and
// all rows of a chunk.  Its phases follow one another, and for a small model,
// whose items hold a few hundred events, their waits are up to two thirds of
// the time; two narrow blocks per SM fill them with one another's work.  They
// hold half the events and up to kNarrowRows rows.
constexpr uint32_t kNarrowRows = 831;
namespace wide {
constexpr uint32_t kVoteThreads = 1024, kEvents = 7168, kSlots = 2048, kGroupLimit = 640, kMaxRows = kMaxChunk;
constexpr int kBlocksPerSm = 1;
#include "vote_kernel.cuh"
}  // namespace wide
namespace narrow {
constexpr uint32_t kVoteThreads = 512, kEvents = 3584, kSlots = 1024, kGroupLimit = 320, kMaxRows = kNarrowRows;
constexpr int kBlocksPerSm = 2;
#include "vote_kernel.cuh"
}  // namespace narrow

// The narrow shape where the chunks of all requests fit it, there are more
// items than SMs (an item alone on an SM is done sooner by a wide block) and no
// scene is so large that its events would often need a second list.  Time of
// the vote pass in wide blocks over narrow ones, models in scenes of 3 to 8
// times their points, two quanta:
//   model points                    100        300        511        700        831
//   superellipsoid, torus, capsules 1.30-1.63  1.26-1.48  1.18-1.37  1.11-1.31  1.07-1.28
//   spheres on a slab               1.31-1.38  1.16-1.25  1.00-1.14  0.96-1.08  0.87-1.07
// The flat model's lists outgrow a narrow block from about 700 points in 5600
// on; its longer groups gain most from the grouping itself.  Past the scene
// bound 700 in 60000 / 51 takes 2515 us wide and 2402 narrow, a flat model 3715
// and 4051.
constexpr uint32_t kNarrowScene = 8 * narrow::kEvents;
bool narrow_blocks(uint32_t rows, uint32_t scene, size_t items) {
  return rows <= kNarrowRows && scene <= kNarrowScene && items > (size_t)sm_count();
}

void launch_votes(const VoteArgs& a, bool check, cudaStream_t stream) {
  if (narrow_blocks(a.chunk, a.n_s, a.n_items)) {
    auto kernel = check ? narrow::vote_kernel<true> : narrow::vote_kernel<false>;
    const size_t grid = std::min<size_t>(a.n_items, (size_t)sm_count() * narrow::kBlocksPerSm);
    kernel<<<(unsigned)grid, narrow::kVoteThreads, narrow::kVoteSmemBytes, stream>>>(a);
  } else {
    auto kernel = check ? wide::vote_kernel<true> : wide::vote_kernel<false>;
    const size_t grid = std::min<size_t>(a.n_items, (size_t)sm_count());
    kernel<<<(unsigned)grid, wide::kVoteThreads, wide::kVoteSmemBytes, stream>>>(a);
  }
  PPF_CUDA(cudaGetLastError());
}

void launch_votes(const BatchArgs& b, uint32_t rows, uint32_t scene, bool check, cudaStream_t stream) {
  if (narrow_blocks(rows, scene, b.n_items)) {
    auto kernel = check ? narrow::vote_batch_kernel<true> : narrow::vote_batch_kernel<false>;
    const size_t grid = std::min<size_t>(b.n_items, (size_t)sm_count() * narrow::kBlocksPerSm);
    kernel<<<(unsigned)grid, narrow::kVoteThreads, narrow::kVoteSmemBytes, stream>>>(b);
  } else {
    auto kernel = check ? wide::vote_batch_kernel<true> : wide::vote_batch_kernel<false>;
    const size_t grid = std::min<size_t>(b.n_items, (size_t)sm_count());
    kernel<<<(unsigned)grid, wide::kVoteThreads, wide::kVoteSmemBytes, stream>>>(b);
  }
  PPF_CUDA(cudaGetLastError());
}

// counts[r * n_s + i]: model run length of a matching scene pair (r, i).
__global__ void pair_vote_counts_kernel(VoteArgs a, unsigned long long* __restrict__ out) {
  for (uint32_t r = blockIdx.y; r < a.n_s; r += gridDim.y) {
    unsigned long long* row = out + (size_t)r * a.n_s;
    const bool ref_row = (r % a.ref_df) == 0 && a.n_s > 1;
    float4 p4 = a.s_pts[r], n4 = a.s_nrm[r];
    float3 pr = make_float3(p4.x, p4.y, p4.z), nr = make_float3(n4.x, n4.y, n4.z);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < a.n_s;
         i += gridDim.x * blockDim.x) {
      unsigned long long cnt = 0;
      if (ref_row && i != r) {
        float4 q4 = a.s_pts[i], m4 = a.s_nrm[i];
        float4 f = pair_feature(pr, nr, make_float3(q4.x, q4.y, q4.z),
                                make_float3(m4.x, m4.y, m4.z), a.d_dist);
        uint32_t key = feature_key(f);
        if (key) {
          uint32_t run = ht_lookup(a.ht_keys, a.ht_runs, a.ht_mask, key);
          if (run != kNoRun) cnt = a.run_count[run];
        }
      }
      row[i] = cnt;
    }
  }
}

uint32_t gcd_u32(uint32_t x, uint32_t y) {
  while (y) {
    uint32_t t = x % y;
    x = y;
    y = t;
  }
  return x;
}

// Chunks per work item.  One item per scene reference point walks the scene
// once for all chunks; with few reference points the chunks are shared out
// until there are about 16 items per SM (8 / 16 / 32: 71.8 / 69.0 / 69.5 ms over
// the bench's four models at ref_point_df 50).
void set_items(VoteArgs& a, size_t refs_in_launch) {
  const size_t want = 16 * (size_t)sm_count();
  size_t split = refs_in_launch ? (want + refs_in_launch - 1) / refs_in_launch : 1;
  split = std::min<size_t>(std::max<size_t>(split, 1), a.n_chunks);
  a.cpi = (uint32_t)((a.n_chunks + split - 1) / split);
  a.n_cg = (a.n_chunks + a.cpi - 1) / a.cpi;
}

VoteArgs make_args(const Model& m, const SceneData& s) {
  const ModelTables& t = m.t;
  VoteArgs a{};
  a.entries = t.entries.as<uint32_t>();
  a.epairs = t.epairs.as<uint32_t>();
  a.split = t.split.as<uint32_t>();
  a.run_count = t.count.as<uint32_t>();
  a.run_flags = t.run_flags.as<uint8_t>();
  a.ht_keys = t.ht_keys.as<uint32_t>();
  a.ht_runs = t.ht_runs.as<uint32_t>();
  a.ht_mask = t.ht_mask;
  a.P = t.P;
  a.K = t.K;
  a.m_r1 = t.frame_r1.as<float4>();
  a.m_r2 = t.frame_r2.as<float4>();
  a.m_pts = t.pts.as<float4>();
  a.n_m = t.n;
  a.chunk = t.chunk;
  a.n_chunks = t.n_chunks;
  a.run_maxl = t.run_maxl.as<uint32_t>();
  if (t.lut_quantum > 0.f && t.lut_quantum == s.d_dist) {
    a.lut = t.lut.as<uint32_t>();
    a.row_flags = t.row_flags.as<uint32_t>();
  }
  a.r_shift = t.r_shift;
  // a unit of the vote phase is a quarter of a segment, at least one block
  const uint32_t segment = vote_segment_shift(*m.ctx);
  a.unit_shift = segment < 9 ? 7 : segment - 2;
  a.s_pts = s.pts.as<float4>();
  a.s_nrm = s.nrm.as<float4>();
  a.n_s = s.n;
  a.ref_df = s.ref_df ? s.ref_df : 1;
  a.n_ref = (s.n + a.ref_df - 1) / a.ref_df;
  a.d_dist = s.d_dist;  // scene pair features use the scene's quantum
  a.thr = m.vote_count_threshold;
  // ref visiting order: j -> j * perm_mul mod n_ref (a bijection)
  uint32_t pm = a.n_ref > 1 ? (0x9E3779B1u % a.n_ref) : 1u;
  if (pm == 0) pm = 1;
  while (a.n_ref > 1 && gcd_u32(pm, a.n_ref) != 1) ++pm;
  a.perm_mul = pm;
  return a;
}

}  // namespace

void init_vote_kernels(int smem_limit) {
  PPF_REQUIRE((size_t)smem_limit >= std::max(wide::kVoteSmemBytes, narrow::kVoteSmemBytes), PPF_ERR_CUDA,
              "vote accumulator too large for this device");
  auto set = [&](auto kernel, size_t bytes) {
    PPF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    PPF_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared));
  };
  set(wide::vote_kernel<false>, wide::kVoteSmemBytes);
  set(wide::vote_kernel<true>, wide::kVoteSmemBytes);
  set(wide::vote_batch_kernel<false>, wide::kVoteSmemBytes);
  set(wide::vote_batch_kernel<true>, wide::kVoteSmemBytes);
  set(narrow::vote_kernel<false>, narrow::kVoteSmemBytes);
  set(narrow::vote_kernel<true>, narrow::kVoteSmemBytes);
  set(narrow::vote_batch_kernel<false>, narrow::kVoteSmemBytes);
  set(narrow::vote_batch_kernel<true>, narrow::kVoteSmemBytes);
}

void reserve_vote_spill(Context& ctx) {
  const size_t words = std::max(wide::kSpillWords, narrow::kBlocksPerSm * narrow::kSpillWords);
  ctx.vote_spill.reserve(sm_count() * words * sizeof(uint2));
}

VoteResult run_votes(Context& ctx, const Model& m, const SceneData& s, bool emit_all, float floor) {
  VoteResult r;
  cudaStream_t stream = ctx.stream;
  VoteArgs a = make_args(m, s);
  a.emit_all = emit_all ? 1 : 0;
  a.floor = floor;
  set_items(a, a.n_ref);
  reserve_vote_spill(ctx);
  a.spill = ctx.vote_spill.as<uint2>();
  const uint32_t n_items = a.n_ref * a.n_cg;
  if (s.n < 2 || n_items == 0) return r;
  // counters: [0] work, [1] max, [2] n_cand, [3] n_redo, [4..9] 3 x u64 stats,
  // [10..11] u64 n_needed, [12] work counter and [14..15] n_needed of the
  // second launch
  ctx.counters.reserve(64);
  PPF_CUDA(cudaMemsetAsync(ctx.counters.ptr, 0, 64, stream));
  // flags word and the bad-index record at byte 32 (site, value, bound, 7 words of detail)
  PPF_CUDA(cudaMemsetAsync(ctx.flags.ptr, 0, 32 + 80, stream));
  uint32_t* cnt = ctx.counters.as<uint32_t>();
  a.work_counter = cnt + 0;
  a.global_max = cnt + 1;
  a.n_cand = cnt + 2;
  a.n_redo = cnt + 3;
  a.stats = reinterpret_cast<unsigned long long*>(cnt + 4);
  a.n_needed = reinterpret_cast<unsigned long long*>(cnt + 10);
  a.flags = ctx.flags.as<uint32_t>();
  ctx.cand_codes.reserve(ctx.cand_cap * sizeof(unsigned long long));
  ctx.cand_counts.reserve(ctx.cand_cap * sizeof(uint32_t));
  ctx.redo_items.reserve((size_t)a.n_ref * a.n_chunks * sizeof(uint32_t));
  a.cand_code = ctx.cand_codes.as<unsigned long long>();
  a.cand_count = ctx.cand_counts.as<uint32_t>();
  a.cand_cap = (uint32_t)std::min<size_t>(ctx.cand_cap, 0xffffffffu);
  a.redo_items = ctx.redo_items.as<uint32_t>();
  a.item_list = nullptr;
  a.n_items = n_items;
  a.n_items_total = a.n_ref * a.n_chunks;
  const bool check = ctx.checks;
  a.bad = reinterpret_cast<unsigned long long*>(ctx.flags.as<uint32_t>() + 8);

  PPF_CUDA(cudaEventRecord(ctx.ev[0], stream));
  launch_votes(a, check, stream);
  ctx.launches++;
  // counters, flags word and bad-index record, one wait for all
  uint32_t* const h = ctx.host;
  auto read_back = [&]() {
    PPF_CUDA(cudaEventRecord(ctx.ev[1], stream));
    PPF_CUDA(cudaMemcpyAsync(h, ctx.counters.ptr, 64, cudaMemcpyDeviceToHost, stream));
    PPF_CUDA(cudaMemcpyAsync(h + 16, ctx.flags.ptr, 32 + 80, cudaMemcpyDeviceToHost, stream));
    PPF_CUDA(cudaStreamSynchronize(stream));
  };
  read_back();
  if (h[3]) {
    // Items that did not fit: grow the buffer (keeping what was emitted) to
    // what every item asked for, then count those items again.
    unsigned long long needed;
    memcpy(&needed, h + 10, sizeof(needed));
    r.n_needed = needed;
    const size_t want = std::max<size_t>(needed, 2 * ctx.cand_cap);
    PPF_REQUIRE(want < 0xffffffffull, PPF_ERR_OUT_OF_MEMORY, "more than 2^32 vote candidates");
    DevBuf nc, nn, items;
    nc.reserve(want * sizeof(unsigned long long));
    nn.reserve(want * sizeof(uint32_t));
    items.reserve((size_t)h[3] * sizeof(uint32_t));
    PPF_CUDA(cudaMemcpyAsync(nc.ptr, ctx.cand_codes.ptr, (size_t)h[2] * 8, cudaMemcpyDeviceToDevice, stream));
    PPF_CUDA(cudaMemcpyAsync(nn.ptr, ctx.cand_counts.ptr, (size_t)h[2] * 4, cudaMemcpyDeviceToDevice, stream));
    PPF_CUDA(cudaMemcpyAsync(items.ptr, ctx.redo_items.ptr, (size_t)h[3] * 4, cudaMemcpyDeviceToDevice, stream));
    ctx.cand_codes = std::move(nc);
    ctx.cand_counts = std::move(nn);
    ctx.cand_cap = want;
    a.cand_code = ctx.cand_codes.as<unsigned long long>();
    a.cand_count = ctx.cand_counts.as<uint32_t>();
    a.cand_cap = (uint32_t)want;
    a.item_list = items.as<uint32_t>();
    a.n_items = h[3];
    a.work_counter = cnt + 12;
    a.n_needed = reinterpret_cast<unsigned long long*>(cnt + 14);
    a.cand_base = h[2];
    PPF_CUDA(cudaMemsetAsync(a.n_redo, 0, 4, stream));
    launch_votes(a, check, stream);
    ctx.launches++;
    r.n_redo = h[3];
    read_back();
    PPF_REQUIRE(h[3] == 0, PPF_ERR_INTERNAL, "vote candidates still do not fit");
  }
  {
    if (h[16] & kFlagBadIndex) {
      unsigned long long bad[10];
      memcpy(bad, h + 16 + 8, sizeof(bad));
      std::string detail;
      for (int k = 3; k < 10; ++k)
        detail += " " + std::to_string(bad[k] >> 32) + ":" + std::to_string(bad[k] & 0xffffffffu);
      throw Error(PPF_ERR_INTERNAL, "vote kernel index out of range: site " + std::to_string(bad[0]) +
                                        " value " + std::to_string(bad[1]) + " bound " +
                                        std::to_string(bad[2]) + " |" + detail);
    }
  }
  PPF_CUDA(cudaEventElapsedTime(&r.vote_ms, ctx.ev[0], ctx.ev[1]));
  r.max_count = h[1];
  r.n_cand = h[2];
  unsigned long long* s64 = reinterpret_cast<unsigned long long*>(h + 4);
  r.n_votes = s64[0];
  r.n_matched = s64[1];
  r.n_exact = s64[2];
  return r;
}

void run_votes_batch(Context& ctx, std::vector<BatchVote>& reqs) {
  cudaStream_t stream = ctx.stream;
  const size_t n = reqs.size();
  if (n == 0) return;
  PPF_REQUIRE(n < (1u << 24), PPF_ERR_INVALID_ARGUMENT, "too many requests in one batch");
  std::vector<VoteArgs> args(n);
  std::vector<uint32_t> item_off(n + 1, 0);
  // per request 16 counter words ([1] max, [2] n_cand, [3] n_redo, [4..9]
  // stats, [10..11] n_needed, [12] work counter and [14..15] n_needed of its
  // redo launch), then the batch's own work counter
  ctx.batch_counters.reserve((n + 1) * 64);
  PPF_CUDA(cudaMemsetAsync(ctx.batch_counters.ptr, 0, (n + 1) * 64, stream));
  PPF_CUDA(cudaMemsetAsync(ctx.flags.ptr, 0, 32 + 80, stream));
  uint32_t* cnt0 = ctx.batch_counters.as<uint32_t>();
  size_t total = 0, refs = 0;
  uint32_t rows = 0, scene = 0;  // of the longest chunk, points of the largest scene
  std::vector<size_t> redo_off(n + 1, 0);
  for (size_t i = 0; i < n; ++i) {
    args[i] = make_args(*reqs[i].m, *reqs[i].s);
    if (reqs[i].s->n >= 2) refs += args[i].n_ref;
  }
  for (size_t i = 0; i < n; ++i) {
    set_items(args[i], refs);
    rows = std::max(rows, args[i].chunk);
    scene = std::max(scene, args[i].n_s);
    const bool any = reqs[i].s->n >= 2;
    total += any ? (uint64_t)args[i].n_ref * args[i].n_cg : 0;
    redo_off[i + 1] = redo_off[i] + (any ? (uint64_t)args[i].n_ref * args[i].n_chunks : 0);
    PPF_REQUIRE(redo_off[i + 1] < 0xffffffffull, PPF_ERR_INVALID_ARGUMENT,
                "more than 2^32 work items in one batch");
    item_off[i + 1] = (uint32_t)total;
  }
  ctx.batch_redo.reserve(std::max<size_t>(redo_off[n], 1) * sizeof(uint32_t));
  reserve_vote_spill(ctx);
  for (size_t i = 0; i < n; ++i) {
    VoteArgs& a = args[i];
    a.spill = ctx.vote_spill.as<uint2>();
    a.emit_all = 0;
    a.floor = -1.f;
    uint32_t* cnt = cnt0 + 16 * i;
    a.work_counter = nullptr;
    a.global_max = cnt + 1;
    a.n_cand = cnt + 2;
    a.n_redo = cnt + 3;
    a.stats = reinterpret_cast<unsigned long long*>(cnt + 4);
    a.n_needed = reinterpret_cast<unsigned long long*>(cnt + 10);
    a.flags = ctx.flags.as<uint32_t>();
    a.bad = reinterpret_cast<unsigned long long*>(ctx.flags.as<uint32_t>() + 8);
    reqs[i].cap = std::max<size_t>(reqs[i].cap, 1024);
    PPF_REQUIRE(reqs[i].cap < 0xffffffffull, PPF_ERR_INVALID_ARGUMENT, "candidate capacity beyond 2^32");
    reqs[i].codes.reserve(reqs[i].cap * sizeof(unsigned long long));
    reqs[i].counts.reserve(reqs[i].cap * sizeof(uint32_t));
    a.cand_code = reqs[i].codes.as<unsigned long long>();
    a.cand_count = reqs[i].counts.as<uint32_t>();
    a.cand_cap = (uint32_t)reqs[i].cap;
    a.redo_items = ctx.batch_redo.as<uint32_t>() + redo_off[i];
    a.item_list = nullptr;
    a.n_items = item_off[i + 1] - item_off[i];
    a.n_items_total = (uint32_t)(redo_off[i + 1] - redo_off[i]);
  }
  ctx.batch_args.reserve(n * sizeof(VoteArgs));
  ctx.batch_off.reserve((n + 1) * sizeof(uint32_t));
  PPF_CUDA(cudaMemcpyAsync(ctx.batch_args.ptr, args.data(), n * sizeof(VoteArgs), cudaMemcpyHostToDevice, stream));
  PPF_CUDA(cudaMemcpyAsync(ctx.batch_off.ptr, item_off.data(), (n + 1) * sizeof(uint32_t), cudaMemcpyHostToDevice,
                           stream));
  BatchArgs b;
  b.reqs = ctx.batch_args.as<VoteArgs>();
  b.item_off = ctx.batch_off.as<uint32_t>();
  b.n_reqs = (uint32_t)n;
  b.n_items = (uint32_t)total;
  b.work_counter = cnt0 + 16 * n;
  const bool check = ctx.checks;
  PPF_CUDA(cudaEventRecord(ctx.ev[0], stream));
  if (total) {
    launch_votes(b, rows, scene, check, stream);
    ctx.launches++;
  }
  std::vector<uint32_t> h((n + 1) * 16);
  unsigned long long rec[14];  // flags word and bad-index record
  auto read_flags = [&]() {
    PPF_CUDA(cudaEventRecord(ctx.ev[1], stream));
    PPF_CUDA(cudaMemcpyAsync(ctx.host, ctx.flags.ptr, sizeof(rec), cudaMemcpyDeviceToHost, stream));
  };
  read_flags();
  PPF_CUDA(cudaMemcpyAsync(h.data(), cnt0, (n + 1) * 64, cudaMemcpyDeviceToHost, stream));
  PPF_CUDA(cudaStreamSynchronize(stream));
  // Requests whose cells did not all fit: grow their buffers (keeping what was
  // emitted) and count their remaining items again, one request at a time.
  for (size_t i = 0; i < n; ++i) {
    uint32_t* hc = h.data() + 16 * i;
    reqs[i].r.n_redo = hc[3];
    if (!hc[3]) continue;
    unsigned long long needed;
    memcpy(&needed, hc + 10, sizeof(needed));
    reqs[i].r.n_needed = needed;
    const size_t want = std::max<size_t>(needed, 2 * reqs[i].cap);
    PPF_REQUIRE(want < 0xffffffffull, PPF_ERR_OUT_OF_MEMORY, "more than 2^32 vote candidates");
    DevBuf nc, nn, items;
    nc.reserve(want * sizeof(unsigned long long));
    nn.reserve(want * sizeof(uint32_t));
    items.reserve((size_t)hc[3] * sizeof(uint32_t));
    PPF_CUDA(cudaMemcpyAsync(nc.ptr, reqs[i].codes.ptr, (size_t)hc[2] * 8, cudaMemcpyDeviceToDevice, stream));
    PPF_CUDA(cudaMemcpyAsync(nn.ptr, reqs[i].counts.ptr, (size_t)hc[2] * 4, cudaMemcpyDeviceToDevice, stream));
    PPF_CUDA(cudaMemcpyAsync(items.ptr, args[i].redo_items, (size_t)hc[3] * 4, cudaMemcpyDeviceToDevice, stream));
    reqs[i].codes = std::move(nc);
    reqs[i].counts = std::move(nn);
    reqs[i].cap = want;
    VoteArgs a = args[i];
    a.cand_code = reqs[i].codes.as<unsigned long long>();
    a.cand_count = reqs[i].counts.as<uint32_t>();
    a.cand_cap = (uint32_t)want;
    a.item_list = items.as<uint32_t>();
    a.n_items = hc[3];
    a.work_counter = cnt0 + 16 * i + 12;
    a.n_needed = reinterpret_cast<unsigned long long*>(cnt0 + 16 * i + 14);
    a.cand_base = hc[2];
    PPF_CUDA(cudaMemsetAsync(a.n_redo, 0, 4, stream));
    launch_votes(a, check, stream);
    ctx.launches++;
    read_flags();
    PPF_CUDA(cudaMemcpyAsync(hc, cnt0 + 16 * i, 64, cudaMemcpyDeviceToHost, stream));
    PPF_CUDA(cudaStreamSynchronize(stream));
    PPF_REQUIRE(hc[3] == 0, PPF_ERR_INTERNAL, "vote candidates still do not fit");
  }
  {
    memcpy(rec, ctx.host, sizeof(rec));
    if ((uint32_t)(rec[0] & 0xffffffffu) & kFlagBadIndex)
      throw Error(PPF_ERR_INTERNAL, "vote kernel index out of range: site " + std::to_string(rec[4]) +
                                        " value " + std::to_string(rec[5]) + " bound " + std::to_string(rec[6]));
  }
  float ms = 0;
  PPF_CUDA(cudaEventElapsedTime(&ms, ctx.ev[0], ctx.ev[1]));
  for (size_t i = 0; i < n; ++i) {
    const uint32_t* hc = h.data() + 16 * i;
    VoteResult& r = reqs[i].r;
    r.max_count = hc[1];
    r.n_cand = hc[2];
    unsigned long long s64[3];
    memcpy(s64, hc + 4, sizeof(s64));
    r.n_votes = s64[0];
    r.n_matched = s64[1];
    r.n_exact = s64[2];
    // the batch's device time, split by work items
    r.vote_ms = total ? ms * (float)(item_off[i + 1] - item_off[i]) / (float)total : 0.f;
  }
}

void pair_vote_counts(Context& ctx, const Model& m, const SceneData& s, uint64_t* out_dev) {
  VoteArgs a = make_args(m, s);
  dim3 grid((s.n + 255) / 256, std::min<uint32_t>(s.n, 65535u));
  pair_vote_counts_kernel<<<grid, 256, 0, ctx.stream>>>(a, reinterpret_cast<unsigned long long*>(out_dev));
  PPF_CUDA(cudaGetLastError());
  ctx.launches++;
}

// ---- allocation-free vote pass (ppf_model_vote_cells_noalloc)
//
// The same vote kernel as run_votes, for callers that must not allocate
// device memory while they run: a serving process whose device-memory budget
// was reserved at start-up (its own pool holds the rest of the device, so a
// further cudaMalloc fails or takes memory the budget does not have) and
// latency-bound loops that cannot take cudaMalloc/cudaFree latency or the
// device-wide synchronisation that cudaFree implies.  Everything the pass
// needs besides the caller's inputs and outputs lives in the context's 32-bit
// counters, reserved when its models are built, and in one static device
// array of this file, which every GPU that loads the library holds until the
// process exits:
//   [0, 256)        counters (the run_votes layout), the flags word at byte
//                   64 and the bad-index record at byte 96
//   items           the work items that did not fit the caller's output
//   points, normals the scene packed to float4
constexpr uint32_t kNoAllocMaxScenePoints = 65536;
constexpr uint32_t kNoAllocMaxItems = 262144;  // scene reference points x model chunks
constexpr size_t kNoAllocHeader = 256;
constexpr size_t kNoAllocItemsOff = kNoAllocHeader;
constexpr size_t kNoAllocPtsOff = kNoAllocItemsOff + (size_t)kNoAllocMaxItems * 4;
constexpr size_t kNoAllocNrmOff = kNoAllocPtsOff + (size_t)kNoAllocMaxScenePoints * 16;
constexpr size_t kNoAllocBytes = kNoAllocNrmOff + (size_t)kNoAllocMaxScenePoints * 16;  // 3 MiB + 256 B
static_assert(kNoAllocPtsOff % 256 == 0 && kNoAllocNrmOff % 256 == 0, "scratch sections stay aligned");

static __device__ __align__(256) unsigned char g_vote_scratch[kNoAllocBytes];

namespace {

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_vote_scratch_mutex;
unsigned char* g_vote_scratch_ptr[kNoAllocMaxDevices] = {};

// Device address of g_vote_scratch on `device`, which must be current.  The
// first call per device looks it up; later calls reuse it.
unsigned char* vote_scratch(int device) {
  PPF_REQUIRE(device >= 0 && device < kNoAllocMaxDevices, PPF_ERR_INVALID_ARGUMENT,
              "device index beyond the allocation-free path's table of 64 devices");
  std::lock_guard<std::mutex> lock(g_vote_scratch_mutex);
  if (!g_vote_scratch_ptr[device]) {
    void* ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_vote_scratch);
    if (e != cudaSuccess || !ptr)
      throw Error(PPF_ERR_CUDA, std::string("cudaGetSymbolAddress(vote scratch): ") + cudaGetErrorString(e));
    g_vote_scratch_ptr[device] = static_cast<unsigned char*>(ptr);
  }
  return g_vote_scratch_ptr[device];
}

__global__ void pack_scene_kernel(const float* __restrict__ xyz, const float* __restrict__ nxyz,
                                  uint32_t n, float4* __restrict__ pts, float4* __restrict__ nrm) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    pts[i] = make_float4(xyz[3 * (size_t)i], xyz[3 * (size_t)i + 1], xyz[3 * (size_t)i + 2], 0.f);
    nrm[i] = make_float4(nxyz[3 * (size_t)i], nxyz[3 * (size_t)i + 1], nxyz[3 * (size_t)i + 2], 0.f);
  }
}

}  // namespace

void vote_cells_noalloc(Context& ctx, const Model& m, const float* xyz, const float* nxyz,
                        uint64_t n, uint32_t ref_df, float vote_floor, uint64_t* codes,
                        uint32_t* counts, uint64_t capacity, uint64_t* n_out, uint32_t* max_out) {
  *n_out = 0;
  if (max_out) *max_out = 0;
  PPF_REQUIRE(n <= kNoAllocMaxScenePoints, PPF_ERR_INVALID_ARGUMENT,
              "scene of " + std::to_string(n) + " points exceeds the allocation-free limit of " +
                  std::to_string(kNoAllocMaxScenePoints));
  if (n < 2) return;
  PPF_REQUIRE(xyz && nxyz && is_device_pointer(xyz, ctx.device) && is_device_pointer(nxyz, ctx.device),
              PPF_ERR_INVALID_ARGUMENT, "scene points and normals must be device memory");
  PPF_REQUIRE(capacity == 0 || (codes && counts && is_device_pointer(codes, ctx.device) &&
                                   is_device_pointer(counts, ctx.device)),
              PPF_ERR_INVALID_ARGUMENT, "vote cell outputs must be device memory");
  PPF_REQUIRE(capacity <= 0xffffffffull, PPF_ERR_INVALID_ARGUMENT, "capacity beyond 2^32 - 1 cells");
  ref_df = ref_df ? ref_df : 1;
  const uint64_t n_ref = (n + ref_df - 1) / ref_df;
  const uint64_t n_items = n_ref * m.t.n_chunks;
  PPF_REQUIRE(n_items <= kNoAllocMaxItems, PPF_ERR_INVALID_ARGUMENT,
              std::to_string(n_ref) + " scene reference points x " + std::to_string(m.t.n_chunks) +
                  " model chunks exceed the allocation-free limit of " + std::to_string(kNoAllocMaxItems) +
                  " work items");
  PPF_REQUIRE(ctx.vote_spill.ptr, PPF_ERR_INTERNAL, "vote counters not reserved");

  unsigned char* scratch = vote_scratch(ctx.device);
  cudaStream_t stream = ctx.stream;
  float4* pts = reinterpret_cast<float4*>(scratch + kNoAllocPtsOff);
  float4* nrm = reinterpret_cast<float4*>(scratch + kNoAllocNrmOff);
  // the counter header is the only part of the scratch that must start at zero
  PPF_CUDA(cudaMemsetAsync(scratch, 0, kNoAllocHeader, stream));
  pack_scene_kernel<<<grid_for(n, 256), 256, 0, stream>>>(xyz, nxyz, (uint32_t)n, pts, nrm);
  PPF_CUDA(cudaGetLastError());
  ctx.launches++;

  // scene with no storage of its own: make_args takes n, d_dist and ref_df from it
  SceneData s;
  s.n = (uint32_t)n;
  s.d_dist = m.t.d_dist;  // ppf_registration builds each scene with its model's d_dist
  s.ref_df = ref_df;
  VoteArgs a = make_args(m, s);
  a.s_pts = pts;
  a.s_nrm = nrm;
  a.emit_all = 0;
  a.floor = vote_floor;
  uint32_t* cnt = reinterpret_cast<uint32_t*>(scratch);
  a.work_counter = cnt + 0;
  a.global_max = cnt + 1;
  a.n_cand = cnt + 2;
  a.n_redo = cnt + 3;
  a.stats = reinterpret_cast<unsigned long long*>(cnt + 4);
  a.n_needed = reinterpret_cast<unsigned long long*>(cnt + 10);
  a.flags = cnt + 16;
  a.bad = reinterpret_cast<unsigned long long*>(cnt + 24);
  a.cand_code = reinterpret_cast<unsigned long long*>(codes);
  a.cand_count = counts;
  a.cand_cap = (uint32_t)capacity;
  a.redo_items = reinterpret_cast<uint32_t*>(scratch + kNoAllocItemsOff);
  a.n_items_total = kNoAllocMaxItems;
  a.item_list = nullptr;
  set_items(a, n_ref);
  a.spill = ctx.vote_spill.as<uint2>();
  a.n_items = (uint32_t)n_ref * a.n_cg;
  launch_votes(a, ctx.checks, stream);
  ctx.launches++;

  unsigned long long h[22];  // bytes [0, 176): counters, flags, bad-index record
  PPF_CUDA(cudaMemcpyAsync(h, scratch, sizeof(h), cudaMemcpyDeviceToHost, stream));
  PPF_CUDA(cudaStreamSynchronize(stream));
  const uint32_t* h32 = reinterpret_cast<const uint32_t*>(h);
  if (h32[16] & kFlagBadIndex) {
    const unsigned long long* bad = h + 12;
    throw Error(PPF_ERR_INTERNAL, "vote kernel index out of range: site " + std::to_string(bad[0]) +
                                      " value " + std::to_string(bad[1]) + " bound " +
                                      std::to_string(bad[2]));
  }
  if (max_out) *max_out = h32[1];
  if (h32[3]) {
    const unsigned long long needed = h[5];
    *n_out = needed;
    throw Error(PPF_ERR_OUT_OF_MEMORY,
                "vote cell output of " + std::to_string(capacity) + " entries is too small: this call needed " +
                    std::to_string(needed) + " (the cells of the items that fit were written)");
  }
  *n_out = h32[2];
}

}  // namespace ppf
