// Engine objects behind the C ABI: context, resident model hash arrays,
// resident scenes, and the device-side layout the kernels consume.
#pragma once

#include <atomic>
#include <string>
#include <unordered_map>
#include <vector>

#include "common.cuh"
#include "sort_scan.cuh"

struct ppf_context_s;

namespace ppf {

// Most m_r rows of a chunk: m_r mod chunk takes the 11 bits above an entry's
// 21-bit angle, and ppf_model_num_chunks reports the chunks.  (1659 rows of
// 31 32-bit counters were what one block's shared memory held; at 64 bytes a
// row they now share it with the scene pairs of one reference point.)
constexpr uint32_t kMaxChunk = 1659;
// Feature table of a model (ModelTables::lut): distance rows with a run per
// angle combination, and rows whose flag says whether any key of theirs
// belongs to the model.
constexpr uint32_t kLutRows = 128;
constexpr uint32_t kFlagRows = 1024;
// Angle quantum on the host (include/kernel.h:16 evaluated in float).
#define PPF_D_ANGLE_HOST ((2.0f * 3.141592654f) / float(30))

constexpr size_t kHostBytes = 4096;  // of Context::host

// Every DevBuf member must be released in ~Context (capi.cu) before the
// stream its blocks are freed on is destroyed.
struct Context {
  int device = 0;
  cudaStream_t stream = nullptr;
  RadixSorter<uint32_t> sort32;
  RadixSorter<unsigned long long> sort64;
  DevBuf flags;      // uint32 device flags (kFlag*)
  DevBuf counters;   // small device counters for kernels
  // Host memory that small results are copied to (kHostBytes).  Pinned in a
  // context that is kept: a copy to pageable memory is staged and waits on its
  // own (about 5 us each).  Pinning takes 0.5 ms, so a context made for one
  // call does without.
  uint32_t* host = nullptr;
  bool host_pinned = false;
  DevBuf scratch;    // run-table scratch
  // vote-pass candidate cells (code, count), kept and grown across lookups
  DevBuf cand_codes, cand_counts, redo_items;
  DevBuf batch_args, batch_off, batch_counters, batch_redo;  // batched vote pass
  // candidate cells the last vote pass of a model with this signature
  // (points, d_dist, threshold) emitted; sizes the next batch's buffers when
  // the same model is built again
  std::unordered_map<uint64_t, size_t> cand_hints;
  uint32_t forced_seg_shift = 0;  // PPF_B200_VOTE_SEGMENT=<2^k>: every model uses it
  DevBuf vote_spill;  // per vote block: 32-bit counters of one chunk (reserve_vote_spill)
  size_t cand_cap = size_t(1) << 24;
  cudaEvent_t ev[4] = {nullptr, nullptr, nullptr, nullptr};
  int vote_smem_limit = 0;  // max dynamic shared memory per vote block
  size_t launches = 0;      // kernels launched (running total)
  bool checks = false;      // self-checking kernels (PPF_B200_CHECKS=1)
  bool cluster_split = true; // exact-sum split clustering allowed (PPF_B200_CLUSTER_SPLIT=0: never)
  bool cluster_sqrt = false; // PPF_B200_CLUSTER_SQRT=1: translation test with the square root
  ~Context();
};

// Model hash array resident in HBM (built once by ppf_model_create).
struct ModelTables {
  uint32_t n = 0;        // model points
  float d_dist = 0;
  // per model point
  DevBuf pts, nrm;       // float4 (x, y, z, 0)
  DevBuf frame_r1, frame_r2;  // rows 1 and 2 of the point's reference frame
  DevBuf angles;         // float2 (roty, rotz) of the frame
  DevBuf weights;        // float vote weights (default 1)
  // all ordered pairs, sorted by feature key (stable: pair index order)
  size_t P = 0;
  DevBuf keys;           // uint32 run of each pair in map order (kept for the self-checks only)
  DevBuf pairs;          // uint32 pair index r*n + i (the hash array's data map)
  // Vote order: by run, then chunk of m_r, then buckets of 2^r_shift of
  // R = 30 x angle mod 2^21 (the angle's position inside an alpha bin), each
  // block of 128 dealt to lanes by m_r mod 32
  DevBuf entries;        // uint32 (m_r mod chunk) << 21 | 21-bit angle of u
  DevBuf epairs;         // uint32 pair index of each entry (vote order)
  uint32_t r_shift = 0;
  // runs
  size_t K = 0;
  DevBuf uniq, first, count;  // uint32 each
  DevBuf run_maxl;            // uint32: most entries of the run that share one m_r
  DevBuf run_flags;           // uint8: 1 = run holds a degenerate pair (exact bins only)
  // key -> run open-addressing table (key 0 is the empty marker)
  DevBuf ht_keys, ht_runs;
  uint32_t ht_mask = 0;
  // Runs of quantised features, for scenes with the model's own quantum:
  // lut[nd * 4913 + angles] for nd < kLutRows (pair_angles; 0xffffffff: none),
  // row_flags bit nd set if any feature of distance index nd < kFlagRows has a
  // run.  lut_quantum: the quantum they hold for (0: no table)
  DevBuf lut, row_flags;
  float lut_quantum = 0;
  // |t - s|^2 < x_star equals sqrtf(|t - s|^2) < d_dist on the device
  // (dist_threshold_kernel), if x_star_ok
  float x_star = 0;
  bool x_star_ok = false;
  // m_r chunking of the vote accumulator
  uint32_t chunk = 0, n_chunks = 0;
  DevBuf split;  // uint32 [K * (n_chunks + 1)] first run position per chunk
};

struct SceneData {
  uint32_t n = 0;
  float d_dist = 0;
  uint32_t ref_df = 1;
  DevBuf pts, nrm;  // float4
};

// Results of the last lookup, kept on the device for the inspection calls.
struct LookupState {
  size_t U = 0;
  DevBuf codes;       // uint64 kept vote codes, reference order
  DevBuf counts;      // uint32
  DevBuf weighted;    // float
  DevBuf transforms;  // float U*16
  DevBuf trans;       // float U*3 (after clustering)
  DevBuf trans0;      // float U*3 (before clustering)
  DevBuf quats;       // float U*4
  DevBuf scores;      // float U
  DevBuf cells_sorted, cells_map, cells_uniq, cells_first, cells_count;
  DevBuf cells3;      // int4 U: integer cell of each pose
  DevBuf qs, tws, adjrun, item_off;  // cell-major clustering tables
  DevBuf item_off32;  // split clustering: (32-target tile, neighbour) items per run
  DevBuf tmp64, tmp32a, tmp32b, tmp32c, perm;
  DevBuf tperm;       // clustering target order (cell, rotation bucket)
  DevBuf best;        // float[16] pose + int idx
  DevBuf argmax_v, argmax_i;  // per-block partial maxima of the scores
  uint32_t cluster_path = 0;  // ppf_stats::cluster_path of the last clustering
  std::vector<float> cpu_poses;
};

struct Model {
  Context* ctx = nullptr;
  ModelTables t;
  float vote_count_threshold = 0.4f;
  bool cpu_clustering = false, use_l1_norm = false, use_averaged_clusters = false;
  size_t cand_hint = 0;  // candidate cells of the last vote pass (sizes batch buffers)
  LookupState last;
};

// ---- model build (model.cu)
void build_model(Context& ctx, ModelTables& t, const float* xyz, const float* nxyz, size_t n,
                 float d_dist);
// keys of all n*n ordered pairs of a cloud held as float4 device arrays
void pair_keys_device(Context& ctx, const float4* pts, const float4* nrm, uint32_t n,
                      uint32_t ref_df, float d_dist, uint32_t* keys);
// upload n x 3 floats (host or device) into a float4 device array
void upload_points(Context& ctx, const float* xyz, size_t n, DevBuf& dst);
// Device memory of `device` or managed memory: true; host memory: false.
// Device memory of another GPU raises PPF_ERR_INVALID_ARGUMENT.
bool is_device_pointer(const void* p, int device);
// Device or managed memory of any GPU.
bool is_any_device_pointer(const void* p);

// ---- voting (vote.cu)
struct VoteResult {
  uint32_t max_count = 0;
  uint64_t n_votes = 0, n_matched = 0, n_exact = 0;
  uint64_t n_cand = 0;
  uint32_t n_redo = 0;  // items emitted by a second launch after the buffer grew
  uint64_t n_needed = 0;  // cells the first launch's items asked for (sizes the next buffer)
  float vote_ms = 0;
};
// Shared-memory sizes of the vote kernels, the same for every launch.
void init_vote_kernels(int smem_limit);
// The vote blocks' 32-bit counters (ctx.vote_spill).
void reserve_vote_spill(Context& ctx);
// Runs the vote pass.  emit_all: emit every nonzero cell (no threshold);
// floor >= 0 forces the emission floor.  Candidates land in
// ctx.cand_codes / ctx.cand_counts.
VoteResult run_votes(Context& ctx, const Model& m, const SceneData& s, bool emit_all, float floor);
// One request of a batched vote pass: its candidate cells land in its own
// buffers (cap cells, grown if they do not fit).
struct BatchVote {
  const Model* m = nullptr;
  const SceneData* s = nullptr;
  size_t cap = 0;
  DevBuf codes, counts;
  VoteResult r;
};
// The vote passes of all requests in one persistent launch (threshold x
// running maximum emission, as run_votes with emit_all = false).
void run_votes_batch(Context& ctx, std::vector<BatchVote>& reqs);
void pair_vote_counts(Context& ctx, const Model& m, const SceneData& s, uint64_t* out_dev);
// The vote pass with no device allocation: scene and outputs are the
// caller's device arrays, everything else lives in a static device array of
// vote.cu (ppf_model_vote_cells_noalloc).
void vote_cells_noalloc(Context& ctx, const Model& m, const float* xyz, const float* nxyz,
                        uint64_t n, uint32_t ref_df, float vote_floor, uint64_t* codes,
                        uint32_t* counts, uint64_t capacity, uint64_t* n_out, uint32_t* max_out);

// log2 of the vote pass's segment length: 4096 entries unless
// PPF_B200_VOTE_SEGMENT says otherwise.  A unit of the vote phase is a quarter
// of it and shrinks where units are few, so the length hardly matters any
// more (2048 / 4096 / 8192: 5.99 / 5.87 / 5.86 ms for a 2000-point model's
// vote pass); it used to be timed per model on the first lookup, which cost
// up to three lookups' worth of launches.
constexpr uint32_t kSegShiftDefault = 12;
inline uint32_t vote_segment_shift(const Context& ctx) {
  return ctx.forced_seg_shift ? ctx.forced_seg_shift : kSegShiftDefault;
}
uint64_t model_signature(const Model& m);

// ---- poses and clustering (pose.cu)
// Filters the candidates to the kept votes and orders them (count desc,
// code asc); returns U.
size_t select_votes(Context& ctx, const Model& m, const SceneData& s, LookupState& st,
                    const unsigned long long* cand_code, const uint32_t* cand_count, size_t n_cand,
                    float min_votecount, uint32_t max_count);
// Orders arbitrary (code, count) pairs by code ascending (all-votes dump).
void sort_by_code(Context& ctx, LookupState& st, size_t n);
void compute_poses(Context& ctx, const Model& m, const SceneData& s, LookupState& st);
// GPU clustering + argmax; writes the best pose (16 floats) and its score and
// returns the index.  Records ctx.ev[3] and waits for the stream; *flags
// receives the device flags as of then.
size_t cluster_poses_gpu(Context& ctx, const Model& m, LookupState& st, float* pose, float* best_score,
                         uint32_t* flags);
// Threshold of the clustering's translation test for cells of size d: out[0]
// its float bits, out[1] nonzero if it cannot be used (both zero before).
void calibrate_distance(Context& ctx, float d, uint32_t* out_dev);

// ---- driver preprocessing (preprocess.cu)
// per-axis min / max over finite points (false when there is none)
bool cloud_extent(Context& ctx, const float* xyz_dev, size_t n, float lo[3], float hi[3]);
// pcl::VoxelGrid centroids of an n x 3 cloud; returns the voxel count
size_t voxel_downsample(Context& ctx, const float* xyz_dev, const float* nxyz_dev, size_t n, float leaf,
                        DevBuf& out_xyz, DevBuf& out_nxyz);

// ---- PLY files (ply.cpp)
ppf_status ply_read(const char* path, float* xyz, float* nxyz, uint64_t cap, uint64_t* n_out, std::string* err);
ppf_status ply_write(const char* path, const float* xyz, const float* nxyz, uint64_t n);

// ---- lookups (capi.cu)
struct LookupOut {
  ppf_status status = PPF_OK;
  float pose[16] = {0};
  ppf_stats stats{};
  size_t cand_hint = 0;  // candidate cells to provide for the next pass of this model
};
void init_context(Context& c, int device, bool kept = true);
// Candidate cells that a batch provides for a request whose model's last pass
// had `hint` of them (0: no pass yet).
inline size_t batch_cells(size_t hint) { return hint ? hint + hint / 4 + 65536 : size_t(1) << 22; }
// Lookups of (models[i], scenes[i]) with one batched vote pass.  states:
// per-request lookup state (nullptr: each model's own `last`); caps:
// per-request candidate capacity hints (nullptr: the models' last passes).
std::vector<LookupOut> lookup_batch(Context& ctx, const std::vector<Model*>& models,
                                    const std::vector<const SceneData*>& scenes, LookupState* states,
                                    const size_t* caps);

// ---- request loop (serve.cu)
struct Server;
Server* server_create(int device, const std::vector<Model*>& models, size_t memory_budget,
                      uint32_t n_workers, uint32_t max_batch);
uint64_t server_submit(Server* srv, const float* xyz, const float* nxyz, uint64_t n, uint32_t ref_df,
                       const uint32_t* model_ids, uint64_t n_ids);
ppf_status server_wait(Server* srv, uint64_t ticket, float* poses, ppf_stats* stats, double* latency_ms,
                       std::string* error);
void server_destroy(Server* srv);

// ---- greedy clustering of the cpu_clustering path on the device (greedy.cu)
int cluster_poses_greedy_gpu(Context& ctx, const float* transforms_dev, const uint32_t* votes_dev, size_t U,
                             float trans_thresh, float rot_thresh, float out_poses[3 * 16], uint32_t out_votes[3]);

int cluster_poses_sorted_gpu(Context& ctx, const float* transforms_dev, const uint32_t* votes_dev, size_t U,
                             float trans_thresh, float rot_thresh, float out_poses[3 * 16], uint32_t out_votes[3]);

}  // namespace ppf

// Handles are reference-counted: the caller's handle is one reference, and
// every model, scene and server made on a context holds one on it (a server
// also holds one on each library model).  A destroy call drops the caller's
// reference; the object goes when the last one does, so handles can be
// destroyed in any order.
struct ppf_context_s {
  ppf::Context c;
  std::atomic<int> refs{1};
};
struct ppf_model_s {
  ppf::Model m;
  ppf_context_s* owner = nullptr;
  std::atomic<int> refs{1};
};
struct ppf_scene_s {
  ppf::Context* ctx = nullptr;
  ppf_context_s* owner = nullptr;
  ppf::SceneData s;
};
struct ppf_server_s {
  ppf::Server* srv = nullptr;
  std::vector<ppf_model_s*> library;
};
