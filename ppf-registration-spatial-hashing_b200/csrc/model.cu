// Model hash array build (the work of Model::Model, src/cuda/model.cu:43-82):
// pair features and keys of all ordered model pairs, a stable key sort, run
// tables, per-pair vote entries and the key -> run lookup table.
#include <algorithm>
#include <cstring>

#include "engine.h"
#include "ppf_math.cuh"

namespace ppf {
namespace {

__global__ void pack_points_kernel(const float* __restrict__ xyz, size_t n,
                                   float4* __restrict__ out) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = make_float4(xyz[3 * i], xyz[3 * i + 1], xyz[3 * i + 2], 0.f);
}

// Per model point: rows 1-2 of its reference frame and the frame angles.
__global__ void model_points_kernel(const float4* __restrict__ pts, const float4* __restrict__ nrm,
                                    uint32_t n, float4* __restrict__ r1, float4* __restrict__ r2,
                                    float2* __restrict__ ang) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    float4 p4 = pts[i], n4 = nrm[i];
    float3 p = make_float3(p4.x, p4.y, p4.z), q = make_float3(n4.x, n4.y, n4.z);
    FrameYZ f = frame_yz(p, q);
    r1[i] = f.r1;
    r2[i] = f.r2;
    FrameAngles a = frame_angles(q);
    ang[i] = make_float2(a.roty, a.rotz);
  }
}

// Keys of ordered pairs (row r, column i) -> keys[r * n + i]; rows with
// r % ref_df != 0 and self pairs get 0 (src/cuda/kernel.cu:404-477).
// grid.y walks rows, x-blocks walk columns (coalesced key writes).
__global__ void pair_keys_kernel(const float4* __restrict__ pts, const float4* __restrict__ nrm,
                                 uint32_t n, uint32_t ref_df, float d_dist,
                                 uint32_t* __restrict__ keys) {
  for (uint32_t r = blockIdx.y; r < n; r += gridDim.y) {
    uint32_t* row = keys + (size_t)r * n;
    const bool ref_row = (r % ref_df) == 0 && n > 1;
    float4 pr4 = pts[r], nr4 = nrm[r];
    float3 pr = make_float3(pr4.x, pr4.y, pr4.z), nr = make_float3(nr4.x, nr4.y, nr4.z);
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      uint32_t k = 0;
      if (ref_row && i != r) {
        float4 pi4 = pts[i], ni4 = nrm[i];
        float4 f = pair_feature(pr, nr, make_float3(pi4.x, pi4.y, pi4.z),
                                make_float3(ni4.x, ni4.y, ni4.z), d_dist);
        k = feature_key(f);
      }
      row[i] = k;
    }
  }
}

// Angle word of model pair pr: (m_r mod chunk) << 21 | angle21(u), u = the
// pair's second point in the frame of the first.  A u that is (numerically)
// zero cannot be binned from angles; its run is flagged for exact binning.
__device__ __forceinline__ uint32_t pair_entry(uint32_t pr, uint32_t n, uint32_t chunk, const float4* __restrict__ pts,
                                               const float4* __restrict__ r1, const float4* __restrict__ r2,
                                               bool& degenerate) {
  const uint32_t mr = pr / n, mi = pr - mr * n;
  FrameYZ f;
  f.r1 = r1[mr];
  f.r2 = r2[mr];
  const float4 q4 = pts[mi];
  const float2 u = frame_point_yz(f, make_float3(q4.x, q4.y, q4.z));
  degenerate = fabsf(u.x) + fabsf(u.y) < 1e-12f || !isfinite(u.x) || !isfinite(u.y);
  return ((mr % chunk) << PPF_ANGLE_BITS) | angle21(u);
}

// ---- runs by feature index
//
// The pairs' quantised features take few values (nd x 17^3 angle combinations,
// a few ten thousand of them present), so the runs of the hash array can be
// found from the values: note which occur, hash and sort those, and give every
// pair the run of its value.  The pairs then need two radix passes by run
// instead of four by 32-bit key, and the vote order's words come in pair order,
// without gathering points through the sorted pairs.  A 14003-point model
// builds in 16.9 ms this way, 25.7 ms by sorted keys (which remain for models
// with pairs beyond kLutRows quanta), a 5711-point one in 3.1 and 4.4 ms.
constexpr uint32_t kNoFeature = kLutRows * kAngleCombos;  // self pairs and NaN distances: key 0
constexpr uint32_t kFeatures = kNoFeature + 1;

// feature[r * n + i] of ordered pair (r, i), and present[feature] = 1;
// *beyond is set if a pair lies past the table's rows.
__global__ void pair_features_kernel(const float4* __restrict__ pts, const float4* __restrict__ nrm, uint32_t n,
                                     float d_dist, uint32_t* __restrict__ feature, uint8_t* __restrict__ present,
                                     uint32_t* __restrict__ beyond) {
  const float inv_d = 1.0f / d_dist;
  for (uint32_t r = blockIdx.y; r < n; r += gridDim.y) {
    const float4 pr4 = pts[r], nr4 = nrm[r];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
      uint32_t f = kNoFeature;
      if (i != r) {
        const float4 pi4 = pts[i], ni4 = nrm[i];
        const float3 d = make_float3(pi4.x - pr4.x, pi4.y - pr4.y, pi4.z - pr4.z);
        const float len = norm3(d);
        if (len < (float)(kLutRows - 1) * d_dist) {
          f = (uint32_t)quant_index(len, d_dist, inv_d) * kAngleCombos +
              pair_angles(make_float3(nr4.x, nr4.y, nr4.z), make_float3(ni4.x, ni4.y, ni4.z), d, len);
        } else if (isfinite(len)) {
          *beyond = 1u;  // (an infinite distance has the feature NaN, as a NaN one)
        }
      }
      feature[(size_t)r * n + i] = f;
      if (!present[f]) present[f] = 1;
    }
  }
}

// Keys of the features that occur, with their index, in no particular order.
__global__ void feature_keys_kernel(const uint8_t* __restrict__ present, float d_dist, uint32_t* __restrict__ keys,
                                    uint32_t* __restrict__ index, uint32_t* __restrict__ n_out) {
  const uint32_t lane = threadIdx.x & 31;
  for (uint32_t b = blockIdx.x * blockDim.x; b < kFeatures; b += gridDim.x * blockDim.x) {
    const uint32_t f = b + threadIdx.x;
    const bool in = f < kFeatures && present[f];
    const uint32_t lanes = __ballot_sync(0xffffffffu, in);
    if (!lanes) continue;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(n_out, (uint32_t)__popc(lanes));
    at = __shfl_sync(0xffffffffu, at, 0) + __popc(lanes & ((1u << lane) - 1u));
    if (in) {
      uint32_t key = 0;
      if (f != kNoFeature) {
        const uint32_t c = f % kAngleCombos;
        key = fnv1a_word(PPF_FNV_BASIS, __float_as_uint(__fmul_rn((float)(f / kAngleCombos), d_dist)));
        key = fnv1a_word(key, angle_word(c / (kAngleValues * kAngleValues)));
        key = fnv1a_word(key, angle_word(c / kAngleValues % kAngleValues));
        key = fnv1a_word(key, angle_word(c % kAngleValues));
      }
      keys[at] = key;
      index[at] = f;
    }
  }
}

// run_of[feature] for the features of every run.
__global__ void feature_runs_kernel(const uint32_t* __restrict__ index, const uint32_t* __restrict__ first,
                                    const uint32_t* __restrict__ count, size_t K, uint32_t* __restrict__ run_of) {
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < K; r += (size_t)gridDim.x * blockDim.x)
    for (uint32_t j = 0; j < count[r]; ++j) run_of[index[first[r] + j]] = (uint32_t)r;
}

// Sorted keys to runs: keys[j] becomes its run, and run[pair] the run of each
// pair.
__global__ void key_runs_kernel(uint32_t* __restrict__ keys, const uint32_t* __restrict__ pairs, size_t P,
                                const uint32_t* __restrict__ uniq, const uint32_t* __restrict__ first, size_t K,
                                uint32_t* __restrict__ run) {
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < P; j += (size_t)gridDim.x * blockDim.x) {
    size_t lo = 0, hi = K;  // last run start <= j
    while (hi - lo > 1) {
      const size_t mid = (lo + hi) >> 1;
      if (first[mid] <= j) lo = mid;
      else hi = mid;
    }
    keys[j] = (uint32_t)lo;
    run[pairs[j]] = (uint32_t)lo;
  }
}

// Sort word of each pair, in pair order, for the vote order: run, chunk of
// m_r, then the top r_bits of R = 30 x angle mod 2^21.  run_of maps in[pair] to
// the pair's run, which then also goes to run_out (null: in[] holds runs).
// Also the runs' exact flags.
template <typename W>
__global__ void order_words_kernel(const uint32_t* __restrict__ in, const uint32_t* __restrict__ run_of, size_t P,
                                   uint32_t n, uint32_t chunk, const float4* __restrict__ pts,
                                   const float4* __restrict__ r1, const float4* __restrict__ r2, int chunk_bits,
                                   int r_bits, W* __restrict__ words, uint32_t* __restrict__ run_out,
                                   uint8_t* __restrict__ run_flags) {
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < P; j += (size_t)gridDim.x * blockDim.x) {
    const uint32_t pr = (uint32_t)j;
    uint32_t run = in[j];
    if (run_of) {
      run = run_of[run];
      run_out[j] = run;
    }
    bool degenerate;
    const uint32_t e = pair_entry(pr, n, chunk, pts, r1, r2, degenerate);
    if (degenerate) run_flags[run] = 1;
    const uint32_t r = ((e & ((1u << PPF_ANGLE_BITS) - 1u)) * PPF_N_ANGLE) & ((1u << PPF_ANGLE_BITS) - 1u);
    words[j] = (((W)run << chunk_bits | (W)(pr / n / chunk)) << r_bits) | (W)(r >> (PPF_ANGLE_BITS - r_bits));
  }
}

// From the pairs sorted by run (and pair index): the runs' first positions and
// the most pairs of each that share one m_r.  A group of such pairs reaches to
// the next start, or, for the warp's last group, is counted 32 pairs at a time
// beyond it.
__global__ void run_bounds_kernel(const uint32_t* __restrict__ runs, const uint32_t* __restrict__ pairs, size_t P,
                                  uint32_t n, uint32_t* __restrict__ first, uint32_t* __restrict__ run_maxl) {
  const uint32_t lane = threadIdx.x & 31;
  for (size_t j0 = blockIdx.x * (size_t)blockDim.x + (threadIdx.x & ~31u); j0 < P;
       j0 += (size_t)gridDim.x * blockDim.x) {
    const size_t j = j0 + lane;
    if (j >= P) continue;
    const uint32_t lanes = P - j0 >= 32 ? 0xffffffffu : (1u << (P - j0)) - 1u;
    const uint32_t run = runs[j], mr = pairs[j] / n;
    const bool head = j == 0 || runs[j - 1] != run;
    if (head) first[run] = (uint32_t)j;
    const bool start = head || pairs[j - 1] / n != mr;
    const uint32_t starts = __ballot_sync(lanes, start);
    if (!starts) continue;
    const int last = 31 - __clz(starts);
    const uint32_t last_run = __shfl_sync(lanes, run, last), last_mr = __shfl_sync(lanes, mr, last);
    uint32_t tail = __popc(lanes) - last;
    for (size_t b = j0 + 32;; b += 32) {
      const bool same = b + lane < P && runs[b + lane] == last_run && pairs[b + lane] / n == last_mr;
      const uint32_t other = ~__ballot_sync(lanes, same) & lanes;
      tail += other ? __ffs(other) - 1 : 32;
      if (other) break;
    }
    if (start) {
      const uint32_t later = starts & ~(0xffffffffu >> (31u - lane));
      const uint32_t l = later ? __ffs(later) - 1 - lane : tail;
      if (l > run_maxl[run]) atomicMax(run_maxl + run, l);
    }
  }
}

__global__ void run_counts_kernel(const uint32_t* __restrict__ first, size_t K, size_t P,
                                  uint32_t* __restrict__ count) {
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < K; r += (size_t)gridDim.x * blockDim.x)
    count[r] = (uint32_t)((r + 1 < K ? first[r + 1] : P) - first[r]);
}

// Vote entries of each sub-run (run, chunk), from the sorted pairs.  The warp
// that takes a whole block of 128 adds 32 of its entries at a time to rows
// m_r of the vote pass's accumulator, in bank m_r mod 32.  The block is
// ordered by m_r mod 32 and dealt round to four such passes, so that a value
// with n entries costs at most ceil(n / 4) accesses a pass: 8.9 accesses a
// block on average where the order of R gives 14.1 and no order less than the
// most frequent value's 8.6 (random values).  A warp per sub-run and
// blockIdx.y; it reads and writes only its own blocks.
constexpr int kEntryBlock = 128;
__global__ void entries_kernel(uint32_t* __restrict__ epairs, uint32_t n, uint32_t chunk,
                               const float4* __restrict__ pts, const float4* __restrict__ r1,
                               const float4* __restrict__ r2, const uint32_t* __restrict__ split, size_t K,
                               uint32_t n_chunks, uint32_t* __restrict__ entries) {
  const uint32_t lane = threadIdx.x & 31;
  const size_t n_sub = K * n_chunks;
  for (size_t s = (blockIdx.x * (size_t)blockDim.x + threadIdx.x) >> 5; s < n_sub;
       s += ((size_t)gridDim.x * blockDim.x) >> 5) {
    const size_t run = s / n_chunks;
    const uint32_t* sp = split + run * (n_chunks + 1) + (s - run * n_chunks);
    const size_t lo = sp[0], hi = sp[1];
    for (size_t b = lo + (size_t)blockIdx.y * kEntryBlock; b < hi; b += (size_t)gridDim.y * kEntryBlock) {
      uint32_t pr[4], e[4], at[4];
      const bool whole = b + kEntryBlock <= hi;
      bool degenerate;
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        at[k] = 32u * k + lane;
        pr[k] = b + at[k] < hi ? epairs[b + at[k]] : 0u;
        e[k] = pair_entry(pr[k], n, chunk, pts, r1, r2, degenerate);
      }
      if (whole) {
        // counting sort by m_r mod 32: lane v holds the number of entries with
        // value v
        uint32_t have = 0, rank[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t v = (e[k] >> PPF_ANGLE_BITS) & 31u;
          const uint32_t peers = __match_any_sync(0xffffffffu, v);
          rank[k] = __shfl_sync(0xffffffffu, have, v) + __popc(peers & ((1u << lane) - 1u));
          uint32_t same = 0xffffffffu;  // lanes whose value is this lane's index
#pragma unroll
          for (int bit = 0; bit < 5; ++bit) {
            const uint32_t set = __ballot_sync(0xffffffffu, (v >> bit) & 1u);
            same &= (lane >> bit) & 1u ? set : ~set;
          }
          have += __popc(same);
        }
        uint32_t below = have;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, below, o);
          if (lane >= (uint32_t)o) below += y;
        }
        below -= have;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          const uint32_t r = __shfl_sync(0xffffffffu, below, (e[k] >> PPF_ANGLE_BITS) & 31u) + rank[k];
          at[k] = 32u * (r & 3u) + (r >> 2);
        }
      }
      __syncwarp();  // the block is read before it is rewritten
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        if (b + at[k] < hi) {
          entries[b + at[k]] = e[k];
          epairs[b + at[k]] = pr[k];
        }
      }
      __syncwarp();
    }
  }
}

__device__ __forceinline__ uint32_t ht_slot(uint32_t key, uint32_t mask) {
  return (key * 0x9E3779B1u) & mask;
}

__global__ void ht_build_kernel(const uint32_t* __restrict__ uniq, size_t K, uint32_t mask,
                                uint32_t* __restrict__ ht_keys, uint32_t* __restrict__ ht_runs) {
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < K;
       r += (size_t)gridDim.x * blockDim.x) {
    uint32_t key = uniq[r];
    if (key == 0) continue;  // key 0 never votes (src/cuda/kernel.cu:491)
    uint32_t s = ht_slot(key, mask);
    for (uint32_t probe = 0; probe <= mask; ++probe) {
      uint32_t prev = atomicCAS(&ht_keys[s], 0u, key);
      if (prev == 0u || prev == key) {
        ht_runs[s] = (uint32_t)r;
        break;
      }
      s = (s + 1) & mask;
    }
  }
}

// The feature table (ModelTables::lut): a block per distance index nd, every
// combination of three angle indices looked up by its key.  Exact, collisions
// of the 32-bit keys included, so a scene pair need not be hashed, and pairs
// whose row has no run (most pairs of a large scene are further apart than
// any model pair) need no angles at all.
__global__ void __launch_bounds__(256) lut_kernel(const uint32_t* __restrict__ ht_keys,
                                                  const uint32_t* __restrict__ ht_runs, uint32_t mask, float d_dist,
                                                  uint32_t* __restrict__ lut, uint32_t* __restrict__ row_flags) {
  const uint32_t nd = blockIdx.x;
  const uint32_t h1 = fnv1a_word(PPF_FNV_BASIS, __float_as_uint(__fmul_rn((float)nd, d_dist)));
  bool any = false;
  for (uint32_t c = threadIdx.x; c < kAngleCombos; c += blockDim.x) {
    const uint32_t y = c / (kAngleValues * kAngleValues), z = c / kAngleValues % kAngleValues, w = c % kAngleValues;
    const uint32_t key = fnv1a_word(fnv1a_word(fnv1a_word(h1, angle_word(y)), angle_word(z)), angle_word(w));
    uint32_t run = 0xffffffffu;
    uint32_t s = ht_slot(key, mask);
    for (uint32_t probe = 0; key != 0u && probe <= mask; ++probe) {
      const uint32_t k = ht_keys[s];
      if (k == key) run = ht_runs[s];
      if (k == key || k == 0u) break;
      s = (s + 1) & mask;
    }
    if (nd < kLutRows) lut[nd * kAngleCombos + c] = run;
    any = any || run != 0xffffffffu;
  }
  __syncwarp();  // the lanes leave the loop at different times
  if (__syncthreads_or(any) && threadIdx.x == 0) atomicOr(row_flags + nd / 32, 1u << (nd % 32));
}

// split[r*(C+1) + c] = first position of run r whose m_r >= c*chunk
// (entries of a run are in chunk order).
__global__ void split_kernel(const uint32_t* __restrict__ epairs, uint32_t n,
                             const uint32_t* __restrict__ first,
                             const uint32_t* __restrict__ count, size_t K, uint32_t chunk,
                             uint32_t n_chunks, uint32_t* __restrict__ split) {
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < K;
       r += (size_t)gridDim.x * blockDim.x) {
    uint32_t b = first[r], e = b + count[r];
    uint32_t* out = split + r * (n_chunks + 1);
    out[0] = b;
    for (uint32_t c = 1; c < n_chunks; ++c) {
      uint32_t bound = c * chunk;
      uint32_t lo = b, hi = e;  // first position with m_r >= bound
      while (lo < hi) {
        uint32_t mid = lo + ((hi - lo) >> 1);
        if (epairs[mid] / n < bound) lo = mid + 1;
        else hi = mid;
      }
      out[c] = lo;
    }
    out[n_chunks] = e;
  }
}

// Self-checking build (PPF_B200_CHECKS=1): verifies the invariants the vote
// pass relies on and records the first violation as (site, index) in bad[].
__global__ void validate_tables_kernel(const uint32_t* __restrict__ keys, size_t P,
                                       const uint32_t* __restrict__ uniq, const uint32_t* __restrict__ first,
                                       const uint32_t* __restrict__ count, size_t K,
                                       const uint32_t* __restrict__ epairs,
                                       const uint32_t* __restrict__ entries, uint32_t n, uint32_t chunk,
                                       uint32_t n_chunks, const uint32_t* __restrict__ split,
                                       unsigned long long* bad, uint32_t* flags) {
  auto report = [&](unsigned long long site, unsigned long long idx) {
    if (atomicCAS(&bad[0], 0ull, site) == 0ull) bad[1] = idx;
    atomicOr(flags, (uint32_t)kFlagBadIndex);
  };
  for (size_t j = blockIdx.x * (size_t)blockDim.x + threadIdx.x; j < P;
       j += (size_t)gridDim.x * blockDim.x) {
    if (j + 1 < P && keys[j] > keys[j + 1]) report(101, j);
    const uint32_t pr = epairs[j];
    if (pr >= (uint32_t)(n * n)) report(102, j);
    const uint32_t mr = pr / n;
    if ((entries[j] >> PPF_ANGLE_BITS) != mr % chunk) report(103, j);
  }
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < K;
       r += (size_t)gridDim.x * blockDim.x) {
    const uint32_t b = first[r], e = b + count[r];
    if (e > P || count[r] == 0) report(104, r);
    if (r + 1 < K && (uniq[r] >= uniq[r + 1] || first[r + 1] != e)) report(105, r);
    if (keys[b] != (uint32_t)r) report(106, r);
    for (uint32_t j = b + 1; j < e && j < P; ++j)
      if (epairs[j] / n / chunk < epairs[j - 1] / n / chunk) {
        report(107, r);
        break;
      }
    const uint32_t* sp = split + r * (n_chunks + 1);
    if (sp[0] != b || sp[n_chunks] != e) report(108, r);
    for (uint32_t c = 0; c < n_chunks; ++c) {
      if (sp[c] > sp[c + 1]) report(109, r);
      for (uint32_t j = sp[c]; j < sp[c + 1] && j < P; ++j) {
        const uint32_t mr = epairs[j] / n;
        if (mr < c * chunk || mr >= (c + 1) * chunk) {
          report(110, r);
          break;
        }
      }
    }
  }
}

__global__ void fill_f32(float* p, size_t n, float v) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    p[i] = v;
}

}  // namespace

bool is_any_device_pointer(const void* p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

bool is_device_pointer(const void* p, int device) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type == cudaMemoryTypeManaged) return true;
  if (a.type != cudaMemoryTypeDevice) return false;
  // A kernel of this context would read another GPU's memory as a peer
  // without peer access enabled: refused before any launch.
  PPF_REQUIRE(a.device == device, PPF_ERR_INVALID_ARGUMENT,
              "device pointer on GPU " + std::to_string(a.device) + " passed to a context on GPU " +
                  std::to_string(device));
  return true;
}

void upload_points(Context& ctx, const float* xyz, size_t n, DevBuf& dst) {
  dst.reserve(n * sizeof(float4));
  if (n == 0) return;
  DevBuf tmp;
  const float* src = xyz;
  if (!is_device_pointer(xyz, ctx.device)) {
    tmp.reserve(n * 3 * sizeof(float));
    PPF_CUDA(cudaMemcpyAsync(tmp.ptr, xyz, n * 3 * sizeof(float), cudaMemcpyHostToDevice,
                             ctx.stream));
    src = tmp.as<float>();
  }
  pack_points_kernel<<<grid_for(n, 256), 256, 0, ctx.stream>>>(src, n, dst.as<float4>());
  PPF_CUDA(cudaGetLastError());
  ctx.launches++;
}

void pair_keys_device(Context& ctx, const float4* pts, const float4* nrm, uint32_t n,
                      uint32_t ref_df, float d_dist, uint32_t* keys) {
  if (n == 0) return;
  dim3 block(256);
  dim3 grid((n + 255) / 256, std::min<uint32_t>(n, 65535u));
  pair_keys_kernel<<<grid, block, 0, ctx.stream>>>(pts, nrm, n, ref_df ? ref_df : 1, d_dist, keys);
  PPF_CUDA(cudaGetLastError());
  ctx.launches++;
}

void build_model(Context& ctx, ModelTables& t, const float* xyz, const float* nxyz, size_t n,
                 float d_dist) {
  PPF_REQUIRE(n >= 2 && n <= 65535, PPF_ERR_INVALID_ARGUMENT,
              "model size must be in [2, 65535] points");
  PPF_REQUIRE(d_dist > 0.f && std::isfinite(d_dist), PPF_ERR_INVALID_ARGUMENT,
              "d_dist must be a positive finite number");
  cudaStream_t st = ctx.stream;
  t.n = (uint32_t)n;
  t.d_dist = d_dist;
  upload_points(ctx, xyz, n, t.pts);
  upload_points(ctx, nxyz, n, t.nrm);
  t.frame_r1.reserve(n * sizeof(float4));
  t.frame_r2.reserve(n * sizeof(float4));
  t.angles.reserve(n * sizeof(float2));
  t.weights.reserve(n * sizeof(float));
  fill_f32<<<grid_for(n, 256), 256, 0, st>>>(t.weights.as<float>(), n, 1.0f);
  model_points_kernel<<<grid_for(n, 128), 128, 0, st>>>(
      t.pts.as<float4>(), t.nrm.as<float4>(), t.n, t.frame_r1.as<float4>(),
      t.frame_r2.as<float4>(), t.angles.as<float2>());
  PPF_CUDA(cudaGetLastError());
  ctx.launches += 2;

  t.P = n * n;
  t.keys.reserve(t.P * sizeof(uint32_t));
  t.pairs.reserve(t.P * sizeof(uint32_t));
  t.entries.reserve(t.P * sizeof(uint32_t));
  t.epairs.reserve(t.P * sizeof(uint32_t));
  PPF_CUDA(cudaMemsetAsync(ctx.flags.ptr, 0, sizeof(uint32_t), st));
  auto sorted = [&](auto& sorter, auto* keys, uint32_t* vals, bool iota, size_t count, int bits) {
    const size_t l0 = sorter.launches();
    sorter.sort(keys, vals, iota, count, 0, bits, st, ctx.flags.as<uint32_t>());
    ctx.launches += sorter.launches() - l0;
  };
  auto bits_for = [](uint64_t x) {
    int b = 0;
    while (b < 64 && (x >> b) != 0) ++b;
    return b;
  };

  // the runs (the hash array's unique keys): by feature index, or by the sort
  // of all pairs' keys
  DevBuf run_of;  // run of each feature index; empty: epairs holds each pair's run
  bool by_feature = d_dist >= kQuantMin;
  if (by_feature) {
    DevBuf present, fkeys, findex, ffirst, fcount;
    present.reserve(kFeatures);
    fkeys.reserve(kFeatures * sizeof(uint32_t));
    findex.reserve(kFeatures * sizeof(uint32_t));
    PPF_CUDA(cudaMemsetAsync(present.ptr, 0, kFeatures, st));
    PPF_CUDA(cudaMemsetAsync(ctx.counters.ptr, 0, 8, st));
    uint32_t* cnt = ctx.counters.as<uint32_t>();  // features, pairs beyond the table
    const dim3 grid((t.n + 255) / 256, std::min<uint32_t>(t.n, 65535u));
    pair_features_kernel<<<grid, 256, 0, st>>>(t.pts.as<float4>(), t.nrm.as<float4>(), t.n, d_dist,
                                               t.epairs.as<uint32_t>(), present.as<uint8_t>(), cnt + 1);
    feature_keys_kernel<<<grid_for(kFeatures, 256), 256, 0, st>>>(present.as<uint8_t>(), d_dist,
                                                                  fkeys.as<uint32_t>(), findex.as<uint32_t>(), cnt);
    PPF_CUDA(cudaGetLastError());
    ctx.launches += 2;
    PPF_CUDA(cudaMemcpyAsync(ctx.host, cnt, 8, cudaMemcpyDeviceToHost, st));
    PPF_CUDA(cudaStreamSynchronize(st));
    const size_t n_features = ctx.host[0];
    by_feature = ctx.host[1] == 0;
    if (by_feature) {
      sorted(ctx.sort32, fkeys.as<uint32_t>(), findex.as<uint32_t>(), false, n_features, 32);
      t.K = build_runs(fkeys.as<uint32_t>(), n_features, t.uniq, ffirst, fcount, ctx.scratch, st, &ctx.launches);
      run_of.reserve(kFeatures * sizeof(uint32_t));
      feature_runs_kernel<<<grid_for(t.K, 128), 128, 0, st>>>(findex.as<uint32_t>(), ffirst.as<uint32_t>(),
                                                              fcount.as<uint32_t>(), t.K, run_of.as<uint32_t>());
      PPF_CUDA(cudaGetLastError());
      ctx.launches++;
    }
  }
  if (!by_feature) {
    pair_keys_device(ctx, t.pts.as<float4>(), t.nrm.as<float4>(), t.n, 1, d_dist, t.keys.as<uint32_t>());
    sorted(ctx.sort32, t.keys.as<uint32_t>(), t.pairs.as<uint32_t>(), true, t.P, 32);
    t.K = build_runs(t.keys.as<uint32_t>(), t.P, t.uniq, t.first, t.count, ctx.scratch, st, &ctx.launches);
    key_runs_kernel<<<grid_for(t.P, 256), 256, 0, st>>>(t.keys.as<uint32_t>(), t.pairs.as<uint32_t>(), t.P,
                                                        t.uniq.as<uint32_t>(), t.first.as<uint32_t>(), t.K,
                                                        t.epairs.as<uint32_t>());
    PPF_CUDA(cudaGetLastError());
    ctx.launches++;
  }

  // m_r chunks: an accumulator of the vote kernel's shared memory each
  t.n_chunks = (t.n + kMaxChunk - 1) / kMaxChunk;
  t.chunk = (t.n + t.n_chunks - 1) / t.n_chunks;

  t.first.reserve(t.K * sizeof(uint32_t));
  t.count.reserve(t.K * sizeof(uint32_t));
  t.run_flags.reserve(t.K);
  t.run_maxl.reserve(t.K * sizeof(uint32_t));
  t.split.reserve(t.K * (t.n_chunks + 1) * sizeof(uint32_t));
  PPF_CUDA(cudaMemsetAsync(t.run_flags.ptr, 0, t.K, st));
  PPF_CUDA(cudaMemsetAsync(t.run_maxl.ptr, 0, t.K * sizeof(uint32_t), st));
  {
    // Sort word: run and chunk in as many bits as they need, and R in what is
    // left of the next whole digit, at least 9 bits (512 buckets over an
    // alpha bin; a block of 128 entries spans more than one of them unless
    // its sub-run has over 65536 entries).  24 bits for the bench's first
    // model, 32 for a 40000-point one: 3 or 4 passes over 8-byte elements.
    const int run_bits = bits_for(t.K - 1), chunk_bits = bits_for(t.n_chunks - 1);
    const int word_bits = (run_bits + chunk_bits + 9 + 7) / 8 * 8;
    const int r_bits = std::min(word_bits - run_bits - chunk_bits, PPF_ANGLE_BITS);
    t.r_shift = PPF_ANGLE_BITS - r_bits;
    auto order = [&](auto& sorter, auto* words) {
      order_words_kernel<<<grid_for(t.P, 256), 256, 0, st>>>(
          t.epairs.as<uint32_t>(), by_feature ? run_of.as<uint32_t>() : nullptr, t.P, t.n, t.chunk,
          t.pts.as<float4>(), t.frame_r1.as<float4>(), t.frame_r2.as<float4>(), chunk_bits, r_bits, words,
          t.keys.as<uint32_t>(), t.run_flags.as<uint8_t>());
      PPF_CUDA(cudaGetLastError());
      ctx.launches++;
      // the hash array's map: pairs by run, in pair order
      if (by_feature)
        sorted(ctx.sort32, t.keys.as<uint32_t>(), t.pairs.as<uint32_t>(), true, t.P, std::max(run_bits, 1));
      run_bounds_kernel<<<grid_for(t.P, 256), 256, 0, st>>>(t.keys.as<uint32_t>(), t.pairs.as<uint32_t>(), t.P, t.n,
                                                            t.first.as<uint32_t>(), t.run_maxl.as<uint32_t>());
      run_counts_kernel<<<grid_for(t.K, 256), 256, 0, st>>>(t.first.as<uint32_t>(), t.K, t.P, t.count.as<uint32_t>());
      PPF_CUDA(cudaGetLastError());
      ctx.launches += 2;
      // vote entries in vote order; epairs keeps each entry's pair index
      sorted(sorter, words, t.epairs.as<uint32_t>(), true, t.P, run_bits + chunk_bits + r_bits);
    };
    // (the words borrow the entries' buffer when they are 32-bit)
    if (word_bits <= 32) {
      order(ctx.sort32, t.entries.as<uint32_t>());
    } else {
      DevBuf words;
      words.reserve(t.P * sizeof(unsigned long long));
      order(ctx.sort64, words.as<unsigned long long>());
    }
    // chunk boundaries of every run (entries are in chunk order within a run)
    split_kernel<<<grid_for(t.K, 256), 256, 0, st>>>(t.epairs.as<uint32_t>(), t.n, t.first.as<uint32_t>(),
                                                      t.count.as<uint32_t>(), t.K, t.chunk, t.n_chunks,
                                                      t.split.as<uint32_t>());
    PPF_CUDA(cudaGetLastError());
    ctx.launches++;
    const dim3 grid(grid_for(t.K * t.n_chunks, 8, 16), 8);
    entries_kernel<<<grid, 256, 0, st>>>(t.epairs.as<uint32_t>(), t.n, t.chunk, t.pts.as<float4>(),
                                         t.frame_r1.as<float4>(), t.frame_r2.as<float4>(), t.split.as<uint32_t>(),
                                         t.K, t.n_chunks, t.entries.as<uint32_t>());
    PPF_CUDA(cudaGetLastError());
    ctx.launches++;
  }
  reserve_vote_spill(ctx);

  // key -> run table, load factor <= 0.5
  uint32_t cap = 1024;
  while (cap < 2 * t.K) cap <<= 1;
  t.ht_mask = cap - 1;
  t.ht_keys.reserve(cap * sizeof(uint32_t));
  t.ht_runs.reserve(cap * sizeof(uint32_t));
  PPF_CUDA(cudaMemsetAsync(t.ht_keys.ptr, 0, cap * sizeof(uint32_t), st));
  ht_build_kernel<<<grid_for(t.K, 256), 256, 0, st>>>(t.uniq.as<uint32_t>(), t.K, t.ht_mask,
                                                       t.ht_keys.as<uint32_t>(),
                                                       t.ht_runs.as<uint32_t>());
  PPF_CUDA(cudaGetLastError());

  ctx.launches += 1;
  if (d_dist >= kQuantMin) {
    t.lut.reserve((size_t)kLutRows * kAngleCombos * sizeof(uint32_t));
    t.row_flags.reserve(kFlagRows / 8);
    PPF_CUDA(cudaMemsetAsync(t.row_flags.ptr, 0, kFlagRows / 8, st));
    lut_kernel<<<kFlagRows, 256, 0, st>>>(t.ht_keys.as<uint32_t>(), t.ht_runs.as<uint32_t>(), t.ht_mask, d_dist,
                                          t.lut.as<uint32_t>(), t.row_flags.as<uint32_t>());
    PPF_CUDA(cudaGetLastError());
    ctx.launches += 1;
    t.lut_quantum = d_dist;
  }
  unsigned long long* bad = reinterpret_cast<unsigned long long*>(ctx.flags.as<uint32_t>() + 8);
  if (ctx.checks) {
    PPF_CUDA(cudaMemsetAsync(bad, 0, 24, st));
    validate_tables_kernel<<<grid_for(t.P, 256), 256, 0, st>>>(
        t.keys.as<uint32_t>(), t.P, t.uniq.as<uint32_t>(), t.first.as<uint32_t>(),
        t.count.as<uint32_t>(), t.K, t.epairs.as<uint32_t>(), t.entries.as<uint32_t>(), t.n, t.chunk,
        t.n_chunks, t.split.as<uint32_t>(), bad, ctx.flags.as<uint32_t>());
    PPF_CUDA(cudaGetLastError());
  }
  PPF_CUDA(cudaMemsetAsync(ctx.counters.ptr, 0, 8, st));
  calibrate_distance(ctx, d_dist, ctx.counters.as<uint32_t>());
  unsigned long long badh[2] = {0, 0};
  PPF_CUDA(cudaMemcpyAsync(ctx.host, ctx.flags.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  PPF_CUDA(cudaMemcpyAsync(ctx.host + 2, ctx.counters.ptr, 8, cudaMemcpyDeviceToHost, st));
  if (ctx.checks) PPF_CUDA(cudaMemcpyAsync(badh, bad, 16, cudaMemcpyDeviceToHost, st));
  PPF_CUDA(cudaStreamSynchronize(st));
  const uint32_t flags = ctx.host[0];
  std::memcpy(&t.x_star, ctx.host + 2, sizeof(t.x_star));
  t.x_star_ok = ctx.host[3] == 0;
  PPF_REQUIRE(!(flags & kFlagSpinTimeout), PPF_ERR_TIMEOUT, "radix sort look-back timed out");
  PPF_REQUIRE(!(flags & kFlagBadIndex), PPF_ERR_INTERNAL,
              "model tables inconsistent: check " + std::to_string(badh[0]) + " at " +
                  std::to_string(badh[1]));
  if (!ctx.checks) t.keys.release();  // only the build's sorts used the runs in map order
  // The sorts keep scratch of 8 bytes per sorted pair (21 where the vote
  // order's words need 64 bits) for reuse by later builds; past 2^28 pairs
  // (16k-point models) that is gigabytes, so it goes back to the pool now.
  if (t.P > (size_t(1) << 28)) {
    ctx.sort32.release();
    ctx.sort64.release();
  }
}

}  // namespace ppf
