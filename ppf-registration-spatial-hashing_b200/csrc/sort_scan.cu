#include "sort_scan.cuh"

namespace ppf {
namespace {

constexpr int kRadix = 256;
constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
// Keys per thread of a onesweep tile.  A tile's keys leave it sorted by digit,
// so a digit's share of a tile is what one write covers: 32 keys (128 bytes)
// of 8192 where 2048-key tiles wrote 8 at a time, and the look-back's status
// words are read and written once per 8192 keys.  A pass over 1.96e8 32-bit
// pairs took 2.3 ms with those tiles and takes 1.7.
template <typename K>
constexpr int kItems = sizeof(K) == 4 ? 16 : 8;
template <typename K>
constexpr int kTile = kThreads * kItems<K>;
constexpr int kSpinLimit = 1 << 22;

// Status word of a (tile, digit): epoch << 34 | state << 32 | count.  The
// epoch numbers the pass over the sorter's lifetime, so that a status array
// need not be cleared between passes or sorts.
constexpr unsigned long long kAgg = 1ull << 32;  // tile aggregate only
constexpr unsigned long long kInc = 2ull << 32;  // inclusive prefix

// Status words of other tiles change while a tile waits on them: read them
// with a load the compiler must repeat.
__device__ __forceinline__ unsigned long long load_status(const unsigned long long* p) {
  return *reinterpret_cast<const volatile unsigned long long*>(p);
}
__device__ __forceinline__ void store_status(unsigned long long* p, unsigned long long v) {
  *reinterpret_cast<volatile unsigned long long*>(p) = v;
}

// Exclusive scan of one value per thread over a block of NW warps.
template <int NW>
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  if (warp == 0) {
    uint32_t w = lane < NW ? s_warp[lane] : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
      if (lane >= o) w += y;
    }
    __syncwarp();
    if (lane < NW) s_warp[lane] = w;
  }
  __syncthreads();
  uint32_t warp_excl = warp ? s_warp[warp - 1] : 0;
  if (total) *total = s_warp[NW - 1];
  uint32_t r = warp_excl + x - v;
  __syncthreads();
  return r;
}

// Lanes whose 8-bit digit equals this lane's, among `in`.
__device__ __forceinline__ uint32_t same_digit(uint32_t d, uint32_t in) {
  uint32_t peers = in;
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const bool set = d >> b & 1u;
    const uint32_t lanes = __ballot_sync(0xffffffffu, set);
    peers &= set ? lanes : ~lanes;
  }
  return peers;
}

// Rank of each item among the warp's items of its digit, in input order
// (warp multisplit); s_hist[d] ends as the warp's count of digit d.
template <int N>
__device__ __forceinline__ void warp_ranks(const uint32_t (&dig)[N], const bool (&ok)[N], uint32_t* s_hist,
                                           uint32_t (&rank)[N]) {
  const uint32_t lane = threadIdx.x & 31, lt = (1u << lane) - 1u;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t in = __ballot_sync(0xffffffffu, ok[i]);
    const uint32_t peers = same_digit(dig[i], in);
    const uint32_t before = ok[i] ? s_hist[dig[i]] : 0u;
    __syncwarp();
    if (ok[i] && (peers & lt) == 0u) s_hist[dig[i]] = before + __popc(peers);
    __syncwarp();
    rank[i] = before + __popc(peers & lt);
  }
}

// Digit counts of all passes.  A shared atomic per key and digit: lanes of a
// warp with one digit share an access, so runs of equal digits cost less than
// random ones (ranking the lanes by digit first took 4.0 ms for 1.96e8 keys).
template <typename K>
__global__ void __launch_bounds__(kThreads) rs_histogram(const K* __restrict__ keys, size_t n,
                                                         int begin_bit, int passes,
                                                         uint32_t* __restrict__ hist) {
  __shared__ uint32_t sh[8][kRadix];
  for (int i = threadIdx.x; i < 8 * kRadix; i += blockDim.x) sh[i / kRadix][i % kRadix] = 0;
  __syncthreads();
  constexpr int kBatch = 4;
  const size_t step = (size_t)gridDim.x * kThreads;
  for (size_t i = blockIdx.x * (size_t)kThreads + threadIdx.x; i < n; i += kBatch * step) {
    K k[kBatch];
#pragma unroll
    for (int b = 0; b < kBatch; ++b) k[b] = i + b * step < n ? keys[i + b * step] : K(0);
#pragma unroll
    for (int b = 0; b < kBatch; ++b)
      if (i + b * step < n)
        for (int p = 0; p < passes; ++p) atomicAdd(&sh[p][(uint32_t)(k[b] >> (begin_bit + 8 * p)) & 0xffu], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * kRadix; i += blockDim.x) {
    uint32_t v = sh[i / kRadix][i % kRadix];
    if (v) atomicAdd(&hist[i], v);
  }
}

template <typename K>
constexpr size_t onesweep_smem() {
  return (size_t)kTile<K> * (sizeof(K) + 4) + (size_t)kWarps * kRadix * 4;
}

template <typename K>
__global__ void __launch_bounds__(kThreads, 2) rs_onesweep(
    const K* __restrict__ kin, const uint32_t* __restrict__ vin, bool vin_iota,
    K* __restrict__ kout, uint32_t* __restrict__ vout, size_t n, int shift,
    const uint32_t* __restrict__ pass_hist, unsigned long long* status, unsigned long long epoch,
    uint32_t* tile_counter, uint32_t* flags, uint32_t stall_tile, int spin_limit) {
  constexpr int N = kItems<K>;
  extern __shared__ __align__(16) unsigned char s_raw[];
  K* const s_keys = reinterpret_cast<K*>(s_raw);
  uint32_t* const s_vals = reinterpret_cast<uint32_t*>(s_keys + kTile<K>);
  uint32_t* const s_whist = s_vals + kTile<K>;  // [kWarps][kRadix]
  __shared__ uint32_t s_tile;
  __shared__ uint32_t s_start[kRadix];   // first position of a digit in the tile
  __shared__ uint32_t s_global[kRadix];  // where the tile's keys of a digit go, less s_start
  __shared__ uint32_t s_scan[kWarps];

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) s_tile = atomicAdd(tile_counter, 1u);
  for (int i = tid; i < kWarps * kRadix; i += kThreads) s_whist[i] = 0;
  __syncthreads();
  const uint32_t tile = s_tile;
  const size_t base = (size_t)tile * kTile<K>;
  const size_t remain = n - base;
  const uint32_t valid = remain < (size_t)kTile<K> ? (uint32_t)remain : (uint32_t)kTile<K>;
  const uint32_t first = warp * 32 * N + lane;  // position in the tile of this thread's first key
  kin += base;
  vin += base;

  K key[N];
  uint32_t dig[N], rank[N];
  bool ok[N];
  if (valid == (uint32_t)kTile<K>) {
#pragma unroll
    for (int i = 0; i < N; ++i) key[i] = kin[first + 32 * i];
  } else {
#pragma unroll
    for (int i = 0; i < N; ++i) key[i] = first + 32 * i < valid ? kin[first + 32 * i] : K(0);
  }
#pragma unroll
  for (int i = 0; i < N; ++i) {
    ok[i] = first + 32 * i < valid;
    dig[i] = (uint32_t)(key[i] >> shift) & 0xffu;
  }
  warp_ranks<N>(dig, ok, s_whist + warp * kRadix, rank);
  __syncthreads();
  // Per digit (thread tid = digit): warp exclusive offsets and the tile count.
  uint32_t cnt = 0;
  if (tid < kRadix) {
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      const uint32_t c = s_whist[w * kRadix + tid];
      s_whist[w * kRadix + tid] = cnt;
      cnt += c;
    }
  }
  const bool publish = tile != stall_tile;  // the test hook's silent tile
  unsigned long long* const my = status + (size_t)tile * kRadix + tid;
  if (tid < kRadix && publish) store_status(my, epoch << 34 | (tile ? kAgg : kInc) | cnt);
  const uint32_t start = block_excl_scan<kWarps>(tid < kRadix ? cnt : 0u, s_scan, nullptr);
  const uint32_t pass_base = block_excl_scan<kWarps>(tid < kRadix ? pass_hist[tid] : 0u, s_scan, nullptr);
  if (tid < kRadix) s_start[tid] = start;
  __syncthreads();
  // the tile's keys and values sorted by digit, while earlier tiles publish
#pragma unroll
  for (int i = 0; i < N; ++i) {
    if (ok[i]) {
      const uint32_t pos = s_start[dig[i]] + s_whist[warp * kRadix + dig[i]] + rank[i];
      s_keys[pos] = key[i];
      s_vals[pos] = vin_iota ? (uint32_t)base + first + 32 * i : vin[first + 32 * i];
    }
  }
  // Decoupled look-back for this digit.
  if (tid < kRadix) {
    uint32_t excl = 0;
    if (tile) {
      for (long long t = (long long)tile - 1; t >= 0; --t) {
        const unsigned long long* p = status + (size_t)t * kRadix + tid;
        unsigned long long v = load_status(p);
        int spins = 0;
        while (v >> 34 != epoch) {
          if (++spins > spin_limit) {
            atomicOr(flags, (uint32_t)kFlagSpinTimeout);
            v = kInc;
            break;
          }
          __nanosleep(32);
          v = load_status(p);
        }
        excl += (uint32_t)v;
        if (v & kInc) break;
      }
      if (publish) store_status(my, epoch << 34 | kInc | (excl + cnt));
    }
    s_global[tid] = pass_base + excl - start;
  }
  __syncwarp();  // the lanes leave the look-back at different times
  __syncthreads();
  const uint32_t last = (uint32_t)(n - 1);
  for (uint32_t p = tid; p < valid; p += kThreads) {
    const K k = s_keys[p];
    // (a position past the sort's end, after a look-back that gave up, is dropped)
    const uint32_t o = s_global[(uint32_t)(k >> shift) & 0xffu] + p;
    if (o <= last) {
      kout[o] = k;
      vout[o] = s_vals[p];
    }
  }
}

// All passes of a sort of at most kSmall elements in one block's shared
// memory: one launch where each pass took two or three (a lookup of a small
// scene sorts a few dozen to a few thousand poses three times).
constexpr int kSmallThreads = 1024;
constexpr int kSmallWarps = kSmallThreads / 32;
constexpr int kSmallItems = 4;
constexpr int kSmall = kSmallThreads * kSmallItems;
template <typename K>
constexpr size_t small_smem() {
  return (size_t)kSmall * (sizeof(K) + 4) + (size_t)kSmallWarps * kRadix * 4;
}

template <typename K>
__global__ void __launch_bounds__(kSmallThreads) rs_small(K* __restrict__ keys, uint32_t* __restrict__ vals,
                                                          bool vals_iota, uint32_t n, int begin_bit, int passes) {
  extern __shared__ __align__(16) unsigned char s_raw[];
  K* const s_keys = reinterpret_cast<K*>(s_raw);
  uint32_t* const s_vals = reinterpret_cast<uint32_t*>(s_keys + kSmall);
  uint32_t* const s_whist = s_vals + kSmall;  // [kSmallWarps][kRadix]
  __shared__ uint32_t s_start[kRadix], s_scan[kSmallWarps];
  const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // warps share the n elements evenly, whole 32s each
  const uint32_t share = (n + 32 * kSmallWarps - 1) / (32 * kSmallWarps);  // <= kSmallItems
  const uint32_t first = warp * 32 * share + lane;
  K key[kSmallItems];
  uint32_t val[kSmallItems], dig[kSmallItems], rank[kSmallItems];
  bool ok[kSmallItems];
#pragma unroll
  for (int i = 0; i < kSmallItems; ++i) {
    const uint32_t p = first + 32 * i;
    ok[i] = i < (int)share && p < n;
    key[i] = ok[i] ? keys[p] : K(0);
    val[i] = ok[i] ? (vals_iota ? p : vals[p]) : 0u;
  }
  for (int pass = 0; pass < passes; ++pass) {
    for (uint32_t i = tid; i < kSmallWarps * kRadix; i += kSmallThreads) s_whist[i] = 0;
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) dig[i] = (uint32_t)(key[i] >> (begin_bit + 8 * pass)) & 0xffu;
    __syncthreads();
    warp_ranks<kSmallItems>(dig, ok, s_whist + warp * kRadix, rank);
    __syncthreads();
    uint32_t cnt = 0;
    if (tid < kRadix) {
#pragma unroll
      for (int w = 0; w < kSmallWarps; ++w) {
        const uint32_t c = s_whist[w * kRadix + tid];
        s_whist[w * kRadix + tid] = cnt;
        cnt += c;
      }
    }
    const uint32_t start = block_excl_scan<kSmallWarps>(cnt, s_scan, nullptr);
    if (tid < kRadix) s_start[tid] = start;
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      if (ok[i]) {
        const uint32_t pos = s_start[dig[i]] + s_whist[warp * kRadix + dig[i]] + rank[i];
        s_keys[pos] = key[i];
        s_vals[pos] = val[i];
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < kSmallItems; ++i) {
      if (ok[i]) {
        key[i] = s_keys[first + 32 * i];
        val[i] = s_vals[first + 32 * i];
      }
    }
  }
#pragma unroll
  for (int i = 0; i < kSmallItems; ++i) {
    if (ok[i]) {
      keys[first + 32 * i] = key[i];
      vals[first + 32 * i] = val[i];
    }
  }
}

// ---- run tables --------------------------------------------------------
constexpr int kRunThreads = 256;
constexpr int kRunWarps = kRunThreads / 32;
constexpr int kRunItems = 16;
constexpr int kRunTile = kRunThreads * kRunItems;

__global__ void __launch_bounds__(kRunThreads) runs_count(const uint32_t* __restrict__ k,
                                                           size_t n, uint32_t* __restrict__ tile_heads) {
  __shared__ uint32_t s_scan[kRunWarps];
  size_t base = (size_t)blockIdx.x * kRunTile + (size_t)threadIdx.x * kRunItems;
  uint32_t c = 0;
  for (int i = 0; i < kRunItems; ++i) {
    size_t p = base + i;
    if (p < n && (p == 0 || k[p] != k[p - 1])) ++c;
  }
  uint32_t total;
  block_excl_scan<kRunWarps>(c, s_scan, &total);
  if (threadIdx.x == 0) tile_heads[blockIdx.x] = total;
}

// Exclusive scan of m values by one block (serial chunks).
__device__ __forceinline__ void scan_chunks(uint32_t* __restrict__ v, size_t m, uint32_t* __restrict__ total_out) {
  __shared__ uint32_t s_scan[kRunWarps];
  __shared__ uint32_t s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (size_t b = 0; b < m; b += kRunThreads) {
    size_t i = b + threadIdx.x;
    uint32_t x = i < m ? v[i] : 0u;
    uint32_t tot;
    uint32_t e = block_excl_scan<kRunWarps>(x, s_scan, &tot);
    if (i < m) v[i] = s_carry + e;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += tot;
    __syncthreads();
  }
  if (threadIdx.x == 0) *total_out = s_carry;
}

__global__ void __launch_bounds__(kRunThreads) runs_scan_tiles(uint32_t* __restrict__ v, size_t m,
                                                               uint32_t* __restrict__ total_out) {
  scan_chunks(v, m, total_out);
}

__global__ void __launch_bounds__(kRunThreads) scan_small(uint32_t* __restrict__ a, uint32_t* __restrict__ b, size_t n,
                                                          const uint32_t* __restrict__ n_dev,
                                                          uint32_t* __restrict__ total_out) {
  scan_chunks(blockIdx.x ? b : a, n_dev ? min(n, (size_t)*n_dev) : n, total_out + blockIdx.x);
}

// Run table of at most kRunsSmall keys by one block, 8 keys per thread.
constexpr int kRunsSmallThreads = 1024;
constexpr uint32_t kRunsSmallItems = kRunsSmall / kRunsSmallThreads;
__global__ void __launch_bounds__(kRunsSmallThreads) runs_small(const uint32_t* __restrict__ k, uint32_t n,
                                                                uint32_t* __restrict__ uniq,
                                                                uint32_t* __restrict__ first,
                                                                uint32_t* __restrict__ count,
                                                                uint32_t* __restrict__ k_out) {
  __shared__ uint32_t s_scan[kRunsSmallThreads / 32];
  __shared__ uint32_t s_first[kRunsSmall + 1];
  const uint32_t base = threadIdx.x * kRunsSmallItems;
  uint32_t heads = 0;
  for (uint32_t i = 0; i < kRunsSmallItems; ++i) {
    const uint32_t p = base + i;
    if (p < n && (p == 0 || k[p] != k[p - 1])) heads |= 1u << i;
  }
  uint32_t total;
  uint32_t r = block_excl_scan<kRunsSmallThreads / 32>(__popc(heads), s_scan, &total);
  for (; heads; heads &= heads - 1) s_first[r++] = base + __ffs(heads) - 1;
  if (threadIdx.x == 0) {
    s_first[total] = n;
    *k_out = total;
  }
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < total; i += kRunsSmallThreads) {
    const uint32_t f = s_first[i];
    uniq[i] = k[f];
    first[i] = f;
    count[i] = s_first[i + 1] - f;
  }
}

__global__ void __launch_bounds__(kRunThreads) runs_emit(const uint32_t* __restrict__ k, size_t n,
                                                          const uint32_t* __restrict__ tile_off,
                                                          uint32_t* __restrict__ uniq,
                                                          uint32_t* __restrict__ first) {
  __shared__ uint32_t s_scan[kRunWarps];
  size_t base = (size_t)blockIdx.x * kRunTile + (size_t)threadIdx.x * kRunItems;
  uint32_t c = 0;
  for (int i = 0; i < kRunItems; ++i) {
    size_t p = base + i;
    if (p < n && (p == 0 || k[p] != k[p - 1])) ++c;
  }
  uint32_t r = tile_off[blockIdx.x] + block_excl_scan<kRunWarps>(c, s_scan, nullptr);
  for (int i = 0; i < kRunItems; ++i) {
    size_t p = base + i;
    if (p < n && (p == 0 || k[p] != k[p - 1])) {
      uniq[r] = k[p];
      first[r] = (uint32_t)p;
      ++r;
    }
  }
}

__global__ void runs_lengths(const uint32_t* __restrict__ first, size_t K, size_t n,
                             uint32_t* __restrict__ count) {
  for (size_t r = blockIdx.x * (size_t)blockDim.x + threadIdx.x; r < K;
       r += (size_t)gridDim.x * blockDim.x) {
    size_t end = (r + 1 < K) ? first[r + 1] : n;
    count[r] = (uint32_t)(end - first[r]);
  }
}

}  // namespace

template <typename K>
void RadixSorter<K>::sort(K* keys, uint32_t* vals, bool vals_iota, size_t n, int begin_bit,
                          int end_bit, cudaStream_t st, uint32_t* d_flags) {
  if (n == 0) return;
  PPF_REQUIRE(n < (1ull << 32), PPF_ERR_INVALID_ARGUMENT, "radix sort: more than 2^32 elements");
  const int passes = (end_bit - begin_bit + 7) / 8;
  if (passes <= 0) {
    if (vals_iota) {
      // identity permutation: still produce the values
      PPF_REQUIRE(false, PPF_ERR_INTERNAL, "radix sort with no digits");
    }
    return;
  }
  if (!attributes_) {
    PPF_CUDA(cudaFuncSetAttribute(rs_onesweep<K>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)onesweep_smem<K>()));
    PPF_CUDA(cudaFuncSetAttribute(rs_small<K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)small_smem<K>()));
    attributes_ = true;
  }
  if (n <= (size_t)kSmall) {
    rs_small<K><<<1, kSmallThreads, small_smem<K>(), st>>>(keys, vals, vals_iota, (uint32_t)n, begin_bit, passes);
    PPF_CUDA(cudaGetLastError());
    launches_ += 1;
    return;
  }
  const size_t tiles = (n + kTile<K> - 1) / kTile<K>;
  kalt_.reserve(n * sizeof(K));
  valt_.reserve(n * sizeof(uint32_t));
  // digit counts of up to 8 passes, then a tile counter per pass
  constexpr size_t kCounts = 8 * kRadix + 8;
  hist_.reserve(kCounts * sizeof(uint32_t));
  const size_t status_bytes = tiles * kRadix * sizeof(unsigned long long);
  if (status_bytes > status_.bytes || epoch_ + passes >= (1ull << 30)) {
    status_.reserve(status_bytes);
    PPF_CUDA(cudaMemsetAsync(status_.ptr, 0, status_.bytes, st));
    epoch_ = 0;
  }
  uint32_t* const hist = hist_.as<uint32_t>();
  PPF_CUDA(cudaMemsetAsync(hist, 0, kCounts * sizeof(uint32_t), st));
  rs_histogram<K><<<grid_for(n, kThreads, 4), kThreads, 0, st>>>(keys, n, begin_bit, passes, hist);
  PPF_CUDA(cudaGetLastError());
  launches_ += 1;
  K* kin = keys;
  uint32_t* vin = vals;
  K* kout = kalt_.as<K>();
  uint32_t* vout = valt_.as<uint32_t>();
  bool iota = vals_iota;
  // the test hook (arm_stall) applies to the first pass of a sort with a tile 1
  const bool stall = stall_ && tiles > 1;
  if (stall) stall_ = false;
  for (int p = 0; p < passes; ++p) {
    const bool stall_here = stall && p == 0;
    rs_onesweep<K><<<(unsigned)tiles, kThreads, onesweep_smem<K>(), st>>>(
        kin, vin, iota, kout, vout, n, begin_bit + 8 * p, hist + p * kRadix, status_.as<unsigned long long>(),
        ++epoch_, hist + 8 * kRadix + p, d_flags, stall_here ? 1u : 0xffffffffu, stall_here ? 4096 : kSpinLimit);
    PPF_CUDA(cudaGetLastError());
    launches_ += 1;
    iota = false;
    std::swap(kin, kout);
    std::swap(vin, vout);
  }
  if (kin != keys) {
    PPF_CUDA(cudaMemcpyAsync(keys, kin, n * sizeof(K), cudaMemcpyDeviceToDevice, st));
    PPF_CUDA(cudaMemcpyAsync(vals, vin, n * sizeof(uint32_t), cudaMemcpyDeviceToDevice, st));
  }
  // One tile waits on nothing.  Otherwise a look-back that gave up leaves the
  // order undefined: stop here.
  if (tiles == 1) return;
  uint32_t f = 0;
  PPF_CUDA(cudaMemcpyAsync(&f, d_flags, sizeof(f), cudaMemcpyDeviceToHost, st));
  PPF_CUDA(cudaStreamSynchronize(st));
  if (f & kFlagSpinTimeout) {
    const uint32_t clear = f & ~(uint32_t)kFlagSpinTimeout;
    PPF_CUDA(cudaMemcpyAsync(d_flags, &clear, sizeof(clear), cudaMemcpyHostToDevice, st));
    PPF_CUDA(cudaStreamSynchronize(st));
    throw Error(PPF_ERR_TIMEOUT, "radix sort look-back timed out (" + std::to_string(n) + " keys)");
  }
}

template class RadixSorter<uint32_t>;
template class RadixSorter<unsigned long long>;

void exclusive_scan_small(uint32_t* a, uint32_t* b, size_t n, const uint32_t* n_dev, uint32_t* total_dev,
                          cudaStream_t st) {
  scan_small<<<b ? 2 : 1, kRunThreads, 0, st>>>(a, b, n, n_dev, total_dev);
  PPF_CUDA(cudaGetLastError());
}

void build_runs_small(const uint32_t* sorted_keys, size_t n, uint32_t* uniq, uint32_t* first, uint32_t* count,
                      uint32_t* k_dev, cudaStream_t st) {
  PPF_REQUIRE(n <= kRunsSmall, PPF_ERR_INTERNAL, "too many keys for one block");
  runs_small<<<1, kRunsSmallThreads, 0, st>>>(sorted_keys, (uint32_t)n, uniq, first, count, k_dev);
  PPF_CUDA(cudaGetLastError());
}

namespace {
// Run heads per tile, scanned: scratch[t] = runs before tile t,
// scratch[tiles] = K.  Returns K (one stream synchronisation).
size_t count_runs(const uint32_t* sorted_keys, size_t n, DevBuf& scratch, cudaStream_t st) {
  const size_t tiles = (n + kRunTile - 1) / kRunTile;
  scratch.reserve((tiles + 1) * sizeof(uint32_t));
  uint32_t* th = scratch.as<uint32_t>();
  runs_count<<<(unsigned)tiles, kRunThreads, 0, st>>>(sorted_keys, n, th);
  runs_scan_tiles<<<1, kRunThreads, 0, st>>>(th, tiles, th + tiles);
  PPF_CUDA(cudaGetLastError());
  uint32_t K = 0;
  PPF_CUDA(cudaMemcpyAsync(&K, th + tiles, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
  PPF_CUDA(cudaStreamSynchronize(st));
  return K;
}

void emit_runs(const uint32_t* sorted_keys, size_t n, size_t K, uint32_t* uniq, uint32_t* first, uint32_t* count,
               DevBuf& scratch, cudaStream_t st) {
  const size_t tiles = (n + kRunTile - 1) / kRunTile;
  runs_emit<<<(unsigned)tiles, kRunThreads, 0, st>>>(sorted_keys, n, scratch.as<uint32_t>(), uniq, first);
  runs_lengths<<<grid_for(K, 256), 256, 0, st>>>(first, K, n, count);
  PPF_CUDA(cudaGetLastError());
}
}  // namespace

size_t build_runs(const uint32_t* sorted_keys, size_t n, uint32_t* uniq, uint32_t* first,
                  uint32_t* count, DevBuf& scratch, cudaStream_t st, size_t* launches) {
  if (n == 0) return 0;
  const size_t K = count_runs(sorted_keys, n, scratch, st);
  emit_runs(sorted_keys, n, K, uniq, first, count, scratch, st);
  if (launches) *launches += 4;
  return K;
}

size_t build_runs(const uint32_t* sorted_keys, size_t n, DevBuf& uniq, DevBuf& first, DevBuf& count,
                  DevBuf& scratch, cudaStream_t st, size_t* launches) {
  if (n == 0) return 0;
  const size_t K = count_runs(sorted_keys, n, scratch, st);
  uniq.reserve(K * sizeof(uint32_t));
  first.reserve(K * sizeof(uint32_t));
  count.reserve(K * sizeof(uint32_t));
  emit_runs(sorted_keys, n, K, uniq.as<uint32_t>(), first.as<uint32_t>(), count.as<uint32_t>(), scratch, st);
  if (launches) *launches += 4;
  return K;
}

}  // namespace ppf
