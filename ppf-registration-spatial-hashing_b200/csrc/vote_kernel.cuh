// The vote kernel, included by vote.cu once per block shape (see there), inside
// a namespace that defines kVoteThreads, kEvents, kSlots, kGroupLimit, kMaxRows
// and kBlocksPerSm.

constexpr uint32_t kVoteWarps = kVoteThreads / 32;
// A chunk's units are halved, down to 512 entries, until there are this many.
constexpr uint32_t kMinUnits = 8 * kVoteWarps, kMinUnitShift = 9;

// ---- shared-memory layout of a vote block (dynamic allocation, 32-bit words)
//
// Events of one s_r held at a time; a walk that fills the list is continued
// after its votes are counted.  A warp looks up 32 pairs only while at most
// kGroupLimit groups exist, so that all warps' pairs fit the slots.
constexpr uint32_t kEventsPerThread = kEvents / kVoteThreads;
constexpr uint32_t kMaxPieces = kGroupLimit + kVoteThreads + (kEvents + kPieceEvents - 1) / kPieceEvents;
static_assert(kGroupLimit + kVoteThreads < kSlots, "every warp's groups find a slot");
static_assert(kMaxPieces <= 2 * kVoteThreads, "two pieces per thread");
static_assert(4 * (kMaxPieces + 1) <= kEvents, "per-chunk piece arrays fit the event slot words");

static_assert(2 * kVoteThreads == kSlots, "two slots per thread");

constexpr uint32_t kOffEvW = 0;                          // A = Q << 21 | R of each event
constexpr uint32_t kOffEvI = kOffEvW + kEvents;          // its scene point
constexpr uint32_t kOffEvK = kOffEvI + kEvents;          // slot << 16 | rank in the group, until grouped
constexpr uint32_t kOffSlotKey = kOffEvK + kEvents;      // run | kExactGroup
constexpr uint32_t kOffSlotCnt = kOffSlotKey + kSlots;   // events, then offset of the group
constexpr uint32_t kOffPcRun = kOffSlotCnt + kSlots;     // piece: its run
constexpr uint32_t kOffPcInf = kOffPcRun + kMaxPieces;   // piece: see piece_info
// per warp: (block of the unit << 16 | event of the piece) pairs that hold
// ambiguous votes
constexpr uint32_t kNotesLen = 32;
constexpr uint32_t kOffNotes = kOffPcInf + kMaxPieces;
constexpr uint32_t kOffAcc = (kOffNotes + kVoteWarps * kNotesLen + 31) / 32 * 32;  // counters, see kRowStride
// over the pieces while the list is filled: per warp the scene pairs that
// await their lookup
constexpr uint32_t kNearLen = 96;
constexpr uint32_t kOffNear = kOffPcRun;
static_assert(kVoteWarps * kNearLen <= 2 * kMaxPieces, "the waiting pairs fit the pieces");
// over the event slot words once the list is grouped: the pieces' entries in
// the current chunk (first entry, length, first unit, running counter bound)
constexpr uint32_t kOffPcLo = kOffEvK;
constexpr uint32_t kOffPcLen = kOffPcLo + kMaxPieces + 1;
constexpr uint32_t kOffPcUnit = kOffPcLen + kMaxPieces + 1;
constexpr uint32_t kOffPcInc = kOffPcUnit + kMaxPieces + 1;
// over the slots once the list is grouped: per warp a histogram table and a
// queue of ambiguous votes
constexpr uint32_t kTabWords = 60, kQueueLen = 32;
constexpr uint32_t kOffTab = kOffSlotKey;
constexpr uint32_t kOffQueue = kOffTab + kVoteWarps * kTabWords;
static_assert(kVoteWarps * (kTabWords + 2 * kQueueLen) <= 2 * kSlots, "tables and queues fit the slots");

// Accumulator: plane j holds the 16-bit counters of bins (2j, 2j + 1) of every
// m_r of the chunk, one word each, and a last plane the 32-bit counters of
// bin 30 (only alpha == pi exactly reaches it).  The planes are a multiple of
// 32 words apart, so a counter's bank is its m_r mod 32 whatever the bin, and
// 32 lanes with distinct m_r mod 32 count without bank conflicts.
constexpr uint32_t kPlanes = PPF_N_ANGLE / 2;
constexpr uint32_t kRowStride = (kMaxRows + 31) / 32 * 32;
// A row no chunk has: lanes past a sub-run's end count there, so that the
// adds need no branch.  Never read.
constexpr uint32_t kPadRow = kRowStride - 1;
static_assert(kPadRow >= kMaxRows && kPadRow < (1u << (32 - PPF_ANGLE_BITS)), "a spare row in every plane");

// uint2 counters that a block spills to (spill_acc)
constexpr size_t kSpillWords = (size_t)kPlanes * kRowStride;
constexpr size_t kVoteSmemBytes = (size_t)(kOffAcc + (kPlanes + 1) * kRowStride) * 4;

// Exclusive block scans of one or two values per thread; the totals come
// back by reference.  s_warp is this call site's own scratch; the caller
// places a barrier between two scans on the same scratch.
__device__ __forceinline__ uint2 block_excl_scan(uint2 v, uint2* s_warp, uint2& total) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint2 x = make_uint2(warp_incl_scan(v.x), warp_incl_scan(v.y));
  if (lane == 31) s_warp[warp] = x;
  block_sync();
  if (warp == 0) {
    const uint2 w = s_warp[lane % kVoteWarps];
    const uint2 t = make_uint2(warp_incl_scan(w.x), warp_incl_scan(w.y));
    if (lane < kVoteWarps) s_warp[lane] = t;
  }
  block_sync();
  const uint2 below = warp ? s_warp[warp - 1] : make_uint2(0u, 0u);
  total = s_warp[kVoteWarps - 1];
  return make_uint2(below.x + x.x - v.x, below.y + x.y - v.y);
}

__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t x = warp_incl_scan(v);
  if (lane == 31) s_warp[warp] = x;
  block_sync();
  if (warp == 0) {
    const uint32_t t = warp_incl_scan(s_warp[lane % kVoteWarps]);
    if (lane < kVoteWarps) s_warp[lane] = t;
  }
  block_sync();
  total = s_warp[kVoteWarps - 1];
  return (warp ? s_warp[warp - 1] : 0u) + x - v;
}

// Per-block shared state of a vote kernel besides the dynamic allocation.
struct VoteShared {
  // the item's scene reference point, its normal and rows 1-2 of its frame:
  // read from here by the scene walk of each tile, so that they do not hold
  // 14 registers through the vote passes between walks
  float4 p_r, n_r, f_r1, f_r2;
  uint32_t item, next, max, base;
  uint32_t n_ev, n_gr;  // events and groups of the list
  uint32_t rows[kFlagRows / 32];  // the model's row flags
  uint2 scan2[kVoteWarps];         // scratch of the two-value scans
  uint32_t scan_emit[kVoteWarps];  // scratch of the emission scan
  uint32_t wmax[kVoteWarps];       // per-warp maxima of the accumulator
};

// Fetches the next work item into sh.item (one atomic per block).
__device__ __forceinline__ uint32_t fetch_item(uint32_t* work_counter, VoteShared& sh) {
  if ((threadIdx.x >> 5) == 0) {
    uint32_t next = 0;
    if ((threadIdx.x & 31) == 0) next = atomicAdd(work_counter, 1u);
    next = __shfl_sync(0xffffffffu, next, 0);
    if ((threadIdx.x & 31) == 0) sh.item = next;
  }
  block_sync();
  return sh.item;
}

// Adds the block's statistics to the request's and clears them.  Called by the
// whole block between items, through the words of the event list: one atomic
// per counter and block.  (One per warp were 14000 on three addresses at the
// end of a launch.)
__device__ __forceinline__ void flush_stats(const VoteArgs& a, VoteStats& st) {
  unsigned long long v[3] = {st.votes, st.matched, st.exact};
  unsigned long long* const part = reinterpret_cast<unsigned long long*>(smem + kOffEvW);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  static_assert(kVoteWarps <= 32 && kEvents >= 3 * 32 * 2, "a lane per warp, in the event words");
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    for (int o = 16; o; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
    if (lane == 0) part[32 * k + warp] = v[k];
  }
  block_sync();
  if (warp < 3) {
    unsigned long long t = lane < kVoteWarps ? part[32 * warp + lane] : 0ull;
    for (int o = 16; o; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0 && t) atomicAdd(&a.stats[warp], t);
  }
  block_sync();
  st = VoteStats();
}

// The warp's histogram table and queue.
__device__ __forceinline__ uint32_t* warp_tab() { return smem + kOffTab + (threadIdx.x >> 5) * kTabWords; }
__device__ __forceinline__ uint32_t* warp_notes() { return smem + kOffNotes + (threadIdx.x >> 5) * kNotesLen; }
__device__ __forceinline__ uint32_t* warp_queue() { return smem + kOffQueue + (threadIdx.x >> 5) * 2 * kQueueLen; }

__device__ __forceinline__ uint32_t wrap30(int b) { return (uint32_t)(b < 0 ? b + PPF_N_ANGLE : b); }

// y' of an event word A and an entry: alpha + pi in 2^-32 turns, shifted down
// by the ambiguity margin (the entry's row bits shift out).
constexpr int kAngleShift = 32 - PPF_ANGLE_BITS;
__device__ __forceinline__ uint32_t count_angle(uint32_t w, uint32_t entry) {
  return ((w / PPF_N_ANGLE - PPF_BIN_MARGIN_UNITS) << kAngleShift) - (entry << kAngleShift);
}

// One vote more in (row, bin).
__device__ __forceinline__ void add_cell(uint32_t row, uint32_t bin) {
  uint32_t* const acc = smem + kOffAcc + row;
  if (bin == PPF_N_ANGLE) atomicAdd(acc + kPlanes * kRowStride, 1u);
  else atomicAdd(acc + (bin >> 1) * kRowStride, 1u << (16 * (bin & 1)));
}

// One vote less in (row, bin), bin < 30; the vote was counted there before,
// so the 16-bit counter does not borrow.
__device__ __forceinline__ void sub_cell(uint32_t row, uint32_t bin) {
  atomicSub(smem + kOffAcc + row + (bin >> 1) * kRowStride, 1u << (16 * (bin & 1)));
}

// Votes near a bin edge are counted in a provisional bin and queued per warp:
// (entry, event | provisional bin << 16).  A full queue is binned by the
// reference's exact arithmetic, one vote per lane: the exact path's loads and
// atan2f then run for 32 votes at once (they are 1.7e-4 of all votes, and
// one at a time they cost as much as the sweep itself).
template <bool kCheck>
__device__ __forceinline__ void drain_queue(const VoteArgs& a, const VoteShared& sh, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t* const queue = warp_queue();
  __syncwarp();
  if (lane < n) {
    const uint32_t pos = queue[2 * lane], inf = queue[2 * lane + 1];
    const uint32_t fast = inf >> 16;
    uint32_t i = in_range<kCheck>(a, 17, inf & 0xffffu, kEvents) ? smem[kOffEvI + (inf & 0xffffu)] : 0u;
    if (!in_range<kCheck>(a, 18, i, a.n_s)) i = 0;
    const float4 p4 = a.s_pts[i];
    FrameYZ fs;
    fs.r1 = sh.f_r1;
    fs.r2 = sh.f_r2;
    const uint32_t exact = exact_bin<kCheck>(a, pos, frame_point_yz(fs, make_float3(p4.x, p4.y, p4.z)));
    if (exact != fast && in_range<kCheck>(a, 19, fast, PPF_N_ANGLE) && in_range<kCheck>(a, 23, pos, a.P)) {
      const uint32_t row = __ldg(a.entries + pos) >> PPF_ANGLE_BITS;
      if (in_range<kCheck>(a, 7, row, a.chunk)) {
        sub_cell(row, fast);
        add_cell(row, exact);
      }
    }
  }
  __syncwarp();
}

// Queues the ambiguous votes of one event among the block's entries at pos
// (bit k of a lane's mask: its k-th entry) and returns the queue's new length.
// Called by the whole warp; it is rare and recomputes from the entries what
// its callers hold in registers.
template <bool kCheck>
__device__ __forceinline__ uint32_t queue_votes(const VoteArgs& a, const VoteShared& sh, uint32_t mask, uint32_t pos,
                                             uint32_t ev, bool sweep, uint32_t qn) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t w = smem[kOffEvW + ev];
  uint32_t* const queue = warp_queue();
#pragma unroll 1
  for (int k = 0; k < kPerLane; ++k) {
    const bool amb = mask >> k & 1u;
    const uint32_t lanes = __ballot_sync(0xffffffffu, amb);
    if (!lanes) continue;
    const uint32_t n = __popc(lanes);
    if (qn + n > kQueueLen) {
      drain_queue<kCheck>(a, sh, qn);
      qn = 0;
    }
    if (amb && in_range<kCheck>(a, 27, pos + 32u * k + lane, a.P)) {
      const uint32_t at = qn + __popc(lanes & ((1u << lane) - 1u));
      const uint32_t e = __ldg(a.entries + pos + 32u * k + lane);
      uint32_t bin;
      if (sweep) {
        const uint32_t t = (e & (kTurn - 1u)) * PPF_N_ANGLE;
        const int below = (w & (kTurn - 1u)) < (t & (kTurn - 1u)) ? 1 : 0;
        bin = wrap30((int)(w >> PPF_ANGLE_BITS) - (int)(t >> PPF_ANGLE_BITS) - below);
      } else {
        bin = (uint32_t)((unsigned long long)count_angle(w, e) * PPF_N_ANGLE >> 32);
      }
      queue[2 * at] = pos + 32u * k + lane;
      queue[2 * at + 1] = ev | bin << 16;
    }
    qn += n;
  }
  __syncwarp();
  return qn;
}

// Queues the ambiguous votes of the noted (block, event) pairs of a unit;
// returns the queue's length and the lane's ambiguous votes.  Notes past the
// array's end were not stored: the block that made them, `blk`, whose notes
// start at `own`, is then searched with all events of the piece.  Out of line
// and called about once per 24 notes at a block's end, where its callers hold
// little in registers: inside their loops it spilled a fifth of the sweep's
// shared-memory accesses, and called once per block it still saved and
// restored 6% of them.
template <bool kCheck>
__device__ __noinline__ uint2 queue_noted(const VoteArgs& a, const VoteShared& sh, uint32_t start, uint32_t end,
                                          uint32_t ev0, uint32_t cnt, uint32_t n_notes, uint32_t own, uint32_t blk,
                                          bool sweep, uint32_t qn) {
  const uint32_t* const notes = warp_notes();
  uint32_t n_exact = 0;
  __syncwarp();
  const bool over = n_notes > kNotesLen;
  const uint32_t n = over ? own + cnt : n_notes;
#pragma unroll 1
  for (uint32_t j = 0; j < n; ++j) {
    const uint32_t note = over && j >= own ? blk << 16 | (j - own) : notes[j];
    const uint32_t pos = start + (note >> 16) * kBlock, ev = ev0 + (note & 0xffffu);
    const uint32_t re = smem[kOffEvW + ev] & (kTurn - 1u);
    uint32_t amb = 0;
#pragma unroll
    for (int k = 0; k < kPerLane; ++k) {
      const uint32_t p = pos + 32u * k + (threadIdx.x & 31);
      if (p < end && in_range<kCheck>(a, 28, p, a.P)) {
        const uint32_t r = ((__ldg(a.entries + p) & (kTurn - 1u)) * PPF_N_ANGLE) & (kTurn - 1u);
        if (((re - r + kMargin - 1u) & (kTurn - 1u)) < 2 * kMargin - 1) amb |= 1u << k;
      }
    }
    n_exact += __popc(amb);
    qn = queue_votes<kCheck>(a, sh, amb, pos, ev, sweep, qn);
  }
  __syncwarp();
  return make_uint2(qn, n_exact);
}

// Entries [pos, pos + 128) of a unit that ends at `end`, kPerLane per lane
// (the pad row past the end).
__device__ __forceinline__ void load_block(const uint32_t* entries, uint32_t pos, uint32_t end,
                                           uint32_t (&e)[kPerLane]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < kPerLane; ++k) {
    const uint32_t p = pos + 32u * k + lane;
    e[k] = p < end ? __ldg(entries + p) : kPadRow << PPF_ANGLE_BITS;
  }
}

// A unit of a piece that is swept (sweep_pays): entries [start, end) of
// the piece's sub-run against events [ev0, ev0 + cnt), in ascending R.
//
// The votes of one entry (Q_m, R_m, row) are the histogram
// H[k] = #{events: Q_s - [R_s < R_m] = k}, rotated by Q_m: 30 counters for
// any number of events.  The entries come in ascending R (by buckets of
// 2^r_shift), so H changes only as R_m passes an event.  Per block of 128
// entries the warp keeps H as of the block's first bucket in a table of
// packed quadruples H[k .. k + 3], k = 0..59 modulo 30, and every lane adds it
// to its entry's row: it reads the 8 table words Q_m + 4j (the lanes' words
// lie among 30 consecutive ones: distinct banks or one broadcast) and adds 15
// words of 16-bit pairs, one per plane.  Events that lie inside the block's
// bucket range then move one vote for each entry beyond them.  Returns the
// queue's length and the lane's ambiguous votes.  Out of line (as count_unit),
// so that the block's phases around it do not spill in its loops.
template <bool kCheck>
__device__ __noinline__ uint2 sweep_unit(const VoteArgs& a, const VoteShared& sh, uint32_t start, uint32_t end,
                                           uint32_t ev0, uint32_t cnt, uint32_t qn) {
  uint32_t n_exact = 0;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t* const ev = smem + kOffEvW + ev0;
  uint32_t* const acc = smem + kOffAcc;
  uint32_t* const tab = warp_tab();
  uint32_t* const notes = warp_notes();
  uint32_t n_notes = 0;
  const uint32_t rs = a.r_shift;
  const uint32_t* const entries = a.entries;  // (a copy: a's fields are read anew after every atomic)
  uint32_t passed = 0;  // events of a bucket below the block's first: counted in H as Q_s - 1
  uint32_t done = 0;    // events too far below the block's first bucket to be ambiguous in it or later
  uint32_t h = 0;       // H[lane]
  for (uint32_t pos = start; pos < end; pos += kBlock) {
    const uint32_t n = min((uint32_t)kBlock, end - pos);
    int rm[kPerLane];  // R_m (-kTurn past the end: below every event)
    uint32_t row[kPerLane], qm[kPerLane];
    uint32_t rmin = kTurn, rmax = 0;
    uint32_t e[kPerLane];
    load_block(entries, pos, end, e);
#pragma unroll
    for (int k = 0; k < kPerLane; ++k) {
      const uint32_t t = (e[k] & (kTurn - 1u)) * PPF_N_ANGLE;
      const bool valid = 32u * k + lane < n;
      rm[k] = valid ? (int)(t & (kTurn - 1u)) : -(int)kTurn;
      row[k] = e[k] >> PPF_ANGLE_BITS;
      qm[k] = t >> PPF_ANGLE_BITS;
      if (valid) {
        rmin = min(rmin, (uint32_t)rm[k]);
        rmax = max(rmax, (uint32_t)rm[k]);
      }
    }
    rmin = __reduce_min_sync(0xffffffffu, rmin);
    rmax = __reduce_max_sync(0xffffffffu, rmax);
    const uint32_t b0 = rmin >> rs, b1 = rmax >> rs;
    bool changed = false;
    if (pos == start) {
      tab[lane] = 0u;
      __syncwarp();
      for (uint32_t j0 = 0; j0 < cnt; j0 += 32) {
        bool below = false, far = false;
        if (j0 + lane < cnt) {
          const uint32_t w = ev[j0 + lane], r = w & (kTurn - 1u), q = w >> PPF_ANGLE_BITS;
          below = (r >> rs) < b0;
          far = r + kMargin <= b0 << rs;
          atomicAdd(tab + (below ? (q ? q - 1u : PPF_N_ANGLE - 1u) : q), 1u);
        }
        passed += __popc(__ballot_sync(0xffffffffu, below));
        done += __popc(__ballot_sync(0xffffffffu, far));
      }
      __syncwarp();
      h = tab[lane];
      changed = true;
    } else {
      while (passed < cnt) {
        const uint32_t w = ev[passed], q = w >> PPF_ANGLE_BITS;
        if (((w & (kTurn - 1u)) >> rs) >= b0) break;
        h += (lane == (q ? q - 1u : PPF_N_ANGLE - 1u) ? 1u : 0u) - (lane == q ? 1u : 0u);
        changed = true;
        ++passed;
      }
      while (done < cnt && (ev[done] & (kTurn - 1u)) + kMargin <= b0 << rs) ++done;
    }
    if (changed) {
      const uint32_t k1 = lane + 1 >= PPF_N_ANGLE ? lane + 1 - PPF_N_ANGLE : lane + 1;
      const uint32_t k2 = lane + 2 >= PPF_N_ANGLE ? lane + 2 - PPF_N_ANGLE : lane + 2;
      const uint32_t two = h | __shfl_sync(0xffffffffu, h, k1) << 8;
      const uint32_t four = two | __shfl_sync(0xffffffffu, two, k2) << 16;
      __syncwarp();
      if (lane < PPF_N_ANGLE) {
        tab[lane] = four;
        tab[lane + PPF_N_ANGLE] = four;
      }
      __syncwarp();
    }
#pragma unroll
    for (int k = 0; k < kPerLane; ++k) {
      if (32u * k < n && in_range<kCheck>(a, 8, row[k], kRowStride)) {
        const uint32_t* const tp = tab + qm[k];
        uint32_t* const ap = acc + row[k];
        uint32_t v[(kPlanes + 1) / 2];
#pragma unroll
        for (uint32_t j = 0; j < (kPlanes + 1) / 2; ++j) v[j] = tp[4 * j];
#pragma unroll
        for (uint32_t j = 0; j < kPlanes; ++j)
          atomicAdd(ap + j * kRowStride, __byte_perm(v[j / 2], 0u, j & 1 ? 0x4342 : 0x4140));
      }
    }
    __syncwarp();
    // events among the block's entries, and within the margin of one; a block
    // near R = 0 meets the margin across it and looks at every event
    const bool edge = rmin < kMargin || rmax > kTurn - kMargin;
    const uint32_t own_notes = n_notes;
    for (uint32_t q = edge ? 0u : min(passed, done); q < cnt; ++q) {
      const uint32_t w = ev[q], re = w & (kTurn - 1u), qe = w >> PPF_ANGLE_BITS;
      if (!edge && (re >> rs) > b1 && re >= rmax + kMargin) break;
      uint32_t nearest = kTurn;  // distance above the margin's lower end, modulo a bin
#pragma unroll
      for (int k = 0; k < kPerLane; ++k)
        nearest = min(nearest, (uint32_t)((int)re - rm[k] + (int)kMargin - 1) & (kTurn - 1u));
      if (q >= passed) {
#pragma unroll
        for (int k = 0; k < kPerLane; ++k) {
          if ((int)re < rm[k] && in_range<kCheck>(a, 13, row[k], a.chunk)) {
            // (unsigned minima wrap the bins: below 0 is a large number)
            const uint32_t d = qe - qm[k], b = min(d, d + PPF_N_ANGLE), to = min(b - 1u, PPF_N_ANGLE - 1u);
            atomicAdd(acc + row[k] + (to >> 1) * kRowStride, to & 1 ? 1u << 16 : 1u);
            atomicAdd(acc + row[k] + (b >> 1) * kRowStride, b & 1 ? 0u - (1u << 16) : 0u - 1u);
          }
        }
      }
      if (__any_sync(0xffffffffu, nearest < 2 * kMargin - 1)) {
        if (n_notes < kNotesLen) notes[n_notes] = (pos - start) / kBlock << 16 | q;  // (by all lanes alike)
        ++n_notes;
      }
    }
    if (n_notes > kNotesLen - 8 || (n_notes && pos + kBlock >= end)) {
      const uint2 r = queue_noted<kCheck>(a, sh, start, end, ev0, cnt, n_notes, own_notes, (pos - start) / kBlock, true,
                                          qn);
      qn = r.x;
      n_exact += r.y;
      n_notes = 0;
    }
  }
  return make_uint2(qn, n_exact);
}

// A unit of a piece with few events or entries: every vote on its own.  With
// y' = (x_s - beta_m - margin) << 11 (count_angle), one 32 x 32 -> 64 multiply
// 15 y' gives the plane in its high word, the half of the counter word in the
// top bit of its low word and the position inside the bin in the rest: a vote
// is unambiguous exactly when 2 low is at most kSpan, and the bin is then that
// of y (y' wraps only for ambiguous votes, to bin 29, so every provisional
// bin is in [0, 29]).
template <bool kCheck>
__device__ __noinline__ uint2 count_unit(const VoteArgs& a, const VoteShared& sh, uint32_t start, uint32_t end,
                                           uint32_t ev0, uint32_t cnt, uint32_t qn) {
  uint32_t n_exact = 0;
  constexpr uint32_t kSpan = (kTurn - 2 * kMargin) << kAngleShift;
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t* const entries = a.entries;
  uint32_t* const acc = smem + kOffAcc;
  uint32_t* const notes = warp_notes();
  uint32_t n_notes = 0;
  for (uint32_t pos = start; pos < end; pos += kBlock) {
    const uint32_t n = min((uint32_t)kBlock, end - pos);
    uint32_t c[kPerLane];
    load_block(entries, pos, end, c);
    const uint32_t own_notes = n_notes;
    for (uint32_t g = 0; g < cnt; ++g) {
      const uint32_t base = count_angle(smem[kOffEvW + ev0 + g], 0u);
      bool amb = false;  // (a lane past the end may say so too)
#pragma unroll
      for (int k = 0; k < kPerLane; ++k) {
        if (32u * k < n && in_range<kCheck>(a, 14, c[k] >> PPF_ANGLE_BITS, kRowStride)) {
          const unsigned long long p = (unsigned long long)(base - (c[k] << kAngleShift)) * (PPF_N_ANGLE / 2);
          const uint32_t hi = (uint32_t)(p >> 32), lo = (uint32_t)p;
          atomicAdd(acc + hi * kRowStride + (c[k] >> PPF_ANGLE_BITS), 1u + (lo >> 31) * 65535u);
          amb = amb || (lo << 1) > kSpan;
        }
      }
      if (__any_sync(0xffffffffu, amb)) {
        if (n_notes < kNotesLen) notes[n_notes] = (pos - start) / kBlock << 16 | g;
        ++n_notes;
      }
    }
    if (n_notes > kNotesLen - 8 || (n_notes && pos + kBlock >= end)) {
      const uint2 r = queue_noted<kCheck>(a, sh, start, end, ev0, cnt, n_notes, own_notes, (pos - start) / kBlock,
                                          false, qn);
      qn = r.x;
      n_exact += r.y;
      n_notes = 0;
    }
  }
  return make_uint2(qn, n_exact);
}

// A unit whose votes all take the exact path (a degenerate frame vector of
// the scene pair or of a pair in the run).
template <bool kCheck>
__device__ __noinline__ void exact_unit(const VoteArgs& a, const VoteShared& sh, uint32_t start, uint32_t end,
                                        uint32_t ev0, uint32_t cnt) {
  for (uint32_t g = 0; g < cnt; ++g) {
    const float4 p4 = a.s_pts[smem[kOffEvI + ev0 + g]];
    FrameYZ fs;
    fs.r1 = sh.f_r1;
    fs.r2 = sh.f_r2;
    const float2 v = frame_point_yz(fs, make_float3(p4.x, p4.y, p4.z));
    for (uint32_t pos = start + (threadIdx.x & 31); pos < end; pos += 32) {
      const uint32_t row = __ldg(a.entries + pos) >> PPF_ANGLE_BITS;
      const uint32_t bin = exact_bin<kCheck>(a, pos, v);
      if (in_range<kCheck>(a, 6, row, a.chunk)) add_cell(row, bin);
    }
  }
}

// A warp's place in the walk over the scene: its next points and the pairs of
// its buffer that still await their lookup.
constexpr uint32_t kWalkStep = 2 * kVoteThreads;
static_assert(31 + 64 <= kNearLen && kNearLen == 3 * 32, "a step's pairs fit behind the waiting ones");
struct WalkState {
  uint32_t base = 0, n_near = 0;
  uint32_t waiting[3];  // the waiting pairs, 32 k + lane, while the buffer is in other use
};

// Fills the list with the events of s_r from the warps' places on, until the
// scene ends (false) or the list is full (true; uniform over the block).
//
// Warp w takes points 32 w + lane of every kVoteThreads, two such steps at a time.  With the model's feature
// table it first looks only at the distance: a pair whose distance row has no
// run is dropped, the others wait in the warp's buffer until there are 32, so
// that the angles (three acosf), the table lookup and the frame angle run on
// full warps.  On the bench's scene 9 of 10 pairs are dropped.  Without the
// table every pair's feature is hashed.
template <bool kCheck>
__device__ __forceinline__ bool walk_scene(const VoteArgs& a, uint32_t sr, bool count, WalkState& ws, VoteShared& sh,
                                           VoteStats& st) {
  uint32_t* const slot_key = smem + kOffSlotKey;
  uint32_t* const slot_cnt = smem + kOffSlotCnt;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* const near = smem + kOffNear + warp * kNearLen;
  // (the buffers lie over the pieces, which the list's votes have read)
#pragma unroll
  for (int k = 0; k < 3; ++k)
    if (32u * k + lane < ws.n_near) near[32 * k + lane] = ws.waiting[k];
  for (uint32_t i = tid; i < kSlots; i += kVoteThreads) {
    slot_key[i] = kNoRun;
    slot_cnt[i] = 0u;
  }
  if (tid == 0) sh.n_ev = sh.n_gr = 0u;
  block_sync();
  const float4 p4 = sh.p_r;
  const float3 pr = make_float3(p4.x, p4.y, p4.z);
  const float inv_d = 1.0f / a.d_dist;
  bool full = false;
  for (;;) {
    // gather pairs until 32 wait or the scene ends
    while (ws.n_near < 32 && ws.base < a.n_s) {
      // two points per lane, so that two loads are in flight
      bool keep[2];
      float4 q[2];
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        const uint32_t i = ws.base + kVoteThreads * k + tid;
        keep[k] = i < a.n_s && i != sr;
        if (keep[k] && a.lut) q[k] = a.s_pts[i];
      }
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (keep[k] && a.lut) {
          const float3 d = make_float3(q[k].x - pr.x, q[k].y - pr.y, q[k].z - pr.z);
          const float len = norm3(d);
          // rows past the flags are looked up by key
          keep[k] = !isnan(len);
          if (len < (float)(kFlagRows - 1) * a.d_dist) {
            const uint32_t nd = (uint32_t)quant_index(len, a.d_dist, inv_d);
            keep[k] = sh.rows[nd / 32] >> (nd % 32) & 1u;
          }
        }
        const uint32_t in = __ballot_sync(0xffffffffu, keep[k]);
        if (keep[k]) near[ws.n_near + __popc(in & ((1u << lane) - 1u))] = ws.base + kVoteThreads * k + tid;
        ws.n_near += __popc(in);
      }
      ws.base += kWalkStep;
    }
    __syncwarp();
    const uint32_t n = min(ws.n_near, 32u);
    if (n == 0) break;
    // One lane reads the count for its warp: other warps raise it meanwhile, and
    // lanes that read it for themselves could part here and leave the others
    // in the ballots below.
    uint32_t groups = 0;
    if (lane == 0) groups = *(volatile uint32_t*)&sh.n_gr;
    if (__shfl_sync(0xffffffffu, groups, 0) > kGroupLimit) {
      full = true;
      break;
    }
    // one pair per lane: feature, lookup, frame angle
    uint32_t run = kNoRun, beta = 0, i = 0;
    bool exact = false;
    if (lane < n) {
      i = near[lane];
      const float4 pi4 = a.s_pts[i], ni4 = a.s_nrm[i], n4 = sh.n_r;
      const float3 pi = make_float3(pi4.x, pi4.y, pi4.z), ni = make_float3(ni4.x, ni4.y, ni4.z);
      const float3 nr = make_float3(n4.x, n4.y, n4.z);
      const float3 d = make_float3(pi.x - pr.x, pi.y - pr.y, pi.z - pr.z);
      const float len = norm3(d);
      uint32_t nd = kLutRows;
      if (a.lut && len < (float)(kLutRows - 1) * a.d_dist) nd = (uint32_t)quant_index(len, a.d_dist, inv_d);
      if (nd < kLutRows) {
        run = __ldg(a.lut + nd * kAngleCombos + pair_angles(nr, ni, d, len));
      } else {
        const uint32_t key = feature_key(pair_feature(pr, nr, pi, ni, a.d_dist));
        if (key != 0u) run = ht_lookup(a.ht_keys, a.ht_runs, a.ht_mask, key);
      }
      if (run != kNoRun && in_range<kCheck>(a, 2, run, a.K)) {
        FrameYZ fs;
        fs.r1 = sh.f_r1;
        fs.r2 = sh.f_r2;
        const float2 v = frame_point_yz(fs, pi);
        exact = fabsf(v.x) + fabsf(v.y) < 1e-12f || !isfinite(v.x) || !isfinite(v.y) || __ldg(a.run_flags + run);
        beta = angle21(v);
      }
    }
    __syncwarp();
    const uint32_t hits = __ballot_sync(0xffffffffu, run != kNoRun);
    if (hits) {
      // room for all of them, or none is taken and the pairs stay
      uint32_t at = 0;
      if (lane == 0) {
        at = *(volatile uint32_t*)&sh.n_ev;
        for (;;) {
          if (at + __popc(hits) > kEvents) {
            at = kNoRun;
            break;
          }
          const uint32_t was = atomicCAS(&sh.n_ev, at, at + __popc(hits));
          if (was == at) break;
          at = was;
        }
      }
      at = __shfl_sync(0xffffffffu, at, 0);
      if (at == kNoRun) {
        full = true;
        break;
      }
      if (run != kNoRun) {
        at += __popc(hits & ((1u << lane) - 1u));
        if (count) {
          st.votes += __ldg(a.run_count + run);
          st.matched += 1;
        }
        // the event's slot and its rank in the group
        const uint32_t group = run | (exact ? kExactGroup : 0u);
        uint32_t slot = __umulhi(group * 0x9E3779B1u, kSlots);
        for (uint32_t probe = 0; probe < kSlots; ++probe) {
          uint32_t k = *(volatile uint32_t*)(slot_key + slot);
          if (k == kNoRun) {
            k = atomicCAS(slot_key + slot, kNoRun, group);
            if (k == kNoRun) {
              atomicAdd(&sh.n_gr, 1u);
              break;
            }
          }
          if (k == group) break;
          slot = (slot + 1) & (kSlots - 1);
        }
        const uint32_t rank = atomicAdd(slot_cnt + slot, 1u);
        if (in_range<kCheck>(a, 15, at, kEvents)) {
          smem[kOffEvW + at] = ((beta + (kTurn >> 1)) & (kTurn - 1u)) * PPF_N_ANGLE;
          smem[kOffEvI + at] = i;
          smem[kOffEvK + at] = slot << 16 | rank;
        }
      }
    }
    // the buffer's rest (at most 63 pairs) moves to its front
    __syncwarp();
    const uint32_t rest = ws.n_near - n;
    const uint32_t m0 = lane < rest ? near[n + lane] : 0u, m1 = lane + 32 < rest ? near[n + lane + 32] : 0u;
    __syncwarp();
    if (lane < rest) near[lane] = m0;
    if (lane + 32 < rest) near[lane + 32] = m1;
    ws.n_near = rest;
    __syncwarp();
  }
  // what waits is kept aside while the list's pieces take the buffers' place
  __syncwarp();
#pragma unroll
  for (int k = 0; k < 3; ++k) ws.waiting[k] = 32u * k + lane < ws.n_near ? near[32 * k + lane] : 0u;
  __syncwarp();
  return __syncthreads_or(full);
}

// Ascending bitonic sort of 32 M distinct words over a warp; word 32 m + lane
// is x[m] of the lane.
template <int M>
__device__ __forceinline__ void warp_sort(uint32_t (&x)[M]) {
  const uint32_t lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 2; k <= 32 * M; k <<= 1) {
#pragma unroll
    for (int j = k >> 1; j >= 32; j >>= 1) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const int o = m ^ (j >> 5);
        if (o > m) {
          const uint32_t lo = min(x[m], x[o]), hi = max(x[m], x[o]);
          const bool up = ((32 * m) & k) == 0;  // k > 32: the same for all lanes
          x[m] = up ? lo : hi;
          x[o] = up ? hi : lo;
        }
      }
    }
#pragma unroll
    for (int j = k >> 1 < 16 ? k >> 1 : 16; j > 0; j >>= 1) {
#pragma unroll
      for (int m = 0; m < M; ++m) {
        const uint32_t y = __shfl_xor_sync(0xffffffffu, x[m], j);
        const bool up = (((uint32_t)(32 * m) | lane) & (uint32_t)k) == 0, low = (lane & (uint32_t)j) == 0;
        x[m] = up == low ? min(x[m], y) : max(x[m], y);
      }
    }
  }
}

// The sort of sort_piece for pieces of at most 32 M events: R above the
// event's index, so that the words are distinct and carry their events.
template <int M>
__device__ __forceinline__ void order_events(uint32_t* ew, uint32_t* ei, uint32_t cnt) {
  static_assert(32 * M <= 256, "an index byte below the 21 bits of R");
  const uint32_t lane = threadIdx.x & 31;
  uint32_t x[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const uint32_t j = 32u * m + lane;
    x[m] = j < cnt ? (ew[j] & (kTurn - 1u)) << 8 | j : 0xffffff00u | j;
  }
  warp_sort<M>(x);
  uint32_t w[M], i[M];
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const uint32_t from = x[m] & 0xffu;
    w[m] = from < cnt ? ew[from] : 0u;
    i[m] = from < cnt ? ei[from] : 0u;
  }
  __syncwarp();
#pragma unroll
  for (int m = 0; m < M; ++m) {
    const uint32_t j = 32u * m + lane;
    if (j < cnt) {
      ew[j] = w[m];
      ei[j] = i[m];
    }
  }
}

// Sorts a swept piece's events by R and returns an upper bound of how many of
// them one entry can vote into one bin: its votes for a bin come from one
// bin's width of event angles, plus the margin on both sides for votes near an
// edge, which lies within four neighbouring half bins.
__device__ __forceinline__ uint32_t sort_piece(uint32_t ev0, uint32_t cnt) {
  uint32_t* const tab = warp_tab();
  const uint32_t lane = threadIdx.x & 31;
  uint32_t* const ew = smem + kOffEvW + ev0;
  uint32_t* const ei = smem + kOffEvI + ev0;
  constexpr uint32_t kHalves = 2 * PPF_N_ANGLE;
  static_assert(kHalves <= kTabWords, "a counter per half bin");
  for (uint32_t k = lane; k < kHalves; k += 32) tab[k] = 0u;
  __syncwarp();
  for (uint32_t j = lane; j < cnt; j += 32) atomicAdd(tab + (ew[j] >> (PPF_ANGLE_BITS - 1)), 1u);
  if (cnt <= 32) order_events<1>(ew, ei, cnt);
  else if (cnt <= 64) order_events<2>(ew, ei, cnt);
  else if (cnt <= 128) order_events<4>(ew, ei, cnt);
  else order_events<8>(ew, ei, cnt);
  __syncwarp();
  uint32_t win = 0;
  for (uint32_t k = lane; k < kHalves; k += 32) {
    uint32_t four = 0;
    for (uint32_t o = k; o < k + 4; ++o) four += tab[o >= kHalves ? o - kHalves : o];
    win = max(win, four);
  }
  win = __reduce_max_sync(0xffffffffu, win);
  __syncwarp();
  return win;
}

// Groups the list's events by run (counting sort through registers, in
// place), cuts the groups into pieces and sorts the swept ones.  Returns the
// number of pieces.
template <bool kCheck>
__device__ __forceinline__ uint32_t group_events(const VoteArgs& a, uint32_t n_ev, VoteShared& sh) {
  uint32_t* const slot_key = smem + kOffSlotKey;
  uint32_t* const slot_cnt = smem + kOffSlotCnt;
  const uint32_t tid = threadIdx.x, warp = tid >> 5;
  const uint32_t key0 = slot_key[2 * tid], key1 = slot_key[2 * tid + 1];
  const uint32_t c0 = slot_cnt[2 * tid], c1 = slot_cnt[2 * tid + 1];
  const uint32_t n0 = (c0 + kPieceEvents - 1) / kPieceEvents, n1 = (c1 + kPieceEvents - 1) / kPieceEvents;
  uint2 total;
  const uint2 at = block_excl_scan(make_uint2(c0 + c1, n0 + n1), sh.scan2, total);
  uint32_t w[kEventsPerThread], ei[kEventsPerThread], ek[kEventsPerThread];
#pragma unroll
  for (uint32_t k = 0; k < kEventsPerThread; ++k) {
    const uint32_t j = tid + k * kVoteThreads;
    w[k] = ei[k] = ek[k] = 0;
    if (j < n_ev) {
      w[k] = smem[kOffEvW + j];
      ei[k] = smem[kOffEvI + j];
      ek[k] = smem[kOffEvK + j];
    }
  }
  slot_cnt[2 * tid] = at.x;
  slot_cnt[2 * tid + 1] = at.x + c0;
  uint32_t p = at.y;
  for (uint32_t o = 0; o < c0 && in_range<kCheck>(a, 24, p, kMaxPieces); o += kPieceEvents, ++p) {
    smem[kOffPcRun + p] = key0 & ~kExactGroup;
    const uint32_t n = min(kPieceEvents, c0 - o);
    smem[kOffPcInf + p] = piece_info(at.x + o, n, key0 & kExactGroup, n);
  }
  for (uint32_t o = 0; o < c1 && in_range<kCheck>(a, 24, p, kMaxPieces); o += kPieceEvents, ++p) {
    smem[kOffPcRun + p] = key1 & ~kExactGroup;
    const uint32_t n = min(kPieceEvents, c1 - o);
    smem[kOffPcInf + p] = piece_info(at.x + c0 + o, n, key1 & kExactGroup, n);
  }
  block_sync();  // offsets visible, every event in a register
#pragma unroll
  for (uint32_t k = 0; k < kEventsPerThread; ++k) {
    if (tid + k * kVoteThreads < n_ev) {
      const uint32_t to = slot_cnt[ek[k] >> 16] + (ek[k] & 0xffffu);
      if (in_range<kCheck>(a, 25, to, n_ev)) {
        smem[kOffEvW + to] = w[k];
        smem[kOffEvI + to] = ei[k];
      }
    }
  }
  block_sync();  // the slots are free for the tables from here on
  for (uint32_t q = warp; q < total.y; q += kVoteWarps) {
    const uint32_t inf = smem[kOffPcInf + q];
    const uint32_t ev0 = inf & 0x1fffu, cnt = (inf >> 13) & 0xffu;
    if (cnt < kSweepMin || (inf >> 21 & 1u)) continue;
    const uint32_t win = sort_piece(ev0, cnt);
    if ((tid & 31) == 0) smem[kOffPcInf + q] = piece_info(ev0, cnt, false, win);
  }
  block_sync();
  return total.y;
}

// Adds the accumulator's 16-bit counters to the block's 32-bit counters in
// global memory and clears them (each thread always handles the same rows).
__device__ __forceinline__ void spill_acc(const VoteArgs& a, bool first) {
  uint32_t* const acc = smem + kOffAcc;
  uint2* const sp = a.spill + (size_t)blockIdx.x * kSpillWords;
  block_sync();
  for (uint32_t row = threadIdx.x; row < a.chunk; row += kVoteThreads) {
#pragma unroll
    for (uint32_t j = 0; j < kPlanes; ++j) {
      const uint32_t v = acc[j * kRowStride + row];
      uint2* const at = sp + j * kRowStride + row;
      uint2 s = make_uint2(0u, 0u);
      if (!first) s = *at;
      *at = make_uint2(s.x + (v & 0xffffu), s.y + (v >> 16));
      acc[j * kRowStride + row] = 0u;
    }
  }
  block_sync();
}

// The units [u0, u1) of the current chunk, events [s0, s1) of each piece.
template <bool kCheck>
__device__ __forceinline__ void vote_units(const VoteArgs& a, VoteShared& sh, VoteStats& st, uint32_t n_pieces,
                                           uint32_t u0, uint32_t u1, uint32_t s0, uint32_t s1, uint32_t shift,
                                           uint32_t item) {
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const uint32_t* const pc_unit = smem + kOffPcUnit;
  if (tid == 0) sh.next = u0 + kVoteWarps;
  block_sync();
  uint32_t qn = 0;
  const uint32_t stride = (n_pieces + 31) / 32;
  uint32_t u = u0 + warp;
  while (u < u1) {
    // piece p with pc_unit[p] <= u < pc_unit[p + 1] (pc_unit is
    // nondecreasing): one ballot over every stride-th piece, then over the
    // stride (at most (kMaxPieces + 31) / 32, 53 in a wide block) pieces behind it
    const uint32_t blk =
        31u - __clz(__ballot_sync(0xffffffffu, lane * stride <= n_pieces && pc_unit[min(lane * stride, n_pieces)] <= u));
    uint32_t p = blk * stride;
    uint32_t in = 0;
    for (uint32_t o = 1; o < stride; o += 32)
      in += __popc(__ballot_sync(0xffffffffu, o + lane < stride && p + o + lane <= n_pieces &&
                                                  pc_unit[min(p + o + lane, n_pieces)] <= u));
    p += in;
    const uint32_t inf = smem[kOffPcInf + min(p, n_pieces - 1)];
    const uint32_t lo = smem[kOffPcLo + p], len = smem[kOffPcLen + p];
    const uint32_t skip = (u - pc_unit[p]) << shift;
    const uint32_t start = lo + skip;
    uint32_t end = lo + min(len, skip + (1u << shift));
    // Always-on guard (one compare per unit): a unit outside its sub-run or
    // the entry array is recorded, raises kFlagBadIndex and is skipped, so
    // the lookup fails instead of the kernel reading outside the entries.
    if (p >= n_pieces || skip >= len || end > a.P || start >= end) {
      if (lane == 0) {
        if (atomicCAS(&a.bad[3], 0ull, 1ull) == 0ull) {
          a.bad[4] = ((unsigned long long)p << 32) | u;
          a.bad[5] = ((unsigned long long)n_pieces << 32) | pc_unit[min(p, n_pieces)];
          a.bad[6] = ((unsigned long long)lo << 32) | len;
          a.bad[7] = ((unsigned long long)u0 << 32) | u1;
          a.bad[8] = ((unsigned long long)s0 << 32) | item;
          a.bad[9] = ((unsigned long long)warp << 32) | inf;
        }
        atomicOr(a.flags, (uint32_t)kFlagBadIndex);
      }
      end = start;
    }
    const uint32_t cnt = (inf >> 13) & 0xffu;
    const uint32_t ev0 = (inf & 0x1fffu) + min(s0, cnt), n_ev = min(s1, cnt) - min(s0, cnt);
    if (end > start && n_ev) {
      if (inf >> 21 & 1u) {
        exact_unit<kCheck>(a, sh, start, end, ev0, n_ev);
        if (lane == 0) st.exact += (unsigned long long)(end - start) * n_ev;
      } else {
        const uint2 r = sweep_pays(cnt, len) ? sweep_unit<kCheck>(a, sh, start, end, ev0, n_ev, qn)
                                         : count_unit<kCheck>(a, sh, start, end, ev0, n_ev, qn);
        qn = r.x;
        st.exact += r.y;
      }
    }
    __syncwarp();
    if (lane == 0) u = atomicAdd(&sh.next, 1u);
    u = __shfl_sync(0xffffffffu, u, 0);
  }
  if (qn) drain_queue<kCheck>(a, sh, qn);
  block_sync();
}

// Largest 16-bit counter of the accumulator.
__device__ __forceinline__ uint32_t acc_max(const VoteArgs& a, VoteShared& sh) {
  uint32_t m = 0;
  for (uint32_t row = threadIdx.x; row < a.chunk; row += kVoteThreads) {
#pragma unroll
    for (uint32_t j = 0; j < kPlanes; ++j) {
      const uint32_t v = smem[kOffAcc + j * kRowStride + row];
      m = max(m, max(v & 0xffffu, v >> 16));
    }
  }
  m = __reduce_max_sync(0xffffffffu, m);
  if ((threadIdx.x & 31) == 0) sh.wmax[threadIdx.x >> 5] = m;
  block_sync();
  m = __reduce_max_sync(0xffffffffu, sh.wmax[threadIdx.x % kVoteWarps]);
  block_sync();
  return m;
}

// Votes of the grouped events into chunk c.  `bound` is the largest value a
// 16-bit counter can hold so far.  Pieces that could take one past 65535 go in
// batches; between two the bound is replaced by the largest counter, and the
// accumulator spilled when that is past half the range.
template <bool kCheck>
__device__ __forceinline__ void vote_chunk(const VoteArgs& a, uint32_t c, uint32_t n_pieces, VoteShared& sh,
                                           VoteStats& st, uint32_t& bound, bool& spilled, uint32_t item) {
  if (n_pieces == 0) return;
  const uint32_t tid = threadIdx.x;
  uint32_t shift = a.unit_shift;
  uint32_t lo[2], len[2], units[2], inc[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t p = 2 * tid + k;
    lo[k] = len[k] = units[k] = inc[k] = 0;
    if (p < n_pieces) {
      const uint32_t run = smem[kOffPcRun + p], win = smem[kOffPcInf + p] >> 22;
      if (in_range<kCheck>(a, 16, run, a.K)) {
        const uint32_t* sp = a.split + (size_t)run * (a.n_chunks + 1) + c;
        lo[k] = __ldg(sp);
        len[k] = __ldg(sp + 1) - lo[k];
        if (kCheck && !in_range<kCheck>(a, 3, (unsigned long long)lo[k] + len[k], a.P + 1)) len[k] = 0;
        // win <= 256 events, at most run_maxl <= 65535 entries each
        inc[k] = len[k] ? min(win * __ldg(a.run_maxl + run), kCounterMax + 1u) : 0u;
      }
    }
  }
  uint2 total, at;
  for (;;) {
#pragma unroll
    for (int k = 0; k < 2; ++k) units[k] = (len[k] >> shift) + (len[k] & ((1u << shift) - 1u) ? 1u : 0u);
    at = block_excl_scan(make_uint2(units[0] + units[1], inc[0] + inc[1]), sh.scan2, total);
    // few units leave warps idle at the end of the phase: halve them
    if (total.x >= kMinUnits || shift <= kMinUnitShift) break;
    --shift;
    block_sync();
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const uint32_t p = 2 * tid + k;
    if (p <= n_pieces) {
      smem[kOffPcLo + p] = lo[k];
      smem[kOffPcLen + p] = len[k];
      smem[kOffPcUnit + p] = at.x + (k ? units[0] : 0u);
      smem[kOffPcInc + p] = at.y + (k ? inc[0] : 0u);
    }
  }
  block_sync();
  if (total.x == 0) return;
  auto spill = [&]() {
    if (!bound) return;
    spill_acc(a, !spilled);
    spilled = true;
    bound = 0;
  };
  const uint32_t* const pc_inc = smem + kOffPcInc;
  const uint32_t* const pc_unit = smem + kOffPcUnit;
  for (uint32_t p0 = 0; p0 < n_pieces;) {
    if (bound && bound + (total.y - pc_inc[p0]) > kCounterMax) {
      bound = acc_max(a, sh);
      if (bound > kCounterMax / 2) spill();
    }
    uint32_t p1 = p0, hi = n_pieces;  // the last p1 whose pieces from p0 on fit
    while (p1 < hi) {
      const uint32_t mid = (p1 + hi + 1) / 2;
      if (bound + (pc_inc[mid] - pc_inc[p0]) <= kCounterMax) p1 = mid;
      else hi = mid - 1;
    }
    if (p1 > p0) {
      vote_units<kCheck>(a, sh, st, n_pieces, pc_unit[p0], pc_unit[p1], 0, kPieceEvents, shift, item);
      bound += pc_inc[p1] - pc_inc[p0];
      p0 = p1;
    } else if (bound) {
      spill();  // and try the piece again with all the range
    } else {
      // one piece alone: as many of its events at a time as surely fit
      const uint32_t sub = max(1u, kCounterMax / max(1u, __ldg(a.run_maxl + smem[kOffPcRun + p0])));
      const uint32_t cnt = (smem[kOffPcInf + p0] >> 13) & 0xffu;
      for (uint32_t s0 = 0; s0 < cnt; s0 += sub) {
        spill();
        vote_units<kCheck>(a, sh, st, n_pieces, pc_unit[p0], pc_unit[p0 + 1], s0, min(s0 + sub, cnt), shift, item);
        bound = kCounterMax;
      }
      ++p0;
    }
  }
}

// Running maximum and emission of the accumulator's cells.
template <bool kCheck>
__device__ __forceinline__ void emit_chunk(const VoteArgs& a, uint32_t sr, uint32_t c, uint32_t item, bool spilled,
                                           VoteShared& sh) {
  const uint32_t* const acc = smem + kOffAcc;
  const uint2* const sp = a.spill + (size_t)blockIdx.x * kSpillWords;
  const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // calls f(row, bin, count) for this thread's counters (its own rows)
  auto each = [&](auto f) {
    for (uint32_t row = tid; row < a.chunk; row += kVoteThreads) {
#pragma unroll
      for (uint32_t j = 0; j < kPlanes; ++j) {
        const uint32_t v = acc[j * kRowStride + row];
        uint2 n = make_uint2(v & 0xffffu, v >> 16);
        if (spilled) n = sp[j * kRowStride + row];
        f(row, 2 * j, n.x);
        f(row, 2 * j + 1, n.y);
      }
      f(row, (uint32_t)PPF_N_ANGLE, acc[kPlanes * kRowStride + row]);
    }
  };
  uint32_t lmax = 0;
  each([&](uint32_t, uint32_t, uint32_t cnt) { lmax = max(lmax, cnt); });
  lmax = __reduce_max_sync(0xffffffffu, lmax);
  if (lane == 0) sh.wmax[warp] = lmax;
  block_sync();
  if (warp == 0) {
    const uint32_t m = __reduce_max_sync(0xffffffffu, sh.wmax[lane % kVoteWarps]);
    if (lane == 0) sh.max = max(atomicMax(a.global_max, m), m);
  }
  block_sync();
  const float floor_v = a.floor >= 0.f ? a.floor : a.thr * (float)sh.max;
  auto kept = [&](uint32_t cnt) { return cnt != 0u && (a.emit_all || (float)cnt > floor_v); };
  // All-or-nothing slot reservation for the chunk's cells: a chunk that does
  // not fit writes nothing and is queued for a second launch after the
  // buffer has grown, so the buffer never holds a partial chunk.  Slots are
  // what an atomic addition to the cells asked for returns: that total only
  // grows, so the chunks that fit are the first ones added and lie without
  // gaps, and n_cand is the sum of theirs.  (A compare-and-swap on n_cand took
  // 34000 cycles where 140 blocks emitted at once, a quarter of a launch of
  // one small item per block.)
  uint32_t my_n = 0;
  each([&](uint32_t, uint32_t, uint32_t cnt) { my_n += kept(cnt) ? 1u : 0u; });
  uint32_t item_total;
  const uint32_t my_off = block_excl_scan(my_n, sh.scan_emit, item_total);
  if (item_total == 0) return;  // uniform
  if (tid == 0) {
    const unsigned long long at = a.cand_base + atomicAdd(a.n_needed, (unsigned long long)item_total);
    const bool fits = at + item_total <= a.cand_cap;
    if (fits) {
      atomicAdd(a.n_cand, item_total);
    } else {
      const uint32_t k = atomicAdd(a.n_redo, 1u);
      if (in_range<kCheck>(a, 9, k, a.n_items_total)) a.redo_items[k] = item;
    }
    sh.base = fits ? (uint32_t)at : 0xffffffffu;
  }
  block_sync();
  const uint32_t item_base = sh.base;
  if (item_base == 0xffffffffu) return;
  uint32_t slot = item_base + my_off;
  each([&](uint32_t row, uint32_t bin, uint32_t cnt) {
    if (!kept(cnt)) return;
    const uint32_t mr = c * a.chunk + row;
    if (in_range<kCheck>(a, 10, slot, a.cand_cap)) {
      a.cand_code[slot] = ((unsigned long long)sr << 32) | ((unsigned long long)mr << 6) | bin;
      a.cand_count[slot] = cnt;
    }
    ++slot;
  });
}

// One work item of request `a` (slot_of_item indexes a's items, or
// a.item_list).  Called by every thread of the block.  A scene whose matched
// pairs fit the list is walked once for all chunks of the item; otherwise
// every chunk walks it again in as many parts as it takes.
template <bool kCheck>
__device__ __forceinline__ void vote_item(const VoteArgs& a, uint32_t slot_of_item, VoteShared& sh, VoteStats& st) {
  const uint32_t tid = threadIdx.x;
  uint32_t rq, c0, c1;
  if (a.item_list) {
    const uint32_t item = a.item_list[slot_of_item];
    rq = item / a.n_chunks;
    c0 = item - rq * a.n_chunks;
    c1 = c0 + 1;
  } else {
    rq = slot_of_item / a.n_cg;
    c0 = (slot_of_item - rq * a.n_cg) * a.cpi;
    c1 = min(a.n_chunks, c0 + a.cpi);
  }
  // ref < n_ref, so sr = ref * ref_df < n_s
  const uint32_t ref = (uint32_t)(((unsigned long long)rq * a.perm_mul) % a.n_ref);
  const uint32_t sr = ref * a.ref_df;
  // thread 0 publishes the frame of s_r, warp 1 the model's row flags; the
  // barrier at the start of the walk makes them visible, and the previous item's readers are past the item-fetch
  // barrier before it is overwritten
  if (tid == 0) {
    const float4 p4 = a.s_pts[sr], n4 = a.s_nrm[sr];
    const FrameYZ f = frame_yz(make_float3(p4.x, p4.y, p4.z), make_float3(n4.x, n4.y, n4.z));
    sh.p_r = p4;
    sh.n_r = n4;
    sh.f_r1 = f.r1;
    sh.f_r2 = f.r2;
  }
  static_assert(kFlagRows / 32 == 32, "a row flag word per lane");
  if (tid >= 32 && tid < 64 && a.lut) sh.rows[tid - 32] = __ldg(a.row_flags + tid - 32);
  bool whole = false;  // the list holds all events of s_r
  uint32_t n_pieces = 0;
  for (uint32_t c = c0; c < c1; ++c) {
    const uint32_t item = rq * a.n_chunks + c;
    if (c > c0) block_sync();  // the previous chunk's emission has read the accumulator
    for (uint32_t row = tid; row < a.chunk; row += kVoteThreads) {
#pragma unroll
      for (uint32_t j = 0; j <= kPlanes; ++j) smem[kOffAcc + j * kRowStride + row] = 0u;
    }
    uint32_t bound = 0;
    bool spilled = false;
    if (whole) {
      vote_chunk<kCheck>(a, c, n_pieces, sh, st, bound, spilled, item);
    } else {
      const bool count = c == 0 && !a.item_list;
      WalkState w;
      for (bool first = true;; first = false) {
        const bool more = walk_scene<kCheck>(a, sr, count, w, sh, st);
        const uint32_t n_ev = sh.n_ev;
        n_pieces = n_ev ? group_events<kCheck>(a, n_ev, sh) : 0;
        whole = first && !more;
        vote_chunk<kCheck>(a, c, n_pieces, sh, st, bound, spilled, item);
        if (!more) break;
        block_sync();  // the votes' reads of the list are over
      }
    }
    block_sync();  // all votes of the chunk are counted
    if (spilled && bound) spill_acc(a, false);
    emit_chunk<kCheck>(a, sr, c, item, spilled, sh);
  }
  // The item-fetch barrier of the caller separates these reads of the
  // accumulator from the next item's clear.
}

template <bool kCheck>
__global__ void __launch_bounds__(kVoteThreads, kBlocksPerSm) vote_kernel(const __grid_constant__ VoteArgs a) {
  __shared__ VoteShared sh;
  VoteStats st;
  for (;;) {
    const uint32_t slot = fetch_item(a.work_counter, sh);
    if (slot >= a.n_items) break;
    vote_item<kCheck>(a, slot, sh, st);
  }
  flush_stats(a, st);
}

template <bool kCheck>
__global__ void __launch_bounds__(kVoteThreads, kBlocksPerSm) vote_batch_kernel(BatchArgs b) {
  __shared__ VoteShared sh;
  __shared__ VoteArgs s_args;
  VoteStats st;
  uint32_t cur = 0xffffffffu;
  for (;;) {
    const uint32_t g = fetch_item(b.work_counter, sh);
    if (g >= b.n_items) break;
    uint32_t lo = 0, hi = b.n_reqs;  // request r with item_off[r] <= g < item_off[r + 1]
    while (hi - lo > 1) {
      const uint32_t mid = (lo + hi) >> 1;
      if (__ldg(b.item_off + mid) <= g) lo = mid;
      else hi = mid;
    }
    if (lo != cur) {  // uniform: every thread found the same request
      if (cur != 0xffffffffu) flush_stats(s_args, st);
      block_sync();
      constexpr int kWords = sizeof(VoteArgs) / 4;
      static_assert(sizeof(VoteArgs) % 4 == 0 && kWords <= kVoteThreads, "request arguments fit one copy pass");
      if (threadIdx.x < kWords)
        reinterpret_cast<uint32_t*>(&s_args)[threadIdx.x] = reinterpret_cast<const uint32_t*>(b.reqs + lo)[threadIdx.x];
      block_sync();
      cur = lo;
    }
    vote_item<kCheck>(s_args, g - __ldg(b.item_off + lo), sh, st);
  }
  if (cur != 0xffffffffu) flush_stats(s_args, st);
}
