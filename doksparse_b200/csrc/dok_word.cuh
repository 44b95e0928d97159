// The general set of values that share their word with the number of their row.
//
// Which of several rows with one key comes last is what the stamps of k_set_claim are for: a write of its own per row, to a
// second array where the slot has no room for it, and a second kernel that lets the last row write again.  A value of at
// most 4 bytes needs neither.  In 32-byte slots it has the 8 bytes behind the tag for itself, so {row's number, value} is one
// word, and one atomicMax per row, which nobody waits for, leaves the last row's value.  A slot is claimed by a 128-bit CAS
// of {tag, word}; whoever finds the tag therefore sees in the word whether a row of this batch has put it there, which is
// what the reference's count of an assignment asks for, and there is nothing left for further kernels.  (Slots of 64 and 128
// bytes have other use for that padding: dok_mark_passed.)
//
// Numbers go on from set to set: a table's `sequence` on the device holds the next one, so that a captured set counts on
// when it is replayed.  Before they run out at 2^31 rows k_word_begin clears them.
//
// 4 M-pair assignment to a 2-D tensor: 393 + 56 + 25 us of k_set_claim, k_set_resolve, k_set_count; here 219 + 4.  8.4 M rows of
// 4-byte values in a table of 2^26 keys, a fifth of them new: 688 -> 564; 800 k Zipf ids 97 -> 52.
#pragma once

// row's number (31 bits) | this batch claimed the slot | value (32 bits)
#define DOK_WORD_FRESH (1ULL << 32)
#define DOK_WORD_SHIFT 33
#define DOK_WORD_ROWS 0x7ffffff0LL
enum { DOK_SEQ_NEXT = 0, DOK_SEQ_BASE = 1, DOK_SEQ_TICKET = 2 };

inline bool dok_set_in_word(const DevTable &t, const DevHash &hp, ll_t n) {
  return t.sb == 32 && t.vb <= 4 && hp.dtype < DOK_F16 && n <= DOK_WORD_ROWS;
}

__device__ __forceinline__ void dok_clear_numbers(const DevTable &t) {
  for (ll_t i = (ll_t)blockIdx.x * blockDim.x + threadIdx.x; i < t.n_slots; i += (ll_t)gridDim.x * blockDim.x)
    *(unsigned *)(dok_value_ptr(t, i) + 4) = 0;
}
// The numbers of this set's rows: base + 1 ... base + n.
static __global__ void __launch_bounds__(DOK_TPB) k_word_begin(DevTable t, ll_t *sequence, ll_t n) {
  __shared__ ll_t next;
  if (threadIdx.x == 0) next = *(volatile ll_t *)&sequence[DOK_SEQ_NEXT];
  __syncthreads();
  const bool over = next + n > DOK_WORD_ROWS;
  if (over) dok_clear_numbers(t);
  __syncthreads();
  if (threadIdx.x != 0) return;
  __threadfence();
  if (atomicAdd((ull_t *)&sequence[DOK_SEQ_TICKET], 1ULL) != gridDim.x - 1) return;
  sequence[DOK_SEQ_BASE] = over ? 0 : next;                  // the last block: all have read
  sequence[DOK_SEQ_NEXT] = (over ? 0 : next) + n;
  sequence[DOK_SEQ_TICKET] = 0;
}

__device__ __forceinline__ ulonglong2 dok_cas_pair(char *slot, ulonglong2 expect, ulonglong2 desired) {
  ulonglong2 old;
  asm volatile("{\n\t.reg .b128 e, d, o;\n\tmov.b128 e, {%3, %4};\n\tmov.b128 d, {%5, %6};\n\t"
               "atom.relaxed.gpu.global.cas.b128 o, [%2], e, d;\n\tmov.b128 {%0, %1}, o;\n\t}"
               : "=l"(old.x), "=l"(old.y) : "l"(slot), "l"(expect.x), "l"(expect.y), "l"(desired.x), "l"(desired.y) : "memory");
  return old;
}

struct WordSlot { ll_t slot; int outcome; ull_t word; };     // word: of a slot that was found

// Insert-or-find by one lane, slot by slot, for the lane that has lost its CAS.  Phase 1 walks the chain: a matching tag is a
// hit; at the first empty tag the slot is claimed unless a tombstone was seen.  Phase 2 walks it again and takes the first
// slot that is free.  (Another walk of the whole warp, as in dok_find_or_claim, is a loop around it that the registers of
// k_set_word do not allow: constructor of 10 M rows 777 -> 903 us, 4 M-pair assignment 230 -> 251.)
static __device__ __forceinline__ WordSlot dok_claim_word_serial(const DevTable &t, const ChainKey &key, ull_t word) {
  bool reuse = false;                                        // a tombstone was seen
  for (int phase = 0; phase < 2; phase++) {
    ll_t group = dok_start_group(key, t);
    unsigned chain = key.word;
    bool more = true;
    while (more) {
      for (int i = 0; i < t.spg && more; i++) {
        const ll_t slot = group * t.spg + i;
        ulonglong2 now = dok_load_pair(dok_slot_ptr(t, slot));
        if ((ll_t)now.x == DOK_REMOVED && phase == 0) reuse = true;
        if ((ll_t)now.x == DOK_EMPTY && phase == 0 && reuse) { more = false; break; }
        if ((ll_t)now.x == DOK_EMPTY || ((ll_t)now.x == DOK_REMOVED && phase == 1)) {
          const ulonglong2 old = dok_cas_pair(dok_slot_ptr(t, slot), now, make_ulonglong2((ull_t)key.uuid, word));
          if (old.x == now.x) return WordSlot{slot, (ll_t)now.x == DOK_EMPTY ? DOK_OUT_CLAIMED_EMPTY : DOK_OUT_REUSED, 0};
          now = old;                                         // (the word of a free slot does not change while a set runs)
        }
        if ((ll_t)now.x == key.uuid) return WordSlot{slot, DOK_OUT_FOUND, now.y};
      }
      more = more && dok_next_group<ll_t>(group, chain, t.n_groups);
    }
    if (!reuse) break;
  }
  return WordSlot{-1, DOK_OUT_FAILED, 0};
}

// dok_find_or_claim with words.  Every lane of the warp must call.
template <bool FEW>
__device__ __forceinline__ WordSlot dok_find_or_claim_word(const DevTable &t, const KeyHash &kh, bool active, ull_t word) {
  const ChainKey key = dok_chain(kh, t);
  const Located loc = dok_locate_quad<32, 2, true>(t, key, 0, active, nullptr, NeedsWord<FEW>());
  if (!active) return WordSlot{-1, -1, 0};
  if (loc.found >= 0) return WordSlot{loc.found, DOK_OUT_FOUND, loc.word};
  const bool reuse = loc.tomb >= 0;
  const ll_t slot = reuse ? loc.tomb : loc.empty;
  if (slot < 0) return WordSlot{-1, DOK_OUT_FAILED, 0};
  char *at = dok_slot_ptr(t, slot);
  ulonglong2 free = make_ulonglong2((ull_t)DOK_EMPTY, loc.word);
  if (reuse) free = dok_load_pair(at);
  if ((ll_t)free.x == DOK_EMPTY || (ll_t)free.x == DOK_REMOVED) {
    const ulonglong2 old = dok_cas_pair(at, free, make_ulonglong2((ull_t)key.uuid, word));
    if (old.x == free.x) return WordSlot{slot, reuse ? DOK_OUT_REUSED : DOK_OUT_CLAIMED_EMPTY, 0};
    free = old;
  }
  if ((ll_t)free.x == key.uuid) return WordSlot{slot, DOK_OUT_FOUND, free.y};
  return dok_claim_word_serial(t, key, word);
}

__device__ __forceinline__ ull_t dok_narrow_value(const char *src, int vb) {
  if (vb == 4) return *(const unsigned *)src;
  if (vb == 2) return *(const unsigned short *)src;
  ull_t v = 0;
  for (int b = 0; b < vb; b++) v |= (ull_t)(unsigned char)src[b] << (8 * b);
  return v;
}

// What became of a row that goes to the table.
struct WordOutcome {
  bool claimed, met;       // met: another row of this batch was there before,
  ull_t fresh;             // ... and this batch claimed the slot
};
template <class Keys>
__device__ __forceinline__ WordOutcome dok_write_word(const DevTable &t, const DevHash &hp, const Keys &keys, ll_t e, const WordSlot &found,
                                                      ll_t base, ull_t word) {
  WordOutcome o;
  const ull_t before = found.word >> DOK_WORD_SHIFT;
  o.claimed = found.outcome == DOK_OUT_CLAIMED_EMPTY || found.outcome == DOK_OUT_REUSED;
  o.met = found.outcome == DOK_OUT_FOUND && before > (ull_t)base;
  o.fresh = o.met ? found.word & DOK_WORD_FRESH : 0;
  if (o.claimed) keys.store_key(t, hp, e, dok_slot_ptr(t, found.slot));
  if (found.outcome == DOK_OUT_FOUND && before < word >> DOK_WORD_SHIFT) atomicMax((ull_t *)dok_value_ptr(t, found.slot), word | o.fresh);
  return o;
}

template <bool FEW, class Keys, class Values>
__global__ void __launch_bounds__(DOK_TPB, 6) k_set_word(DevTable t, DevHash hp, Keys keys, Values values, const ll_t *sequence,
                                                         ll_t *counters, ll_t *more) {
  __shared__ BlockTally tally;
  __shared__ BlockTwins twins;
  const unsigned block = gridDim.x - 1 - blockIdx.x;         // from the end of the batch: a popular key's last rows first
  dok_tally_begin(tally);
  const ll_t base = sequence[DOK_SEQ_BASE];
  ll_t e;
  bool active = keys.row(e, block);
  KeyHash kh{0, 0};
  ull_t value = 0;
  if (active) {
    kh = keys.hash(hp, e);
    value = dok_narrow_value(values.row(t, e), t.vb);
  }
  active = dok_in_window(t, kh, active);
  bool any_twins;
  const Twins same = dok_find_twins(twins, kh, active, any_twins);
  const bool last = active && same.last == (int)threadIdx.x;
  const ull_t word = (ull_t)(base + e + 1) << DOK_WORD_SHIFT | value;
  const WordSlot found = dok_find_or_claim_word<FEW>(t, kh, last, word | DOK_WORD_FRESH);
  const WordOutcome o = dok_write_word(t, hp, keys, e, found, base, word);
  int failed = found.outcome == DOK_OUT_FAILED, again = failed || o.fresh != 0, twin = active && !last;
  if (any_twins) {                                           // uniform over the block
    if (last) twins.slot[threadIdx.x] = failed ? 2 : o.claimed || o.fresh;
    __syncthreads();
    if (twin) {
      const ll_t how = twins.slot[same.last];
      failed = how == 2;
      again = how != 0;
    }
  }
  dok_tally_add(tally, DOK_TALLY_EXTRA, again);
  if (counters) {
    dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, found.outcome == DOK_OUT_CLAIMED_EMPTY);
    dok_tally_add(tally, DOK_CNT_REUSED_REMOVED, found.outcome == DOK_OUT_REUSED);
    dok_tally_add(tally, DOK_CNT_FAILED, failed);
    dok_tally_add(tally, DOK_CNT_HITS, (twin && !failed) || found.outcome == DOK_OUT_FOUND);
    dok_tally_add(tally, DOK_CNT_DUPLICATES, twin || o.met);
  }
  dok_tally_flush(tally, counters, more);
}

// The same for a batch that one cluster holds (k_set_small), in one launch: the blocks read the next number together, and the
// first one moves it on when all have.
template <class Keys, class Values>
__global__ void __launch_bounds__(DOK_SMALL_SET_TPB) k_set_word_small(DevTable t, DevHash hp, Keys keys, Values values, ll_t *sequence,
                                                                      ll_t *counters, ll_t *more) {
  __shared__ BlockTally tally;
  dok_tally_begin(tally);
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  ll_t base = *(volatile ll_t *)&sequence[DOK_SEQ_NEXT];
  const bool over = base + keys.count() > DOK_WORD_ROWS;     // uniform over the launch
  if (over) {
    base = 0;
    dok_clear_numbers(t);
    cluster.sync();
  }
  const ll_t e = (ll_t)blockIdx.x * DOK_SMALL_SET_TPB + threadIdx.x;
  const bool active = e < keys.count();
  KeyHash kh{0, 0};
  ull_t value = 0;
  if (active) {
    kh = keys.hash(hp, e);
    value = dok_narrow_value(values.row(t, e), t.vb);
  }
  const ull_t word = (ull_t)(base + e + 1) << DOK_WORD_SHIFT | value;
  const WordSlot found = dok_find_or_claim_word<true>(t, kh, active, word | DOK_WORD_FRESH);
  const WordOutcome o = dok_write_word(t, hp, keys, e, found, base, word);
  const int failed = found.outcome == DOK_OUT_FAILED;
  dok_tally_add(tally, DOK_TALLY_EXTRA, failed || o.fresh != 0);
  if (counters) {
    dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, found.outcome == DOK_OUT_CLAIMED_EMPTY);
    dok_tally_add(tally, DOK_CNT_REUSED_REMOVED, found.outcome == DOK_OUT_REUSED);
    dok_tally_add(tally, DOK_CNT_FAILED, failed);
    dok_tally_add(tally, DOK_CNT_HITS, found.outcome == DOK_OUT_FOUND);
    dok_tally_add(tally, DOK_CNT_DUPLICATES, o.met);
  }
  dok_tally_flush(tally, counters, more);
  cluster.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) sequence[DOK_SEQ_NEXT] = base + keys.count();
}

template <class Keys, class Values>
inline int launch_set_word(const DevTable &t, const DevHash &hp, const Keys &keys, const Values &values, int64_t *sequence, int64_t *counters,
                           int64_t *more, cudaStream_t st) {
  if (dok_set_is_small(t, keys.n))
    return dok_launch_cluster(keys.n, st, k_set_word_small<Keys, Values>, t, hp, keys, values, (ll_t *)sequence, (ll_t *)counters, (ll_t *)more);
  k_word_begin<<<148, DOK_TPB, 0, st>>>(t, (ll_t *)sequence, keys.n);
  int rc = dok_check_launch();
  if (rc != DOK_OK) return rc;
  const dim3 grid = dok_grid(keys);
  DOK_BY_SIZE(grid.x, DOK_FOR_WINDOWS(t, rc, (k_set_word<FEW><<<grid, DOK_TPB, 0, st>>>(wt, hp, keys, values, (const ll_t *)sequence,
                                                                                     (ll_t *)counters, (ll_t *)more))));
  return rc;
}
