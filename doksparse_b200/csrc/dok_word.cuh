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
// Numbers go on from set to set.  The host hands them out (`base` of a launch), so that sets on several streams have ranges of
// their own and whatever is ordered after a set has larger ones; k_word_clear makes a new start when they have run out at
// 2^31 rows.  A set in a graph, whose base would be old when it is replayed, first takes the numbers of the slots that it will
// write away (k_word_release: another walk) and has base 0.
//
// 4 M-pair assignment to a 2-D tensor: 393 + 56 + 25 us of k_set_claim, k_set_resolve, k_set_count; here 219.  8.4 M rows of
// 4-byte values in a table of 2^26 keys, a fifth of them new: 688 -> 564; 800 k Zipf ids 97 -> 52.
#pragma once

// row's number (31 bits) | this batch claimed the slot | value (32 bits)
#define DOK_WORD_FRESH (1ULL << 32)
#define DOK_WORD_SHIFT 33

inline bool dok_values_in_word(const DevTable &t) { return t.sb == 32 && t.vb <= 4; }
inline bool dok_set_in_word(const DevTable &t, const DevHash &hp, ll_t n) {
  return dok_values_in_word(t) && hp.dtype < DOK_F16 && n > 0 && n <= DOK_MAX_NUMBER;
}
inline bool dok_numbers_fit(ll_t base, ll_t n) { return base == DOK_RENUMBER || (base >= 0 && base <= DOK_MAX_NUMBER - n); }

__device__ __forceinline__ unsigned *dok_number_ptr(const DevTable &t, ll_t slot) { return (unsigned *)(dok_value_ptr(t, slot) + 4); }

static __global__ void __launch_bounds__(DOK_TPB) k_word_clear(DevTable t) {
  for (ll_t i = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; i < t.n_slots; i += (ll_t)gridDim.x * DOK_TPB) *dok_number_ptr(t, i) = 0;
}

// The numbers of the slots that hold the batch's keys.
template <bool FEW, class Keys>
__global__ void __launch_bounds__(DOK_TPB) k_word_release(DevTable t, DevHash hp, Keys keys) {
  ll_t e;
  bool active = keys.row(e);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  const Located loc = dok_locate<32, 1, false>(t, kh, e, active, nullptr, NoEmit<FEW>());
  if (active && loc.found >= 0) *dok_number_ptr(t, loc.found) = 0;
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
          if (old.x == now.x && old.y == now.y) return WordSlot{slot, (ll_t)now.x == DOK_EMPTY ? DOK_OUT_CLAIMED_EMPTY : DOK_OUT_REUSED, 0};
          now = old;               // (the word of a free slot stays as it is while sets and removals of one key are in order)
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
    if (old.x == free.x && old.y == free.y) return WordSlot{slot, reuse ? DOK_OUT_REUSED : DOK_OUT_CLAIMED_EMPTY, 0};
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
  if (found.outcome == DOK_OUT_FOUND && before < word >> DOK_WORD_SHIFT)
    o.met |= atomicMax((ull_t *)dok_value_ptr(t, found.slot), word | o.fresh) >> DOK_WORD_SHIFT > (ull_t)base;
  return o;
}

template <bool FEW, class Keys, class Values>
__global__ void __launch_bounds__(DOK_TPB, 6) k_set_word(DevTable t, DevHash hp, Keys keys, Values values, ll_t base, ll_t *counters,
                                                         ll_t *more) {
  __shared__ BlockTally tally;
  __shared__ BlockTwins twins;
  const unsigned block = gridDim.x - 1 - blockIdx.x;         // from the end of the batch: a popular key's last rows first
  dok_tally_begin(tally);
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

// The same for a batch of few rows (k_set_small), which has no popular keys to look for.
template <class Keys, class Values>
__global__ void __launch_bounds__(DOK_TPB, 4) k_set_word_small(DevTable t, DevHash hp, Keys keys, Values values, ll_t base, ll_t *counters,
                                                            ll_t *more) {
  __shared__ BlockTally tally;
  dok_tally_begin(tally);
  ll_t e;
  const bool active = keys.row(e);
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
}

template <class Keys, class Values>
inline int launch_set_word(const DevTable &t, const DevHash &hp, const Keys &keys, const Values &values, int64_t base, int64_t *counters,
                           int64_t *more, cudaStream_t st) {
  const dim3 grid = dok_grid(keys);
  int rc = DOK_OK;
  if (base == DOK_RENUMBER) {
    base = 0;
    DOK_BY_SIZE(grid.x, DOK_FOR_WINDOWS(t, rc, (k_word_release<FEW><<<grid, DOK_TPB, 0, st>>>(wt, hp, keys))));
    if (rc != DOK_OK) return rc;
  }
  if (dok_set_is_small(t, keys.n)) {
    k_set_word_small<<<grid, DOK_TPB, 0, st>>>(t, hp, keys, values, (ll_t)base, (ll_t *)counters, (ll_t *)more);
    return dok_check_launch();
  }
  DOK_BY_SIZE(grid.x, DOK_FOR_WINDOWS(t, rc, (k_set_word<FEW><<<grid, DOK_TPB, 0, st>>>(wt, hp, keys, values, (ll_t)base, (ll_t *)counters,
                                                                                     (ll_t *)more))));
  return rc;
}
