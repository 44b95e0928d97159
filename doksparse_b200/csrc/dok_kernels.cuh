// Kernel templates of the closed-hashing map: batched get / set / remove / exists / count-new and the
// compaction of live slots.  They are templated on the slot width SB (32, 64, 128 bytes: quad-cooperative walk,
// one 128-byte group per request; 0: slots wider than a line, serial walk) and on the key source (contiguous key
// rows, or the index tensors of a DOK selector), so that the map entry points (map_api.cu) and the fused DOK
// entry points (dok_api.cu) share them.  One CUDA thread owns one batch element, as in the reference kernels
// (sparse_dok/components/cuda/closed_hashmap_impl.cu); misses write the fallback from the kernel, and counters
// are accumulated on the device so that the host never has to synchronise.
//
// No thread of a warp returns early: the cooperative walk needs all 32 lanes.
#pragma once
#include <cooperative_groups.h>
#include <type_traits>
#include "dok_stream.cuh"

// ---------------------------------------------------------------------------------------------------------
// get
// ---------------------------------------------------------------------------------------------------------
// One row per thread: for 32-byte slots with values of at most 8 bytes, whose walk fits 32 registers, so that 64 warps are
// resident (8.4 M lookups at load 0.6: 251 us; the form below, with half the instructions but 32 warps: 291), for slots wider
// than a line, and for batches that dok_get_by_rows names.
// For values of more than 8 bytes the walk reads the tags alone, so that 64 warps are resident here too, and the row's own
// lane reads the value where it was found -- from L1, as its sector has just come in, and further sectors of the line from
// L2, up to eight pieces at a time (one after the other: 33.5 M hits of 40-byte values in 8 GB 2294 -> 2050 us, of 28 bytes
// 2339 -> 2052, 1 M of a 128 MB table 53 -> 49).  Against whole lines in the registers of 24 warps: 40-byte values, 300 k lookups
// of a 128 MB table 31 -> 25 us, 8 M 367 -> 263; 16-byte values, 200 k 24 -> 18, 3000 15 -> 11.
// Lines through cp.async and shared memory, 40 warps: 445, 62 and 50 for 40-byte values, 292 for 16-byte ones, and 2053
// instead of 1800 for the churn's, whose popular lines are then not in L1.  Values read and stored by the quad as soon as their
// tag is found, when the line is in L1 for certain: 33.5 M hits 1852, but misses 1405 -> 1480 and 8 M of a 256 MB table 300 -> 343.
template <int SB, int LW, bool PASSED, bool FEW, class Keys>
__global__ void __launch_bounds__(DOK_TPB, SB == 0 ? 1 : SB != 32 && LW == 2 ? 6 : 8)
    k_get_row(DevTable t, DevHash hp, Keys keys, char *__restrict__ out_values, uint8_t *__restrict__ out_found, Fallback fb, ll_t *counters,
              int count_probes) {
  constexpr bool AGAIN = LW == 4;                          // the value is read when its slot is known
  __shared__ BlockTally tally;
  if (keys.idle()) return;
  if (counters) dok_tally_begin(tally);
  ll_t e;
  bool active = keys.row(e);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  int probes = 0;
  Located loc;
  if constexpr (AGAIN) loc = dok_locate<SB, 1, false>(t, kh, e, active, &probes, Probe<FEW>());
  // ... or on a hit the quad writes it from the registers that hold the line
  else loc = dok_locate<SB, LW, false>(t, kh, e, active, &probes, EmitValue<SB, LW, PASSED>{t, out_values});
  const int hit = active && loc.found >= 0;
  if (active) {
    char *dst = out_values + e * (ll_t)t.vb;
    if (AGAIN && hit) {
      if constexpr (SB == 0) dok_load_value(t, loc.found, dst);
      else dok_fetch_value(t, loc.found, dst);
    }
    if (!hit) dok_store_fallback(t, fb, dst);
  }
  if (active && out_found) out_found[e] = (uint8_t)hit;
  if (counters) {
    dok_tally_add(tally, DOK_CNT_HITS, hit);
    dok_tally_flush(tally, counters, nullptr);
    if (count_probes) dok_warp_add(counters + DOK_CNT_PROBES, probes);
  }
}

// A warp's share of the batch (dok_stream.cuh): for larger batches of everything else.  16-byte values need the registers of
// whole lines (3 blocks of 256 per SM in either form), and where a line holds fewer slots the chains are longer, so that a
// warp that waits for its longest chain leaves most of its lanes idle: 8.4 M lookups of 16-byte values 544 -> 303 us, 8.4 M
// misses in 64-byte slots at load 0.69 750 -> 595, selections of 32-byte slots 153 -> 141.
// Values of at most 8 bytes lie behind the tag in the word pair that a lane has loaded: the key's own lane fetches it from
// the lane of the slot that matched, and stores value (or fallback) and flag of its row -- one store for 32 rows of which
// most are neighbours.  16-byte values are written by the lane that holds the slot, others by the lanes of the quad.  Either way
// a hit needs no second access to the table.
template <int SB, int LW, bool PASSED, class Keys>
__global__ void __launch_bounds__(DOK_TPB, LW == 4 ? 3 : 4) k_get(DevTable t, DevHash hp, Keys keys, char *__restrict__ out_values,
                                                                  uint8_t *__restrict__ out_found, Fallback fb, ll_t *counters,
                                                                  int count_probes) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ WarpQueue queues[DOK_WARPS];
  int hits = 0, probes = 0;
  dok_walk_share<LW, true, PASSED>(queues[threadIdx.x >> 5], t, hp, keys, [&](LaneRow &lr, const Lines<LW> &f, const WarpShare &share) {
    const unsigned l = threadIdx.x & 3u, base = threadIdx.x & 28u;
    unsigned m, me, match[4], empty[4];
    ull_t value = 0;
    if constexpr (LW == 2) {
      if constexpr (SB == 32) {
        const unsigned bits = dok_inspect<SB, LW>(lr, f);
        m = dok_matches(bits, l); me = dok_ends(bits, l);
      } else {
        dok_inspect_votes<SB, LW, PASSED>(lr, f, m, me, match, empty);
      }
      const unsigned from = base + (me ? (unsigned)__ffs(me) - 1 : 0u);
#pragma unroll
      for (unsigned r = 0; r < 4; r++) {
        const ull_t v = __shfl_sync(FULL, f.w[r][1], from);
        if (l == r) value = v;
      }
    } else {
      dok_inspect_votes<SB, LW, false>(lr, f, m, me, match, empty);
      const EmitValue<SB, LW, false> emit{t, out_values};
      // 16-byte values: one store
      const bool pairs = t.vb == 16 && ((size_t)out_values & 15) == 0;
      if (pairs) {
#pragma unroll
        for (unsigned r = 0; r < 4; r++) {
          const unsigned row_r = __shfl_sync(FULL, lr.row, base + r);
          const unsigned me_r = ((match[r] | empty[r]) >> base) & 0xfu;
          if ((unsigned)__ffs(me_r) == l + 1 && ((match[r] >> (base + l)) & 1u))
            *(ulonglong2 *)(out_values + keys.elem(share.first + row_r) * 16) = make_ulonglong2(f.w[r][1], f.w[r][2]);
        }
      } else
#pragma unroll
      for (unsigned r = 0; r < 4; r++) {
        const unsigned row_r = __shfl_sync(FULL, lr.row, base + r);
        const unsigned m_r = (match[r] >> base) & 0xfu, me_r = m_r | ((empty[r] >> base) & 0xfu);
        if (me_r) {
          const int lane = __ffs(me_r) - 1;
          if ((m_r >> lane) & 1u) emit(keys.elem(share.first + row_r), lane * 32 / SB, f.w[r]);
        }
      }
    }
    if (!lr.busy()) return;
    const bool hit = me && ((m >> (__ffs(me) - 1)) & 1u);
    probes++;
    if (me || !dok_next_group<unsigned>(lr.group, lr.word, (unsigned)t.n_groups)) {
      const ll_t e = keys.elem(share.first + lr.row);
      char *dst = out_values + e * (ll_t)t.vb;
      if constexpr (LW == 2) {
        if (!hit) value = fb.w[0];
        if (t.vb == 8) *(ull_t *)dst = value;
        else if (t.vb == 4) *(unsigned *)dst = (unsigned)value;
        else dok_store_word(dst, value, t.vb, t.vb & -t.vb);
      } else {
        if (!hit) dok_store_fallback(t, fb, dst);
      }
      if (out_found) out_found[e] = (uint8_t)hit;
      hits += hit;
      lr.done();
    }
  });
  if (counters) {
    dok_warp_add(counters + DOK_CNT_HITS, hits);
    if (count_probes) dok_warp_add(counters + DOK_CNT_PROBES, probes);
  }
}

// Kernels whose walk has a form for few rows (dok_locate_quad): up to four blocks per SM.
#define DOK_FEW_BLOCKS (148 * 4)
#define DOK_BY_SIZE(blocks, CALL)                                    \
  if ((blocks) <= DOK_FEW_BLOCKS) { constexpr bool FEW = true; CALL; } \
  else { constexpr bool FEW = false; CALL; }

#define DOK_DISPATCH_SB(t, CALL)                        \
  switch ((t).sb) {                                     \
    case 32: { constexpr int SB = 32; CALL; break; }    \
    case 64: { constexpr int SB = 64; CALL; break; }    \
    case 128: { constexpr int SB = 128; CALL; break; }  \
    default: { constexpr int SB = 0; CALL; break; }     \
  }

// ... with MARKS (dok_find_or_claim): a walk that looks for them takes 2 % longer
#define DOK_DISPATCH_MARKS(t, CALL)                                                            \
  if (dok_has_passed_bits(t)) DOK_DISPATCH_SB(t, { constexpr bool MARKS = SB >= 64; CALL; })   \
  else DOK_DISPATCH_SB(t, { constexpr bool MARKS = false; CALL; })

// launch grid of a batch: one thread per row; sliced batches put the slice in gridDim.y
inline dim3 dok_grid(const RowKeys &k) {
  if (k.slice_rows == 0) return dim3((unsigned)((k.n + DOK_TPB - 1) / DOK_TPB));
  return dim3((unsigned)((k.slice_rows + DOK_TPB - 1) / DOK_TPB), (unsigned)(k.n / k.slice_rows));
}
inline dim3 dok_grid(const SelKeys &k) { return dim3((unsigned)((k.n + DOK_TPB - 1) / DOK_TPB)); }

// The same for the kernels whose warps share the batch out (dok_stream.cuh): one wave of the blocks that fit, fewer when
// the batch has no row for each of their threads.
template <auto KERNEL, class Keys>
inline dim3 dok_stream_grid(const Keys &keys) {
  static const int per_sm = [] {
    int blocks = 0;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, KERNEL, DOK_TPB, 0) == cudaSuccess && blocks > 0 ? blocks : 4;
  }();
  dim3 grid = dok_grid(keys);
  const unsigned wave = 148u * per_sm, most = grid.y >= wave ? 1u : wave / grid.y;
  if (grid.x > most) grid.x = most;
  return grid;
}

// kernel, then its arguments behind the table; once per window
#define DOK_STREAM(t, rc, st, keys, KERNEL, ...) \
  DOK_FOR_WINDOWS(t, rc, (KERNEL<<<dok_stream_grid<KERNEL>(keys), DOK_TPB, 0, st>>>(wt, __VA_ARGS__)))

// Which batches of key rows go to k_get_row.  Values of at most 8 bytes in 64- and 128-byte slots: with less than two rows for
// each lane of k_get there are too few chains for a lane to take up when its own ends.  k_get / k_get_row, us, 4-byte values in
// 64-byte slots, table of 2^21 slots at load 0.6, all / none of them stored: 64 rows 7.2/6.9 6.9/6.4, 1000 10.2/9.1 8.4/7.8,
// 8000 11.9/9.8 10.8/8.6, 37 k 13.4/11.2 11.5/9.8 (at 0.85 29.4/22.1 29.1/23.5); of 2^22 slots at load 0.8 500 k 47/47 45/46,
// 1 M 62/74 63/75, 4 M 166/240 176/247.
// Wider values: k_get_row looks at the slot a second time, which costs nothing where the batch is all latency or address
// translation covers the table.  In larger tables a batch of hits pays for it, but one with misses has more from the 64 warps
// that walk.  k_get / k_get_row, us, 8 M rows, all / half / none of them stored:
//                                   load 0.5                     load 0.8
//   12 bytes, 32-byte slots  1 GB   305/287 343/254 285/236      359/340 504/424 512/487
//                            4 GB   315/320 347/276 303/250      371/377 514/446 567/510
//   16 bytes, 32-byte slots 256 MB  227/170 258/192 252/192      267/234 373/360 427/428
//                            1 GB   254/305 281/258 281/236      303/350 426/420 508/486
//   28 bytes, 64-byte slots  2 GB   469/473 528/371 430/346      573/563 819/666 815/792
//   40 bytes, 64-byte slots 512 MB  390/371 446/316 421/326      471/446 678/625 752/756
//                            2 GB   399/472 453/358 437/349      488/564 708/664 820/803
//   64 bytes, 128-byte slots 256 MB 430/526 527/504 543/494      565/653 899/944 1034/1149
//                            4 GB   455/727 553/553 569/549      616/862 1002/1061 1295/1305
// Values that a lane of k_get stores at once (16 bytes of a 32-byte slot) and those that fill three sectors of their line have
// less from k_get_row; at 300 k rows these take 41/37 49/39 48/43 and 76/62 125/82 121/85, at 1 M 82/110 98/96 106/96 and
// 139/143 234/191 258/224 in 4 GB.  Selections of a tensor, whose index arithmetic a share does for 32 rows at a time, differ by
// a tenth either way and stay with k_get in 32-byte slots.
inline bool dok_get_by_rows(const DevTable &t, ll_t n) {
  if (t.vb <= 8) return n < 148LL * DOK_TPB * 4 * 2;
  if (t.vb > 56) return n < 1000000;
  return t.sb > 32 || t.vb < 16 || n < 900000 || t.n_slots * t.sb <= 256LL << 20;
}

template <class Keys>
inline int launch_get(const DevTable &t, const DevHash &hp, const Keys &keys, void *out_values, uint8_t *out_found,
                      const void *fallback, int64_t *counters, int count_probes, cudaStream_t st) {
  const ll_t n = keys.n;
  if (n == 0) return DOK_OK;
  Fallback fb;
  memset(&fb, 0, sizeof(fb));
  if (fallback) memcpy(&fb, fallback, (size_t)t.vb);
  int rc = DOK_OK;
  char *values = (char *)out_values;
  ll_t *cnt = (ll_t *)counters;
  // tag and value fit the first 16 bytes of the slot: half the load width
  const bool narrow = t.vb <= 8;
  const dim3 grid = dok_grid(keys);
  const auto launch = [&](auto slot_bytes, auto words, auto passed) {
    constexpr int SB = decltype(slot_bytes)::value, LW = decltype(words)::value;
    constexpr bool PASSED = decltype(passed)::value, ROWS = std::is_same<Keys, RowKeys>::value;
    constexpr bool ONLY_ROWS = SB == 0 || (LW == 4 && (SB == 64 || (SB == 128 && !ROWS))) || (ROWS && SB == 32 && LW == 2);
    if constexpr (ROWS || ONLY_ROWS)
      if (ONLY_ROWS || dok_get_by_rows(t, n)) {
        DOK_BY_SIZE(grid.x * grid.y, DOK_FOR_WINDOWS(t, rc, (k_get_row<SB, LW, PASSED, FEW && LW == 4 && SB != 0, Keys>
                                                             <<<grid, DOK_TPB, 0, st>>>(wt, hp, keys, values, out_found, fb, cnt, count_probes))));
        return;
      }
    if constexpr (!ONLY_ROWS) DOK_STREAM(t, rc, st, keys, (k_get<SB, LW, PASSED, Keys>), hp, keys, values, out_found, fb, cnt, count_probes);
  };
  const auto by_width = [&](auto slot_bytes) {
    if constexpr (decltype(slot_bytes)::value != 32)         // (four slots per group have no marks)
      if (dok_has_passed_bits(t)) return launch(slot_bytes, std::integral_constant<int, 2>(), std::true_type());
    if (narrow) launch(slot_bytes, std::integral_constant<int, 2>(), std::false_type());
    else launch(slot_bytes, std::integral_constant<int, 4>(), std::false_type());
  };
  switch (t.sb) {
    case 32: by_width(std::integral_constant<int, 32>()); break;
    case 64: by_width(std::integral_constant<int, 64>()); break;
    case 128: by_width(std::integral_constant<int, 128>()); break;
    default: launch(std::integral_constant<int, 0>(), std::integral_constant<int, 4>(), std::false_type());
  }
  return rc;
}

// ---------------------------------------------------------------------------------------------------------
// set
// ---------------------------------------------------------------------------------------------------------

// Value row of batch element e into its slot, and the key row too when this row claimed the slot.  A row that
// found its uuid already stored leaves the stored key alone: the reference rewrites it
// (closed_hashmap_impl_class.cu:384-386), but with the same bytes unless two different keys share a uuid, and every
// store to the table costs a request.  Floating-point keys are the exception -- their value cast makes different
// keys share a uuid as a rule -- so they are rewritten like in the reference.
template <class Keys, class Values>
__device__ __forceinline__ void dok_write_row(const DevTable &t, const DevHash &hp, const Keys &keys, const Values &values,
                                              ll_t e, ll_t slot, bool with_key) {
  if (with_key) keys.store_key(t, hp, e, dok_slot_ptr(t, slot));
  dok_store_value(t, slot, values.row(t, e));
}

// One kernel, for batches whose rows have pairwise different uuids.
template <int SB, bool MARKS, class Keys, class Values>
__global__ void __launch_bounds__(DOK_TPB, 6) k_set_unique(DevTable t, DevHash hp, Keys keys, Values values,
                                                        uint8_t *__restrict__ out_stored, ll_t *counters) {
  __shared__ BlockTally tally;
  if (keys.idle()) return;
  if (counters) dok_tally_begin(tally);
  ll_t e;
  bool active = keys.row(e);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  int outcome = -1;
  const ll_t slot = dok_find_or_claim<SB, false, MARKS>(t, kh, active, &outcome);
  if (active) {
    if (slot >= 0) dok_write_row(t, hp, keys, values, e, slot, outcome != DOK_OUT_FOUND || hp.dtype >= DOK_F16);
    if (out_stored) out_stored[e] = (uint8_t)(slot >= 0);
  }
  if (counters) {
    dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, outcome == DOK_OUT_CLAIMED_EMPTY);
    dok_tally_add(tally, DOK_CNT_REUSED_REMOVED, outcome == DOK_OUT_REUSED);
    dok_tally_add(tally, DOK_CNT_FAILED, outcome == DOK_OUT_FAILED);
    dok_tally_add(tally, DOK_CNT_HITS, outcome == DOK_OUT_FOUND);
    dok_tally_flush(tally, counters, nullptr);
  }
}

// Stamp word of a slot during a general set: (epoch << 34) | (row << 2) | fresh << 1 | conflict, unsigned.  The epoch of
// a call is larger than every epoch used on the table before, so an atomicMax leaves the LAST row of this batch that
// targets the slot; the lowest bit records that more than one row of the batch did, the next one (k_set_count only) that
// such a slot was claimed by this batch.
#define DOK_STAMP_CONFLICT 1ULL
#define DOK_STAMP_FRESH 2ULL
// Filter of the slots with a conflict (by 22 bits of a product of the slot index, so a set bit may be another slot's): a
// batch of millions of rows with some repetitions would otherwise read a stamp at random for every row in the second and
// third kernel, 151 us of a 4 M-row assignment; 512 KB that stay in L2 answer for most rows.
#define DOK_FILTER_BITS 22
#define DOK_FILTER_WORDS (1 << (DOK_FILTER_BITS - 6))                       // int64 words behind slot_out[n]
// One block in 16 adds up its rows whose slot another block has stamped, for the blocks that come later; a line of its own,
// and a sample, because every block reads it (all of them adding to a word that all of them read: a 4 M-row assignment
// 488 -> 700 us).
#define DOK_FILTER_SIGNAL (2 * DOK_FILTER_WORDS + 32)                       // unsigned words behind the filter's start
#define DOK_SIGNAL_SAMPLE 16
__device__ __forceinline__ unsigned *dok_signal(unsigned *filter) {         // 16-byte aligned
  return (unsigned *)(((uintptr_t)(filter + DOK_FILTER_SIGNAL) + 15) & ~(uintptr_t)15);
}
#define DOK_FILTER_ALL (DOK_FILTER_WORDS + 32)                              // int64 words, all zeroed
#define DOK_FILTER_FROM 65536                                               // rows; below, clearing it costs more
__device__ __forceinline__ unsigned dok_filter_bit(ll_t slot) { return ((unsigned)slot * 0x9e3779b1u) >> (32 - DOK_FILTER_BITS); }
__device__ __forceinline__ void dok_filter_set(unsigned *filter, ll_t slot) {
  const unsigned b = dok_filter_bit(slot);
  if (filter) atomicOr(filter + (b >> 5), 1u << (b & 31u));
}
__device__ __forceinline__ bool dok_filter_has(const unsigned *filter, ll_t slot) {
  const unsigned b = dok_filter_bit(slot);
  return !filter || ((__ldcg(filter + (b >> 5)) >> (b & 31u)) & 1u);
}
#define DOK_ROW_FRESH (1LL << 62)      // bit of a row's slot index: this row claimed the slot
__device__ __forceinline__ ull_t dok_stamp(ll_t epoch, ll_t row) { return ((ull_t)epoch << 34) | ((ull_t)row << 2); }

// The rows of a block that hold the same key, found in shared memory before the table is touched: only the last of them,
// which is the one whose value stays, goes on.  In a Zipf batch the most popular key is 4 % of the rows, and every one of
// them read, stored and stamped the same line, which the L2 serves one after the other: 12.8 M such rows took 20 ms.
// Same key: same uuid and same chain, so that the rows would have met in one slot.  The set is keyed by the chain's hash;
// rows that share it by chance have different uuids and go on by themselves.
#define DOK_TWIN_SLOTS (2 * DOK_TPB)
struct BlockTwins {
  ll_t chain[DOK_TWIN_SLOTS];              // 55 bits of the chain's hash | 8 bits: thread of the key's last row so far
  ll_t uuid[DOK_TPB], slot[DOK_TPB];       // by thread; inactive rows have no uuid
  uint8_t more[DOK_TPB * 2];               // by place: more than one row
  uint4 signal;                            // see dok_signal
};
struct Twins { int last; bool more; };     // thread of the key's last row; whether there are others

// every thread of the block must call; any: the block has such rows
__device__ __forceinline__ Twins dok_find_twins(BlockTwins &b, const KeyHash &kh, bool active, bool &any) {
#pragma unroll
  for (int i = threadIdx.x; i < DOK_TWIN_SLOTS; i += DOK_TPB) { b.chain[i] = DOK_EMPTY; b.more[i] = 0; }
  b.uuid[threadIdx.x] = active ? kh.uuid : DOK_EMPTY;
  __syncthreads();
  int at = 0;
  bool met = false;
  if (active) {
    const ll_t mine = ((ll_t)dok_chain_hash(kh) & 0x7fffffffffffff00LL) | threadIdx.x;
    at = (int)(mine >> 8) & (DOK_TWIN_SLOTS - 1);
    for (;;) {                             // at most DOK_TPB of the DOK_TWIN_SLOTS places are ever taken
      const ll_t old = (ll_t)atomicCAS((ull_t *)&b.chain[at], (ull_t)DOK_EMPTY, (ull_t)mine);
      if (old == DOK_EMPTY) break;
      if (((old ^ mine) >> 8) == 0) {
        atomicMax(&b.chain[at], mine);
        b.more[at] = 1;
        met = true;
        break;
      }
      at = (at + 1) & (DOK_TWIN_SLOTS - 1);
    }
  }
  asm volatile("cp.async.wait_all;" ::: "memory");              // (k_set_claim: the signal)
  any = __syncthreads_or(met);
  Twins w{(int)threadIdx.x, false};
  if (active) {
    const int last = (int)(b.chain[at] & 255);
    if (b.uuid[last] == kh.uuid) w.last = last;
    w.more = b.more[at] != 0;
  }
  return w;
}

// First kernel of the general set.  Find or claim the slot, store the row there and raise the slot's stamp --
// for a batch without equal uuids that is all there is to do.  A row that finds the slot already stamped in
// this epoch sets the conflict bit and counts a duplicate (in slot_out[n], zeroed by the host before the
// launch); the second kernel then lets the slot's last row rewrite it.
template <int SB, bool FEW, bool MARKS, class Keys, class Values>
__global__ void __launch_bounds__(DOK_TPB, FEW ? 4 : 6) k_set_claim(DevTable t, DevHash hp, Keys keys, Values values,
                                                       ll_t *__restrict__ slot_out, unsigned *filter, ll_t epoch, int mark_fresh,
                                                       uint8_t *__restrict__ out_stored, ll_t *counters) {
  __shared__ BlockTally tally;
  __shared__ BlockTwins twins;
  // from the end of the batch to its beginning, see below
  const unsigned block = gridDim.x - 1 - blockIdx.x;
  if (keys.idle(block)) return;
  dok_tally_begin(tally);
  // on its way while the rows are hashed, and in no register
  if (filter && threadIdx.x == 0)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(&twins.signal)), "l"(dok_signal(filter)) : "memory");
  ll_t e;
  bool active = keys.row(e, block);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  bool any_twins;
  const Twins same = dok_find_twins(twins, kh, active, any_twins);
  const bool last = active && same.last == (int)threadIdx.x;
  int outcome = -1, conflict = 0, dup = 0;
  ll_t slot = dok_find_or_claim<SB, FEW, MARKS>(t, kh, last, &outcome);
  if (last) {
    const bool fresh = outcome == DOK_OUT_CLAIMED_EMPTY || outcome == DOK_OUT_REUSED;
    slot_out[e] = mark_fresh && fresh ? slot | DOK_ROW_FRESH : slot;
    if (slot >= 0) {
      // the row is stored without waiting for the stamp's answer: the two requests travel together.  If the slot
      // turns out to be shared, whatever the racing stores left is rewritten by the second kernel.
      ull_t *stamp = (ull_t *)dok_stamp_ptr(t, slot);
      // A key that the block holds several times is probably all over the batch.  If a later row has already stamped its
      // slot -- blocks start from the batch's end, so one has unless it is still running -- this row has nothing to write,
      // and a line that most of the blocks want is read, not written: writes to one line come 140 ns apart.  In a batch with
      // many repetitions (one row in 16 so far, by a sample) the same goes for the keys that a block holds once: one in a
      // thousand rows of a Zipf batch of 12.8 M is 12,800 writes to one line.  Elsewhere the look would cost every row a round
      // trip for nothing.
      const bool contended = filter && (ull_t)twins.signal.x * DOK_SIGNAL_SAMPLE * 16 > ((ull_t)blockIdx.y * gridDim.x + blockIdx.x) * DOK_TPB;
      ull_t old = (same.more || contended) && !fresh ? __ldcg(stamp) : 0;
      const bool over = old > (dok_stamp(epoch, e) | 3);
      dup = over;
      if (!over) {
        dok_write_row(t, hp, keys, values, e, slot, fresh || hp.dtype >= DOK_F16);
        old = atomicMax(stamp, dok_stamp(epoch, e));
      }
      if (over ? mark_fresh && !(old & DOK_STAMP_CONFLICT) : (old >> 34) == (ull_t)epoch || (mark_fresh && same.more)) {
        atomicOr(stamp, DOK_STAMP_CONFLICT);
        dok_filter_set(filter, slot);
        conflict = dup = 1;
      }
    } else {
      conflict = mark_fresh;          // a row without a place is counted by k_set_count too
    }
    if (out_stored) out_stored[e] = (uint8_t)(slot >= 0);
    if (slot < 0 && same.more && counters) {                        // a full table: its twins, counted as found below,
      ll_t others = -1;                                             // have no place either
      for (int i = 0; i < DOK_TPB; i++) others += twins.uuid[i] == kh.uuid;
      atomicAdd((ull_t *)counters + DOK_CNT_FAILED, (ull_t)others);
      atomicAdd((ull_t *)counters + DOK_CNT_HITS, (ull_t)-others);
    }
  }
  if (out_stored || mark_fresh) {                                   // uniform over the launch
    if (last) twins.slot[threadIdx.x] = slot;
    __syncthreads();
    if (active && !last) {
      slot = twins.slot[same.last];
      slot_out[e] = slot;
      if (out_stored) out_stored[e] = (uint8_t)(slot >= 0);
    }
  } else if (active && !last) {
    slot_out[e] = -1;                                               // nothing to rewrite: a later row of the block may
  }
  dok_tally_add(tally, DOK_TALLY_EXTRA, conflict);
  if (filter && blockIdx.x % DOK_SIGNAL_SAMPLE == 0) {            // uniform over the block
    const unsigned votes = __ballot_sync(0xffffffffu, dup);
    if ((threadIdx.x & 31) == 0 && votes) atomicAdd(dok_signal(filter), __popc(votes));
  }
  if (counters) {
    const bool twin = active && !last;
    dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, outcome == DOK_OUT_CLAIMED_EMPTY);
    dok_tally_add(tally, DOK_CNT_REUSED_REMOVED, outcome == DOK_OUT_REUSED);
    dok_tally_add(tally, DOK_CNT_FAILED, outcome == DOK_OUT_FAILED);
    dok_tally_add(tally, DOK_CNT_HITS, twin || outcome == DOK_OUT_FOUND);
    dok_tally_add(tally, DOK_CNT_DUPLICATES, twin || dup);
  }
  dok_tally_flush(tally, counters, slot_out + keys.count());
}

// Second kernel: does nothing unless the first one counted duplicates.  Then the row that owns a conflicted
// slot's stamp (the last row of the batch for that slot) rewrites key and value: one writer per slot, after
// every first-kernel write has completed, so rows cannot tear and the last row wins.
template <class Keys, class Values>
__global__ void __launch_bounds__(DOK_TPB) k_set_resolve(DevTable t, DevHash hp, Keys keys, Values values,
                                                         const ll_t *__restrict__ slot_in, const unsigned *filter, ll_t epoch) {
  if (slot_in[keys.count()] == 0) return;        // the first kernel met no duplicate: every row is already in place
  if (keys.idle()) return;
  // a few blocks per SM stride over the rows: the usual launch has nothing to do, and a grid of one block per 256
  // rows would cost a millisecond at 2^28 rows just to find that out
  const ll_t span = keys.span(), stride = (ll_t)gridDim.x * DOK_TPB;
  for (ll_t j = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; j < span; j += stride) {
    ll_t e;
    if (!keys.at(j, e)) continue;
    ll_t slot = slot_in[e];
    if (slot < 0) continue;
    const bool fresh = (slot & DOK_ROW_FRESH) != 0;
    slot &= ~DOK_ROW_FRESH;
    if (t.win_hi != 0) {                         // windowed passes: by the slot's own group (each slot has one pass)
      const ll_t g = slot / t.spg;
      if (g < t.win_lo || g >= t.win_hi) continue;
    }
    if (!dok_filter_has(filter, slot)) continue;
    const ull_t stamp = (ull_t)__ldcg(dok_stamp_ptr(t, slot));
    if (!(stamp & DOK_STAMP_CONFLICT)) continue;
    if (fresh) atomicOr((ull_t *)dok_stamp_ptr(t, slot), DOK_STAMP_FRESH);
    if ((stamp & ~DOK_STAMP_FRESH) != (dok_stamp(epoch, e) | DOK_STAMP_CONFLICT)) continue;
    dok_write_row(t, hp, keys, values, e, slot, true);
  }
}

// Third kernel, for callers that count like the reference's DOK assignment does (sparse_dok_tensor_impl.py:461-474): every
// row whose key was not stored before the batch, its repetitions too.  The claims are counted already; this adds the
// other rows of the slots that the batch claimed, and rows that found the table full.  Counting the stored keys in a pass
// of its own before the set, as the reference does, costs a walk per row: 145 of the 800 us of a 4 M-row assignment.
template <class Keys>
__global__ void __launch_bounds__(DOK_TPB) k_set_count(DevTable t, Keys keys, const ll_t *__restrict__ slot_in,
                                                       const unsigned *filter, ll_t epoch,
                                                       ll_t *__restrict__ more) {
  if (slot_in[keys.count()] == 0) return;
  const ll_t span = keys.span(), stride = (ll_t)gridDim.x * DOK_TPB;
  int c = 0;
  for (ll_t j = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; j < span; j += stride) {
    ll_t e;
    if (!keys.at(j, e)) continue;
    const ll_t slot = slot_in[e];
    if (slot < 0) { c++; continue; }
    if ((slot & DOK_ROW_FRESH) || !dok_filter_has(filter, slot)) continue;      // a slot with several rows has a conflict
    const ull_t stamp = (ull_t)__ldcg(dok_stamp_ptr(t, slot));
    c += (stamp >> 34) == (ull_t)epoch && (stamp & DOK_STAMP_FRESH) != 0;
  }
  dok_warp_add(more, c);
}

// The general set of a batch that one cluster holds, one row per thread: the three kernels above as three phases of one
// launch.  Such a batch is all latency: a set of 400 rows was a clearing of the scratch, two or three launches and an
// allocation, 16 us of which the table took 4.  The barrier is the cluster's (up to 8 blocks of 1024 threads), and slots
// stay in registers, so there is no scratch.
#define DOK_SMALL_SET_TPB 1024
#define DOK_SMALL_SET_ROWS (8 * DOK_SMALL_SET_TPB)

template <int SB, class Keys, class Values>
__global__ void __launch_bounds__(DOK_SMALL_SET_TPB) k_set_small(DevTable t, DevHash hp, Keys keys, Values values, ll_t epoch,
                                                                 ll_t *counters, ll_t *more) {
  __shared__ BlockTally tally;
  dok_tally_begin(tally);
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const ll_t e = (ll_t)blockIdx.x * DOK_SMALL_SET_TPB + threadIdx.x;
  const bool active = e < keys.count();
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  int outcome = -1, dup = 0, again = 0;
  const ll_t slot = dok_find_or_claim<SB, true>(t, kh, active, &outcome);
  const bool placed = active && slot >= 0, fresh = outcome == DOK_OUT_CLAIMED_EMPTY || outcome == DOK_OUT_REUSED;
  ull_t *stamp = placed ? (ull_t *)dok_stamp_ptr(t, slot) : nullptr;
  if (placed) {
    dok_write_row(t, hp, keys, values, e, slot, fresh || hp.dtype >= DOK_F16);
    if ((atomicMax(stamp, dok_stamp(epoch, e)) >> 34) == (ull_t)epoch) {
      atomicOr(stamp, DOK_STAMP_CONFLICT);
      dup = 1;
    }
  }
  cluster.sync();
  if (placed) {
    const ull_t now = __ldcg(stamp);
    if (now & DOK_STAMP_CONFLICT) {
      if (more && fresh) atomicOr(stamp, DOK_STAMP_FRESH);
      if ((now & ~DOK_STAMP_FRESH) == (dok_stamp(epoch, e) | DOK_STAMP_CONFLICT)) dok_write_row(t, hp, keys, values, e, slot, true);
    }
  }
  if (more) {                                             // uniform over the launch
    cluster.sync();
    if (placed && !fresh) {
      const ull_t now = __ldcg(stamp);
      again = (now >> 34) == (ull_t)epoch && (now & DOK_STAMP_FRESH) != 0;
    } else {
      again = active && !placed;
    }
  }
  dok_tally_add(tally, DOK_TALLY_EXTRA, again);
  if (counters) {
    dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, outcome == DOK_OUT_CLAIMED_EMPTY);
    dok_tally_add(tally, DOK_CNT_REUSED_REMOVED, outcome == DOK_OUT_REUSED);
    dok_tally_add(tally, DOK_CNT_FAILED, outcome == DOK_OUT_FAILED);
    dok_tally_add(tally, DOK_CNT_HITS, outcome == DOK_OUT_FOUND);
    dok_tally_add(tally, DOK_CNT_DUPLICATES, dup);
  }
  dok_tally_flush(tally, counters, more);
}

template <class Kernel, class... Args>
inline int dok_launch_cluster(ll_t rows, cudaStream_t st, Kernel kernel, Args... args) {
  unsigned blocks = 1;
  while ((ll_t)blocks * DOK_SMALL_SET_TPB < rows) blocks *= 2;
  cudaLaunchAttribute cluster;
  cluster.id = cudaLaunchAttributeClusterDimension;
  cluster.val.clusterDim.x = blocks;
  cluster.val.clusterDim.y = cluster.val.clusterDim.z = 1;
  cudaLaunchConfig_t config = {};
  config.gridDim = dim3(blocks);
  config.blockDim = dim3(blocks > 1 ? DOK_SMALL_SET_TPB : (unsigned)((rows + 63) / 64 * 64));
  config.stream = st;
  config.attrs = &cluster;
  config.numAttrs = 1;
  cudaLaunchKernelEx(&config, kernel, args...);
  return dok_check_launch();
}

inline bool dok_is_sliced(const RowKeys &k) { return k.slice_rows != 0; }
inline bool dok_is_sliced(const SelKeys &) { return false; }
inline bool dok_set_is_small(const DevTable &t, ll_t n) { return n <= DOK_SMALL_SET_ROWS && dok_window_passes(t) == 1; }

#include "dok_word.cuh"

// contiguous value rows [n, value_bytes]
template <class Keys, class Values>
inline int launch_set_general(const DevTable &t, const DevHash &hp, const Keys &keys, const Values &values,
                              int64_t *slot_scratch, int64_t epoch, uint8_t *out_stored, int64_t *counters, cudaStream_t st,
                              int64_t *more = nullptr, int64_t scratch_words = 0) {
  if (!out_stored && !dok_is_sliced(keys) && dok_set_is_small(t, keys.n)) {
    int rc = DOK_OK;
    DOK_DISPATCH_SB(t, (rc = dok_launch_cluster(keys.n, st, k_set_small<SB, Keys, Values>, t, hp, keys, values, (ll_t)epoch, (ll_t *)counters, (ll_t *)more)));
    return rc;
  }
  const bool filtered = keys.n >= DOK_FILTER_FROM && scratch_words >= keys.n + 1 + DOK_FILTER_ALL;
  unsigned *filter = filtered ? (unsigned *)(slot_scratch + keys.n + 1) : nullptr;
  const size_t zeroed = sizeof(int64_t) * (filtered ? 1 + DOK_FILTER_ALL : 1);
  if (cudaMemsetAsync(slot_scratch + keys.n, 0, zeroed, st) != cudaSuccess) return dok_check_launch();
  const dim3 grid = dok_grid(keys);
  int rc = DOK_OK;
  DOK_DISPATCH_MARKS(t, DOK_BY_SIZE(grid.x * grid.y, DOK_FOR_WINDOWS(t, rc, (k_set_claim<SB, FEW, MARKS><<<grid, DOK_TPB, 0, st>>>(wt, hp, keys, values, (ll_t *)slot_scratch, filter,
                                                                                       (ll_t)epoch, more != nullptr, out_stored, (ll_t *)counters)))));
  if (rc != DOK_OK) return rc;
  dim3 few = grid;
  if (few.x > 148 * 8) few.x = 148 * 8;
  DOK_FOR_WINDOWS(t, rc, (k_set_resolve<<<few, DOK_TPB, 0, st>>>(wt, hp, keys, values, (const ll_t *)slot_scratch, filter, (ll_t)epoch)));
  if (rc != DOK_OK || more == nullptr) return rc;
  k_set_count<<<few, DOK_TPB, 0, st>>>(t, keys, (const ll_t *)slot_scratch, filter, (ll_t)epoch, (ll_t *)more);
  return dok_check_launch();
}

inline int launch_set(const DevTable &t, const DevHash &hp, const RowKeys &keys, const char *values, int64_t *slot_scratch,
                      int64_t epoch, uint8_t *out_stored, int64_t *counters, cudaStream_t st, int64_t scratch_words = 0) {
  RowValues rv{values};
  return launch_set_general(t, hp, keys, rv, slot_scratch, epoch, out_stored, counters, st, nullptr, scratch_words);
}

inline int launch_set_unique(const DevTable &t, const DevHash &hp, const RowKeys &keys, const char *values,
                             uint8_t *out_stored, int64_t *counters, cudaStream_t st) {
  RowValues rv{values};
  const dim3 grid = dok_grid(keys);
  int rc = DOK_OK;
  DOK_DISPATCH_MARKS(t, DOK_FOR_WINDOWS(t, rc, (k_set_unique<SB, MARKS><<<grid, DOK_TPB, 0, st>>>(wt, hp, keys, rv, out_stored, (ll_t *)counters))));
  return rc;
}

// ---------------------------------------------------------------------------------------------------------
// remove / exists / count-new
// ---------------------------------------------------------------------------------------------------------

// REMOVE = 1: the tag is swapped to the tombstone by CAS so that equal uuids in one batch report exactly once
// (ClosedHashmap::remove, closed_hashmap_impl_class.cu:459-484, stores it non-atomically).
template <int SB, int REMOVE, bool FEW, class Keys>
__global__ void __launch_bounds__(DOK_TPB) k_find(DevTable t, DevHash hp, Keys keys, uint8_t *__restrict__ out_flags,
                                                  ll_t *counters) {
  __shared__ BlockTally tally;
  if (keys.idle()) return;
  if (counters) dok_tally_begin(tally);
  ll_t e;
  bool active = keys.row(e);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  const Located loc = dok_locate<SB, 1, false>(t, kh, e, active, nullptr, NoEmit<FEW>());
  int hit = active && loc.found >= 0;
  if (REMOVE && hit) hit = dok_cas_tag(t, loc.found, kh.uuid, DOK_REMOVED) == kh.uuid;
  if (active && out_flags) out_flags[e] = (uint8_t)hit;
  if (counters) {
    dok_tally_add(tally, DOK_CNT_HITS, hit);
    dok_tally_flush(tally, counters, nullptr);
  }
}

template <int REMOVE, class Keys>
inline int launch_find(const DevTable &t, const DevHash &hp, const Keys &keys, uint8_t *out_flags, int64_t *counters,
                       cudaStream_t st) {
  const dim3 grid = dok_grid(keys);
  int rc = DOK_OK;
  DOK_DISPATCH_SB(t, DOK_BY_SIZE(grid.x * grid.y, DOK_FOR_WINDOWS(t, rc, (k_find<SB, REMOVE, FEW><<<grid, DOK_TPB, 0, st>>>(wt, hp, keys, out_flags, (ll_t *)counters)))));
  return rc;
}

static __global__ void k_fill_i64(ll_t *p, ll_t n, ll_t v) {
  for (ll_t i = (ll_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (ll_t)gridDim.x * blockDim.x) p[i] = v;
}

// Rows absent from the table insert their uuid into a scratch tag set; the number of successful claims is the
// number of distinct absent uuids.
template <int SB, bool FEW, class Keys>
__global__ void __launch_bounds__(DOK_TPB) k_count_new(DevTable t, DevHash hp, Keys keys, ll_t *__restrict__ scratch,
                                                       ll_t scratch_slots, ll_t *counters) {
  __shared__ BlockTally tally;
  if (keys.idle()) return;
  dok_tally_begin(tally);
  ll_t e;
  bool active = keys.row(e);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  Located loc{-1, -1, -1};
  if (t.n_groups > 0) loc = dok_locate<SB, 1, false>(t, kh, e, active, nullptr, NoEmit<FEW>());      // (0: no table, every row is absent)
  int claimed = 0;
  if (active && loc.found < 0) {
    const ll_t uuid = kh.uuid;
    ll_t slot = (ll_t)__umul64hi(dok_mix64((ull_t)uuid ^ 0x5851f42d4c957f2dULL), (ull_t)scratch_slots);
    for (ll_t i = 0; i < scratch_slots; i++) {
      ll_t tag = __ldcg(&scratch[slot]);
      if (tag == DOK_EMPTY) {
        tag = (ll_t)atomicCAS((ull_t *)&scratch[slot], (ull_t)DOK_EMPTY, (ull_t)uuid);
        if (tag == DOK_EMPTY) { claimed = 1; break; }
      }
      if (tag == uuid) break;
      if (++slot == scratch_slots) slot = 0;
    }
  }
  dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, claimed);
  dok_tally_flush(tally, counters, nullptr);
}

// ---------------------------------------------------------------------------------------------------------
// rehash: live slots of one table straight into another
// ---------------------------------------------------------------------------------------------------------

// One thread per SOURCE slot: the stored key row of a live slot is hashed with the destination's parameters and
// inserted, key bytes and value copied as they are (both tables store key element i in column perm[i]).  Replaces
// the reference's rehash = two boolean-mask gathers plus a full `set` with its pre-get and unique
// (cuda_closed_hashmap.py:456-468) and this library's own compaction + insert.  Live keys are pairwise different,
// so every row claims a fresh slot; tombstones stay behind.
template <int SB, bool FEW, bool MARKS>
__global__ void __launch_bounds__(DOK_TPB, FEW ? 4 : 5) k_reinsert(DevTable src, DevTable dst, DevHash hp, ll_t *counters) {
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB;
  int claimed = 0, failed = 0, found = 0;
  for (ll_t base = (ll_t)blockIdx.x * DOK_TPB; base < src.nb; base += stride) {       // uniform over the block
    const ll_t s = base + threadIdx.x;
    bool active = false;
    if (s < src.nb) active = dok_load_tag(src, s) >= 0;   // uuids are non-negative; empty, tombstone, padding are not
    KeyHash kh{0, 0};
    const char *krow = dok_key_row(src, active ? s : 0);
    if (active) {
      ll_t k = dok_key_elem(krow, hp.dtype, hp.perm[0]);
      ll_t u = dok_uuid_term(k, hp.a[0], hp.b[0], hp.p[0], hp.m[0]);
      ull_t h = (ull_t)k * (ull_t)hp.a1[0] + (ull_t)hp.b1[0];
      for (int i = 1; i < hp.ks; i++) {
        k = dok_key_elem(krow, hp.dtype, hp.perm[i]);
        u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(k, hp.a[i], hp.b[i], hp.p[i], hp.m[i]));
        h *= (ull_t)k * (ull_t)hp.a1[i] + (ull_t)hp.b1[i];
      }
      kh = KeyHash{dok_llabs(u), (ll_t)h};
    }
    active = dok_in_window(dst, kh, active);
    int outcome = -1;
    const ll_t slot = dok_find_or_claim<SB, FEW, MARKS, true>(dst, kh, active, &outcome);
    if (active && slot >= 0) {
      char *drow = dok_key_row(dst, slot);
      if ((dst.kb & 7) == 0) for (int i = 0; i < (dst.kb >> 3); i++) ((ull_t *)drow)[i] = ((const ull_t *)krow)[i];
      else if ((dst.kb & 3) == 0) for (int i = 0; i < (dst.kb >> 2); i++) ((unsigned *)drow)[i] = ((const unsigned *)krow)[i];
      else if ((dst.kb & 1) == 0) for (int i = 0; i < (dst.kb >> 1); i++) ((unsigned short *)drow)[i] = ((const unsigned short *)krow)[i];
      else for (int i = 0; i < dst.kb; i++) drow[i] = krow[i];
      dok_store_value(dst, slot, dok_value_ptr(src, s));
    }
    claimed += outcome == DOK_OUT_CLAIMED_EMPTY || outcome == DOK_OUT_REUSED;
    failed += outcome == DOK_OUT_FAILED;
    found += outcome == DOK_OUT_FOUND;
  }
  if (counters) {
    dok_warp_add(counters + DOK_CNT_CLAIMED_EMPTY, claimed);
    dok_warp_add(counters + DOK_CNT_FAILED, failed);
    dok_warp_add(counters + DOK_CNT_HITS, found);
  }
}

// ---------------------------------------------------------------------------------------------------------
// init / uuid
// ---------------------------------------------------------------------------------------------------------

__device__ __forceinline__ void dok_store_sector(char *p, ll_t first) {
  asm volatile("st.global.v4.u64 [%0], {%1, %2, %2, %2};" ::"l"(p), "l"(first), "l"(0LL) : "memory");
}

static __global__ void k_init(DevTable t, ll_t *state, int state_words) {
  const ll_t stride = (ll_t)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x < state_words) state[threadIdx.x] = 0;
  // whole 32-byte sectors, so that none of them has to be read to be completed: 2^21 64-byte slots 22 -> 14 us
  const int stamp_sector = t.stamp_off & ~31;
  for (ll_t i = (ll_t)blockIdx.x * blockDim.x + threadIdx.x; i < t.n_slots; i += stride) {
    char *slot = dok_slot_ptr(t, i);
    dok_store_sector(slot, i < t.nb ? DOK_EMPTY : DOK_BLOCKED);
    if (t.stamp_off >= 32) dok_store_sector(slot + stamp_sector, 0);
    if (t.stamp_off < 0 && t.stamp) t.stamp[i] = 0;
  }
}

template <class Keys>
__global__ void k_uuid(DevTable t, DevHash hp, Keys keys, ll_t *uuid_out, ll_t *slot_out) {
  const ll_t e = (ll_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= keys.count()) return;
  const KeyHash kh = keys.hash(hp, e);
  if (uuid_out) uuid_out[e] = kh.uuid;
  if (slot_out) slot_out[e] = t.n_groups > 0 ? dok_start_group(kh, t) * t.spg : 0;
}

// ---------------------------------------------------------------------------------------------------------
// compaction of live slots in slot order
// ---------------------------------------------------------------------------------------------------------
#define DOK_COMPACT_ROUNDS 8
#define DOK_COMPACT_TILE (DOK_TPB * DOK_COMPACT_ROUNDS)

__device__ __forceinline__ bool dok_is_live(ll_t tag) { return tag != DOK_EMPTY && tag != DOK_REMOVED && tag != DOK_BLOCKED; }

static __global__ void __launch_bounds__(DOK_TPB) k_compact_count(DevTable t, ll_t *tile_counts) {
  __shared__ int warp_sums[DOK_TPB / 32];
  const ll_t base = (ll_t)blockIdx.x * DOK_COMPACT_TILE;
  int c = 0;
#pragma unroll
  for (int r = 0; r < DOK_COMPACT_ROUNDS; r++) {
    const ll_t slot = base + r * DOK_TPB + threadIdx.x;
    if (slot < t.nb) c += dok_is_live(__ldcs(dok_tag_ptr(t, slot)));
  }
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    int s = 0;
    for (int w = 0; w < DOK_TPB / 32; w++) s += warp_sums[w];
    tile_counts[blockIdx.x] = s;
  }
}

// In-place exclusive scan of a[0..n) by one block; a[n] receives the total.
static __global__ void __launch_bounds__(1024) k_exclusive_scan(ll_t *a, ll_t n) {
  __shared__ ll_t partial[1024];
  const ll_t per = (n + 1023) / 1024;
  const ll_t lo = threadIdx.x * per, hi = lo + per < n ? lo + per : n;
  ll_t s = 0;
  for (ll_t i = lo; i < hi; i++) s += a[i];
  partial[threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    ll_t run = 0;
    for (int i = 0; i < 1024; i++) { const ll_t v = partial[i]; partial[i] = run; run += v; }
    a[n] = run;
  }
  __syncthreads();
  ll_t run = partial[threadIdx.x];
  for (ll_t i = lo; i < hi; i++) { const ll_t v = a[i]; a[i] = run; run += v; }
}

static __global__ void __launch_bounds__(DOK_TPB) k_compact_scatter(DevTable t, DevHash hp, const ll_t *__restrict__ tile_offsets,
                                                             ll_t total_tiles, char *keys_out, int keys_transposed,
                                                             char *values_out, ll_t *uuid_out) {
  __shared__ int warp_sums[DOK_TPB / 32];
  __shared__ int round_base;
  const ll_t base = (ll_t)blockIdx.x * DOK_COMPACT_TILE;
  const ll_t count = tile_offsets[total_tiles];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) round_base = 0;
  __syncthreads();
  const ll_t tile_out = tile_offsets[blockIdx.x];
  for (int r = 0; r < DOK_COMPACT_ROUNDS; r++) {
    const ll_t slot = base + r * DOK_TPB + threadIdx.x;
    ll_t tag = DOK_EMPTY;
    if (slot < t.nb) tag = __ldcs(dok_tag_ptr(t, slot));
    const bool live = dok_is_live(tag);
    const unsigned ballot = __ballot_sync(0xffffffffu, live);
    if (lane == 0) warp_sums[warp] = __popc(ballot);
    __syncthreads();
    int before = round_base;
    for (int w = 0; w < warp; w++) before += warp_sums[w];
    before += __popc(ballot & ((1u << lane) - 1u));
    if (live) {
      const ll_t pos = tile_out + before;
      if (uuid_out) uuid_out[pos] = tag;
      if (values_out) dok_load_value(t, slot, values_out + pos * (ll_t)t.vb);
      if (keys_out) {
        // keys(): column i of the output is storage column key_perm[i] (cuda_closed_hashmap.py:165)
        const char *src = dok_key_row(t, slot);
        for (int i = 0; i < hp.ks; i++) {
          const ll_t o = keys_transposed ? ((ll_t)i * count + pos) : (pos * hp.ks + i);
          switch (hp.elem_bytes) {
            case 8: ((ll_t *)keys_out)[o] = ((const ll_t *)src)[hp.perm[i]]; break;
            case 4: ((int *)keys_out)[o] = ((const int *)src)[hp.perm[i]]; break;
            case 2: ((short *)keys_out)[o] = ((const short *)src)[hp.perm[i]]; break;
            default: keys_out[o] = src[hp.perm[i]]; break;
          }
        }
      }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int s = 0;
      for (int w = 0; w < DOK_TPB / 32; w++) s += warp_sums[w];
      round_base += s;
    }
    __syncthreads();
  }
}

