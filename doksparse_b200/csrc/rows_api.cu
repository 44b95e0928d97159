// Row-wise passes that the reference leaves to `unique(dim=0)`: the count of the distinct new rows of a float-key set
// (cuda_closed_hashmap.py:350-363) and the removal of a batch's sorted unique rows (:438-454).
#include <cstddef>
#include <type_traits>
#include "dok_kernels.cuh"

// ---------------------------------------------------------------------------------------------------------
// element order and row comparison
// ---------------------------------------------------------------------------------------------------------

// Element as an unsigned number of the type's width that sorts like the element: the sign bit flipped for signed
// integers; for floats, the magnitude's bits above or below the middle, which gives the two zeros, equal, one image and
// keeps the mantissa's low zeros of whole numbers of either sign.  *nan is set for a NaN, which compares with nothing.
__device__ __forceinline__ ull_t dok_ordered(const void *keys, int dtype, ll_t idx, bool *nan) {
  switch (dtype) {
    case DOK_I64: return ((const ull_t *)keys)[idx] ^ 0x8000000000000000ULL;
    case DOK_I32: return ((const unsigned *)keys)[idx] ^ 0x80000000u;
    case DOK_I16: return (unsigned)(((const unsigned short *)keys)[idx] ^ 0x8000u);
    case DOK_I8: return (unsigned)(((const unsigned char *)keys)[idx] ^ 0x80u);
    case DOK_U8: return ((const unsigned char *)keys)[idx];
    case DOK_F64: {
      const ull_t b = ((const ull_t *)keys)[idx], size = b & 0x7fffffffffffffffULL;
      *nan |= size > 0x7ff0000000000000ULL;
      return (b >> 63) ? 0x8000000000000000ULL - size : 0x8000000000000000ULL + size;
    }
    case DOK_F32: {
      const unsigned b = ((const unsigned *)keys)[idx], size = b & 0x7fffffffu;
      *nan |= size > 0x7f800000u;
      return (b >> 31) ? 0x80000000u - size : 0x80000000u + size;
    }
    default: {
      const unsigned b = ((const unsigned short *)keys)[idx], size = b & 0x7fffu;
      *nan |= size > (dtype == DOK_F16 ? 0x7c00u : 0x7f80u);
      return (b >> 15) ? 0x8000u - size : 0x8000u + size;
    }
  }
}

// rows a and b of the batch: < 0, 0, > 0 in lexicographic order
__device__ __forceinline__ int dok_compare_rows(const void *keys, int dtype, int ks, ll_t a, ll_t b) {
  bool nan = false;
  for (int i = 0; i < ks; i++) {
    const ull_t x = dok_ordered(keys, dtype, a * ks + i, &nan), y = dok_ordered(keys, dtype, b * ks + i, &nan);
    if (x != y) return x < y ? -1 : 1;
  }
  return 0;
}

// ---------------------------------------------------------------------------------------------------------
// distinct absent rows
// ---------------------------------------------------------------------------------------------------------

// k_count_new for keys whose identity is the ROW, not the uuid (float keys: the value cast gives many rows one uuid).  The
// scratch set holds {32 bits of the row's hash | row index}; a row that meets its hash there compares the rows.  A row with
// a NaN equals none, not even itself, and counts each time.  Replaces a boolean gather and a sort of the absent rows:
// 1 M rows of three floats took 0.5 ms of it.
template <int SB>
__global__ void __launch_bounds__(DOK_TPB) k_count_new_rows(DevTable t, DevHash hp, RowKeys keys, ull_t *__restrict__ scratch,
                                                            ll_t scratch_slots, ll_t *counters) {
  __shared__ BlockTally tally;
  dok_tally_begin(tally);
  ll_t e;
  bool active = keys.row(e);
  KeyHash kh{0, 0};
  if (active) kh = keys.hash(hp, e);
  active = dok_in_window(t, kh, active);
  Located loc{-1, -1, -1};
  if (t.n_groups > 0) loc = dok_locate<SB, 1, false>(t, kh, e, active, nullptr, NoEmit<false>());      // (0: no table, every row is absent)
  int claimed = 0;
  if (active && loc.found < 0) {
    bool nan = false;
    ull_t h = 0x5851f42d4c957f2dULL;
    for (int i = 0; i < hp.ks; i++) h = dok_mix64(h ^ dok_ordered(keys.keys, hp.dtype, e * hp.ks + i, &nan)) + 0x9e3779b97f4a7c15ULL;
    const ull_t mine = (h << 32) | (ull_t)e;
    ll_t slot = (ll_t)__umul64hi(h, (ull_t)scratch_slots);
    claimed = nan;
    for (ll_t i = 0; i < scratch_slots && !nan; i++) {
      ull_t other = __ldcg(&scratch[slot]);
      if (other == ~0ULL) {
        other = atomicCAS(&scratch[slot], ~0ULL, mine);
        if (other == ~0ULL) { claimed = 1; break; }
      }
      if ((other >> 32) == (mine >> 32) && dok_compare_rows(keys.keys, hp.dtype, hp.ks, e, (ll_t)(other & 0xffffffffULL)) == 0) break;
      if (++slot == scratch_slots) slot = 0;
    }
  }
  dok_tally_add(tally, DOK_CNT_CLAIMED_EMPTY, claimed);
  dok_tally_flush(tally, counters, nullptr);
}

// ---------------------------------------------------------------------------------------------------------
// removal of the sorted unique rows: up to DOK_SMALL_ROWS rows in one block
// ---------------------------------------------------------------------------------------------------------

// A batch that one block holds in shared memory is sorted (bitonic network over the first 8 bytes of the rows' images,
// equal prefixes compared by row), made unique and removed by ONE kernel.  Such a batch is all latency: the library's
// sort, select and fill kernels, the removal kernel and their launches took 110 us for 200 rows.
#define DOK_SMALL_ROWS 4096
#define DOK_SMALL_TPB 1024

struct SmallRows {
  ull_t key[DOK_SMALL_ROWS];
  unsigned short row[DOK_SMALL_ROWS];        // 0xffff: padding, behind every row
};

template <int SB>
__global__ void __launch_bounds__(DOK_SMALL_TPB) k_remove_unique_small(DevTable t, DevHash hp, RowKeys keys, int padded,
                                                                       uint8_t *__restrict__ out_removed,
                                                                       ll_t *__restrict__ out_count, ll_t *counters) {
  __shared__ SmallRows s;
  __shared__ int warp_sums[DOK_SMALL_TPB / 32], removed;
  const int n = (int)keys.n, tid = (int)threadIdx.x, threads = (int)blockDim.x;
  const int per = min(hp.ks, 8 / hp.elem_bytes);                 // columns in the prefix
  const bool whole = per == hp.ks;
  bool nan = false;
  for (int i = tid; i < padded; i += threads) {
    ull_t k = ~0ULL;
    if (i < n) {
      k = 0;
      for (int c = 0; c < hp.ks; c++) {
        const ull_t v = dok_ordered(keys.keys, hp.dtype, (ll_t)i * hp.ks + c, &nan);
        if (c < per) k = hp.elem_bytes == 8 ? v : (k << (8 * hp.elem_bytes)) | v;
      }
    }
    s.key[i] = k;
    s.row[i] = i < n ? (unsigned short)i : (unsigned short)0xffff;
  }
  if (tid == 0) removed = 0;
  if (__syncthreads_or(nan)) {                                   // rows that compare with nothing: the caller's way
    if (tid == 0) *out_count = -1;
    return;
  }
  auto before = [&](int a, int b) {                              // element a sorts before element b
    const ull_t x = s.key[a], y = s.key[b];
    if (x != y) return x < y;
    const unsigned short p = s.row[a], q = s.row[b];
    if (p == 0xffff || q == 0xffff) return p != 0xffff && q == 0xffff;
    return !whole && dok_compare_rows(keys.keys, hp.dtype, hp.ks, p, q) < 0;
  };
  for (int size = 2; size <= padded; size <<= 1)
    for (int step = size >> 1; step > 0; step >>= 1) {
      for (int i = tid; i < padded / 2; i += threads) {
        const int a = 2 * i - (i & (step - 1)), b = a + step;
        const bool up = (a & size) == 0;
        if (up ? before(b, a) : before(a, b)) {
          const ull_t k = s.key[a];
          s.key[a] = s.key[b];
          s.key[b] = k;
          const unsigned short r = s.row[a];
          s.row[a] = s.row[b];
          s.row[b] = r;
        }
      }
      // up to a step of 32 each warp keeps to the same 64 elements
      if (step > 32 || (step == 1 && size > 32)) __syncthreads(); else __syncwarp();
    }
  __syncthreads();
  // the first row of each run of equal rows, compacted in order into s.row (a row never moves up, so the last row of a
  // chunk stays in place for the comparison with the next chunk's first)
  int count = 0;
  for (int base = 0; base < n; base += threads) {
    const int i = base + tid;
    const unsigned short row = i < n ? s.row[i] : (unsigned short)0xffff;
    bool head = i < n;
    if (head && i > 0 && s.key[i] == s.key[i - 1])
      head = !whole && dok_compare_rows(keys.keys, hp.dtype, hp.ks, row, s.row[i - 1]) != 0;
    const unsigned votes = __ballot_sync(0xffffffffu, head);
    if ((tid & 31) == 0) warp_sums[tid >> 5] = __popc(votes);
    __syncthreads();
    int at = count, total = 0;
    for (int w = 0; w < threads / 32; w++) {
      if (w < (tid >> 5)) at += warp_sums[w];
      total += warp_sums[w];
    }
    at += __popc(votes & ((1u << (tid & 31)) - 1u));
    if (head && at != i) s.row[at] = row;
    count += total;
    __syncthreads();
  }
  for (int base = 0; base < count; base += threads) {
    const int i = base + tid;
    const bool active = i < count;
    const ll_t e = active ? s.row[i] : 0;
    KeyHash kh{0, 0};
    if (active) kh = keys.hash(hp, e);
    const Located loc = dok_locate<SB, 1, false>(t, kh, 0, active, nullptr, NoEmit<true>());
    int hit = active && loc.found >= 0;
    if (hit) hit = dok_cas_tag(t, loc.found, kh.uuid, DOK_REMOVED) == kh.uuid;
    if (active) out_removed[i] = (uint8_t)hit;
    const unsigned votes = __ballot_sync(0xffffffffu, hit);
    if ((tid & 31) == 0 && votes) atomicAdd(&removed, __popc(votes));
  }
  __syncthreads();
  if (tid == 0) {
    *out_count = count;
    if (removed && counters) atomicAdd((ull_t *)counters + DOK_CNT_HITS, (ull_t)removed);
  }
}

// ---------------------------------------------------------------------------------------------------------
// the same for larger batches: radix sort of 32-bit prefixes, ties by row
// ---------------------------------------------------------------------------------------------------------

// A row's columns are packed, first column on top, each in as many bits as its values differ in: those of the largest less
// the smallest, without the low bits that all rows share (the empty end of the mantissa of whole numbers).  The leading 32
// bits of that are the prefix, and four passes of a single-pass-per-digit radix sort (D. Merrill and M. Garland,
// "Single-pass parallel prefix scan with decoupled look-back", 2016; A. Adinets and D. Merrill, "Onesweep", 2022) bring the
// row numbers into prefix order.  Digits that all rows share are skipped.  Where the packed row has more than 32 bits, runs
// of equal prefixes that hold different rows -- a handful for scattered keys -- are put in order afterwards.  Half the
// passes of a 64-bit sort, and rows of any number of columns at the price of one; a comparison sort of rows took 0.37 ms
// for 250 k rows of three floats.
//
// Where such runs are the rule (ids of a few bits more than 32 of which the small ones are in every batch, few values in the
// first columns), the rows are sorted by every word of the packed row instead, the last word first: the host is told how
// many there are and calls again.  Whether they are the rule is estimated before the first pass, on samples of the batch
// (a call of remove(), 1 M / 6.4 M rows, us.  Ids that are Zipf-distributed over 2^34: 647 / 2023 where a batch with a run of
// more than 64 rows was given back to the library after the passes, 272 / 796 by all words.  Three floats below 1000: 838 /
// 4288, 317 / 1279.  The prefix alone tells three floats below 2^20 well enough apart: 263 at 1 M, 465 by all words).
#define DOK_SORT_TPB 256
#define DOK_SORT_ITEMS 16                  // per thread; a quarter where that leaves SMs without a tile
#define DOK_SORT_SMALL_ITEMS 4
#define DOK_SORT_SMALL (148LL * DOK_SORT_TPB * DOK_SORT_ITEMS)
#define DOK_SORT_MAX_ROWS (1LL << 30)      // counts travel in 30 bits beside two flags
#define DOK_SORT_SPINS (1 << 22)           // bound of every wait for another block; far beyond what one takes
#define DOK_MAX_RUN 16                     // longest run of equal prefixes with different rows that one thread sorts
#define DOK_LONG_RUNS 4096                 // places for longer ones, which a block sorts:
#define DOK_TIES_TPB 1024
#define DOK_BLOCK_RUN 4096                 // by a network up to here, ...
#define DOK_MAX_DISTINCT 32                // ... beyond if they hold no more different rows than this
#define DOK_CLUMP_SLOTS 1024               // rows per block that are looked at for the estimate
#define DOK_CLUMPED_MIN 8
#define DOK_UNIQUE_ROUNDS 8                // rows per thread of the removal; one of them for small batches, likewise

// why nothing was removed
enum { DOK_REFUSED_ROWS = 1, DOK_REFUSED_WAIT = 2, DOK_REFUSED_PREFIX = 3 };

// zeroed before the first kernel
struct SortControl {
  ull_t not_min[DOK_MAX_KEY_SIZE], max[DOK_MAX_KEY_SIZE];     // of the ordered images, ~min so that 0 is neutral
  ull_t varying[DOK_MAX_KEY_SIZE];                            // bits in which a row's image differs from the first row's
  // and again before the first word of a sort by all words
  unsigned final_b;       // the rows in order are in buffer b
  unsigned refused;       // DOK_REFUSED_ROWS: a NaN, or a wait of the sort that ran out; _WAIT: a wait of the removal;
                          // _PREFIX: the sort by prefixes is not worth it, or has left a run that nobody sorts
  // and again before each word
  unsigned hist[4][256];
  unsigned ticket[5];                                         // next tile of each pass, and of the removal
  unsigned n_mixed, n_long, differ;                           // short and long mixed runs; rows of the samples in mixed runs
  unsigned skip[4], from_b[4];                                // plan of the passes
  unsigned long_set[DOK_LONG_RUNS], long_run[DOK_LONG_RUNS];  // the long ones' starts, + 1: as a set, and in a row
};

__device__ __forceinline__ int dok_column_shift(const SortControl *c, int i) {      // (0 in a column of one value)
  const int shift = __ffsll((ll_t)c->varying[i]) - 1;
  return shift < 0 ? 0 : shift;
}
__device__ __forceinline__ int dok_column_bits(const SortControl *c, int i) {
  const ull_t span = (c->max[i] - ~c->not_min[i]) >> dok_column_shift(c, i);
  return span ? 64 - __clzll(span) : 0;
}
__device__ __forceinline__ int dok_row_words(const SortControl *c, int ks) {
  int bits = 0;
  for (int i = 0; i < ks; i++) bits += dok_column_bits(c, i);
  return bits <= 32 ? 1 : (bits + 31) / 32;
}
__device__ __forceinline__ bool dok_prefix_is_row(const SortControl *c, int ks) { return dok_row_words(c, ks) == 1; }

// How a row is packed, in shared memory.
struct RowPack {
  ull_t min[DOK_MAX_KEY_SIZE];
  int shift[DOK_MAX_KEY_SIZE], bits[DOK_MAX_KEY_SIZE];
};
__device__ __forceinline__ void dok_load_pack(RowPack &pack, const SortControl *c, int ks) {
  const int i = threadIdx.x;
  if (i < ks) {
    pack.min[i] = ~c->not_min[i];
    pack.shift[i] = dok_column_shift(c, i);
    pack.bits[i] = dok_column_bits(c, i);
  }
}
// Bits 32 * word .. 32 * word + 31 of the packed row, counted from its leading bit; the last word has what is left.
// HASH: with a hash of the whole row.
template <bool HASH>
__device__ __forceinline__ unsigned dok_row_word(const RowPack &pack, const void *keys, int dtype, int ks, ll_t e, int word, unsigned *rest) {
  bool nan = false;
  ull_t acc = 0, hash = 0;
  const int from = 32 * word, to = from + 32;
  int at = 0;
  for (int i = 0; i < ks && (HASH || at < to); i++) {
    const int end = at + pack.bits[i], lo = at > from ? at : from, hi = end < to ? end : to;
    if (HASH || lo < hi) {
      const ull_t v = (dok_ordered(keys, dtype, e * ks + i, &nan) - pack.min[i]) >> pack.shift[i];
      if (lo < hi) acc = (acc << (hi - lo)) | ((v >> (end - hi)) & ((1ULL << (hi - lo)) - 1ULL));
      if (HASH) hash = (hash ^ v) * 0x9e3779b97f4a7c15ULL;
    }
    at = end;
  }
  if (HASH) *rest = (unsigned)(hash >> 32);
  return (unsigned)acc;
}

// The loop below knows the type, so that four loads are on their way at a time.
template <class F>
__device__ __forceinline__ void dok_with_dtype(int dtype, const F &f) {
  switch (dtype) {
    case DOK_I64: f(std::integral_constant<int, DOK_I64>()); break;
    case DOK_I32: f(std::integral_constant<int, DOK_I32>()); break;
    case DOK_I16: f(std::integral_constant<int, DOK_I16>()); break;
    case DOK_I8: f(std::integral_constant<int, DOK_I8>()); break;
    case DOK_U8: f(std::integral_constant<int, DOK_U8>()); break;
    case DOK_F64: f(std::integral_constant<int, DOK_F64>()); break;
    case DOK_F32: f(std::integral_constant<int, DOK_F32>()); break;
    case DOK_F16: f(std::integral_constant<int, DOK_F16>()); break;
    default: f(std::integral_constant<int, DOK_BF16>()); break;
  }
}

struct ColumnRange { ull_t not_min, max, varying; };

#define DOK_RANGE_BLOCKS 5                 // per SM, resident
__global__ void __launch_bounds__(DOK_TPB, DOK_RANGE_BLOCKS) k_row_range(RowKeys keys, int dtype, int ks, SortControl *c) {
  __shared__ ull_t lo_hi[3 * DOK_MAX_KEY_SIZE];
  if (threadIdx.x < 3 * DOK_MAX_KEY_SIZE) lo_hi[threadIdx.x] = 0;
  __syncthreads();
  bool nan = false;
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB, n = keys.n;
  for (int i = 0; i < ks; i++) {
    ColumnRange r{0, 0, 0};
    dok_with_dtype(dtype, [&](auto type) {
      constexpr int TYPE = decltype(type)::value;
      const ull_t first = dok_ordered(keys.keys, TYPE, i, &nan);
      const auto add = [&](ull_t v) {
        r.not_min = ~v > r.not_min ? ~v : r.not_min;
        r.max = v > r.max ? v : r.max;
        r.varying |= v ^ first;
      };
      ll_t e = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x;
      for (; e + 3 * stride < n; e += 4 * stride) {
        ull_t v[4];
#pragma unroll
        for (int k = 0; k < 4; k++) v[k] = dok_ordered(keys.keys, TYPE, (e + k * stride) * ks + i, &nan);
#pragma unroll
        for (int k = 0; k < 4; k++) add(v[k]);
      }
      for (; e < n; e += stride) add(dok_ordered(keys.keys, TYPE, e * ks + i, &nan));
    });
    for (int o = 16; o > 0; o >>= 1) {
      const ull_t a = __shfl_xor_sync(0xffffffffu, r.not_min, o), b = __shfl_xor_sync(0xffffffffu, r.max, o);
      r.not_min = a > r.not_min ? a : r.not_min;
      r.max = b > r.max ? b : r.max;
      r.varying |= __shfl_xor_sync(0xffffffffu, r.varying, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicMax(&lo_hi[3 * i], r.not_min);
      atomicMax(&lo_hi[3 * i + 1], r.max);
      atomicOr(&lo_hi[3 * i + 2], r.varying);
    }
  }
  nan = __syncthreads_or(nan);
  if (threadIdx.x < ks) {
    atomicMax(&c->not_min[threadIdx.x], lo_hi[3 * threadIdx.x]);
    atomicMax(&c->max[threadIdx.x], lo_hi[3 * threadIdx.x + 1]);
    atomicOr(&c->varying[threadIdx.x], lo_hi[3 * threadIdx.x + 2]);
  }
  if (threadIdx.x == 0 && nan) c->refused = DOK_REFUSED_ROWS;
}

__device__ __forceinline__ void dok_count_digits(unsigned (&hist)[4][256], unsigned word) {
#pragma unroll
  for (int d = 0; d < 4; d++) atomicAdd(&hist[d][(word >> (8 * d)) & 255u], 1u);
}
__device__ __forceinline__ void dok_add_digits(SortControl *c, const unsigned (&hist)[4][256]) {
  for (int i = threadIdx.x; i < 1024; i += DOK_TPB)
    if (((const unsigned *)hist)[i]) atomicAdd((unsigned *)c->hist + i, ((const unsigned *)hist)[i]);
}

__device__ __forceinline__ void dok_warp_count(unsigned *counter, int v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd(counter, (unsigned)v);
}

// The prefixes of the rows, and how many rows of the block's first DOK_CLUMP_SLOTS meet their prefix there with another
// row: by a table that keeps the last row of each prefix (of each place, which two prefixes may share).
__global__ void __launch_bounds__(DOK_TPB, 8) k_row_prefix(RowKeys keys, int dtype, int ks, SortControl *c, unsigned *prefix, unsigned *row) {
  __shared__ unsigned hist[4][256];
  __shared__ ull_t seen[DOK_CLUMP_SLOTS];
  __shared__ RowPack pack;
  dok_load_pack(pack, c, ks);
  for (int i = threadIdx.x; i < 1024; i += DOK_TPB) ((unsigned *)hist)[i] = 0;
  for (int i = threadIdx.x; i < DOK_CLUMP_SLOTS; i += DOK_TPB) seen[i] = ~0ULL;
  __syncthreads();
  int bits = 0;
  for (int i = 0; i < ks; i++) bits += pack.bits[i];
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB;
  ll_t e = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x;
  const auto put = [&](unsigned p) {
    prefix[e] = p;
    row[e] = (unsigned)e;
    dok_count_digits(hist, p);
  };
  if (bits > 32) {
    int differ = 0;
    for (int looked = 0; e < keys.n && looked < DOK_CLUMP_SLOTS; e += stride, looked += DOK_TPB) {
      unsigned rest;
      const unsigned p = dok_row_word<true>(pack, keys.keys, dtype, ks, e, 0, &rest);
      const ull_t mine = (ull_t)p << 32 | rest, other = atomicExch(&seen[(p * 0x9e3779b1u) >> 22], mine);
      differ += (unsigned)(other >> 32) == p && other != mine && other != ~0ULL;
      put(p);
    }
    dok_warp_count(&c->differ, differ);
  }
  for (; e < keys.n; e += stride) put(dok_row_word<false>(pack, keys.keys, dtype, ks, e, 0, nullptr));
  __syncthreads();
  dok_add_digits(c, hist);
}

// One word of the packed rows, in the order that the rows have so far (first: their own).
__global__ void __launch_bounds__(DOK_TPB, 8) k_row_word(RowKeys keys, int dtype, int ks, SortControl *c, int word, bool first, unsigned *key_a,
                                                      unsigned *row_a, unsigned *key_b, unsigned *row_b) {
  __shared__ unsigned hist[4][256];
  __shared__ RowPack pack;
  dok_load_pack(pack, c, ks);
  for (int i = threadIdx.x; i < 1024; i += DOK_TPB) ((unsigned *)hist)[i] = 0;
  __syncthreads();
  unsigned *key = c->final_b ? key_b : key_a, *row = c->final_b ? row_b : row_a;
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB;
  for (ll_t i = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; i < keys.n; i += stride) {
    if (first) row[i] = (unsigned)i;
    const unsigned e = first ? (unsigned)i : row[i];
    if (e >= keys.n) continue;                                // (a wait of an earlier pass ran out: nothing is removed)
    const unsigned w = dok_row_word<false>(pack, keys.keys, dtype, ks, e, word, nullptr);
    key[i] = w;
    dok_count_digits(hist, w);
  }
  __syncthreads();
  dok_add_digits(c, hist);
}

// digit counts -> exclusive offsets; which passes move anything, and from which buffer each one reads.  None does where the
// sort by prefixes gives up: `clumped` rows of the samples or more are in mixed runs (0: no limit).
__global__ void __launch_bounds__(256) k_sort_plan(SortControl *c, unsigned n, unsigned clumped) {
  __shared__ unsigned sums[8];
  const bool give_up = c->refused != 0 || (clumped && c->differ >= clumped);
  unsigned in_b = c->final_b;
  for (int d = 0; d < 4; d++) {
    const unsigned own = c->hist[d][threadIdx.x];
    unsigned v = own;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
      if ((threadIdx.x & 31) >= o) v += u;
    }
    if ((threadIdx.x & 31) == 31) sums[threadIdx.x >> 5] = v;
    const bool same = __syncthreads_or(own == n) || give_up;
    for (int w = 0; w < (int)(threadIdx.x >> 5); w++) v += sums[w];
    c->hist[d][threadIdx.x] = v - own;
    if (threadIdx.x == 0) { c->skip[d] = same; c->from_b[d] = in_b; }
    if (!same) in_b ^= 1;
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    c->final_b = in_b;
    if (give_up && c->refused == 0) c->refused = DOK_REFUSED_PREFIX;
  }
}

#define DOK_LB_LOCAL 0x40000000u           // a tile's own count
#define DOK_LB_TOTAL 0x80000000u           // the count up to and including the tile
#define DOK_LB_VALUE 0x3fffffffu

__device__ __forceinline__ unsigned dok_peek(const unsigned *p) { return *(const volatile unsigned *)p; }
__device__ __forceinline__ void dok_post(unsigned *p, unsigned v) { *(volatile unsigned *)p = v; }

// One digit.  A tile of 4096 or 1024 (prefix, row) pairs is ranked by digit with warp votes, its digit counts are posted, the
// counts of the tiles before it are summed up by looking back (tiles are handed out in order, so all of them have started),
// and the pairs leave through shared memory in digit order, a run of the output at a time.  80 us for 6.4 M pairs: bound by
// the latency of the ranking (shared memory, votes), not by the 102 MB it moves nor by the looking back; neither eight
// predecessors at a time (80 us) nor 32 instead of 24 warps per SM (83 us) changes it.
template <int ITEMS>
__global__ void __launch_bounds__(DOK_SORT_TPB) k_sort_pass(SortControl *c, int digit, unsigned n, unsigned *key_a, unsigned *row_a,
                                                            unsigned *key_b, unsigned *row_b, unsigned *look) {
  constexpr int TILE = DOK_SORT_TPB * ITEMS;
  if (c->skip[digit]) return;
  __shared__ unsigned keys[TILE], rows[TILE];
  __shared__ unsigned counts[DOK_SORT_TPB / 32][256];
  __shared__ unsigned start[256], shift_by[256], sums[8], tile_id;
  const bool b = c->from_b[digit];
  const unsigned *key_in = b ? key_b : key_a, *row_in = b ? row_b : row_a;
  unsigned *key_out = b ? key_a : key_b, *row_out = b ? row_a : row_b;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, shift = 8 * digit;
  if (tid == 0) tile_id = atomicAdd(&c->ticket[digit], 1u);
  for (int i = tid; i < (DOK_SORT_TPB / 32) * 256; i += DOK_SORT_TPB) ((unsigned *)counts)[i] = 0;
  __syncthreads();
  const unsigned tile = tile_id;
  const unsigned first = tile * TILE, size = min((unsigned)TILE, n - first);
  unsigned key[ITEMS], row[ITEMS], rank[ITEMS];
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const unsigned i = warp * 32 * ITEMS + k * 32 + lane;
    key[k] = i < size ? key_in[first + i] : 0;
    row[k] = i < size ? row_in[first + i] : 0;
  }
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const unsigned i = warp * 32 * ITEMS + k * 32 + lane;
    const unsigned digit_of = i < size ? (key[k] >> shift) & 255u : 256u;
    const unsigned peers = __match_any_sync(0xffffffffu, digit_of);
    unsigned base = 0;
    if (lane == __ffs(peers) - 1 && i < size) { base = counts[warp][digit_of]; counts[warp][digit_of] = base + __popc(peers); }
    base = __shfl_sync(0xffffffffu, base, __ffs(peers) - 1);
    rank[k] = base + __popc(peers & ((1u << lane) - 1u));
    __syncwarp();
  }
  __syncthreads();
  // thread d owns digit d
  unsigned total = 0;
  for (int w = 0; w < DOK_SORT_TPB / 32; w++) {
    const unsigned v = counts[w][tid];
    counts[w][tid] = total;
    total += v;
  }
  dok_post(look + (size_t)tile * 256 + tid, (tile == 0 ? DOK_LB_TOTAL : DOK_LB_LOCAL) | total);
  unsigned v = total;
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  if (lane == 31) sums[warp] = v;
  __syncthreads();
  for (int w = 0; w < warp; w++) v += sums[w];
  start[tid] = v - total;
  unsigned before = 0;
  int spins = 0;
  for (unsigned p = tile; p > 0;) {
    const unsigned s = dok_peek(look + (size_t)(p - 1) * 256 + tid);
    if (s == 0) {
      if (++spins < DOK_SORT_SPINS) continue;
      c->refused = DOK_REFUSED_ROWS;
      break;
    }
    before += s & DOK_LB_VALUE;
    if (s & DOK_LB_TOTAL) break;
    p--;
  }
  if (tile > 0) dok_post(look + (size_t)tile * 256 + tid, DOK_LB_TOTAL | (before + total));
  shift_by[tid] = c->hist[digit][tid] + before - (v - total);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < ITEMS; k++) {
    const unsigned i = warp * 32 * ITEMS + k * 32 + lane;
    if (i < size) {
      const unsigned d = (key[k] >> shift) & 255u, at = start[d] + counts[warp][d] + rank[k];
      keys[at] = key[k];
      rows[at] = row[k];
    }
  }
  __syncthreads();
  for (unsigned i = tid; i < size; i += DOK_SORT_TPB) {
    const unsigned k = keys[i], to = i + shift_by[(k >> shift) & 255u];
    if (to < n) { key_out[to] = k; row_out[to] = rows[i]; }
  }
}

// first place of [lo, hi) whose key is >= k, of a sorted array
__device__ __forceinline__ unsigned dok_lower_bound(const unsigned *key, unsigned lo, unsigned hi, unsigned k) {
  while (lo < hi) {
    const unsigned mid = lo + (hi - lo) / 2;
    if (key[mid] < k) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Runs of equal prefixes that hold different rows are listed by their start: at the first place where two neighbours differ,
// in a run of more than DOK_MAX_RUN rows by each such place that has none in the DOK_MAX_RUN rows before it.
__global__ void __launch_bounds__(DOK_TPB) k_list_ties(SortControl *c, RowKeys keys, int dtype, int ks, unsigned *key_a, const unsigned *row_a,
                                                       unsigned *key_b, const unsigned *row_b) {
  const unsigned n = (unsigned)keys.n;
  if (c->refused || dok_prefix_is_row(c, ks)) return;
  const unsigned *key = c->final_b ? key_b : key_a, *row = c->final_b ? row_b : row_a;
  unsigned *list = c->final_b ? key_a : key_b;
  const unsigned stride = gridDim.x * DOK_TPB;
  for (unsigned i = blockIdx.x * DOK_TPB + threadIdx.x; i + 1 < n; i += stride) {
    if (key[i] != key[i + 1] || dok_compare_rows(keys.keys, dtype, ks, row[i], row[i + 1]) == 0) continue;
    unsigned lo = i;
    bool first = true;
    while (first && lo > 0 && key[lo - 1] == key[i] && i - lo < DOK_MAX_RUN) {
      first = dok_compare_rows(keys.keys, dtype, ks, row[lo - 1], row[lo]) == 0;
      lo--;
    }
    if (!first) continue;                          // an earlier place lists the run
    if (n - lo <= DOK_MAX_RUN || key[lo + DOK_MAX_RUN] != key[i]) {
      list[atomicAdd(&c->n_mixed, 1u)] = lo;
      continue;
    }
    lo = dok_lower_bound(key, 0, i, key[i]);
    unsigned at = lo * 0x9e3779b1u % DOK_LONG_RUNS, tries = 0;
    for (; tries < DOK_LONG_RUNS; tries++) {
      const unsigned old = atomicCAS(&c->long_set[at], 0u, lo + 1);
      if (old == 0) c->long_run[atomicAdd(&c->n_long, 1u)] = lo + 1;
      if (old == 0 || old == lo + 1) break;
      at = (at + 1) % DOK_LONG_RUNS;
    }
    if (tries == DOK_LONG_RUNS) { c->refused = DOK_REFUSED_PREFIX; return; }
  }
}

// The smallest row of a block's threads, and how many hold one that equals it.
struct SmallestRow { unsigned row, count; };
#define DOK_NO_ROW 0xffffffffu
__device__ __forceinline__ SmallestRow dok_smaller(const RowKeys &keys, int dtype, int ks, SmallestRow a, SmallestRow b) {
  if (a.row == DOK_NO_ROW) return b;
  if (b.row == DOK_NO_ROW) return a;
  const int order = dok_compare_rows(keys.keys, dtype, ks, a.row, b.row);
  if (order) return order < 0 ? a : b;
  return SmallestRow{min(a.row, b.row), a.count + b.count};
}

// A listed run of up to DOK_MAX_RUN rows is sorted by insertion, by one thread (each step waits for the one before: 64 rows
// took 0.3 ms).  A longer one is sorted by a block: by a bitonic network where its rows fit; beyond that it is most often a
// key that the batch repeats and another that shares its prefix, and the block looks for the smallest row, the next larger
// one and so on, and writes each as often as it occurs (which of several equal rows it is makes no difference).  A batch of
// 6.4 M rows with 2.5 M different keys, Zipf-distributed, has about ten long runs.
__global__ void __launch_bounds__(DOK_TIES_TPB) k_sort_ties(SortControl *c, RowKeys keys, int dtype, int ks, const unsigned *key_a, unsigned *row_a,
                                                       const unsigned *key_b, unsigned *row_b) {
  __shared__ SmallestRow best_of[DOK_TIES_TPB / 32];
  __shared__ unsigned run[DOK_BLOCK_RUN];
  const unsigned n = (unsigned)keys.n;
  if (c->refused == DOK_REFUSED_ROWS || dok_prefix_is_row(c, ks)) return;      // (_PREFIX: set before, or by a block of this kernel)
  const unsigned *key = c->final_b ? key_b : key_a;
  const unsigned *list = c->final_b ? key_a : key_b;
  unsigned *row = c->final_b ? row_b : row_a, *sorted = c->final_b ? row_a : row_b;
  const unsigned n_long = c->n_long;
  for (unsigned r = blockIdx.x; r < n_long; r += gridDim.x) {
    const unsigned lo = c->long_run[r] - 1, k = key[lo], hi = k == 0xffffffffu ? n : dok_lower_bound(key, lo, n, k + 1);
    if (hi - lo <= DOK_BLOCK_RUN) {                                             // uniform over the block
      unsigned padded = 2;
      while (padded < hi - lo) padded *= 2;
      for (unsigned i = threadIdx.x; i < padded; i += DOK_TIES_TPB) run[i] = lo + i < hi ? row[lo + i] : DOK_NO_ROW;
      __syncthreads();
      const auto before = [&](unsigned a, unsigned b) {                         // the padding is behind every row
        if (a == DOK_NO_ROW || b == DOK_NO_ROW) return a < b;
        return dok_compare_rows(keys.keys, dtype, ks, a, b) < 0;
      };
      for (unsigned size = 2; size <= padded; size *= 2)
        for (unsigned step = size / 2; step > 0; step /= 2) {
          for (unsigned i = threadIdx.x; i < padded / 2; i += DOK_TIES_TPB) {
            const unsigned p = 2 * i - (i & (step - 1)), q = p + step, a = run[p], b = run[q];
            if ((p & size) == 0 ? before(b, a) : before(a, b)) { run[p] = b; run[q] = a; }
          }
          __syncthreads();
        }
      for (unsigned i = threadIdx.x; i < hi - lo; i += DOK_TIES_TPB) row[lo + i] = run[i];
      __syncthreads();
      continue;
    }
    unsigned out = lo, last = 0;
    for (int d = 0; out < hi; d++) {
      SmallestRow best{DOK_NO_ROW, 0};
      if (d < DOK_MAX_DISTINCT)
        for (unsigned i = lo + threadIdx.x; i < hi; i += DOK_TIES_TPB)
          if (d == 0 || dok_compare_rows(keys.keys, dtype, ks, row[i], last) > 0)
            best = dok_smaller(keys, dtype, ks, best, SmallestRow{row[i], 1});
      for (int o = 16; o > 0; o >>= 1)
        best = dok_smaller(keys, dtype, ks, best, SmallestRow{__shfl_xor_sync(0xffffffffu, best.row, o), __shfl_xor_sync(0xffffffffu, best.count, o)});
      __syncthreads();
      if ((threadIdx.x & 31) == 0) best_of[threadIdx.x >> 5] = best;
      __syncthreads();
      best = best_of[0];
      for (int w = 1; w < DOK_TIES_TPB / 32; w++) best = dok_smaller(keys, dtype, ks, best, best_of[w]);
      if (best.row == DOK_NO_ROW) {                                             // too many different rows
        if (threadIdx.x == 0) c->refused = DOK_REFUSED_PREFIX;
        break;
      }
      last = best.row;
      for (unsigned i = out + threadIdx.x; i < out + best.count; i += DOK_TIES_TPB) sorted[i] = last;
      out += best.count;
    }
    __syncthreads();
    if (out == hi)
      for (unsigned i = lo + threadIdx.x; i < hi; i += DOK_TIES_TPB) row[i] = sorted[i];
  }
  const unsigned stride = gridDim.x * DOK_TIES_TPB, mixed = c->n_mixed;
  for (unsigned m = blockIdx.x * DOK_TIES_TPB + threadIdx.x; m < mixed; m += stride) {
    const unsigned lo = list[m];
    unsigned hi = lo + 1;
    while (hi < n && hi - lo <= DOK_MAX_RUN && key[hi] == key[lo]) hi++;
    for (unsigned i = lo + 1; i < hi; i++) {
      const unsigned r = row[i];
      unsigned j = i;
      for (; j > lo && dok_compare_rows(keys.keys, dtype, ks, r, row[j - 1]) < 0; j--) row[j] = row[j - 1];
      row[j] = r;
    }
  }
}

// The first rows of runs of equal rows, as a key source for the walk.
struct HeadKeys {
  const RowKeys &keys;
  const unsigned *rows;
  __device__ __forceinline__ ll_t elem(unsigned i) const { return (ll_t)rows[i]; }
  __device__ __forceinline__ KeyHash hash(const DevHash &hp, ll_t e) const { return keys.hash(hp, e); }
};

// First row of each run of equal rows: looked up, its slot turned into a tombstone, its flag written at the run's number.
// Runs are counted across tiles by looking back like in the sort, when the tile's own lookups are done.  A tile's runs are
// gathered first and each warp walks its eighth of them with a lane taking the next when its chain ends (dok_stream.cuh):
// walked row by row, half the lanes of a batch that holds each key twice were idle, and all but the longest chain's of keys
// that are no longer there (64 M-operation churn, a table at load 0.9: 5.03 -> 4.64 ms; 4 rows per thread 4.85, 16 spill).
template <int SB, int ROUNDS>
__global__ void __launch_bounds__(DOK_TPB, 4) k_remove_unique(DevTable t, DevHash hp, RowKeys keys, SortControl *c, const unsigned *key_a,
                                                              const unsigned *row_a, const unsigned *key_b, const unsigned *row_b,
                                                              unsigned *look, unsigned tiles, uint8_t *__restrict__ out_removed,
                                                              ll_t *__restrict__ out_count, ll_t *counters) {
  constexpr unsigned TILE = DOK_TPB * ROUNDS;
  __shared__ unsigned sums[ROUNDS][DOK_WARPS], tile_id, base_of_tile;
  __shared__ unsigned head_row[TILE];
  __shared__ uint8_t hit_of[TILE];
  __shared__ WarpQueue queues[DOK_WARPS];
  __shared__ int removed;
  const unsigned n = (unsigned)keys.n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned refused = *(volatile unsigned *)&c->refused;
  if (refused == DOK_REFUSED_ROWS || refused == DOK_REFUSED_PREFIX) {      // set before this kernel: nothing has been removed
    if (blockIdx.x == 0 && tid == 0) *out_count = refused == DOK_REFUSED_ROWS ? -1 : -DOK_SORT_ALL_WORDS - dok_row_words(c, hp.ks);
    return;
  }
  if (tid == 0) { tile_id = atomicAdd(&c->ticket[4], 1u); removed = 0; }
  __syncthreads();
  const unsigned tile = tile_id;
  const unsigned *key = c->final_b ? key_b : key_a, *row = c->final_b ? row_b : row_a;
  const bool whole = dok_prefix_is_row(c, hp.ks);
  unsigned votes[ROUNDS], e[ROUNDS];
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    const unsigned i = tile * TILE + r * DOK_TPB + tid;
    bool head = i < n;
    e[r] = i < n ? row[i] : 0;
    if (head && i > 0 && key[i] == key[i - 1])
      head = !whole && dok_compare_rows(keys.keys, hp.dtype, hp.ks, e[r], row[i - 1]) != 0;
    votes[r] = __ballot_sync(0xffffffffu, head);
    if (lane == 0) sums[r][warp] = __popc(votes[r]);
  }
  __syncthreads();
  unsigned total = 0;
#pragma unroll
  for (int r = 0; r < ROUNDS; r++) {
    unsigned mine = total;
    for (int w = 0; w < DOK_WARPS; w++) {
      if (w < warp) mine += sums[r][w];
      total += sums[r][w];
    }
    if ((votes[r] >> lane) & 1u) head_row[mine + __popc(votes[r] & ((1u << lane) - 1u))] = e[r];
  }
  if (tid == 0) dok_post(look + tile, (tile == 0 ? DOK_LB_TOTAL : DOK_LB_LOCAL) | total);
  __syncthreads();
  int hits = 0;
  if constexpr (SB == 0) {
    for (unsigned i = tid; i < total; i += DOK_TPB) {
      const KeyHash kh = keys.hash(hp, head_row[i]);
      const Located loc = dok_locate_serial(t, kh, nullptr);
      const int hit = loc.found >= 0 && dok_cas_tag(t, loc.found, kh.uuid, DOK_REMOVED) == kh.uuid;
      hit_of[i] = (uint8_t)hit;
      hits += hit;
    }
  } else {
    const unsigned first = total * warp / DOK_WARPS, last = total * (warp + 1) / DOK_WARPS;
    dok_walk_share<1, false, false>(queues[warp], WarpShare{first, last - first, 0, 0, 0}, t, hp, HeadKeys{keys, head_row},
                      [&](LaneRow &lr, const Lines<1> &f, const WarpShare &share) {
      const unsigned bits = dok_inspect<SB, 1>(lr, f), m = dok_matches(bits, tid & 3), me = dok_ends(bits, tid & 3);
      if (!lr.busy()) return;
      const unsigned pos = me ? (unsigned)__ffs(me) - 1 : 0;
      const unsigned slot = lr.group * (128 / SB) + pos;
      if (me || !dok_next_group<unsigned>(lr.group, lr.word, (unsigned)t.n_groups)) {
        const int hit = ((m >> pos) & 1u) && dok_cas_tag(t, slot, lr.uuid, DOK_REMOVED) == lr.uuid;
        hit_of[share.first + lr.row] = (uint8_t)hit;
        hits += hit;
        lr.done();
      }
    });
  }
  for (int o = 16; o > 0; o >>= 1) hits += __shfl_xor_sync(0xffffffffu, hits, o);
  if (lane == 0 && hits) atomicAdd(&removed, hits);
  __syncthreads();
  if (warp == 0) {                                 // 32 predecessors at a time
    unsigned before = 0;
    int spins = 0;
    for (ll_t end = tile; end > 0;) {
      const ll_t p = end - 1 - lane;
      const unsigned s = p >= 0 ? dok_peek(look + p) : DOK_LB_TOTAL;
      if (__any_sync(0xffffffffu, s == 0)) {
        if (++spins < DOK_SORT_SPINS) continue;
        if (lane == 0) c->refused = DOK_REFUSED_WAIT;
        break;
      }
      const unsigned totals = __ballot_sync(0xffffffffu, (s & DOK_LB_TOTAL) != 0);
      const int stop = totals ? __ffs(totals) - 1 : 31;
      unsigned v = lane <= stop ? s & DOK_LB_VALUE : 0;
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      before += v;
      if (totals) break;
      end -= 32;
    }
    if (lane == 0) {
      if (tile > 0) dok_post(look + tile, DOK_LB_TOTAL | (before + total));
      base_of_tile = before;
      if (tile == tiles - 1) *out_count = *(volatile unsigned *)&c->refused == DOK_REFUSED_WAIT ? -2 : (ll_t)before + total;
      if (removed && counters) atomicAdd((ull_t *)counters + DOK_CNT_HITS, (ull_t)removed);
    }
  }
  __syncthreads();
  for (unsigned i = tid; i < total; i += DOK_TPB)
    if (base_of_tile + i < n) out_removed[base_of_tile + i] = hit_of[i];
}

struct SortWork {
  SortControl *control;
  unsigned *look, *unique_look, *key_a, *row_a, *key_b, *row_b;
  size_t zeroed, bytes;
  unsigned tiles, unique_tiles;
  bool small;
};

static SortWork sort_work(void *base, ll_t n) {
  SortWork w;
  size_t at = 0;
  const auto take = [&](size_t bytes) { const size_t from = at; at += (bytes + 255) / 256 * 256; return (char *)base + from; };
  w.small = n < DOK_SORT_SMALL;
  const ll_t tile = DOK_SORT_TPB * (w.small ? DOK_SORT_SMALL_ITEMS : DOK_SORT_ITEMS), unique_tile = DOK_TPB * (w.small ? 1 : DOK_UNIQUE_ROUNDS);
  w.tiles = (unsigned)((n + tile - 1) / tile);
  w.unique_tiles = (unsigned)((n + unique_tile - 1) / unique_tile);
  w.control = (SortControl *)take(sizeof(SortControl));
  w.look = (unsigned *)take((size_t)w.tiles * 256 * 4 * sizeof(unsigned));
  w.unique_look = (unsigned *)take((size_t)w.unique_tiles * sizeof(unsigned));
  w.zeroed = at;
  w.key_a = (unsigned *)take((size_t)n * sizeof(unsigned));
  w.row_a = (unsigned *)take((size_t)n * sizeof(unsigned));
  w.key_b = (unsigned *)take((size_t)n * sizeof(unsigned));
  w.row_b = (unsigned *)take((size_t)n * sizeof(unsigned));
  w.bytes = at;
  return w;
}

static unsigned rows_grid(ll_t n, ll_t per_sm = 8) {
  const ll_t blocks = (n + DOK_TPB - 1) / DOK_TPB, quarter = (n + 4 * DOK_TPB - 1) / (4 * DOK_TPB);
  // one per SM first, then four rows per thread: each block adds a thousand digit counts to the batch's
  return (unsigned)(blocks < 148 ? blocks : quarter < 148 ? 148 : quarter < 148 * per_sm ? quarter : 148 * per_sm);
}

// the four passes over one word
static int sort_rows(const SortWork &w, ll_t n, unsigned clumped, cudaStream_t st) {
  int rc;
  k_sort_plan<<<1, 256, 0, st>>>(w.control, (unsigned)n, clumped);
  if ((rc = dok_check_launch()) != DOK_OK) return rc;
  for (int d = 0; d < 4; d++) {
    const auto pass = w.small ? k_sort_pass<DOK_SORT_SMALL_ITEMS> : k_sort_pass<DOK_SORT_ITEMS>;
    pass<<<w.tiles, DOK_SORT_TPB, 0, st>>>(w.control, d, (unsigned)n, w.key_a, w.row_a, w.key_b, w.row_b,
                                           w.look + (size_t)d * w.tiles * 256);
    if ((rc = dok_check_launch()) != DOK_OK) return rc;
  }
  return DOK_OK;
}

static int remove_sorted(const DevTable &dt, const DevHash &dh, const RowKeys &rk, const SortWork &w, uint8_t *out_removed, int64_t *out_count,
                         int64_t *counters, cudaStream_t st) {
  const auto remove = [&](auto kernel) {
    kernel<<<w.unique_tiles, DOK_TPB, 0, st>>>(dt, dh, rk, w.control, w.key_a, w.row_a, w.key_b, w.row_b, w.unique_look, w.unique_tiles,
                                               out_removed, (ll_t *)out_count, (ll_t *)counters);
  };
  DOK_DISPATCH_SB(dt, (w.small ? remove(k_remove_unique<SB, 1>) : remove(k_remove_unique<SB, DOK_UNIQUE_ROUNDS>)));
  return dok_check_launch();
}

extern "C" {

int dok_map_count_new_rows(const dok_table *t, const dok_hash_params *hp, const void *keys, int64_t n,
                           int64_t *scratch, int64_t scratch_slots, int64_t *counters, void *stream) {
  DevHash dh;
  DevTable dt;
  memset(&dt, 0, sizeof(dt));
  if (!dok_make_hash(hp, &dh) || (t && (!dok_make_table(t, &dt) || dt.kb != dh.ks * dh.elem_bytes)) || n < 0 || n > DOK_MAX_BATCH) return DOK_BAD_ARG;
  if (n == 0) return DOK_OK;
  if (!keys || !scratch || !counters || scratch_slots < 2 * n) return DOK_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  if (cudaMemsetAsync(scratch, 0xff, (size_t)scratch_slots * 8, st) != cudaSuccess) return dok_check_launch();
  RowKeys rk{keys, n};
  int rc = DOK_OK;
  DOK_DISPATCH_SB(dt, DOK_FOR_WINDOWS(dt, rc, (k_count_new_rows<SB><<<dok_grid(rk), DOK_TPB, 0, st>>>(
                                                  wt, dh, rk, (ull_t *)scratch, scratch_slots, (ll_t *)counters))));
  return rc;
}

int64_t dok_map_remove_unique_bytes(int64_t n) {
  return n <= DOK_SMALL_ROWS ? 0 : n > DOK_SORT_MAX_ROWS ? -1 : (int64_t)sort_work(nullptr, n).bytes;
}

int dok_map_remove_unique(const dok_table *t, const dok_hash_params *hp, const void *keys, int64_t n, uint8_t *out_removed,
                          void *work, int64_t *out_count, int64_t *counters, void *stream) {
  DevHash dh;
  DevTable dt;
  if (!dok_make_hash(hp, &dh) || !dok_make_table(t, &dt) || dt.kb != dh.ks * dh.elem_bytes || n < 1 || !keys || !out_removed || !out_count)
    return DOK_BAD_ARG;
  if (n > DOK_SORT_MAX_ROWS || dok_window_passes(dt) > 1) return DOK_TOO_LARGE;
  cudaStream_t st = (cudaStream_t)stream;
  RowKeys rk{keys, n};
  if (n <= DOK_SMALL_ROWS) {
    int padded = 1;
    while (padded < n) padded *= 2;
    const int threads = padded < 64 ? 64 : padded < DOK_SMALL_TPB ? padded : DOK_SMALL_TPB;      // fewer wait at the barriers
    DOK_DISPATCH_SB(dt, (k_remove_unique_small<SB><<<1, threads, 0, st>>>(dt, dh, rk, padded, out_removed, (ll_t *)out_count, (ll_t *)counters)));
    return dok_check_launch();
  }
  if (!work) return DOK_BAD_ARG;
  const SortWork w = sort_work(work, n);
  if (cudaMemsetAsync(work, 0, w.zeroed, st) != cudaSuccess) return dok_check_launch();
  int rc;
  const unsigned grid = rows_grid(n);
  k_row_range<<<rows_grid(n, DOK_RANGE_BLOCKS), DOK_TPB, 0, st>>>(rk, dh.dtype, dh.ks, w.control);
  if ((rc = dok_check_launch()) != DOK_OK) return rc;
  k_row_prefix<<<grid, DOK_TPB, 0, st>>>(rk, dh.dtype, dh.ks, w.control, w.key_a, w.row_a);
  if ((rc = dok_check_launch()) != DOK_OK) return rc;
  // A row with m mates (other rows of its prefix) finds one among the rows before it of a block's sample of s rows in
  // s / 2n * m of the cases.  The sort by all words is taken from four mates per row on, on average: below, the runs cost
  // less than the further passes; and from as many as one run of more than DOK_BLOCK_RUN rows gives, which might be refused
  // in the end (at DOK_CLUMPED_MIN such rows chance is out of the question).
  const double block_rows = n < (ll_t)grid * DOK_CLUMP_SLOTS ? (double)n / grid : DOK_CLUMP_SLOTS, samples = block_rows * grid;
  const double one_run = (double)DOK_BLOCK_RUN * DOK_BLOCK_RUN / n, clumped = (one_run < 4 ? one_run : 4) * samples * block_rows / (2.0 * n);
  if ((rc = sort_rows(w, n, clumped < DOK_CLUMPED_MIN ? DOK_CLUMPED_MIN : (unsigned)clumped, st)) != DOK_OK) return rc;
  k_list_ties<<<grid, DOK_TPB, 0, st>>>(w.control, rk, dh.dtype, dh.ks, w.key_a, w.row_a, w.key_b, w.row_b);
  if ((rc = dok_check_launch()) != DOK_OK) return rc;
  k_sort_ties<<<grid < 148 ? grid : 148, DOK_TIES_TPB, 0, st>>>(w.control, rk, dh.dtype, dh.ks, w.key_a, w.row_a, w.key_b, w.row_b);
  if ((rc = dok_check_launch()) != DOK_OK) return rc;
  return remove_sorted(dt, dh, rk, w, out_removed, out_count, counters, st);
}

int dok_map_remove_unique_words(const dok_table *t, const dok_hash_params *hp, const void *keys, int64_t n, uint8_t *out_removed,
                                void *work, int words, int64_t *out_count, int64_t *counters, void *stream) {
  DevHash dh;
  DevTable dt;
  if (!dok_make_hash(hp, &dh) || !dok_make_table(t, &dt) || dt.kb != dh.ks * dh.elem_bytes || n <= DOK_SMALL_ROWS || n > DOK_SORT_MAX_ROWS ||
      !keys || !out_removed || !out_count || !work || words < 2 || words > 2 * DOK_MAX_KEY_SIZE || dok_window_passes(dt) > 1)
    return DOK_BAD_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  RowKeys rk{keys, n};
  const SortWork w = sort_work(work, n);
  const unsigned grid = rows_grid(n);
  int rc;
  for (int word = words - 1; word >= 0; word--) {
    const bool first = word == words - 1;
    const size_t from = first ? offsetof(SortControl, final_b) : offsetof(SortControl, hist);
    if (cudaMemsetAsync((char *)work + from, 0, w.zeroed - from, st) != cudaSuccess) return dok_check_launch();
    k_row_word<<<grid, DOK_TPB, 0, st>>>(rk, dh.dtype, dh.ks, w.control, word, first, w.key_a, w.row_a, w.key_b, w.row_b);
    if ((rc = dok_check_launch()) != DOK_OK) return rc;
    if ((rc = sort_rows(w, n, 0, st)) != DOK_OK) return rc;
  }
  return remove_sorted(dt, dh, rk, w, out_removed, out_count, counters, st);
}

}  // extern "C"
