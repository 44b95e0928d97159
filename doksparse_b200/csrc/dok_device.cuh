// Device-side building blocks shared by the kernels of libdoksparse.so (sm_100a).
//
// Semantics follow the reference's ClosedHashmap class
// (sparse_dok/components/cuda/closed_hashmap_impl_class.cu): key identity is the 64-bit uuid, tags are
// uuid / -1 (empty) / -3 (tombstone), a lookup stops at the first empty tag of its chain and steps over
// tombstones.  What differs on purpose is the memory layout, the start slot and the order of the chain.
//
// Layout.  On B200, when the table is much larger than L2, every load / store / atomic INSTRUCTION-LANE that
// touches it costs the same (~48 G per second over the whole GPU, measured; a second access to a sector that
// was just read costs as much as a new random line), while lanes of one instruction that fall into the same
// 128-byte line count once.  So an operation should touch its line with as few instructions as possible, and
// adjacent lanes should share them.  A slot is {int64 tag | value | key row | stamp (if room)} padded to 32, 64
// or 128 bytes (tag first, value right behind it), a 128-byte line is a GROUP of 4, 2 or 1 slots, and probing
// starts at a group boundary.  The four
// lanes of a quad read one group with ONE coalesced 128-byte request (32 bytes per lane) and resolve a lookup
// from registers: tags, value and key of all its slots are then on chip.  The probe order is a sequence of groups
// (dok_next_group), slot by slot inside each.
#pragma once
#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>
#include "../../include/doksparse.h"

typedef long long ll_t;
typedef unsigned long long ull_t;

#define DOK_EMPTY (-1LL)
#define DOK_REMOVED (-3LL)
#define DOK_TPB 256

// ---------------------------------------------------------------------------------------------------------
// Hash parameters in device-ready form: already permuted by key_perm (element i of the caller's key row uses
// a[i], b[i], p[i]) and with a magic reciprocal per prime so that the truncated remainder needs no division.
// ---------------------------------------------------------------------------------------------------------
struct DevHash {
  int ks;                       // key elements per row
  int dtype;                    // dok_dtype of the key rows
  int elem_bytes;               // bytes of one key element
  int in_order;                 // key_perm is the identity
  ll_t a[DOK_MAX_KEY_SIZE];     // alpha2[key_perm[i]]   -- second hash: the uuid (key identity)
  ll_t b[DOK_MAX_KEY_SIZE];     // beta2[key_perm[i]]
  ull_t p[DOK_MAX_KEY_SIZE];    // |prime2[key_perm[i]]|  (>= 2)
  ull_t m[DOK_MAX_KEY_SIZE];    // floor(2^64 / p)
  ll_t a1[DOK_MAX_KEY_SIZE];    // alpha1[key_perm[i]], forced odd -- first-hash terms: they only decorrelate the
  ll_t b1[DOK_MAX_KEY_SIZE];    // beta1[key_perm[i]]                 probe chains of keys whose uuids collide
  int perm[DOK_MAX_KEY_SIZE];   // storage column of key element i
};

struct KeyHash { ll_t uuid; ll_t hash1; };   // hash1: product of the linear first-hash terms (see dok_start_group)

struct DevTable {
  char *slots;      // n_slots * sb bytes, 128-byte aligned
  ll_t *stamp;      // [n_slots] duplicate-resolution stamps when they do not fit in the slot, else nullptr
  ll_t nb;          // slots the caller sees (0 .. nb-1); slots nb .. n_slots-1 are blocked padding
  ll_t n_slots;     // n_groups * spg
  ll_t n_groups;    // probe groups: 128-byte lines of spg slots (sb <= 128), single slots otherwise
  int sb;           // slot bytes: 32, 64, 128, or a larger multiple of 128
  int spg;          // slots per group: 128 / sb, or 1 for sb > 128
  int vb;           // value bytes
  int kb;           // key row bytes
  int val_off;      // slot offset of the value: always 8, right behind the tag
  int key_off;      // slot offset of the key row: 8 + round_up(vb, 8)
  int stamp_off;    // slot offset of the stamp (behind the key row), -1 when `stamp` is a separate array
  int vwords;       // ceil(vb / 8)
  // Window of probe groups served by this launch; win_hi == 0: the whole table.  A slot array larger than the
  // reach of the GPU's TLB (64 GiB of 2 MiB pages on B200: random reads fall from 45 G/s to 13 G/s at 114 GB) is
  // worked through in passes, each pass taking only the rows whose chain STARTS inside its window, so that one
  // pass touches a range the TLB covers.
  ll_t win_lo, win_hi;
};

#define DOK_BLOCKED (-2LL)   // tag of padding slots: never empty, never a tombstone, never a uuid (uuids are >= 0)

// One factor of the uuid product: ((int64)k * a + b) % p with wrapping arithmetic and the C remainder
// (sign of the dividend), closed_hashmap_impl_class.cu:100,103.  q = mulhi(|x|, floor(2^64/p)) is
// floor(|x|/p) or one less, so a single conditional subtraction finishes the remainder.
__device__ __forceinline__ ll_t dok_uuid_term(ll_t k, ll_t a, ll_t b, ull_t p, ull_t m) {
  const ll_t x = (ll_t)((ull_t)k * (ull_t)a + (ull_t)b);
  const ull_t ux = x < 0 ? (0ULL - (ull_t)x) : (ull_t)x;
  const ull_t q = __umul64hi(ux, m);
  ull_t r = ux - q * p;
  if (r >= p) r -= p;
  return x < 0 ? -(ll_t)r : (ll_t)r;
}

__device__ __forceinline__ ll_t dok_llabs(ll_t v) {  // llabs; INT64_MIN stays INT64_MIN like the device's
  return v < 0 ? (ll_t)(0ULL - (ull_t)v) : v;
}

// `(ll_t) key[i]`: the reference converts key elements by VALUE (closed_hashmap_impl_class.cu:89-103), so a
// float key is truncated toward zero.  The plain C++ casts below compile to the same conversions the
// reference's JIT build uses.
__device__ __forceinline__ ll_t dok_key_elem(const void *keys, int dtype, ll_t idx) {
  switch (dtype) {
    case DOK_I64: return ((const ll_t *)keys)[idx];
    case DOK_I32: return (ll_t)((const int *)keys)[idx];
    case DOK_F32: return (ll_t)((const float *)keys)[idx];
    case DOK_I16: return (ll_t)((const short *)keys)[idx];
    case DOK_I8: return (ll_t)((const signed char *)keys)[idx];
    case DOK_U8: return (ll_t)((const unsigned char *)keys)[idx];
    case DOK_F64: return (ll_t)((const double *)keys)[idx];
    case DOK_F16: return __half2ll_rz(((const __half *)keys)[idx]);
    default: return (ll_t)__bfloat162float(((const __nv_bfloat16 *)keys)[idx]);
  }
}

// Mixer (the 64-bit finaliser of MurmurHash3); with a multiply-high range reduction of its upper half (a table that fits
// a GPU has fewer than 2^31 groups) any table size works without a modulo.
__device__ __forceinline__ ull_t dok_mix64(ull_t h) {
  h ^= h >> 33; h *= 0xff51afd7ed558ccdULL;
  h ^= h >> 33; h *= 0xc4ceb9fe1a85ec53ULL;
  h ^= h >> 33;
  return h;
}
// Start group.  In the reference two keys whose uuids collide are still told apart as long as their probe
// chains (first hash modulo n_buckets) do not meet; a uuid collision is not rare there, because alpha2 may be
// drawn as 0 (cuda_closed_hashmap.py:100), which makes one key element drop out of the uuid.  To keep that
// property the start group mixes the uuid with a second function of the key built from the first hash's
// parameters, prod_i (key_i * (alpha1_i | 1) + beta1_i) (wrapping, no modulo: it only has to differ where the
// keys differ): keys that collide in the uuid alone get unrelated chains.
__device__ __forceinline__ ull_t dok_chain_hash(const KeyHash &h) {
  return dok_mix64((ull_t)h.uuid ^ ((ull_t)h.hash1 * 0x9e3779b97f4a7c15ULL));
}
__device__ __forceinline__ ll_t dok_start_group(const KeyHash &h, const DevTable &t) {
  return (ll_t)__umulhi((unsigned)(dok_chain_hash(h) >> 32), (unsigned)t.n_groups);
}
// Order of a chain's groups.  Plain linear probing piles full groups up into long runs, and every miss walks its run to
// the end: at load 0.9 with 4 slots per group a miss inspects 13.2 groups on average and 300 at most, a hit 2.0; at 0.745
// with 2 slots 4.4 and 1.6.  Here the first DOK_CHAIN_STRIDED steps go by a stride of 1 .. 64 groups taken from the low
// bits of the key's hash (the start comes from the high ones), so that keys which meet in a full group part again: 4.3 /
// 67 / 1.4 groups and 2.6 / 1.4 (simulated over 2^20 groups).  On B200, 44.8 M Zipf lookups of a table at load 0.9 with
// linear probing took 18.9 ms.  The stride is short because a chain has to stay inside the window of a windowed pass, and
// what the TLB covers: at most 64 * 64 groups = 512 KiB from its start.  Then every group is visited in turn, so the walk
// is complete; a table of no more than 64 groups has no room for strides and is walked linearly from the start.
// `word`: bit 31 clear: groups inspected << 6 | stride - 1;  set: groups inspected since the linear part began.
#define DOK_CHAIN_STRIDED 64u
#define DOK_CHAIN_LINEAR 0x80000000u
__device__ __forceinline__ unsigned dok_chain_word(const KeyHash &h, const DevTable &t) {
  return t.n_groups > 64 ? (unsigned)dok_chain_hash(h) & 63u : DOK_CHAIN_LINEAR;
}
// The chain of a key, its hash mixed: for walks that come back to where the chain starts.
struct ChainKey { ll_t uuid; unsigned hash, word; };
__device__ __forceinline__ ChainKey dok_chain(const KeyHash &h, const DevTable &t) {
  const ull_t mixed = dok_chain_hash(h);
  return ChainKey{h.uuid, (unsigned)(mixed >> 32), t.n_groups > 64 ? (unsigned)mixed & 63u : DOK_CHAIN_LINEAR};
}
__device__ __forceinline__ ll_t dok_start_group(const ChainKey &k, const DevTable &t) { return (ll_t)__umulhi(k.hash, (unsigned)t.n_groups); }
__device__ __forceinline__ unsigned dok_chain_word(const ChainKey &k, const DevTable &) { return k.word; }
// steps to the next group of the chain; false when every group has been inspected
template <class Index>
__device__ __forceinline__ bool dok_next_group(Index &group, unsigned &word, Index n_groups) {
  Index step = 1;
  if (word & DOK_CHAIN_LINEAR) {
    if ((Index)(++word & ~DOK_CHAIN_LINEAR) == n_groups) return false;
  } else {
    step += (Index)(word & 63u);
    word += 64u;
    if (word >> 6 == DOK_CHAIN_STRIDED) word = DOK_CHAIN_LINEAR;
  }
  group += step;
  if (group >= n_groups) group -= n_groups;
  return true;
}
// Groups that a key went past.  Lookups of absent keys would inspect every group up to one with an empty slot: at load 0.745
// with 2 slots per group 2.6 of them.  Most full groups hold just the keys that start there, so each group remembers whether a
// key was ever placed behind it: in the highest bit of its first slot's value word, where values of at most 7 bytes leave
// padding and where a lookup has it in a register already.  Insertion sets it, and nothing clears it but a new table; a walk
// that looks for a place ignores it.  A key that was found is marked too: a key of the same uuid whose hash differs has been
// placed from another start (alpha2 = 0 in a column), and a lookup has to get past the groups that this walk went past.
// 8.4 M lookups of a 4-D selection, nearly all misses: 587 -> 402 us; 4 M lookups at load 0.8, 30 % hits: 335 -> 210.  What it
// costs: filling a 4-D tensor with 50 M rows 8.02 -> 8.29 ms (8.63 where the groups are read again for their marks), a table of
// 2 slots per group up to load 0.8 1.60 -> 1.69, of one 2.53 -> 2.71, rebuilt 1.87 -> 2.18 and 2.75 -> 3.14; general sets of
// stored keys 2 to 3 %.  With 4 slots per group fewer keys go past one: at load 0.36 4 M lookups went from 140 to 127 us, but a
// table that grows to 300 k rows from 880 to 910 and a dense tensor's conversion from 348 to 359 (398 where the bit is written
// without a look), so those stay without.
#define DOK_PASSED 0x8000000000000000ULL
__host__ __device__ __forceinline__ bool dok_has_passed_bits(const DevTable &t) { return t.vb < 8 && t.spg <= 2; }
// a key was placed or found in `slot`: marks the groups before it on its chain that the walk saw without the mark (bit k of
// `missing`: the chain's group k; 31: some group from there on)
__device__ __forceinline__ void dok_mark_passed(const DevTable &t, const ChainKey &kh, ll_t slot, unsigned missing) {
  if (!dok_has_passed_bits(t)) return;
  const unsigned placed = (unsigned)slot / (unsigned)t.spg, n_groups = (unsigned)t.n_groups;
  unsigned group = (unsigned)dok_start_group(kh, t), word = dok_chain_word(kh, t);
  while (group != placed) {
    const unsigned step = min(word >> 6, 31u);
    ull_t *first = (ull_t *)(t.slots + (ull_t)group * 128u + 8u);       // (no slot with such a value is wider than a line)
    if (((missing >> step) & 1u) && (step < 31 || !(__ldcg(first) & DOK_PASSED))) atomicOr(first, DOK_PASSED);
    if (!dok_next_group<unsigned>(group, word, n_groups)) break;
  }
}
// does this launch serve the row?  (rows outside the window belong to another pass over the same batch)
__device__ __forceinline__ bool dok_in_window(const DevTable &t, const KeyHash &h, bool active) {
  if (t.win_hi == 0 || !active) return active;
  const ll_t g = dok_start_group(h, t);
  return g >= t.win_lo && g < t.win_hi;
}
#define DOK_SHARD_SALT 0x9e3779b97f4a7c15ULL
__device__ __forceinline__ int dok_owner_shard(ll_t uuid, int n_shards) {
  return (int)__umul64hi(dok_mix64((ull_t)uuid ^ DOK_SHARD_SALT), (ull_t)n_shards);
}

// `n` 8-byte words word(0), word(1), ... to `off` bytes (a multiple of 8) behind a slot's start, which is 32-byte aligned:
// two at a time wherever that is 16-byte aligned.  Every store instruction to a table beyond L2 costs a request per lane,
// so a 40-byte value goes in three instead of five.
template <class Word>
__device__ __forceinline__ void dok_store_words(char *slot, int off, int n, const Word &word) {
  int i = 0;
  if ((off & 8) && n > 0) { *(ull_t *)(slot + off) = word(0); i = 1; }
  for (; i + 1 < n; i += 2) *(ulonglong2 *)(slot + off + 8 * i) = make_ulonglong2(word(i), word(i + 1));
  if (i < n) *(ull_t *)(slot + off + 8 * i) = word(i);
}

// ---------------------------------------------------------------------------------------------------------
// Key sources.  A key source yields, for batch element e, the uuid of its key and can write the key's raw
// bytes into a table key row.  Keys are never held in a register array (key_size is a run-time value):
// elements are re-read where needed, which stays in L1.
// ---------------------------------------------------------------------------------------------------------
struct RowKeys {          // contiguous [n, ks] rows of the key dtype (closed_hashmap_impl.cu:51-60)
  const void *keys;
  ll_t n;
  // Sliced batches (the inbox of a sharded table): the rows come as gridDim.y slices of `slice_rows` rows each, of
  // which only the first slice_counts[y] are in use -- a count that only the DEVICE knows at launch time (another
  // GPU wrote it), so the grid covers whole slices and blocks beyond the count leave at once.  A non-zero *abort
  // (the exchange overflowed somewhere) turns the launch into a no-op.  Batch element e = y * slice_rows + row.
  ll_t slice_rows = 0;
  const ll_t *slice_counts = nullptr;
  const ll_t *abort = nullptr;
  __device__ __forceinline__ ll_t count() const { return n; }
  // batch element of the calling thread and whether it exists
  __device__ __forceinline__ bool row(ll_t &e) const {
    const ll_t j = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x;
    if (slice_rows == 0) { e = j; return j < n; }
    e = (ll_t)blockIdx.y * slice_rows + j;
    return j < slice_rows && j < slice_counts[blockIdx.y];
  }
  __device__ __forceinline__ bool row(ll_t &e, unsigned block) const { return at((ll_t)block * DOK_TPB + threadIdx.x, e); }
  // the same for position j of the batch (of slice blockIdx.y), for kernels that stride over the rows
  __device__ __forceinline__ bool at(ll_t j, ll_t &e) const {
    if (slice_rows == 0) { e = j; return j < n; }
    e = (ll_t)blockIdx.y * slice_rows + j;
    return j < slice_rows && j < slice_counts[blockIdx.y];
  }
  __device__ __forceinline__ ll_t span() const { return slice_rows == 0 ? n : slice_rows; }
  // rows in use (of slice blockIdx.y), and the batch element of one of them
  __device__ __forceinline__ ll_t total() const {
    if (slice_rows == 0) return n;
    if (abort != nullptr && *abort != 0) return 0;
    const ll_t used = slice_counts[blockIdx.y];
    return used < slice_rows ? used : slice_rows;
  }
  __device__ __forceinline__ ll_t elem(unsigned row) const {
    return slice_rows == 0 ? (ll_t)row : (ll_t)blockIdx.y * slice_rows + row;
  }
  // block-uniform: nothing for this block to do
  __device__ __forceinline__ bool idle() const { return idle(blockIdx.x); }
  __device__ __forceinline__ bool idle(unsigned block) const {
    if (slice_rows == 0) return false;
    if (abort != nullptr && *abort != 0) return true;
    return (ll_t)block * DOK_TPB >= slice_counts[blockIdx.y];
  }
  // get_uuid of the reference (closed_hashmap_impl_class.cu:98-107) and the chain-decorrelating product, in one
  // pass over the key
  __device__ __forceinline__ KeyHash hash(const DevHash &hp, ll_t e) const {
    if (hp.ks == 1 && hp.dtype == DOK_I64) {          // the common case, kept free of loops and type dispatch
      const ll_t k = ((const ll_t *)keys)[e];
      return KeyHash{dok_llabs(dok_uuid_term(k, hp.a[0], hp.b[0], hp.p[0], hp.m[0])),
                     (ll_t)((ull_t)k * (ull_t)hp.a1[0] + (ull_t)hp.b1[0])};
    }
    ll_t k = dok_key_elem(keys, hp.dtype, e * hp.ks);
    ll_t u = dok_uuid_term(k, hp.a[0], hp.b[0], hp.p[0], hp.m[0]);
    ull_t h = (ull_t)k * (ull_t)hp.a1[0] + (ull_t)hp.b1[0];
    for (int i = 1; i < hp.ks; i++) {
      k = dok_key_elem(keys, hp.dtype, e * hp.ks + i);
      u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(k, hp.a[i], hp.b[i], hp.p[i], hp.m[i]));
      h *= (ull_t)k * (ull_t)hp.a1[i] + (ull_t)hp.b1[i];
    }
    return KeyHash{dok_llabs(u), (ll_t)h};
  }
  // set_key_permuted (closed_hashmap_impl_class.cu:144-150): storage column perm[i] <- key element i
  __device__ __forceinline__ void store_key(const DevTable &t, const DevHash &hp, ll_t e, char *slot) const {
    const char *src = (const char *)keys + e * (ll_t)hp.ks * hp.elem_bytes;
    char *dst_row = slot + t.key_off;
    if (hp.in_order && hp.elem_bytes >= 4) {
      if (hp.elem_bytes == 8) { dok_store_words(slot, t.key_off, hp.ks, [&](int i) { return ((const ull_t *)src)[i]; }); return; }
      const unsigned *s4 = (const unsigned *)src;
      dok_store_words(slot, t.key_off, hp.ks >> 1, [&](int i) { return (ull_t)s4[2 * i] | (ull_t)s4[2 * i + 1] << 32; });
      if (hp.ks & 1) ((unsigned *)dst_row)[hp.ks - 1] = s4[hp.ks - 1];
      return;
    }
    switch (hp.elem_bytes) {
      case 8: for (int i = 0; i < hp.ks; i++) ((ll_t *)dst_row)[hp.perm[i]] = ((const ll_t *)src)[i]; break;
      case 4: for (int i = 0; i < hp.ks; i++) ((int *)dst_row)[hp.perm[i]] = ((const int *)src)[i]; break;
      case 2: for (int i = 0; i < hp.ks; i++) ((short *)dst_row)[hp.perm[i]] = ((const short *)src)[i]; break;
      default: for (int i = 0; i < hp.ks; i++) dst_row[hp.perm[i]] = src[i]; break;
    }
  }
};

// ndim int64 index tensors (or affine index functions) broadcast to one shape; element e of the row-major linearisation of `sizes`.
// Replaces StrictTensorAccessor::get_index_from_offset + get (tensor_accessor.cu:70-87) as used by
// sparse_dok_tensor_impl.cu:36-42.
struct SelKeys {
  dok_selectors s;
  ll_t n;
  __device__ __forceinline__ ll_t count() const { return n; }
  __device__ __forceinline__ bool row(ll_t &e) const { e = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; return e < n; }
  __device__ __forceinline__ bool at(ll_t j, ll_t &e) const { e = j; return j < n; }
  __device__ __forceinline__ ll_t span() const { return n; }
  __device__ __forceinline__ ll_t total() const { return n; }
  __device__ __forceinline__ ll_t elem(unsigned row) const { return (ll_t)row; }
  __device__ __forceinline__ bool idle(unsigned = 0) const { return false; }
  __device__ __forceinline__ bool row(ll_t &e, unsigned block) const { return at((ll_t)block * DOK_TPB + threadIdx.x, e); }
  __device__ __forceinline__ ll_t index(int d, ll_t off) const { return s.ptr[d] ? s.ptr[d][off] : s.base[d] + off; }
  // Element offsets of batch element e into each of the N index tensors.  N is the number of dims, or the most there can be:
  // the loops are unrolled so that `off` stays in registers, and every dim that is not there would cost its instructions all
  // the same (8 instead of 2: a third of those of a 2-D lookup).
  template <int N>
  __device__ __forceinline__ void offsets(ll_t e, ll_t (&off)[N]) const {
    if (s.selector_ndim == 1) {        // one index tensor per dim, most often: nothing to unravel
#pragma unroll
      for (int d = 0; d < N; d++) off[d] = d < s.ndim ? e * s.strides[d][0] : 0;
      return;
    }
#pragma unroll
    for (int d = 0; d < N; d++) off[d] = 0;
    unsigned rem = (unsigned)e;        // batches have fewer than 2^32 elements; the outermost index is what is left
    for (int j = s.selector_ndim - 1; j >= 0; j--) {
      const unsigned size = (unsigned)s.sizes[j];
      const unsigned q = j > 0 ? rem / size : 0;
      const ll_t idx = (ll_t)(rem - q * size);
      rem = q;
#pragma unroll
      for (int d = 0; d < N; d++) if (d < s.ndim) off[d] += idx * s.strides[d][j];
    }
  }
  template <int N>
  __device__ __forceinline__ KeyHash hash_dims(const DevHash &hp, ll_t e) const {
    ll_t off[N], k[N];
    offsets<N>(e, off);
#pragma unroll
    for (int d = 0; d < N; d++) k[d] = d < s.ndim ? index(d, off[d]) : 0;          // on their way together
    ll_t u = dok_uuid_term(k[0], hp.a[0], hp.b[0], hp.p[0], hp.m[0]);
    ull_t h = (ull_t)k[0] * (ull_t)hp.a1[0] + (ull_t)hp.b1[0];
#pragma unroll
    for (int d = 1; d < N; d++)
      if (d < s.ndim) {
        u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(k[d], hp.a[d], hp.b[d], hp.p[d], hp.m[d]));
        h *= (ull_t)k[d] * (ull_t)hp.a1[d] + (ull_t)hp.b1[d];
      }
    return KeyHash{dok_llabs(u), (ll_t)h};
  }
  __device__ __forceinline__ KeyHash hash(const DevHash &hp, ll_t e) const {
    return s.ndim <= 2 ? hash_dims<2>(hp, e) : s.ndim <= 4 ? hash_dims<4>(hp, e) : hash_dims<DOK_MAX_KEY_SIZE>(hp, e);
  }
  template <int N>
  __device__ __forceinline__ void store_key_dims(const DevTable &t, const DevHash &hp, ll_t e, char *slot) const {
    ll_t off[N];
    offsets<N>(e, off);
    char *dst_row = slot + t.key_off;
    if (hp.in_order && (t.key_off & 8) == 0) {
#pragma unroll
      for (int d = 0; d < N; d += 2) {
        if (d + 1 < s.ndim) *(longlong2 *)(dst_row + 8 * d) = make_longlong2(index(d, off[d]), index(d + 1, off[d + 1]));
        else if (d < s.ndim) *(ll_t *)(dst_row + 8 * d) = index(d, off[d]);
      }
      return;
    }
#pragma unroll
    for (int d = 0; d < N; d++)
      if (d < s.ndim) ((ll_t *)dst_row)[hp.perm[d]] = index(d, off[d]);
  }
  __device__ __forceinline__ void store_key(const DevTable &t, const DevHash &hp, ll_t e, char *slot) const {
    if (s.ndim <= 2) store_key_dims<2>(t, hp, e, slot);
    else store_key_dims<DOK_MAX_KEY_SIZE>(t, hp, e, slot);
  }
};

// ---------------------------------------------------------------------------------------------------------
// Slot access
// ---------------------------------------------------------------------------------------------------------
__device__ __forceinline__ char *dok_slot_ptr(const DevTable &t, ll_t slot) { return t.slots + slot * (ll_t)t.sb; }
__device__ __forceinline__ ll_t *dok_tag_ptr(const DevTable &t, ll_t slot) { return (ll_t *)dok_slot_ptr(t, slot); }
__device__ __forceinline__ ll_t dok_load_tag(const DevTable &t, ll_t slot) {
  return __ldcg(dok_tag_ptr(t, slot));   // L2 is the point of coherence for the CAS claims
}
__device__ __forceinline__ ll_t dok_cas_tag(const DevTable &t, ll_t slot, ll_t expect, ll_t desired) {
  return (ll_t)atomicCAS((ull_t *)dok_tag_ptr(t, slot), (ull_t)expect, (ull_t)desired);
}
__device__ __forceinline__ ll_t *dok_stamp_ptr(const DevTable &t, ll_t slot) {
  return t.stamp_off >= 0 ? (ll_t *)(dok_slot_ptr(t, slot) + t.stamp_off) : t.stamp + slot;
}
__device__ __forceinline__ char *dok_value_ptr(const DevTable &t, ll_t slot) { return dok_slot_ptr(t, slot) + t.val_off; }
__device__ __forceinline__ char *dok_key_row(const DevTable &t, ll_t slot) { return dok_slot_ptr(t, slot) + t.key_off; }

// `nbytes` (1..8) of the little-endian word `w` to dst, with the widest stores the alignment `align` (a power
// of two that divides both dst and nbytes' positions) allows
__device__ __forceinline__ void dok_store_word(char *dst, ull_t w, int nbytes, int align) {
  if (nbytes == 8 && align >= 8) { *(ull_t *)dst = w; return; }
  if (align >= 4) {
    *(unsigned *)dst = (unsigned)w;
    if (nbytes > 4) *(unsigned *)(dst + 4) = (unsigned)(w >> 32);
    return;
  }
  if (align >= 2) {
    for (int i = 0; i < nbytes; i += 2) *(unsigned short *)(dst + i) = (unsigned short)(w >> (8 * i));
    return;
  }
  for (int i = 0; i < nbytes; i++) dst[i] = (char)(w >> (8 * i));
}

// What a walk of one key's chain found.  found >= 0: the slot holding the uuid.  Otherwise `empty` is the first
// empty slot of the chain (-1: the whole table was walked without meeting one) and `tomb` the first tombstone
// met before it (-1: none) -- the two places ClosedHashmap::set may claim (closed_hashmap_impl_class.cu:368-427).
// word: the value word of the slot that ended the walk, for handlers that ask for it.
struct Located { ll_t found, empty, tomb; ull_t word = 0; };

// Walk by ONE lane, the reference's loop (closed_hashmap_impl_class.cu:280-312, 368-407) over this library's chain.
// Used for slots wider than a line (one slot per group).
template <class Key>
__device__ __forceinline__ Located dok_locate_serial(const DevTable &t, const Key &kh, int *probes) {
  Located r{-1, -1, -1};
  ll_t group = dok_start_group(kh, t);
  unsigned word = dok_chain_word(kh, t);
  int n = 0;
  do {
    const ll_t slot = group * t.spg;
    const ll_t tag = dok_load_tag(t, slot);
    n++;
    if (tag == kh.uuid) { r.found = slot; break; }
    if (tag == DOK_EMPTY) { r.empty = slot; break; }
    if (tag == DOK_REMOVED && r.tomb < 0) r.tomb = slot;
  } while (dok_next_group<ll_t>(group, word, t.n_groups));
  if (probes) *probes = n;
  return r;
}

// No-op hit handler for walks that only need the slot.
template <bool FEW>
struct NoEmit {
  static constexpr bool L1 = false, ENDS = false, WORD = false, BOTH = FEW, MARKS = false;
  template <int LW>
  __device__ __forceinline__ void operator()(ll_t, int, const ull_t (&)[LW]) const {}
};

// {tag, value word} of a slot, in one piece: what a 128-bit CAS has written is seen as a whole
__device__ __forceinline__ ulonglong2 dok_load_pair(const char *slot) {
  ulonglong2 v;
  asm volatile("{\n\t.reg .b128 v;\n\tld.relaxed.gpu.global.b128 v, [%2];\n\tmov.b128 {%0, %1}, v;\n\t}" : "=l"(v.x), "=l"(v.y) : "l"(slot));
  return v;
}

// A lookup that only needs the slot.
template <bool FEW>
struct Probe {
  static constexpr bool L1 = true, ENDS = false, WORD = false, BOTH = FEW, MARKS = false;
  template <int LW>
  __device__ __forceinline__ void operator()(ll_t, int, const ull_t (&)[LW]) const {}
};

// A walk whose owner lanes get the value word of the slot that was found, or of the empty one (of 32-byte slots).
template <bool FEW>
struct NeedsWord {
  static constexpr bool L1 = false, ENDS = false, WORD = true, BOTH = FEW, MARKS = false;
  template <int LW>
  __device__ __forceinline__ void operator()(ll_t, int, const ull_t (&)[LW]) const {}
};

// A walk of 64- or 128-byte slots that ends with dok_mark_passed: Located::word has its `missing`.  Lane 1 of the quad, whose part of the line has no tag, reads the word with the mark.
template <bool FEW>
struct Marks {
  static constexpr bool L1 = false, ENDS = false, WORD = false, BOTH = FEW, MARKS = true;
  template <int LW>
  __device__ __forceinline__ void operator()(ll_t, int, const ull_t (&)[LW]) const {}
};

// LW 8-byte words of a line chunk with one load.  Walks that claim or remove read through L2, the point of coherence for
// their CAS.  Lookups change nothing and go through L1: batches of real ids are skewed, and the lines of the popular ones,
// which otherwise come from a single L2 slice each, stay there (39.5 M Zipf(0.99) hits of 16-byte values: 1255 -> 1050 us;
// 33.5 M uniform ones: 987 us either way).
template <int LW, bool L1>
__device__ __forceinline__ void dok_load_words(const char *p, ull_t (&w)[LW]) {
  if constexpr (LW == 4) {
    if constexpr (L1) asm volatile("ld.global.ca.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3]) : "l"(p));
    else asm volatile("ld.global.cg.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(w[0]), "=l"(w[1]), "=l"(w[2]), "=l"(w[3]) : "l"(p));
  } else if constexpr (LW == 2) {
    const ulonglong2 v = L1 ? __ldca((const ulonglong2 *)p) : __ldcg((const ulonglong2 *)p);
    w[0] = v.x; w[1] = v.y;
  } else {
    w[0] = L1 ? __ldca((const ull_t *)p) : __ldcg((const ull_t *)p);
  }
}

// The same walk for the 32 keys of a warp, one 128-byte group per request.  Lane i owns key i.  The four lanes of
// a quad serve the quad's four keys together, in PASSES: in a pass each lane loads, for every key of the quad that
// is still unresolved, the first LW words of its 32 bytes of that key's current group (one coalesced request per
// line: 1 word = the tags only, 2 = tag and an 8-byte value, 4 = everything; all requests of a pass are issued
// before any answer is looked at), compares its tag, and packs one match bit and one empty bit per key and slot
// into ONE 32-bit word (byte r = key r: bits 0-3 match, bits 4-7 empty, by slot).  Two xor-shuffles OR the quad's
// words together; every lane then knows the outcome of all four keys, and the owner lanes advance their own
// state once per pass.  With TOMB the tombstone bits travel in a second word (set needs them, lookups do not).
// The number of dependent memory round trips of a warp is the longest chain among its 32 keys (in groups), and
// rounds in which no quad of the warp has work are skipped (the decision is warp-uniform).
// On a hit, `emit(e_r, slot_in_group, words)` runs on all four lanes while they still hold the line: e_r is the
// batch element of the key, words the calling lane's chunk.
// Every lane of the warp must call this (inactive lanes pass active = false), with CONSECUTIVE batch elements e in
// consecutive lanes.  SB = slot bytes (32, 64, 128).  Slot indices are 32-bit here: the host refuses cooperative
// tables of 2^32 - 1 slots or more.
template <class Emit, int LW>
__device__ __forceinline__ void dok_load_line(const char *p, ull_t (&w)[LW]) {
  if constexpr (Emit::WORD) {
    const ulonglong2 v = dok_load_pair(p);
    w[0] = v.x; w[1] = v.y;
  } else {
    dok_load_words<LW, Emit::L1>(p, w);
  }
}
template <int SB, int LW, bool TOMB, class Key, class Emit>
__device__ __forceinline__ Located dok_locate_quad(const DevTable &t, const Key &kh, ll_t e, bool active,
                                                   int *probes, const Emit &emit) {
  constexpr int SPG = 128 / SB;
  constexpr unsigned FULL = 0xffffffffu;
  constexpr unsigned NONE = 0xffffffffu;              // group index of a lane with nothing (left) to do
  const unsigned lane = threadIdx.x & 31u, l = lane & 3u, base = lane & ~3u;
  const bool has_tag = ((32u * l) % SB) == 0;         // does this lane's chunk start with a slot's tag?
  const unsigned my_slot = (32u * l) / SB;            // slot (within the group) the chunk belongs to
  const ll_t e_quad = e - l;                          // batch element of the quad's first lane (elements are consecutive)
  const unsigned n_groups = (unsigned)t.n_groups;     // < 2^32 (checked on the host)
  static_assert(!Emit::MARKS || (SB >= 64 && LW == 1));
  const char *my_base = t.slots + (Emit::MARKS && l == 1 ? 8 : 32 * l);
  constexpr unsigned SLOTS = Emit::MARKS ? (1u << SPG) - 1u : 0xfu, UNMARKED = 8u;
  ull_t word_of = 0;
  // results as 32-bit group-relative codes until the end: slot = group * SPG + position
  unsigned found = NONE, empty = NONE, tomb = NONE;
  unsigned group = NONE, word = 0, walked = 0;
  if (active) {
    group = (unsigned)dok_start_group(kh, t);
    word = dok_chain_word(kh, t);
  }

  // a group that no key went past ends a chain like an empty last slot (in the bits of its first slot's lane)
  auto ends = [&](const ull_t (&w)[LW]) -> unsigned { return l == 0 && !(w[LW > 1 ? 1 : 0] & DOK_PASSED) ? 1u << (3 + SPG) : 0u; };

  // what the owner lane does with the outcome of one inspected group: m / me / tb = match, match-or-empty and
  // tombstone bits by slot
  auto advance = [&](unsigned m, unsigned me, unsigned tb) {
    const int pos = (me & SLOTS) ? __ffs(me & SLOTS) - 1 : -1;
    if (Emit::MARKS && pos < 0 && (m & UNMARKED)) word_of |= 1u << min(word >> 6, 31u);
    const unsigned first_slot = group * SPG;
    if (probes) walked++;
    if (TOMB && tomb == NONE) {
      const unsigned before = pos >= 0 ? (tb & ((1u << pos) - 1u)) : tb;
      if (before) tomb = first_slot + __ffs(before) - 1;
    }
    if (pos >= 0) {
      if ((m >> pos) & 1u) found = first_slot + pos; else empty = first_slot + pos;
      group = NONE;
    } else if (!dok_next_group<unsigned>(group, word, n_groups)) {
      group = NONE;                                   // every group inspected: no empty slot anywhere
    }
  };

  // ---- a group of each of the quad's four keys: four requests in flight, one packed exchange
  auto inspect_all = [&]() {
    ull_t w[4][LW];
    unsigned g[4];
#pragma unroll
    for (unsigned r = 0; r < 4; r++) {
      g[r] = __shfl_sync(FULL, group, base + r);
      if (g[r] != NONE) dok_load_line<Emit>(my_base + (ull_t)g[r] * 128u, w[r]);
    }
    unsigned bits = 0, tbits = 0;
#pragma unroll
    for (unsigned r = 0; r < 4; r++) {
      const ll_t uuid_r = __shfl_sync(FULL, kh.uuid, base + r);
      if (has_tag && g[r] != NONE) {
        const ll_t tag = (ll_t)w[r][0];
        bits |= ((unsigned)(tag == uuid_r) | ((unsigned)(tag == DOK_EMPTY) << 4)) << (8u * r + my_slot);
        if constexpr (Emit::ENDS) bits |= ends(w[r]) << (8u * r);
        if (TOMB) tbits |= (unsigned)(tag == DOK_REMOVED) << (4u * r + my_slot);
      }
      if constexpr (Emit::MARKS) if (l == 1 && g[r] != NONE && !(w[r][0] & DOK_PASSED)) bits |= UNMARKED << (8u * r);
    }
    bits |= __shfl_xor_sync(FULL, bits, 1);
    bits |= __shfl_xor_sync(FULL, bits, 2);
    if (TOMB) {
      tbits |= __shfl_xor_sync(FULL, tbits, 1);
      tbits |= __shfl_xor_sync(FULL, tbits, 2);
    }
#pragma unroll
    for (unsigned r = 0; r < 4; r++) {                // hits: hand the line to the emitter while it is in registers
      const unsigned m = (bits >> (8u * r)) & 0xfu, me = (m | (bits >> (8u * r + 4u))) & 0xfu;
      if (me) {
        const int pos = __ffs(me) - 1;
        if ((m >> pos) & 1u) emit(e_quad + r, pos, w[r]);
      }
    }
    if constexpr (Emit::WORD) {
#pragma unroll
      for (unsigned r = 0; r < 4; r++) {
        const unsigned me = ((bits >> (8u * r)) | (bits >> (8u * r + 4u))) & 0xfu;
        const ull_t v = __shfl_sync(FULL, w[r][LW - 1], base + (me ? __ffs(me) - 1 : 0));
        if (l == r && group != NONE) word_of = v;
      }
    }
    if (group != NONE) {
      const unsigned mine = bits >> (8u * l);
      advance(mine & 0xfu, (mine | (mine >> 4)) & 0xfu, TOMB ? (tbits >> (4u * l)) & 0xfu : 0u);
    }
  };

  // ---- of one of them
  auto inspect_one = [&](unsigned pend) {
    const unsigned quad = (pend >> base) & 0xfu;
    const unsigned r = quad ? (unsigned)(__ffs(quad) - 1) : 0u;     // the quad's lowest unfinished key
    unsigned g_r = __shfl_sync(FULL, group, base + r);
    if (!quad) g_r = NONE;
    const ll_t uuid_r = __shfl_sync(FULL, kh.uuid, base + r);
    ull_t wl[LW];
    if (g_r != NONE) dok_load_line<Emit>(my_base + (ull_t)g_r * 128u, wl);
    const ll_t tag = (has_tag && g_r != NONE) ? (ll_t)wl[0] : DOK_BLOCKED;
    unsigned bits = ((unsigned)(tag == uuid_r) | ((unsigned)(tag == DOK_EMPTY) << 4) |
                     (TOMB ? (unsigned)(tag == DOK_REMOVED) << 8 : 0u)) << my_slot;
    if constexpr (Emit::ENDS) if (g_r != NONE) bits |= ends(wl);
    if constexpr (Emit::MARKS) if (l == 1 && g_r != NONE && !(wl[0] & DOK_PASSED)) bits |= UNMARKED;
    bits |= __shfl_xor_sync(FULL, bits, 1);
    bits |= __shfl_xor_sync(FULL, bits, 2);
    const unsigned m = bits & 0xfu, me = (bits | (bits >> 4)) & 0xfu;
    if (me) {
      const int pos = __ffs(me) - 1;
      if ((m >> pos) & 1u) emit(e_quad + r, pos, wl);
    }
    if constexpr (Emit::WORD) {
      const ull_t v = __shfl_sync(FULL, wl[LW - 1], base + (me ? __ffs(me) - 1 : 0));
      if (l == r && group != NONE) word_of = v;
    }
    if (l == r && group != NONE) advance(m, me, (bits >> 8) & 0xfu);
  };

  // Keys whose chain runs into further groups.  A large batch, which keeps the memory busy, has the fewest instructions with
  // one key per quad and iteration.  A small one waits for the iterations: all of the quad's keys at once while a quad has
  // more than one (sets of 30 k rows of 64-byte slots at load 0.65 55 -> 49 us, lookups 31 -> 27; no difference at 300 k rows;
  // sets of 33.5 M rows 2694 -> 2713).
  if constexpr (Emit::BOTH) {
    unsigned pend = FULL;
    for (bool all = true;;) {
      if (all) inspect_all(); else inspect_one(pend);
      pend = __ballot_sync(FULL, group != NONE);
      if (pend == 0) break;
      const unsigned per_quad = (pend & 0x11111111u) + ((pend >> 1) & 0x11111111u) + ((pend >> 2) & 0x11111111u) + ((pend >> 3) & 0x11111111u);
      all = (per_quad & 0x66666666u) != 0;
    }
  } else {
    inspect_all();
    while (const unsigned pend = __ballot_sync(FULL, group != NONE)) inspect_one(pend);
  }
  if (probes) *probes = (int)walked;
  Located res;
  res.found = found == NONE ? -1 : (ll_t)found;
  res.empty = empty == NONE ? -1 : (ll_t)empty;
  res.tomb = tomb == NONE ? -1 : (ll_t)tomb;
  res.word = word_of;
  return res;
}

// Hit handler of `get` (PASSED: of a table whose groups remember that a key went past them): the lane that holds the slot
// writes the value straight from its registers, so a hit needs no second access to the table.  LW = 2 serves values of at
// most 8 bytes, one word behind the tag, LW = 4 whole slots, each lane of the quad with its part of the value.
template <int SB, int LW, bool PASSED>
struct EmitValue {
  static constexpr bool L1 = true, ENDS = PASSED, WORD = false, BOTH = false, MARKS = false;
  const DevTable &t;
  char *out_values;
  __device__ __forceinline__ void operator()(ll_t e_r, int pos, const ull_t (&w)[LW]) const {
    char *dst = out_values + e_r * (ll_t)t.vb;
    if constexpr (LW == 4 && SB != 32) {                   // (128-byte slots of values that fill more than half of them)
      const int start = pos * SB + 8 - 32 * (int)(threadIdx.x & 3u);      // of the value, from this lane's part of the line
      const int align = (t.vb & 7) ? t.vb & -t.vb : 8;
#pragma unroll
      for (int j = 0; j < LW; j++) {
        const int at = 8 * j - start;
        if ((unsigned)at >= (unsigned)t.vb) continue;
        if (align == 8) *(ull_t *)(dst + at) = w[j];
        else dok_store_word(dst + at, w[j], t.vb - at < 8 ? t.vb - at : 8, align);
      }
      return;
    }
    if ((int)(threadIdx.x & 3u) != pos * (SB / 32)) return;
    if constexpr (LW == 2) {
      if (t.vb == 8) *(ull_t *)dst = w[1];
      else dok_store_word(dst, w[1], t.vb, (t.vb & -t.vb));
    } else if ((t.vb & 7) == 0) {
#pragma unroll
      for (int j = 1; j < LW; j++) if (8 * j <= t.vb) *(ull_t *)(dst + 8 * j - 8) = w[j];
    } else if ((t.vb & 3) == 0) {
#pragma unroll
      for (int j = 1; j < LW; j++) {
        if (8 * j - 4 <= t.vb) *(unsigned *)(dst + 8 * j - 8) = (unsigned)w[j];
        if (8 * j <= t.vb) *(unsigned *)(dst + 8 * j - 4) = (unsigned)(w[j] >> 32);
      }
    } else {
      const int align = t.vb & -t.vb;
#pragma unroll
      for (int j = 1; j < LW; j++)
        if (8 * j - 8 < t.vb) dok_store_word(dst + 8 * j - 8, w[j], t.vb - 8 * j + 8 < 8 ? t.vb - 8 * j + 8 : 8, align);
    }
  }
};

// SB == 0 selects the serial walk (slots wider than one line); emit is not called there.
template <int SB, int LW, bool TOMB, class Key, class Emit>
__device__ __forceinline__ Located dok_locate(const DevTable &t, const Key &kh, ll_t e, bool active, int *probes,
                                              const Emit &emit) {
  if constexpr (SB == 0) {
    if (probes) *probes = 0;
    Located r{-1, -1, -1};
    if (active) r = dok_locate_serial(t, kh, probes);
    // The lanes leave the walk one by one; what comes next is for all of them together.  Without this, the copy of a
    // 160-byte value ran in several turns: 10,000 lookups at load 0.6 made 43 requests per warp instead of 30.
    __syncwarp();
    return r;
  } else {
    return dok_locate_quad<SB, LW, TOMB>(t, kh, e, active, probes, emit);
  }
}

enum { DOK_OUT_FOUND = 0, DOK_OUT_CLAIMED_EMPTY = 1, DOK_OUT_REUSED = 2, DOK_OUT_FAILED = 3 };

// Insert-or-find by one lane, slot by slot.  Phase 1 walks the chain: a matching tag is a hit; at the first empty tag the slot
// is claimed by CAS unless a tombstone was seen.  Phase 2 walks it again and takes the first slot that is free, tombstone or
// empty.  missing: of dok_mark_passed.
template <bool MARKS>
static __device__ __forceinline__ ll_t dok_find_or_claim_serial(const DevTable &t, const KeyHash &kh, int *outcome, unsigned *missing) {
  const ll_t uuid = kh.uuid;
  bool reuse = false;                                    // a tombstone was seen
  for (int phase = 0; phase < 2; phase++) {
    ll_t group = dok_start_group(kh, t);
    unsigned word = dok_chain_word(kh, t);
    *missing = 0;
    bool more = true;
    while (more) {
      for (int i = 0; i < t.spg && more; i++) {
        const ll_t slot = group * t.spg + i;
        ll_t tag = dok_load_tag(t, slot);
        if (tag == DOK_REMOVED && phase == 0) reuse = true;
        if (tag == DOK_EMPTY && phase == 0 && reuse) { more = false; break; }
        if (tag == DOK_EMPTY || (tag == DOK_REMOVED && phase == 1)) {
          const ll_t old = dok_cas_tag(t, slot, tag, uuid);
          if (old == tag) { *outcome = tag == DOK_EMPTY ? DOK_OUT_CLAIMED_EMPTY : DOK_OUT_REUSED; return slot; }
          tag = old;
        }
        if (tag == uuid) { *outcome = DOK_OUT_FOUND; return slot; }
      }
      if (MARKS && more && !(__ldcg((const ull_t *)(t.slots + (ull_t)group * 128u + 8u)) & DOK_PASSED)) *missing |= 1u << min(word >> 6, 31u);
      more = more && dok_next_group<ll_t>(group, word, t.n_groups);
    }
    if (!reuse) break;
  }
  *outcome = DOK_OUT_FAILED;
  return -1;
}

// Insert-or-find for the 32 keys of a warp (ClosedHashmap::set, closed_hashmap_impl_class.cu:368-427, without the row
// stores): one cooperative walk tells every owner lane where its uuid is or where the chain offers a place (first tombstone,
// else first empty slot); the owner claims that place with one CAS.  Losing the CAS to the same uuid means a twin row of the
// batch claimed it: join.  Losing it to another uuid means another walk for that lane: no slot becomes free while a set runs,
// so each lost CAS is a slot taken.  In a table that fills up that is no exception -- the rows that are on their way at a time
// see the same first places -- and a lane that went on by itself, slot by slot, held its warp up: sets of a fifth new rows,
// 300 k rows of 32-byte slots 60 -> 54 us, 1 M 113 -> 107, 30 k rows of 64-byte slots 59 -> 48.  Every lane of the warp must call.
// ORDERED: keys in the order of the table, whose lanes compete for the places of their group on every walk: those that lose go
// on by themselves (rebuild of 11.7 M rows in 32-byte slots 1535 -> 1430 us, in 64-byte slots 2020 -> 1904).
// MARKS: the table may be one with marks.
template <int SB, bool FEW = false, bool MARKS = (SB >= 64), bool ORDERED = false>
__device__ __forceinline__ ll_t dok_find_or_claim(const DevTable &t, const KeyHash &kh, bool active, int *outcome) {
  ll_t slot = -1;
  do {
    const Located loc = dok_locate<SB, 1, true>(t, kh, 0, active, nullptr, std::conditional_t<MARKS, Marks<FEW>, NoEmit<FEW>>());
    if (active) {
      active = false;
      slot = loc.found;
      *outcome = DOK_OUT_FOUND;
      unsigned missing = (unsigned)loc.word;
      if (slot < 0) {
        slot = loc.tomb >= 0 ? loc.tomb : loc.empty;
        const ll_t expect = loc.tomb >= 0 ? DOK_REMOVED : DOK_EMPTY;
        if (slot < 0) {
          *outcome = DOK_OUT_FAILED;                     // no match, no tombstone, no empty slot: the table is full
        } else {
          const ll_t old = dok_cas_tag(t, slot, expect, kh.uuid);
          if (old == expect) {
            *outcome = expect == DOK_EMPTY ? DOK_OUT_CLAIMED_EMPTY : DOK_OUT_REUSED;
          } else {
            active = old != kh.uuid;
            if constexpr (ORDERED)
              if (active) {
                slot = dok_find_or_claim_serial<MARKS>(t, kh, outcome, &missing);
                active = false;
              }
          }
        }
      }
      if constexpr (MARKS) if (missing && !active && slot >= 0) dok_mark_passed(t, dok_chain(kh, t), slot, missing);
    }
  } while (__any_sync(0xffffffffu, active));
  return slot;
}

// value row (vb bytes at `src`, alignment of the widest power of two dividing vb, capped at 8) -> slot
__device__ __forceinline__ void dok_store_value(const DevTable &t, ll_t slot, const char *src) {
  char *dst = dok_value_ptr(t, slot);
  if (t.vb == 8) { *(ull_t *)dst = *(const ull_t *)src; return; }
  if (t.vb == 4) { *(unsigned *)dst = *(const unsigned *)src; return; }
  if ((t.vb & 7) == 0) {
    dok_store_words(dok_slot_ptr(t, slot), t.val_off, t.vwords, [&](int i) { return ((const ull_t *)src)[i]; });
  } else if ((t.vb & 3) == 0) {
    const unsigned *s4 = (const unsigned *)src;
    dok_store_words(dok_slot_ptr(t, slot), t.val_off, t.vb >> 3, [&](int i) { return (ull_t)s4[2 * i] | (ull_t)s4[2 * i + 1] << 32; });
    ((unsigned *)dst)[(t.vb >> 2) - 1] = s4[(t.vb >> 2) - 1];
  } else if ((t.vb & 1) == 0) {
    unsigned short *d16 = (unsigned short *)dst;
    for (int w = 0; w < (t.vb >> 1); w++) d16[w] = ((const unsigned short *)src)[w];
  } else {
    for (int w = 0; w < t.vb; w++) dst[w] = src[w];
  }
}

// slot -> value row
__device__ __forceinline__ void dok_load_value(const DevTable &t, ll_t slot, char *dst) {
  const ull_t *src = (const ull_t *)dok_value_ptr(t, slot);
  if (t.vb == 8) { *(ull_t *)dst = __ldcg(src); return; }
  if (t.vb == 4) { *(unsigned *)dst = __ldcg((const unsigned *)src); return; }
  if ((t.vb & 7) == 0) {
    for (int w = 0; w < t.vwords; w++) ((ull_t *)dst)[w] = __ldcg(src + w);
  } else if ((t.vb & 3) == 0) {
    for (int w = 0; w < (t.vb >> 2); w++) ((unsigned *)dst)[w] = __ldcg((const unsigned *)src + w);
  } else if ((t.vb & 1) == 0) {
    for (int w = 0; w < (t.vb >> 1); w++) ((unsigned short *)dst)[w] = __ldcg((const unsigned short *)src + w);
  } else {
    for (int w = 0; w < t.vb; w++) dst[w] = __ldcg((const char *)src + w);
  }
}
// ... of more than 8 bytes, for slots found at random: through L1, up to eight pieces on their way together
template <class T>
__device__ __forceinline__ void dok_fetch_pieces(const T *src, T *dst, int n) {
  for (int i = 0; i < n; i += 8) {
    T v[8];
#pragma unroll
    for (int k = 0; k < 8; k++) if (i + k < n) v[k] = __ldca(src + i + k);
#pragma unroll
    for (int k = 0; k < 8; k++) if (i + k < n) dst[i + k] = v[k];
  }
}
__device__ __forceinline__ void dok_fetch_value(const DevTable &t, ll_t slot, char *dst) {
  const char *src = (const char *)dok_value_ptr(t, slot);
  if ((t.vb & 7) == 0) dok_fetch_pieces((const ull_t *)src, (ull_t *)dst, t.vwords);
  else if ((t.vb & 3) == 0) dok_fetch_pieces((const unsigned *)src, (unsigned *)dst, t.vb >> 2);
  else if ((t.vb & 1) == 0) dok_fetch_pieces((const unsigned short *)src, (unsigned short *)dst, t.vb >> 1);
  else dok_fetch_pieces((const unsigned char *)src, (unsigned char *)dst, t.vb);
}

struct Fallback { ull_t w[DOK_MAX_VALUE_BYTES / 8]; };   // miss fill, passed by value

__device__ __forceinline__ void dok_store_fallback(const DevTable &t, const Fallback &fb, char *dst) {
  const char *src = (const char *)fb.w;
  if (t.vb == 8) { *(ull_t *)dst = fb.w[0]; return; }
  if (t.vb == 4) { *(unsigned *)dst = (unsigned)fb.w[0]; return; }
  if ((t.vb & 7) == 0) {
    for (int w = 0; w < t.vwords; w++) ((ull_t *)dst)[w] = fb.w[w];
  } else if ((t.vb & 3) == 0) {
    for (int w = 0; w < (t.vb >> 2); w++) ((unsigned *)dst)[w] = ((const unsigned *)src)[w];
  } else if ((t.vb & 1) == 0) {
    for (int w = 0; w < (t.vb >> 1); w++) ((unsigned short *)dst)[w] = ((const unsigned short *)src)[w];
  } else {
    for (int w = 0; w < t.vb; w++) dst[w] = src[w];
  }
}

// Per-launch counters.  The counters of a launch are a handful of global addresses, and atomics on one address are
// served one after the other, so a million per-warp atomics on one word cost about as much as the probing itself.
// A block therefore tallies in shared memory (one vote and one shared atomic per warp and counter) and the LAST warp
// of the block to finish adds the block's totals to global memory: one global atomic per block and counter, and no
// barrier at the end of the kernel, where warps finish at very different times.
// Slots 0 .. 7 go to counters[slot] (the dok_counter indices), slot 8 to `extra`.  Every thread of the block must
// call begin and flush, and every lane of a warp must call add together.
#define DOK_TALLY_SLOTS 9
#define DOK_TALLY_EXTRA 8
struct BlockTally { int v[DOK_TALLY_SLOTS]; int done; };

__device__ __forceinline__ void dok_tally_begin(BlockTally &b) {
  if (threadIdx.x < DOK_TALLY_SLOTS) b.v[threadIdx.x] = 0;
  if (threadIdx.x == DOK_TALLY_SLOTS) b.done = 0;
  __syncthreads();
}
__device__ __forceinline__ void dok_tally_add(BlockTally &b, int slot, int pred) {
  const unsigned m = __ballot_sync(0xffffffffu, pred);
  if ((threadIdx.x & 31) == 0 && m) atomicAdd(&b.v[slot], __popc(m));
}
__device__ __forceinline__ void dok_tally_flush(BlockTally &b, ll_t *counters, ll_t *extra) {
  __syncwarp();
  int last = 0;
  if ((threadIdx.x & 31) == 0) {
    __threadfence_block();
    last = atomicAdd(&b.done, 1) == (int)(blockDim.x >> 5) - 1;
  }
  last = __shfl_sync(0xffffffffu, last, 0);
  if (!last) return;
  const int k = threadIdx.x & 31;
  if (k < DOK_TALLY_SLOTS) {
    const int c = ((volatile int *)b.v)[k];
    ll_t *dst = k < DOK_TALLY_EXTRA ? (counters ? counters + k : nullptr) : extra;
    if (c && dst) atomicAdd((ull_t *)dst, (ull_t)c);
  }
}

// warp sum + one atomicAdd per warp (replaces warp_sum + atomicAdd of sparse_dok_tensor_impl.cu:52-55).
// Every lane of the warp must call it.
__device__ __forceinline__ void dok_warp_add(ll_t *counter, int v) {
  if (counter == nullptr) return;
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0 && v) atomicAdd((ull_t *)counter, (ull_t)v);
}
