// C-ABI entry points of the fused DOK tensor paths (declared in include/doksparse.h): the keys of a batch are
// formed on the fly from broadcast index tensors (or from the position of a non-zero element of a dense
// tensor) instead of being materialised as an int64[n, ndim] matrix first.
#include "dok_kernels.cuh"

// dense source of __setitem__ viewed through the selector's common shape (strides in elements, 0 = broadcast);
// replaces the extra StrictTensorAccessor of sparse_dok_set_items_dense (sparse_dok_tensor_impl.cu:290,309).
struct StridedValues {
  const char *src;
  int selector_ndim;
  ll_t sizes[DOK_MAX_SELECTOR_NDIM];
  ll_t strides[DOK_MAX_SELECTOR_NDIM];
  __device__ __forceinline__ const char *row(const DevTable &t, ll_t e) const {
    if (selector_ndim == 1) return src + e * strides[0] * (ll_t)t.vb;
    unsigned rem = (unsigned)e;        // batches have fewer than 2^32 elements
    ll_t off = 0;
    for (int j = selector_ndim - 1; j >= 0; j--) {
      const unsigned size = (unsigned)sizes[j];
      const unsigned q = j > 0 ? rem / size : 0;
      off += (ll_t)(rem - q * size) * strides[j];
      rem = q;
    }
    return src + off * (ll_t)t.vb;
  }
};

static bool prepare(const dok_table *t, const dok_hash_params *hp, DevTable *dt, DevHash *dh) {
  if (!dok_make_hash(hp, dh) || !dok_make_table(t, dt)) return false;
  return dt->kb == dh->ks * dh->elem_bytes;
}


static bool make_sel(const dok_selectors *sel, const DevHash &dh, SelKeys *out) {
  if (!sel || sel->ndim != dh.ks || dh.dtype != DOK_I64) return false;
  if (sel->selector_ndim < 0 || sel->selector_ndim > DOK_MAX_SELECTOR_NDIM) return false;
  ll_t n = 1;
  for (int j = 0; j < sel->selector_ndim; j++) {
    if (sel->sizes[j] < 0) return false;
    n *= sel->sizes[j];
  }
  out->s = *sel;
  out->n = n;
  return n <= DOK_MAX_BATCH;
}

// ---- from_dense ------------------------------------------------------------------------------------------

template <typename T>
__device__ __forceinline__ bool dok_nonzero(T bits, int is_float) {
  // `x != 0`: for floating types both signed zeros compare equal to zero, NaN does not
  return is_float ? (T)(bits << 1) != 0 : bits != 0;
}

template <typename T>
__global__ void __launch_bounds__(DOK_TPB) k_dense_count(const T *__restrict__ dense, ll_t numel, int is_float, ll_t *count_out) {
  int c = 0;
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB;
  for (ll_t i = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; i < numel; i += stride) c += dok_nonzero<T>(__ldcs(dense + i), is_float);
  dok_warp_add(count_out, c);
}

struct DenseShape { int ndim; ll_t sizes[DOK_MAX_KEY_SIZE]; };

// The count that keeps what it finds: positions and values of the non-zeros, in no particular order, as far as the list
// goes.  The insertion then reads the list, not the tensor, and every thread of it has a row: 8192^2 f32 at 1 %, count 47 and
// insertion 127 us; here 59 and 52.  A lane reads 32 bytes of its warp's span at a time (16 of bytes), the next ones on their
// way meanwhile; the non-zeros collect in the warp's list and leave from DOK_COLLECT_FLUSH on, with one atomic.
// A list that will not hold them all is of no use and takes longer than the count: from_dense of 8192^2 f32 at 20 % 1,925 us
// with it, 1,874 without.  So the launch before, which sets the count to zero, looks at 16-byte pieces that are spread over the
// tensor, and where they hold an eighth more than the list would, its mark in the count says to count only: 1,872.  (The look
// by a block of this kernel, and a loop that ends when the mark appears or the list is full: 59 -> 62 us.)
#define DOK_COLLECT_FLUSH 128
#define DOK_COLLECT_BLOCKS 6

#define DOK_LOOK_PIECES 1024

template <typename T>
__global__ void __launch_bounds__(DOK_LOOK_PIECES) k_dense_look(const T *__restrict__ dense, ll_t numel, int is_float, ll_t capacity, ll_t *count) {
  constexpr int EACH = 16 / (int)sizeof(T);
  __shared__ int sampled;
  if (threadIdx.x == 0) sampled = 0;
  __syncthreads();
  if (numel > capacity && numel >= DOK_LOOK_PIECES * EACH) {
    const ull_t spacing = (ull_t)(numel / EACH) / DOK_LOOK_PIECES;      // each piece lies anywhere in its share of the tensor
    union { uint4 q; T v[EACH]; } look;
    look.q = __ldg((const uint4 *)dense + (threadIdx.x * spacing + (spacing * (threadIdx.x * 0x9e3779b1u) >> 32)));
    int c = 0;
#pragma unroll
    for (int j = 0; j < EACH; j++) c += dok_nonzero<T>(look.v[j], is_float);
    c = __reduce_add_sync(0xffffffffu, c);
    if ((threadIdx.x & 31) == 0) atomicAdd(&sampled, c);
  }
  __syncthreads();
  if (threadIdx.x == 0) *count = (ll_t)sampled * numel > (capacity + capacity / 8) * (DOK_LOOK_PIECES * EACH) ? DOK_UNLISTED : 0;
}

template <typename T>
__global__ void __launch_bounds__(DOK_TPB, DOK_COLLECT_BLOCKS) k_dense_collect(const T *__restrict__ dense, ll_t numel, int is_float, unsigned *__restrict__ at_out,
                                                                               T *__restrict__ value_out, ll_t capacity, ll_t *count) {
  constexpr int PIECES = sizeof(T) == 1 ? 1 : 2, EACH = 16 / (int)sizeof(T), SPAN = 32 * PIECES * EACH;
  __shared__ unsigned list_at[DOK_WARPS][DOK_COLLECT_FLUSH + SPAN];
  __shared__ T list_value[DOK_WARPS][DOK_COLLECT_FLUSH + SPAN];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  unsigned *const found_at = list_at[warp];
  T *const found_value = list_value[warp];
  const ll_t first = ((ll_t)blockIdx.x * DOK_WARPS + warp) * SPAN, stride = (ll_t)gridDim.x * DOK_WARPS * SPAN;
  union Piece { uint4 q; T v[EACH]; };
  Piece p[PIECES];
  int total = 0;
  const auto fetch = [&](ll_t base) {
#pragma unroll
    for (int k = 0; k < PIECES; k++) {
      const ll_t i = base + (k * 32 + lane) * EACH;
      if (i + EACH <= numel) {
        p[k].q = __ldcs((const uint4 *)(dense + i));
      } else {
#pragma unroll
        for (int j = 0; j < EACH; j++) p[k].v[j] = i + j < numel ? dense[i + j] : (T)0;
      }
    }
  };
  const auto flush = [&]() {
    __syncwarp();
    ll_t to = 0;
    if (lane == 0) to = (ll_t)atomicAdd((ull_t *)count, (ull_t)total);
    to = __shfl_sync(0xffffffffu, to, 0);
    for (int i = lane; i < total; i += 32)
      if (to + i < capacity) {
        at_out[to + i] = found_at[i];
        value_out[to + i] = found_value[i];
      }
    __syncwarp();
    total = 0;
  };
  const ll_t mark = __ldca(count);       // through L1: from L2 the one line takes 7104 warps 2 us
  fetch(first);
  if (mark & DOK_UNLISTED) {
    int c = 0;
    for (ll_t i = ((ll_t)blockIdx.x * DOK_TPB + threadIdx.x) * EACH; i < numel; i += (ll_t)gridDim.x * DOK_TPB * EACH) {
      union { uint4 q; T v[EACH]; } piece;
      if (i + EACH <= numel) {
        piece.q = __ldcs((const uint4 *)(dense + i));
#pragma unroll
        for (int j = 0; j < EACH; j++) c += dok_nonzero<T>(piece.v[j], is_float);
      } else {
        for (ll_t k = i; k < numel; k++) c += dok_nonzero<T>(dense[k], is_float);
      }
    }
    dok_warp_add(count, c);
    return;
  }
  for (ll_t base = first; base < numel; base += stride) {                                 // uniform over the warp
    Piece now[PIECES];
    unsigned nonzero = 0;
#pragma unroll
    for (int k = 0; k < PIECES; k++) {
      now[k].q = p[k].q;
#pragma unroll
      for (int j = 0; j < EACH; j++) nonzero |= (unsigned)dok_nonzero<T>(now[k].v[j], is_float) << (k * EACH + j);
    }
    fetch(base + stride);
    if (!__any_sync(0xffffffffu, nonzero)) continue;
    const int own = __popc(nonzero);
    int upto = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int u = __shfl_up_sync(0xffffffffu, upto, o);
      if (lane >= o) upto += u;
    }
    int at = total + upto - own;
#pragma unroll
    for (int k = 0; k < PIECES; k++)
#pragma unroll
      for (int j = 0; j < EACH; j++)
        if ((nonzero >> (k * EACH + j)) & 1u) {
          found_value[at] = now[k].v[j];
          found_at[at++] = (unsigned)(base + (k * 32 + lane) * EACH + j);
        }
    total += __shfl_sync(0xffffffffu, upto, 31);
    if (total >= DOK_COLLECT_FLUSH) flush();
  }
  if (total > 0) flush();
}

// Keys given as positions of a dense tensor.
struct ListKeys {
  const unsigned *at;
  ll_t n;
  DenseShape shape;
  __device__ __forceinline__ bool idle() const { return false; }
  __device__ __forceinline__ bool row(ll_t &e) const { e = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; return e < n; }
  __device__ __forceinline__ void unravel(ll_t e, unsigned (&idx)[DOK_MAX_KEY_SIZE]) const {
    unsigned rem = at[e];
#pragma unroll
    for (int d = DOK_MAX_KEY_SIZE - 1; d >= 0; d--) {
      idx[d] = 0;
      if (d < shape.ndim) {
        const unsigned size = (unsigned)shape.sizes[d], q = d > 0 ? rem / size : 0;
        idx[d] = rem - q * size;
        rem = q;
      }
    }
  }
  __device__ __forceinline__ KeyHash hash(const DevHash &hp, ll_t e) const {
    unsigned idx[DOK_MAX_KEY_SIZE];
    unravel(e, idx);
    ll_t u = dok_uuid_term(idx[0], hp.a[0], hp.b[0], hp.p[0], hp.m[0]);
    ull_t h = (ull_t)idx[0] * (ull_t)hp.a1[0] + (ull_t)hp.b1[0];
#pragma unroll
    for (int d = 1; d < DOK_MAX_KEY_SIZE; d++)
      if (d < shape.ndim) {
        u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(idx[d], hp.a[d], hp.b[d], hp.p[d], hp.m[d]));
        h *= (ull_t)idx[d] * (ull_t)hp.a1[d] + (ull_t)hp.b1[d];
      }
    return KeyHash{dok_llabs(u), (ll_t)h};
  }
  __device__ __forceinline__ void store_key(const DevTable &t, const DevHash &hp, ll_t e, char *slot) const {
    unsigned idx[DOK_MAX_KEY_SIZE];
    unravel(e, idx);
    ll_t *krow = (ll_t *)(slot + t.key_off);
#pragma unroll
    for (int d = 0; d < DOK_MAX_KEY_SIZE; d++) if (d < shape.ndim) krow[hp.perm[d]] = (ll_t)idx[d];
  }
};

// A warp takes DOK_DENSE_SPAN consecutive elements at a time, DOK_DENSE_ROUNDS per lane (coalesced, and requested while the
// span before is worked on); the non-zero ones are collected in the warp's list in shared memory (position and value), and
// whenever 32 have come together the warp inserts them with every lane busy; what is left over waits for the next span.
// Inserting span by span took 530 us for the 671 k non-zeros of 8192^2 elements, with lists of whole blocks, whose warps
// wait for one another three times a span, 144.
#define DOK_DENSE_ROUNDS 8
#define DOK_DENSE_SPAN (32 * DOK_DENSE_ROUNDS)

template <int SB, typename T>
__global__ void __launch_bounds__(DOK_TPB, 4) k_dense_insert(DevTable t, DevHash hp, const T *__restrict__ dense, ll_t numel,
                                                          int is_float, DenseShape shape, ll_t *counters) {
  __shared__ ll_t list_at[DOK_WARPS][DOK_DENSE_SPAN + 32];
  __shared__ T list_value[DOK_WARPS][DOK_DENSE_SPAN + 32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ll_t *const found_at = list_at[warp];
  T *const found_value = list_value[warp];
  const ll_t first = ((ll_t)blockIdx.x * DOK_WARPS + warp) * DOK_DENSE_SPAN, stride = (ll_t)gridDim.x * DOK_WARPS * DOK_DENSE_SPAN;
  int claimed = 0, reused = 0, failed = 0, hits = 0, total = 0;
  const auto unravel = [&](auto rem, ll_t (&idx)[DOK_MAX_KEY_SIZE]) {          // a 64-bit division costs four of 32 bits
    using U = decltype(rem);
#pragma unroll
    for (int d = DOK_MAX_KEY_SIZE - 1; d >= 0; d--) {
      idx[d] = 0;
      if (d < shape.ndim) {
        const U size = (U)shape.sizes[d], q = rem / size;
        idx[d] = (ll_t)(rem - q * size);
        rem = q;
      }
    }
  };
  T v[DOK_DENSE_ROUNDS];
  const auto fetch = [&](ll_t base) {
#pragma unroll
    for (int r = 0; r < DOK_DENSE_ROUNDS; r++) {
      const ll_t i = base + r * 32 + lane;
      v[r] = i < numel ? __ldcs(dense + i) : (T)0;
    }
  };
  fetch(first);
  for (ll_t base = first; base < numel; base += stride) {                                 // uniform over the warp
#pragma unroll
    for (int r = 0; r < DOK_DENSE_ROUNDS; r++) {
      const bool nz = dok_nonzero<T>(v[r], is_float);
      const unsigned votes = __ballot_sync(0xffffffffu, nz);
      if (nz) {
        const int at = total + __popc(votes & ((1u << lane) - 1u));
        found_value[at] = v[r];
        found_at[at] = base + r * 32 + lane;
      }
      total += __popc(votes);
    }
    fetch(base + stride);
    __syncwarp();
    const bool at_end = base + stride >= numel;
    while (total >= 32 || (at_end && total > 0)) {                                        // uniform over the warp
      const int k = total - 1 - lane;                                                     // from the end of the list
      bool active = k >= 0;
      int outcome = -1;
      T value = 0;
      ll_t idx[DOK_MAX_KEY_SIZE];
      KeyHash kh{0, 0};
      if (active) {
        value = found_value[k];
        // unravel the row-major position into the index tuple; each index is one factor of the hash products
        if (numel <= 0xffffffffLL) unravel((unsigned)found_at[k], idx);
        else unravel((ull_t)found_at[k], idx);
        ll_t u = dok_uuid_term(idx[0], hp.a[0], hp.b[0], hp.p[0], hp.m[0]);
        ull_t h = (ull_t)idx[0] * (ull_t)hp.a1[0] + (ull_t)hp.b1[0];
#pragma unroll
        for (int d = 1; d < DOK_MAX_KEY_SIZE; d++)
          if (d < shape.ndim) {
            u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(idx[d], hp.a[d], hp.b[d], hp.p[d], hp.m[d]));
            h *= (ull_t)idx[d] * (ull_t)hp.a1[d] + (ull_t)hp.b1[d];
          }
        kh = KeyHash{dok_llabs(u), (ll_t)h};
      }
      active = dok_in_window(t, kh, active);
      const ll_t slot = dok_find_or_claim<SB>(t, kh, active, &outcome);
      if (active && slot >= 0) {
        ll_t *krow = (ll_t *)dok_key_row(t, slot);
#pragma unroll
        for (int d = 0; d < DOK_MAX_KEY_SIZE; d++) if (d < shape.ndim) krow[hp.perm[d]] = idx[d];
        *(T *)dok_value_ptr(t, slot) = value;
      }
      claimed += outcome == DOK_OUT_CLAIMED_EMPTY;
      reused += outcome == DOK_OUT_REUSED;
      failed += outcome == DOK_OUT_FAILED;
      hits += outcome == DOK_OUT_FOUND;
      total = total > 32 ? total - 32 : 0;
    }
    __syncwarp();                                        // the list is added to by the next span
  }
  if (counters) {
    dok_warp_add(counters + DOK_CNT_CLAIMED_EMPTY, claimed);
    dok_warp_add(counters + DOK_CNT_REUSED_REMOVED, reused);
    dok_warp_add(counters + DOK_CNT_FAILED, failed);
    dok_warp_add(counters + DOK_CNT_HITS, hits);
  }
}

// ---- flatten / reshape: re-key + re-insert in one pass ----------------------------------------------------

struct Rekey {
  int old_ndim, new_ndim;
  int old_perm[DOK_MAX_KEY_SIZE];       // storage column of logical index d in the source table
  ll_t old_strides[DOK_MAX_KEY_SIZE];   // row-major strides of the source shape (logical order)
  ll_t new_sizes[DOK_MAX_KEY_SIZE];     // destination shape
};

// One thread per SOURCE slot: a live slot's index tuple is linearised in the old shape, unravelled in the new one
// and inserted with its value into the destination table -- no compaction of the source, no intermediate tensors
// (the reference goes through indices()/values() and, for reshape, through a whole intermediate flattened tensor:
// sparse_dok_tensor.py:479-514).  Distinct positions stay distinct, so every insert claims a fresh slot.
template <int SB>
__global__ void __launch_bounds__(DOK_TPB) k_rekey_insert(DevTable src, DevTable dst, DevHash hp, Rekey rk, ll_t *counters) {
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB;
  int claimed = 0, failed = 0, found = 0;
  for (ll_t base = (ll_t)blockIdx.x * DOK_TPB; base < src.nb; base += stride) {       // uniform over the block
    const ll_t s = base + threadIdx.x;
    bool active = false;
    ll_t idx[DOK_MAX_KEY_SIZE];
    KeyHash kh{0, 0};
    if (s < src.nb) {
      const ll_t tag = dok_load_tag(src, s);
      active = tag >= 0;                                  // uuids are non-negative; empty, tombstone, padding are not
    }
    if (active) {
      const ll_t *krow = (const ll_t *)dok_key_row(src, s);
      ull_t linear = 0;
#pragma unroll
      for (int d = 0; d < DOK_MAX_KEY_SIZE; d++)
        if (d < rk.old_ndim) linear += (ull_t)krow[rk.old_perm[d]] * (ull_t)rk.old_strides[d];
#pragma unroll
      for (int d = DOK_MAX_KEY_SIZE - 1; d >= 0; d--) {
        idx[d] = 0;
        if (d < rk.new_ndim) {
          const ull_t size = (ull_t)rk.new_sizes[d];
          const ull_t q = linear / size;
          idx[d] = (ll_t)(linear - q * size);
          linear = q;
        }
      }
      ll_t u = dok_uuid_term(idx[0], hp.a[0], hp.b[0], hp.p[0], hp.m[0]);
      ull_t h = (ull_t)idx[0] * (ull_t)hp.a1[0] + (ull_t)hp.b1[0];
#pragma unroll
      for (int d = 1; d < DOK_MAX_KEY_SIZE; d++)
        if (d < rk.new_ndim) {
          u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(idx[d], hp.a[d], hp.b[d], hp.p[d], hp.m[d]));
          h *= (ull_t)idx[d] * (ull_t)hp.a1[d] + (ull_t)hp.b1[d];
        }
      kh = KeyHash{dok_llabs(u), (ll_t)h};
    }
    active = dok_in_window(dst, kh, active);
    int outcome = -1;
    const ll_t slot = dok_find_or_claim<SB>(dst, kh, active, &outcome);
    if (active && slot >= 0) {
      ll_t *krow = (ll_t *)dok_key_row(dst, slot);
#pragma unroll
      for (int d = 0; d < DOK_MAX_KEY_SIZE; d++) if (d < rk.new_ndim) krow[hp.perm[d]] = idx[d];
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

// ---- sparse gather: lookup over the selectors and insert of the hits into a second table, one kernel -----

// One thread per selector element: the key formed from the selectors is looked up in `src`; a hit is inserted into
// `dst` under the element's POSITION in the selection (its index tuple in the selection's shape, int64), with the
// stored value.  Positions are pairwise different, so every insert claims a fresh slot.  Replaces
// sparse_dok_get_items (sparse_dok_tensor_impl.cu:110-160), which does the same per thread.
template <int SBS, int SBD>
__global__ void __launch_bounds__(DOK_TPB) k_gather_insert(DevTable src, DevHash shp, SelKeys sel, DevTable dst, DevHash dhp,
                                                           ll_t *counters) {
  ll_t e;
  const bool active = sel.row(e);
  KeyHash kh{0, 0};
  if (active) kh = sel.hash(shp, e);
  const Located loc = dok_locate<SBS, 1, false>(src, kh, e, active, nullptr, NoEmit<false>());
  const bool hit = active && loc.found >= 0;
  ll_t idx[DOK_MAX_KEY_SIZE];
  KeyHash kd{0, 0};
  if (hit) {
    // the element's index tuple in the selection's shape (row-major); a 0-dim selection is position (0,)
    ull_t rem = (ull_t)e;
#pragma unroll
    for (int d = DOK_MAX_KEY_SIZE - 1; d >= 0; d--) {
      idx[d] = 0;
      if (d < sel.s.selector_ndim) {
        const ull_t size = (ull_t)sel.s.sizes[d];
        const ull_t q = rem / size;
        idx[d] = (ll_t)(rem - q * size);
        rem = q;
      }
    }
    ll_t u = dok_uuid_term(idx[0], dhp.a[0], dhp.b[0], dhp.p[0], dhp.m[0]);
    ull_t h = (ull_t)idx[0] * (ull_t)dhp.a1[0] + (ull_t)dhp.b1[0];
#pragma unroll
    for (int d = 1; d < DOK_MAX_KEY_SIZE; d++)
      if (d < dhp.ks) {
        u = (ll_t)((ull_t)u * (ull_t)dok_uuid_term(idx[d], dhp.a[d], dhp.b[d], dhp.p[d], dhp.m[d]));
        h *= (ull_t)idx[d] * (ull_t)dhp.a1[d] + (ull_t)dhp.b1[d];
      }
    kd = KeyHash{dok_llabs(u), (ll_t)h};
  }
  int outcome = -1;
  const ll_t slot = dok_find_or_claim<SBD>(dst, kd, hit, &outcome);
  if (hit && slot >= 0) {
    ll_t *krow = (ll_t *)dok_key_row(dst, slot);
#pragma unroll
    for (int d = 0; d < DOK_MAX_KEY_SIZE; d++) if (d < dhp.ks) krow[dhp.perm[d]] = idx[d];
    dok_store_value(dst, slot, dok_value_ptr(src, loc.found));
  }
  if (counters) {
    dok_warp_add(counters + DOK_CNT_HITS, hit);
    dok_warp_add(counters + DOK_CNT_CLAIMED_EMPTY, outcome == DOK_OUT_CLAIMED_EMPTY || outcome == DOK_OUT_REUSED);
    dok_warp_add(counters + DOK_CNT_FAILED, outcome == DOK_OUT_FAILED);
  }
}

// ---- to_dense ---------------------------------------------------------------------------------------------

struct DenseTarget {
  int ndim;
  int perm[DOK_MAX_KEY_SIZE];            // storage column of logical index d
  ll_t sizes[DOK_MAX_KEY_SIZE], strides[DOK_MAX_KEY_SIZE];
};

// One thread per slot: a live slot's value goes to its position of the dense tensor (zeroed before); positions outside of
// it are left out.  Replaces the compaction to index and value lists, their flattening and an indexed add.
template <typename T>
__global__ void __launch_bounds__(DOK_TPB) k_to_dense(DevTable t, DenseTarget d, T *__restrict__ dense) {
  const ll_t stride = (ll_t)gridDim.x * DOK_TPB;
  for (ll_t s = (ll_t)blockIdx.x * DOK_TPB + threadIdx.x; s < t.nb; s += stride) {
    if (dok_load_tag(t, s) < 0) continue;
    const ll_t *krow = (const ll_t *)dok_key_row(t, s);
    ll_t at = 0;
    bool inside = true;
#pragma unroll
    for (int i = 0; i < DOK_MAX_KEY_SIZE; i++)
      if (i < d.ndim) {
        const ll_t x = krow[d.perm[i]];
        inside = inside && (ull_t)x < (ull_t)d.sizes[i];
        at += x * d.strides[i];
      }
    if (inside) dense[at] = *(const T *)dok_value_ptr(t, s);
  }
}

static unsigned streaming_grid(ll_t numel) {
  const ll_t blocks = (numel + DOK_TPB - 1) / DOK_TPB;
  const ll_t cap = 148 * 8;   // 8 resident blocks of 256 threads per SM
  return (unsigned)(blocks < cap ? (blocks < 1 ? 1 : blocks) : cap);
}

extern "C" {

int dok_dok_get(const dok_table *t, const dok_hash_params *hp, const dok_selectors *sel, void *out_values,
                uint8_t *out_found, const void *fallback, int64_t *counters, void *stream) {
  DevHash dh;
  DevTable dt;
  SelKeys sk;
  if (!prepare(t, hp, &dt, &dh) || !make_sel(sel, dh, &sk)) return DOK_BAD_ARG;
  if (sk.n > 0 && !out_values) return DOK_BAD_ARG;
  return launch_get(dt, dh, sk, out_values, out_found, fallback, counters, 0, (cudaStream_t)stream);
}

int dok_dok_count_exists(const dok_table *t, const dok_hash_params *hp, const dok_selectors *sel, int64_t *counters,
                         void *stream) {
  DevHash dh;
  DevTable dt;
  SelKeys sk;
  if (!prepare(t, hp, &dt, &dh) || !make_sel(sel, dh, &sk) || !counters) return DOK_BAD_ARG;
  if (sk.n == 0) return DOK_OK;
  return launch_find<0>(dt, dh, sk, nullptr, counters, (cudaStream_t)stream);
}

int dok_dok_zero_items(const dok_table *t, const dok_hash_params *hp, const dok_selectors *sel, int64_t *counters,
                       void *stream) {
  DevHash dh;
  DevTable dt;
  SelKeys sk;
  if (!prepare(t, hp, &dt, &dh) || !make_sel(sel, dh, &sk) || !counters) return DOK_BAD_ARG;
  if (sk.n == 0) return DOK_OK;
  return launch_find<1>(dt, dh, sk, nullptr, counters, (cudaStream_t)stream);
}

int dok_dok_set_dense(const dok_table *t, const dok_hash_params *hp, const dok_selectors *sel, const void *src,
                      const int64_t *src_strides, int64_t *slot_scratch, int64_t epoch, int64_t *counters,
                      void *stream) {
  if (!slot_scratch) return DOK_BAD_ARG;
  int64_t n = 1;
  for (int j = 0; sel && j < sel->selector_ndim && j < DOK_MAX_SELECTOR_NDIM; j++) n *= sel->sizes[j];
  return dok_dok_assign(t, hp, sel, src, src_strides, slot_scratch, n + 1, epoch, counters, nullptr, stream);
}

static StridedValues strided(const dok_selectors *sel, const void *src, const int64_t *src_strides) {
  StridedValues sv;
  sv.src = (const char *)src;
  sv.selector_ndim = sel->selector_ndim;
  for (int j = 0; j < DOK_MAX_SELECTOR_NDIM; j++) {
    sv.sizes[j] = j < sel->selector_ndim ? sel->sizes[j] : 1;
    sv.strides[j] = j < sel->selector_ndim ? src_strides[j] : 0;
  }
  return sv;
}

int dok_dok_assign(const dok_table *t, const dok_hash_params *hp, const dok_selectors *sel, const void *src,
                   const int64_t *src_strides, int64_t *scratch, int64_t scratch_words, int64_t epoch, int64_t *counters,
                   int64_t *more, void *stream) {
  DevHash dh;
  DevTable dt;
  SelKeys sk;
  if (!prepare(t, hp, &dt, &dh) || !make_sel(sel, dh, &sk)) return DOK_BAD_ARG;
  if (sk.n == 0) return DOK_OK;
  if (!dok_set_is_small(dt, sk.n) && (!scratch || scratch_words < sk.n + 1)) return DOK_BAD_ARG;
  if (!src || !src_strides || !dok_has_stamps(dt) || epoch < 1 || epoch > DOK_MAX_EPOCH) return DOK_BAD_ARG;
  return launch_set_general(dt, dh, sk, strided(sel, src, src_strides), scratch, epoch, nullptr, counters, (cudaStream_t)stream, more, scratch_words);
}

int dok_dok_assign_numbered(const dok_table *t, const dok_hash_params *hp, const dok_selectors *sel, const void *src,
                            const int64_t *src_strides, int64_t base, int64_t *counters, int64_t *more, void *stream) {
  DevHash dh;
  DevTable dt;
  SelKeys sk;
  if (!prepare(t, hp, &dt, &dh) || !make_sel(sel, dh, &sk) || !dok_set_in_word(dt, dh, sk.n) || !dok_numbers_fit(base, sk.n) || !src ||
      !src_strides)
    return DOK_BAD_ARG;
  return launch_set_word(dt, dh, sk, strided(sel, src, src_strides), base, counters, more, (cudaStream_t)stream);
}

int dok_dok_gather_insert(const dok_table *src, const dok_hash_params *src_hp, const dok_selectors *sel,
                          const dok_table *dst, const dok_hash_params *dst_hp, int64_t *counters, void *stream) {
  DevHash sh, dh;
  DevTable st_, dt;
  SelKeys sk;
  if (!prepare(src, src_hp, &st_, &sh) || !prepare(dst, dst_hp, &dt, &dh) || !make_sel(sel, sh, &sk)) return DOK_BAD_ARG;
  if (dh.dtype != DOK_I64 || st_.vb != dt.vb || dh.ks != (sel->selector_ndim > 0 ? sel->selector_ndim : 1)) return DOK_BAD_ARG;
  if (st_.sb > 128 || dt.sb > 128) return DOK_BAD_ARG;                 // DOK tables: int64 index keys, one value element
  if (dok_window_passes(st_) > 1 || dok_window_passes(dt) > 1) return DOK_TOO_LARGE;   // callers take the two-step route
  if (sk.n == 0) return DOK_OK;
  const unsigned grid = (unsigned)((sk.n + DOK_TPB - 1) / DOK_TPB);
  cudaStream_t st = (cudaStream_t)stream;
#define DOK_GATHER(SBS) \
  switch (dt.sb) { \
    case 32: k_gather_insert<SBS, 32><<<grid, DOK_TPB, 0, st>>>(st_, sh, sk, dt, dh, (ll_t *)counters); break; \
    case 64: k_gather_insert<SBS, 64><<<grid, DOK_TPB, 0, st>>>(st_, sh, sk, dt, dh, (ll_t *)counters); break; \
    default: k_gather_insert<SBS, 128><<<grid, DOK_TPB, 0, st>>>(st_, sh, sk, dt, dh, (ll_t *)counters); break; \
  }
  switch (st_.sb) {
    case 32: DOK_GATHER(32); break;
    case 64: DOK_GATHER(64); break;
    default: DOK_GATHER(128); break;
  }
#undef DOK_GATHER
  return dok_check_launch();
}

int dok_dok_rekey_insert(const dok_table *src, const dok_hash_params *src_hp, const int64_t *src_sizes,
                         const dok_table *dst, const dok_hash_params *dst_hp, const int64_t *dst_sizes,
                         int64_t *counters, void *stream) {
  DevHash sh, dh;
  DevTable st_, dt;
  if (!prepare(src, src_hp, &st_, &sh) || !prepare(dst, dst_hp, &dt, &dh)) return DOK_BAD_ARG;
  if (sh.dtype != DOK_I64 || dh.dtype != DOK_I64 || !src_sizes || !dst_sizes || st_.vb != dt.vb) return DOK_BAD_ARG;
  Rekey rk;
  memset(&rk, 0, sizeof(rk));
  rk.old_ndim = sh.ks;
  rk.new_ndim = dh.ks;
  ll_t old_total = 1, new_total = 1;
  for (int d = sh.ks - 1; d >= 0; d--) {
    if (src_sizes[d] < 1) return DOK_BAD_ARG;
    rk.old_strides[d] = old_total;
    rk.old_perm[d] = sh.perm[d];
    old_total *= src_sizes[d];
  }
  for (int d = 0; d < dh.ks; d++) {
    if (dst_sizes[d] < 1) return DOK_BAD_ARG;
    rk.new_sizes[d] = dst_sizes[d];
    new_total *= dst_sizes[d];
  }
  if (old_total != new_total) return DOK_BAD_ARG;
  const unsigned grid = streaming_grid(st_.nb);
  int rc = DOK_OK;
  DOK_DISPATCH_SB(dt, DOK_FOR_WINDOWS(dt, rc, (k_rekey_insert<SB><<<grid, DOK_TPB, 0, (cudaStream_t)stream>>>(st_, wt, dh, rk, (ll_t *)counters))));
  return rc;
}

int dok_dok_to_dense(const dok_table *t, const dok_hash_params *hp, const int64_t *sizes, void *dense, void *stream) {
  DevHash dh;
  DevTable dt;
  if (!prepare(t, hp, &dt, &dh) || dh.dtype != DOK_I64 || !sizes || !dense) return DOK_BAD_ARG;
  DenseTarget d;
  memset(&d, 0, sizeof(d));
  d.ndim = dh.ks;
  ll_t total = 1;
  for (int i = dh.ks - 1; i >= 0; i--) {
    if (sizes[i] < 0) return DOK_BAD_ARG;
    d.sizes[i] = sizes[i];
    d.strides[i] = total;
    d.perm[i] = dh.perm[i];
    total *= sizes[i];
  }
  const unsigned grid = streaming_grid(dt.nb);
  cudaStream_t st = (cudaStream_t)stream;
  switch (dt.vb) {
    case 1: k_to_dense<<<grid, DOK_TPB, 0, st>>>(dt, d, (unsigned char *)dense); break;
    case 2: k_to_dense<<<grid, DOK_TPB, 0, st>>>(dt, d, (unsigned short *)dense); break;
    case 4: k_to_dense<<<grid, DOK_TPB, 0, st>>>(dt, d, (unsigned *)dense); break;
    case 8: k_to_dense<<<grid, DOK_TPB, 0, st>>>(dt, d, (ull_t *)dense); break;
    default: return DOK_BAD_ARG;
  }
  return dok_check_launch();
}

int dok_dense_count_nonzero(const void *dense, int64_t numel, int elem_bytes, int is_float, int64_t *count_out,
                            void *stream) {
  if (numel < 0 || !count_out || (numel > 0 && !dense)) return DOK_BAD_ARG;
  if (numel == 0) return DOK_OK;
  const unsigned grid = streaming_grid(numel);
  cudaStream_t st = (cudaStream_t)stream;
  switch (elem_bytes) {
    case 1: k_dense_count<unsigned char><<<grid, DOK_TPB, 0, st>>>((const unsigned char *)dense, numel, is_float, (ll_t *)count_out); break;
    case 2: k_dense_count<unsigned short><<<grid, DOK_TPB, 0, st>>>((const unsigned short *)dense, numel, is_float, (ll_t *)count_out); break;
    case 4: k_dense_count<unsigned><<<grid, DOK_TPB, 0, st>>>((const unsigned *)dense, numel, is_float, (ll_t *)count_out); break;
    case 8: k_dense_count<ull_t><<<grid, DOK_TPB, 0, st>>>((const ull_t *)dense, numel, is_float, (ll_t *)count_out); break;
    default: return DOK_BAD_ARG;
  }
  return dok_check_launch();
}

int dok_dense_collect_nonzero(const void *dense, int64_t numel, int elem_bytes, int is_float, void *list, int64_t capacity,
                              int64_t *count_out, void *stream) {
  if (numel < 0 || numel > 0xffffffffLL || !count_out || capacity < 0 || (capacity & 1) || (capacity > 0 && !list)) return DOK_BAD_ARG;
  if (numel > 0 && (!dense || ((uintptr_t)dense & 15) != 0)) return DOK_BAD_ARG;
  if (numel == 0) return cudaMemsetAsync(count_out, 0, sizeof(int64_t), (cudaStream_t)stream) == cudaSuccess ? DOK_OK : dok_check_launch();
  const ll_t spans = (numel * elem_bytes + (elem_bytes == 1 ? 512 : 1024) * DOK_WARPS - 1) / ((elem_bytes == 1 ? 512 : 1024) * DOK_WARPS);
  const unsigned grid = (unsigned)(spans < 148 * DOK_COLLECT_BLOCKS ? spans : 148 * DOK_COLLECT_BLOCKS);
  cudaStream_t st = (cudaStream_t)stream;
  int rc = DOK_OK;
  const auto collect = [&](auto *typed) {
    k_dense_look<<<1, DOK_LOOK_PIECES, 0, st>>>(typed, numel, is_float, capacity, (ll_t *)count_out);
    if ((rc = dok_check_launch()) != DOK_OK) return;
    k_dense_collect<<<grid, DOK_TPB, 0, st>>>(typed, numel, is_float, (unsigned *)list,
                                              (std::remove_const_t<std::remove_pointer_t<decltype(typed)>> *)((char *)list + 4 * capacity), capacity, (ll_t *)count_out);
    rc = dok_check_launch();
  };
  switch (elem_bytes) {
    case 1: collect((const unsigned char *)dense); break;
    case 2: collect((const unsigned short *)dense); break;
    case 4: collect((const unsigned *)dense); break;
    case 8: collect((const ull_t *)dense); break;
    default: return DOK_BAD_ARG;
  }
  return rc;
}

int dok_dense_insert_list(const dok_table *t, const dok_hash_params *hp, const void *list, int64_t capacity, int64_t n, const int64_t *sizes,
                          int64_t *counters, void *stream) {
  DevHash dh;
  DevTable dt;
  if (!prepare(t, hp, &dt, &dh) || dh.dtype != DOK_I64 || !sizes || n < 0 || n > capacity || (capacity & 1)) return DOK_BAD_ARG;
  if (n == 0) return DOK_OK;
  if (!list) return DOK_BAD_ARG;
  ListKeys keys{(const unsigned *)list, n, {}};
  keys.shape.ndim = dh.ks;
  for (int d = 0; d < DOK_MAX_KEY_SIZE; d++) {
    keys.shape.sizes[d] = d < dh.ks ? sizes[d] : 1;
    if (keys.shape.sizes[d] < 1 || keys.shape.sizes[d] > 0xffffffffLL) return DOK_BAD_ARG;
  }
  const RowValues values{(const char *)list + 4 * capacity};
  const unsigned grid = (unsigned)((n + DOK_TPB - 1) / DOK_TPB);
  int rc = DOK_OK;
  DOK_DISPATCH_MARKS(dt, DOK_FOR_WINDOWS(dt, rc, (k_set_unique<SB, MARKS><<<grid, DOK_TPB, 0, (cudaStream_t)stream>>>(wt, dh, keys, values, (uint8_t *)nullptr, (ll_t *)counters))));
  return rc;
}

int dok_dense_insert_nonzero(const dok_table *t, const dok_hash_params *hp, const void *dense, const int64_t *sizes,
                             int64_t numel, int is_float, int64_t *counters, void *stream) {
  DevHash dh;
  DevTable dt;
  if (!prepare(t, hp, &dt, &dh) || dh.dtype != DOK_I64 || !sizes || numel < 0) return DOK_BAD_ARG;
  if (numel == 0) return DOK_OK;
  if (!dense) return DOK_BAD_ARG;
  DenseShape shape;
  shape.ndim = dh.ks;
  ll_t prod = 1;
  for (int d = 0; d < DOK_MAX_KEY_SIZE; d++) {
    shape.sizes[d] = d < dh.ks ? sizes[d] : 1;
    if (shape.sizes[d] < 1) return DOK_BAD_ARG;
    prod *= shape.sizes[d];
  }
  if (prod != numel) return DOK_BAD_ARG;
  const ll_t blocks = (numel + DOK_DENSE_SPAN * DOK_WARPS - 1) / (DOK_DENSE_SPAN * DOK_WARPS);
  const unsigned grid = (unsigned)(blocks < 148 * 4 ? blocks : 148 * 4);        // one wave: each warp ends with a list that is not full
  cudaStream_t st = (cudaStream_t)stream;
  int rc = DOK_OK;
  switch (dt.vb) {
    case 1: DOK_DISPATCH_SB(dt, DOK_FOR_WINDOWS(dt, rc, (k_dense_insert<SB, unsigned char><<<grid, DOK_TPB, 0, st>>>(wt, dh, (const unsigned char *)dense, numel, is_float, shape, (ll_t *)counters)))); break;
    case 2: DOK_DISPATCH_SB(dt, DOK_FOR_WINDOWS(dt, rc, (k_dense_insert<SB, unsigned short><<<grid, DOK_TPB, 0, st>>>(wt, dh, (const unsigned short *)dense, numel, is_float, shape, (ll_t *)counters)))); break;
    case 4: DOK_DISPATCH_SB(dt, DOK_FOR_WINDOWS(dt, rc, (k_dense_insert<SB, unsigned><<<grid, DOK_TPB, 0, st>>>(wt, dh, (const unsigned *)dense, numel, is_float, shape, (ll_t *)counters)))); break;
    case 8: DOK_DISPATCH_SB(dt, DOK_FOR_WINDOWS(dt, rc, (k_dense_insert<SB, ull_t><<<grid, DOK_TPB, 0, st>>>(wt, dh, (const ull_t *)dense, numel, is_float, shape, (ll_t *)counters)))); break;
    default: return DOK_BAD_ARG;
  }
  return rc;
}

}  // extern "C"
