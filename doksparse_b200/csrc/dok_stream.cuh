// The walk of a large batch: a warp keeps 32 chains in flight and takes the next row whenever one of them ends.
//
// With one row per thread a warp walks until the longest of its 32 chains ends.  At load 0.6 one row in six needs a second
// group, so nearly every warp made one to three more dependent round trips to DRAM for a handful of lanes: a row stayed on
// its SM for 10 us, five times the latency of one access, and DRAM ran at 74 % of what a copy reaches.  Here a warp has a
// share of the batch.  It hashes 32 rows at a time (coalesced) into a queue in shared memory; a lane whose chain has ended
// takes the queue's next row; and every round of the loop inspects one group for each of the 32 lanes, the four lanes of a
// quad reading the line of each of the quad's four keys together (dok_device.cuh).  Rows that belong to another window of a
// windowed launch never enter the queue, so they cost their hash and nothing else.
//
// Small batches have one row per lane and no refill; the code is the same.
#pragma once
#include "dok_host.cuh"

#define DOK_QUEUE 64                     // entries per warp: up to 31 waiting plus 32 new ones
#define DOK_WARPS (DOK_TPB / 32)
#define DOK_NONE 0xffffffffu

struct WarpQueue { ulonglong2 entry[DOK_QUEUE]; };      // uuid | group, row of the share (26 bits), stride - 1 (6 bits)

// What a lane works on.  row (of the warp's share) == DOK_NONE: nothing; its uuid then matches no tag, and the group it
// reads is the one of its last row (or group 0).
struct LaneRow {
  ll_t uuid;
  unsigned group, word, row;
  __device__ __forceinline__ bool busy() const { return row != DOK_NONE; }
  __device__ __forceinline__ void done() { row = DOK_NONE; uuid = -4; }
};
#define DOK_IDLE_LANE LaneRow{-4, 0, 0, DOK_NONE}

// A warp's share of the batch (of the block's slice): one range of rows.  (Every warp taking each so-many-th piece of 32
// rows, so that the grid works on neighbouring rows, was 3 % slower.)
struct WarpShare {
  unsigned first, rows, next;            // range; row of it that is hashed next
  unsigned head, waiting;                // queue position, entries
};

__device__ __forceinline__ WarpShare dok_share(ll_t total) {
  const ll_t warps = (ll_t)gridDim.x * DOK_WARPS, w = (ll_t)blockIdx.x * DOK_WARPS + (threadIdx.x >> 5);
  ll_t per = (total + warps - 1) / warps;
  if (per < 32) per = 32;                // a short batch: whole warps first
  ll_t first = w * per, end = first + per;
  if (end > total) end = total;
  if (first > end) first = end;
  return WarpShare{(unsigned)first, (unsigned)(end - first), 0, 0, 0};
}

// Fills the queue until 32 rows wait or the share is used up.
template <class Keys>
__device__ __forceinline__ void dok_fill_queue(WarpQueue &q, WarpShare &s, const DevTable &t, const DevHash &hp, const Keys &keys) {
  const unsigned lane = threadIdx.x & 31u;
  while (s.waiting < 32 && s.next < s.rows) {
    const unsigned k = s.next + lane;
    s.next += 32;
    KeyHash kh{0, 0};
    bool enter = k < s.rows;
    if (enter) {
      kh = keys.hash(hp, keys.elem(s.first + k));
      enter = dok_in_window(t, kh, true);
    }
    const unsigned votes = __ballot_sync(0xffffffffu, enter);
    if (enter) {
      const ull_t h = dok_chain_hash(kh);
      const unsigned group = __umulhi((unsigned)(h >> 32), (unsigned)t.n_groups);
      const unsigned at = (s.head + s.waiting + __popc(votes & ((1u << lane) - 1u))) & (DOK_QUEUE - 1);
      q.entry[at] = make_ulonglong2((ull_t)kh.uuid, (ull_t)group << 32 | (k << 6 | ((unsigned)h & 63u)));
    }
    s.waiting += __popc(votes);
  }
  __syncwarp();
}

// Lanes without a row take the next ones; false when no lane of the warp has a row.
__device__ __forceinline__ bool dok_refill(const WarpQueue &q, WarpShare &s, LaneRow &r, const DevTable &t) {
  const unsigned idle = __ballot_sync(0xffffffffu, !r.busy());
  if (idle == 0) return true;
  const unsigned rank = __popc(idle & ((1u << (threadIdx.x & 31u)) - 1u));
  if (!r.busy() && rank < s.waiting) {
    const ulonglong2 e = q.entry[(s.head + rank) & (DOK_QUEUE - 1)];
    r.uuid = (ll_t)e.x;
    r.group = (unsigned)(e.y >> 32);
    r.word = t.n_groups > 64 ? (unsigned)e.y & 63u : DOK_CHAIN_LINEAR;
    r.row = (unsigned)e.y >> 6;
  }
  const unsigned n = __popc(idle), taken = n < s.waiting ? n : s.waiting;
  s.head += taken;
  s.waiting -= taken;
  __syncwarp();
  return n < 32 || taken > 0;
}

// One group for each lane: four requests, each for the lines of a quad's key in its turn.
template <int LW>
struct Lines { ull_t w[4][LW]; };
// MARKS (of 64- and 128-byte slots): the last lane, whose part of the line has no tag, reads the group's mark.
template <int LW, bool L1, bool MARKS>
__device__ __forceinline__ void dok_request(const DevTable &t, const LaneRow &lr, Lines<LW> &f) {
  const unsigned l = threadIdx.x & 3u;
  const char *my_base = t.slots + (MARKS && l == 3 ? 0 : 32 * l);
#pragma unroll
  for (unsigned r = 0; r < 4; r++)
    dok_load_words<LW, L1>(my_base + (ull_t)__shfl_sync(0xffffffffu, lr.group, (threadIdx.x & 28u) + r) * 128u, f.w[r]);
}

// What the lines of a quad's four keys hold: byte r = key r, bits 0-3 match, 4-7 empty, by slot of the group.
template <int SB, int LW>
__device__ __forceinline__ unsigned dok_inspect(const LaneRow &lr, const Lines<LW> &f) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned l = threadIdx.x & 3u, base = threadIdx.x & 28u;
  const bool has_tag = ((32u * l) % SB) == 0;
  unsigned bits = 0;
#pragma unroll
  for (unsigned r = 0; r < 4; r++) {
    const ll_t uuid_r = __shfl_sync(FULL, lr.uuid, base + r), tag = (ll_t)f.w[r][0];
    if (has_tag) bits |= ((unsigned)(tag == uuid_r) | ((unsigned)(tag == DOK_EMPTY) << 4)) << (8u * r + 32u * l / SB);
  }
  bits |= __shfl_xor_sync(FULL, bits, 1);
  bits |= __shfl_xor_sync(FULL, bits, 2);
  return bits;
}
// The same by votes, bits by LANE of the quad (the slot at lane p is p * 32 / SB).  MARKS: a group that no key went past counts
// as one with an empty slot at the last lane (dok_mark_passed).
template <int SB, int LW, bool MARKS>
__device__ __forceinline__ void dok_inspect_votes(const LaneRow &lr, const Lines<LW> &f, unsigned &m, unsigned &me, unsigned (&match)[4],
                                                  unsigned (&empty)[4]) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned l = threadIdx.x & 3u, base = threadIdx.x & 28u;
  const bool has_tag = ((32u * l) % SB) == 0;
  unsigned own_m = 0, own_e = 0;
#pragma unroll
  for (unsigned r = 0; r < 4; r++) {
    const ll_t uuid_r = __shfl_sync(FULL, lr.uuid, base + r), tag = (ll_t)f.w[r][0];
    match[r] = __ballot_sync(FULL, has_tag && tag == uuid_r);
    empty[r] = __ballot_sync(FULL, (has_tag && tag == DOK_EMPTY) || (MARKS && l == 3 && !(f.w[r][LW > 1 ? 1 : 0] & DOK_PASSED)));
    if (l == r) { own_m = match[r]; own_e = empty[r]; }
  }
  m = (own_m >> base) & 0xfu;
  me = ((own_m | own_e) >> base) & 0xfu;
}
__device__ __forceinline__ unsigned dok_matches(unsigned bits, unsigned r) { return (bits >> (8u * r)) & 0xfu; }
__device__ __forceinline__ unsigned dok_ends(unsigned bits, unsigned r) { return ((bits >> (8u * r)) | (bits >> (8u * r + 4u))) & 0xfu; }

// The loop.  `step(lane's row, lines, share)` inspects the lines, lets the row go to its next group (dok_next_group) or ends
// it (done()).
template <int LW, bool L1, bool MARKS, class Keys, class Step>
__device__ __forceinline__ void dok_walk_share(WarpQueue &queue, WarpShare share, const DevTable &t, const DevHash &hp, const Keys &keys,
                                               const Step &step) {
  LaneRow lr = DOK_IDLE_LANE;
  Lines<LW> lines;
  for (;;) {
    dok_fill_queue(queue, share, t, hp, keys);
    if (!dok_refill(queue, share, lr, t)) break;
    dok_request<LW, L1, MARKS>(t, lr, lines);
    step(lr, lines, share);
  }
}
// ... of the warp's part of the whole batch
template <int LW, bool L1, bool MARKS, class Keys, class Step>
__device__ __forceinline__ void dok_walk_share(WarpQueue &queue, const DevTable &t, const DevHash &hp, const Keys &keys, const Step &step) {
  dok_walk_share<LW, L1, MARKS>(queue, dok_share(keys.total()), t, hp, keys, step);
}
