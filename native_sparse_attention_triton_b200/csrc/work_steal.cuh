// Persistent CTAs that take over the thread blocks of their own grid that have not started yet (clusterlaunchcontrol).
//
// The grid is launched as if every work item had a CTA of its own; a CTA that runs asks the hardware to cancel one pending CTA and
// does its item instead.  So items are handed out dynamically, in the grid's order, without a counter in memory that each launch
// would have to clear, and what a CTA sets up once (tensor memory, barriers, pipelines) serves all the items it gets.
//
// One warp (the loads' producer) sends the requests, one item ahead, looks the items up and publishes them in a small ring in
// shared memory, from which the other warps take them in order.
#pragma once
#include "common.cuh"

namespace nsa {

// ---- the request to the hardware: one outstanding at a time, sent and read by one warp ----
struct StealSlot {
  uint4 answer;  // 16-byte aligned
  uint64_t full;
  uint64_t pad;
};

// One thread; only after the request before it was answered with a block: asking again after a refusal is undefined.
__device__ __forceinline__ void steal_request(StealSlot* s) {
  fence_proxy_async();  // the last answer was read through the generic proxy, the next one is written through the async proxy
  mbar_expect_tx(&s->full, 16);
  asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];\n"
               ::"r"(smem_u32(&s->answer)), "r"(smem_u32(&s->full)) : "memory");
}
// Answer to request number n (0, 1, ...): false if no block was left (or the wait gave up), else its index.  All lanes call it.
__device__ __forceinline__ bool steal_answer(StealSlot* s, int n, uint3& block, const Status& st) {
  const bool ok = mbar_wait(&s->full, n & 1, st);
  uint32_t got, x, y, z;
  asm volatile(
      "{\n .reg .b128 a;\n .reg .pred p;\n ld.shared.b128 a, [%4];\n"
      " clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, a;\n"
      " selp.u32 %0, 1, 0, p;\n mov.u32 %1, 0;\n mov.u32 %2, 0;\n mov.u32 %3, 0;\n"
      " @p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%1, %2, %3, _}, a;\n}\n"
      : "=r"(got), "=r"(x), "=r"(y), "=r"(z) : "r"(smem_u32(&s->answer)) : "memory");
  block = make_uint3(x, y, z);
  return __all_sync(0xffffffffu, ok && got != 0);  // every lane has read the answer before the next request may overwrite it
}

// ---- the items, from the producer to the other warps ----
constexpr int kItemSlots = 4;

// One work item of a dense attention pass: row tiles of one sequence and KV head.  head < 0: no further item.
struct AttnItem {
  int qs, Lq, ksq, Lk;    // first row and length of the sequence, queries and keys
  int head, q0;           // KV head, first token of the item in its sequence
  int kt0, ntiles;        // first key tile any of its rows sees, number of key tiles
};

struct ItemRing {
  AttnItem item[kItemSlots];
  uint64_t full[kItemSlots];
  uint64_t empty[kItemSlots];
};

// one thread, before the CTA's first barrier; `readers` warps take every item
__device__ __forceinline__ void items_init(ItemRing* r, StealSlot* s, int readers) {
  for (int i = 0; i < kItemSlots; ++i) {
    mbar_init(r->full + i, 1);
    mbar_init(r->empty + i, readers);
  }
  mbar_init(&s->full, 1);
}
// item number n (0, 1, ...); one thread
__device__ __forceinline__ void item_publish(ItemRing* r, int n, const AttnItem& w, const Status& st) {
  const int s = n % kItemSlots;
  if (n >= kItemSlots) mbar_wait(r->empty + s, ((n / kItemSlots) - 1) & 1, st);
  r->item[s] = w;
  mbar_arrive(r->full + s);
}
// a whole warp; false when there is no further item (or a wait gave up)
__device__ __forceinline__ bool item_take(ItemRing* r, int n, AttnItem& w, const Status& st) {
  const int s = n % kItemSlots;
  const bool ok = mbar_wait(r->full + s, (n / kItemSlots) & 1, st);
  w = r->item[s];
  w.ntiles = __shfl_sync(0xffffffffu, w.ntiles, 0);  // (warp-uniform for the compiler)
  const bool more = __all_sync(0xffffffffu, ok && w.head >= 0);
  if (lane_id() == 0) mbar_arrive(r->empty + s);
  return more;
}
// a whole warp: item number n can be taken without waiting
__device__ __forceinline__ bool item_ready(ItemRing* r, int n) {
  return mbar_test_warp(r->full + n % kItemSlots, (n / kItemSlots) & 1);
}

// Row tiles of 2^log_per tokens in a grid that knows no length: sequence b owns the slots from (cu[b] + b (per - 1)) / per on, room for its
// tiles whatever its length (floor(x + y) >= floor(x) + floor(y)), at most one of which stands for nothing.
__host__ __device__ __forceinline__ long long row_tile_slots(long long tokens, long long sequences, int log_per) {
  return (tokens + sequences * ((1 << log_per) - 1)) >> log_per;
}
// The sequence of a slot is searched for, 32 ways a turn: two dependent loads for 1024 sequences.  (Counting tiles through the sequences,
// 32 a turn, made 4096 sequences of 16 tokens, 64q/4kv, causal, take 6020 us; with a search it is 770, with a CTA per item and the
// sequence in the grid it was 1010.)
// A whole warp looks up slot `want`; false for a slot without a tile.
__device__ __forceinline__ bool find_row_tile(const int* __restrict__ cu, int nseq, int log_per, int want, int& b, int& start, int& len,
                                              int& tile) {
  const int lane = lane_id();
  int span = nseq, first = 0, next = 0, src = 0;
  b = 0;
  for (int step = 0; step != 1;) {
    step = (span + 31) >> 5;
    const int mine = b + lane * step;
    const bool in = lane * step < span;
    if (in) {
      first = __ldg(cu + mine);
      if (step == 1) next = __ldg(cu + mine + 1);
    }
    const unsigned hit = __ballot_sync(0xffffffffu, in && row_tile_slots(first, mine, log_per) <= want);
    if (!hit) return false;
    src = 31 - __clz(hit);
    b += src * step;
    span = min(step, span - src * step);
  }
  start = __shfl_sync(0xffffffffu, first, src);
  len = __shfl_sync(0xffffffffu, next, src) - start;
  tile = want - (int)row_tile_slots(start, b, log_per);
  return ((long long)tile << log_per) < len;
}

// The producer warp's loop.  The next item is asked for before the loads of the present one are issued and looked up after them: its
// first loads follow at once, and a CTA never holds more than one item that another could have started.  `lookup(block, item)` says
// whether the block stands for an item; `load(item)` issues its loads.  The whole warp calls both.
template <typename Lookup, typename Load>
__device__ __forceinline__ void produce_items(StealSlot* steal, ItemRing* ring, const Status& st, Lookup lookup, Load load) {
  const bool first_lane = lane_id() == 0;
  uint3 blk = blockIdx;
  AttnItem w;
  int out = 0;
  bool more = true;
  for (int req = 0; more; ++req) {
    if (first_lane) steal_request(steal);
    if (lookup(blk, w)) {
      if (first_lane) item_publish(ring, out, w, st);
      __syncwarp();
      ++out;
      load(w);
    }
    more = steal_answer(steal, req, blk, st);
  }
  w.head = -1;
  if (first_lane) item_publish(ring, out, w, st);
  __syncwarp();
}

}  // namespace nsa
