// dK/dV pass of the top-k sparse attention on the 5th-generation tensor cores (head_dim 64 and 128).
//
// Work item = one tile of 64 keys of a selected block (K and V tile resident in SMEM) x a stream of row tiles taken from
// the block's inverted index (the tokens that selected it); a row tile is 128 rows = (128/G tokens) x (G query
// heads).  All five products have M = 128:
//     S    = Q  K^T          [128 rows x 64 keys]   A = Q  (K-major),  B = K tile (K-major)
//     dP   = dO V^T          [128 rows x 64 keys]   A = dO (K-major),  B = V tile (K-major)
//     dV^T = dO^T P          [128 d    x 64 keys]   A = dO (MN-major), B = P  [rows][keys] (MN-major)
//     dK^T = Q^T  dS         [128 d    x 64 keys]   A = Q  (MN-major), B = dS [rows][keys] (MN-major)
//     dQ^T = K^T  dS^T       [128 d    x 128 rows]  A = K tile (MN-major), B = dS [rows][keys] (K-major)
// so the token/head rows are the reduction dimension of dV and dK and the G heads of a KV group are summed
// inside the MMA.  dV^T and dK^T stay in TMEM for the whole item and are added to the fp32 accumulators in global memory at
// its end; S and dP have one TMEM buffer each (the softmax threads read them into registers at once), dQ has two.
//
// dQ comes out of this pass because the K tile is resident and dS already sits in shared memory: the contribution of a
// key tile to the rows' dQ costs one more product (4 MMAs of 128 x 128 x 16) and no operand
// traffic.  A per-token kernel would fetch the 64-key tile again for every token that selected it (32 KB per token and
// block through the L2-to-SM path, the bound of such a kernel); here the tile is shared by every token of the list and
// what leaves the SM is the 128 x 128 fp32 partial result, added to the dQ accumulator with red.global.add.f32.  The
// product is computed TRANSPOSED (d on the TMEM lanes) so that the 32 lanes of a warp hold 32 consecutive d of one
// (token, head) row: one reduction instruction then covers one whole 128-byte line.  Measured on this part, reductions
// into L2-resident lines run at 24 bytes a clock and SM when a warp instruction covers whole lines (scalar or v4 alike; copy-engine
// reductions of 8 KB: 23), 2.8 TB/s when each lane hits its own line (a thread owning a row), and 10 bytes a clock when the lines
// live in HBM: the work items are ordered by token window (index_scan) so that the accumulator rows being reduced into stay
// resident in L2.
//
// The rows of a tile are scattered tokens (4 KB of Q and of dO each at G = 16); a token's G heads are one TMA box per panel of
// 64 d.  Boxes of 2 KB arrive at 26 bytes a clock and SM, cp.async at more than 60, but cp.async shares the load/store path with
// the reductions, which hold it for 2700 clocks of every tile, and takes four warps to issue.  The Q ring has three stages (a Q
// tile lives from its S product to its dK product), the dO ring two.
//   warps 0..7  : two threads per row (32 of the 64 key columns each).  P phase (after S): P = exp2(S*scale - lse)
//                 -> 16-bit SMEM tile; dS phase (after dP): dS = P (dP - delta) scale -> SMEM tile.  The per-row
//                 (lse, delta) come straight from global memory, fetched one tile ahead.  At the end they drain
//                 dV / dK from TMEM
//   warps 8, 9  : Q and dO rows (warps 10, 11: idle)
//   warp 12     : S and dP products (converged warp, one elected lane issues)
//   warps 13..16: dQ drain: warp w owns the TMEM lanes (= d) of quarter w % 4 and adds the 128 rows of
//                 every tile's dQ^T to the fp32 accumulator
//   warp 17     : dV, dQ and dK products
//   warp 18     : claims items, describes them to the others, loads their K and V tiles
//
// What bounds it: the reductions.  65 536 tokens, 64q/4kv, top-16, clocks of a row tile and SM: 3750, of which the drain warps are
// in their reductions 3300; 2300 with the reductions left out (timing-only build).  One warp that issued all five products was
// busy all the time, 700 to 850 clocks a product (250 of them in waits, commits and addresses, with the pipe running dry), and a
// tile took 4600 clocks.  Same GPU, one buffer for dQ, one issuing warp, cp.async and items of 64 tiles -> this, items of 32 tiles
// (attn_bwd.cu): 65 536 tokens 9.8 -> 9.0 ms (the clock falls under the power cap: 1.5 GHz), 16 384 in three sequences 2132 ->
// 1840 us, 8192 tokens 32q/8kv 678 -> 601, 16q/2kv 308 -> 264 us.  With dQ staged in shared memory for the copy engine (Q ring of
// two) the four staging warps bound a tile at 5000 clocks: 11.7 ms.
// TMEM columns: S [0,64) dP [64,128) dV^T [128,192) dK^T [192,256) dQ0 [256,384) dQ1 [384,512).
//
// head_dim 64: d alone is half a row dimension, so two operands are stacked to fill it.  A stage holds a tile's dO and Q rows as
// two panels of one 128-row operand and a P/dS pair its two tiles as panels of one 128-column operand, and ONE product
//     [dO^T; Q^T] [P dS]     [128 x 128]           dV^T is its upper left quadrant, dK^T its lower right one
// takes the place of two with M = 64 (512 clocks; the other two quadrants are computed and never read); [K^T; V^T] dS^T gives
// dQ^T in its upper half.  Tiles and stages are half as large, so P/dS pairs are double-buffered and both row rings have three
// stages.  Measured against the mma.sync kernels that served head_dim 64 before (16 rows per warp, dQ by a per-token kernel of its
// own): 7833 tokens, 16q/2kv, top-8: 516 -> 128 us, now 105.
#include <algorithm>

#include "attn_bwd.h"
#include "host_util.h"
#include "tc5.cuh"

namespace nsa {

namespace {
constexpr int kSpRowPanel = 128 * 128;      // [128 rows][64 d]
constexpr int kSpKvPanel = 64 * 128;        // [64 keys][64 d]
constexpr int kSpPdBytes = 128 * 64 * 2;    // P or dS tile [128 rows][64 keys]: one panel
constexpr int kSpItemQ = 2;                // entries of a CTA's queue of work items
template <int D>
struct SpCfg {
  static constexpr int kPanels = D / 64;
  static constexpr int kQStages = 3, kDoStages = D == 128 ? 2 : 3;
  static constexpr int kPdBufs = D == 128 ? 1 : 2;             // P/dS pairs
  static constexpr int kRowBytes = kPanels * kSpRowPanel;      // Q or dO rows of one tile
  static constexpr int kKvBytes = kPanels * kSpKvPanel;        // K or V tile
  static constexpr int kQStride = D == 128 ? kRowBytes : 2 * kRowBytes, kDoStride = kQStride;  // from a stage to the next
  static constexpr int kRings = (kQStages + kDoStages) * kRowBytes;
  static constexpr size_t kSmem = 2 * kKvBytes + kPdBufs * 2 * kSpPdBytes + kRings + 48 * sizeof(uint64_t) + 16 + kSpItemQ * 32;  // rows, barriers, TMEM address, item queue
};
constexpr int kTmS = 0, kTmDp = 64, kTmAcc = 128, kTmDq = 256;  // TMEM columns: logits, dP, dV and dK (64 each), two buffers for dQ
constexpr int kSpWarps = 19, kSpThreads = kSpWarps * 32;
}  // namespace

// One work item: a 64-key tile of a selected block and (a chunk of) the list of tokens that selected the block.
struct alignas(16) SpItem {
  int h, qs, kpos, krow0, kvalid, tok_begin, tok_count;
  int ntiles;  // 0: nothing to do (past the end of the sequence, or an empty chunk); in a queue entry -1: no more items
};

template <typename T, int LOGG, int D>
__global__ void __launch_bounds__(kSpThreads, 1)
sparse_dkdv_tc_kernel(const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmQ,
                      const __grid_constant__ CUtensorMap tmDO, DkdvParams p) {
  constexpr int logG = LOGG;
  constexpr int G = 1 << LOGG;
  constexpr int KT = 64;
  using C = SpCfg<D>;
  constexpr int PANELS = C::kPanels, NB = C::kPdBufs;
  constexpr int kLoaders = 2;                         // loader warps
  constexpr int kItemReaders = kSpWarps - 3;          // warps that read an entry of the item queue: all but the one that writes it and two idle ones
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* k_sm = smem;
  uint8_t* v_sm = k_sm + C::kKvBytes;
  uint8_t* p_sm = v_sm + C::kKvBytes;              // [NB] pairs of a P and a dS tile
  uint8_t* ds_sm = p_sm + kSpPdBytes;
  uint8_t* rings = p_sm + NB * 2 * kSpPdBytes;
  uint8_t* q_ring = D == 128 ? rings : rings + C::kRowBytes;                      // head_dim 64: dO and Q of a stage side by side
  uint8_t* do_ring = D == 128 ? rings + C::kQStages * C::kRowBytes : rings;
  SpItem* item_q = reinterpret_cast<SpItem*>(rings + C::kRings);   // [kSpItemQ]
  uint64_t* bars = reinterpret_cast<uint64_t*>(item_q + kSpItemQ);
  uint64_t* k_full = bars;
  uint64_t* v_full = bars + 1;
  uint64_t* kv_empty = bars + 2;              // [0] K (head_dim 64: and V) tile no longer read, [1] V tile
  uint64_t* q_full = bars + 4;
  uint64_t* q_empty = q_full + C::kQStages;
  uint64_t* do_full = q_empty + C::kQStages;
  uint64_t* do_empty = do_full + C::kDoStages;
  uint64_t* s_full = do_empty + C::kDoStages;
  uint64_t* s_empty = s_full + 1;
  uint64_t* dp_full = s_empty + 1;
  uint64_t* dp_empty = dp_full + 1;
  uint64_t* p_full = dp_empty + 1;            // [NB] each
  uint64_t* p_empty = p_full + NB;
  uint64_t* ds_full = p_empty + NB;
  uint64_t* ds_empty = ds_full + NB;
  uint64_t* all_done = ds_empty + NB;
  uint64_t* dq_full = all_done + 1;           // [2]
  uint64_t* dq_empty = dq_full + 2;           // [2]
  uint64_t* acc_free = dq_empty + 2;          // the dV / dK accumulators of the previous item have been read out
  uint64_t* iq_full = acc_free + 1;           // [kSpItemQ] an entry of the CTA's item queue has been written
  uint64_t* iq_empty = iq_full + kSpItemQ;    // [kSpItemQ] all warps have read it
  uint64_t* iq_begun = iq_empty + kSpItemQ;   // the loaders have begun an item: the next one may be claimed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(iq_begun + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int TPT = 128 >> logG;  // tokens per row tile
  if (smem_u32(smem) & 1023u) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) p.st.raise(kErrSmemLayout);
    return;
  }

  // ---- the CTA is persistent: it takes items from a grid-wide counter, in list order ----
  // (In order, because the list is sorted by token window: CTAs that run together then reduce into the same L2-resident part
  // of the dQ accumulator.  A fixed stride per CTA let them drift windows apart: 15.8 ms against 10.2 ms.)  A warp of its own
  // claims the CTA's next item, works out what it is (a chain of dependent loads) and leaves the description in a small
  // shared-memory queue that all other warps read, each at its own pace; it also loads the items' K and V tiles.
  // Tensor memory, barriers and the warps' roles are set up once; the rings, the TMEM buffers and every barrier phase run
  // on across items (tile index j counts the tiles of all items of this CTA), so that the gathers, the first logits and the
  // P phase of an item overlap the last products and the dV / dK read-out of the item before it.
  const int total_x = p.Hkv * p.NW * p.TB;
  const int nsub = p.block_size / KT;                          // 64-key tiles per selected block
  const int n_items = __ldg(p.item_base + total_x) * nsub;     // work items: (entry of the list, tile of the block)
  if (n_items <= 0) return;
  auto load_item = [&](int work) -> SpItem {
    SpItem it;
    const int item = work / nsub, ysub = work - item * nsub;
    const int x = __ldg(p.item_bin + item);  // the item's bin, written by index_scan
    const int base = __ldg(p.item_base + x), off0 = __ldg(p.offsets + x), off1 = __ldg(p.offsets + x + 1);
    it.h = x / (p.NW * p.TB);
    const int gb = x % p.TB;
    const int b = find_block_sequence(p.cu_q, p.B, gb, p.block_size);
    it.qs = __ldg(p.cu_q + b);
    const int Lq = __ldg(p.cu_q + b + 1) - it.qs;
    const int blk = gb - block_base(it.qs, b, p.block_size);
    it.kpos = blk * p.block_size + ysub * KT;
    it.krow0 = it.qs + it.kpos;
    it.kvalid = min(KT, Lq - it.kpos);
    const int c = item - base;
    it.tok_begin = off0 + c * p.chunk;
    it.tok_count = min(p.chunk, (off1 - off0) - c * p.chunk);
    it.ntiles = (it.kvalid > 0 && it.tok_count > 0) ? (it.tok_count + TPT - 1) / TPT : 0;
    return it;
  };

  if (threadIdx.x == 0) {
    mbar_init(k_full, 1);
    mbar_init(v_full, 1);
    mbar_init(kv_empty, 1);
    mbar_init(kv_empty + 1, 1);
    for (int s = 0; s < C::kQStages; ++s) {
      mbar_init(q_full + s, 1);
      mbar_init(q_empty + s, 1);
    }
    for (int s = 0; s < C::kDoStages; ++s) {
      mbar_init(do_full + s, 1);
      mbar_init(do_empty + s, D == 128 ? 2 : 1);  // read by dP and dV, which come from two warps (head_dim 64: see issue_pair)
    }
    mbar_init(s_full, 1);
    mbar_init(s_empty, 8);
    mbar_init(dp_full, 1);
    mbar_init(dp_empty, 8);
    for (int s = 0; s < NB; ++s) {
      mbar_init(p_full + s, 8);
      mbar_init(p_empty + s, 1);
      mbar_init(ds_full + s, 8);
      mbar_init(ds_empty + s, 2);  // dK and dQ read the dS tile
    }
    mbar_init(all_done, 1);
    for (int s = 0; s < 2; ++s) {
      mbar_init(dq_full + s, 1);
      mbar_init(dq_empty + s, D / 32);  // the warps that drain it
    }
    mbar_init(acc_free, 8);
    for (int s = 0; s < kSpItemQ; ++s) {
      mbar_init(iq_full + s, 1);
      mbar_init(iq_empty + s, kItemReaders);
    }
    mbar_init(iq_begun, kLoaders);
    fence_barrier_init();
  }
  if (warp == 12) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  // k-th item of this CTA, read once by every warp that works on items; ntiles < 0 ends the sequence
  auto take = [&](int k) -> SpItem {
    const int s = k % kSpItemQ;
    SpItem it;
    it.ntiles = -1;
    if (!mbar_wait(iq_full + s, (k / kSpItemQ) & 1, p.st)) return it;
    const int4* e = reinterpret_cast<const int4*>(item_q + s);
    const int4 a = e[0], c = e[1];
    it.h = a.x; it.qs = a.y; it.kpos = a.z; it.krow0 = a.w;
    it.kvalid = c.x; it.tok_begin = c.y; it.tok_count = c.z; it.ntiles = c.w;
    __syncwarp();
    if (lane == 0) mbar_arrive(iq_empty + s);
    return it;
  };

  // every role walks the same list of items; `gt` is the number of tiles of the items before the current one
  if (warp == 8 || warp == 9) {
    // ===================== loaders: warp 8 the Q rows, warp 9 the dO rows; a token's heads are one TMA box per panel =====================
    const bool is_q = warp == 8;
    const CUtensorMap* tm = is_q ? &tmQ : &tmDO;
    uint64_t* full = is_q ? q_full : do_full;
    uint64_t* empty = is_q ? q_empty : do_empty;
    uint8_t* ring = is_q ? q_ring : do_ring;
    const int stages = is_q ? C::kQStages : C::kDoStages;
    // a lane's boxes: one token of the tile (32 is a multiple of their number), every kPnStep-th panel
    constexpr int kPnStep = G / 4;
    const int pn0 = lane >> (7 - LOGG), slot = lane & (TPT - 1);
    const uint32_t off = slot * (G * 128);
    int s = 0;
    uint32_t round = 0;  // parity of the ring's round
    bool first = true;
    for (int k = 0;; ++k) {
      const SpItem cur = take(k);
      if (cur.ntiles < 0) break;
      if (lane == 0) mbar_arrive(iq_begun);
      auto token_of = [&](int i) {
        const int ti = i * TPT + slot;
        return ti < cur.tok_count ? __ldg(p.list + cur.tok_begin + ti) : -1;  // a missing token: out of range, zero fill
      };
      int n = token_of(0);
      for (int i = 0; i < cur.ntiles; ++i) {
        const int next_n = token_of(i + 1);
        if (!first) mbar_wait(empty + s, round ^ 1u, p.st);
        if (lane == 0) mbar_expect_tx(full + s, C::kRowBytes);
        __syncwarp();
#pragma unroll
        for (int pb = 0; pb < PANELS; pb += kPnStep) {
          const int pn = pb + pn0;
          if (pn < PANELS) tma_load_3d(ring + s * C::kQStride + off + pn * kSpRowPanel, tm, full + s, pn * 64, cur.h * G, n);
        }
        n = next_n;
        if (++s == stages) {
          s = 0;
          round ^= 1u;
          first = false;
        }
      }
    }
  } else if (warp == 18) {
    // ===================== items: claimed, described and queued; their K and V tiles =====================
    if (lane == 0) {
      int n_begun = 0;
      for (int k = 0;; ++k) {
        // one item ahead of the loaders, no more: what a CTA has claimed no other can take
        if (k > 0 && !mbar_wait(iq_begun, n_begun++ & 1, p.st)) break;
        SpItem it;
        it.ntiles = -1;
        for (int item; (item = atomicAdd(p.item_counter, 1)) < n_items;) {
          it = load_item(item);
          if (it.ntiles > 0) break;
          it.ntiles = -1;
        }
        const int s = k % kSpItemQ;
        if (k >= kSpItemQ && !mbar_wait(iq_empty + s, ((k / kSpItemQ) - 1) & 1, p.st)) break;
        int4* e = reinterpret_cast<int4*>(item_q + s);
        e[0] = make_int4(it.h, it.qs, it.kpos, it.krow0);
        e[1] = make_int4(it.kvalid, it.tok_begin, it.tok_count, it.ntiles);
        mbar_arrive(iq_full + s);
        if (it.ntiles < 0) break;
        // V is read by the item's dP products alone (head_dim 64: by dQ as well), K by S and dQ
        if (k > 0 && !mbar_wait(kv_empty + (D == 128 ? 1 : 0), (k - 1) & 1, p.st)) break;
        mbar_expect_tx(v_full, C::kKvBytes);
#pragma unroll
        for (int pn = 0; pn < PANELS; ++pn) tma_load_3d(v_sm + pn * kSpKvPanel, &tmV, v_full, pn * 64, it.h, it.krow0);
        if (D == 128 && k > 0 && !mbar_wait(kv_empty, (k - 1) & 1, p.st)) break;
        mbar_expect_tx(k_full, C::kKvBytes);
#pragma unroll
        for (int pn = 0; pn < PANELS; ++pn) tma_load_3d(k_sm + pn * kSpKvPanel, &tmK, k_full, pn * 64, it.h, it.krow0);
      }
    }
  } else if (warp == 12) {
    // ===================== S and dP products (converged warp, elected lane issues) =====================
    const uint32_t idesc_s = umma_idesc<T>(128, KT, false, false);
    const uint32_t k_addr = smem_u32(k_sm), v_addr = smem_u32(v_sm), q_base = smem_u32(q_ring), do_base = smem_u32(do_ring);
    // A = rows (two [128][64] panels), B = K or V tile (two [64][64] panels)
    auto issue_logits = [&](uint32_t a_addr, uint32_t b_addr, uint32_t d_tmem) {
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk)
        umma_ss(d_tmem, umma_desc_kmajor(a_addr + (kk >> 2) * kSpRowPanel + (kk & 3) * 32),
                umma_desc_kmajor(b_addr + (kk >> 2) * kSpKvPanel + (kk & 3) * 32), idesc_s, kk > 0);
    };
    int j = 0;
    bool alive = true;
    for (int k = 0; alive; ++k) {
      const SpItem cur = take(k);
      if (cur.ntiles < 0) break;
      for (int i = 0; i < cur.ntiles; ++i, ++j) {
        const int sq = j % C::kQStages, sd = j % C::kDoStages;
        alive = (i > 0 || mbar_wait(k_full, k & 1, p.st)) && mbar_wait(q_full + sq, (j / C::kQStages) & 1, p.st) &&
                (j == 0 || mbar_wait(s_empty, (j - 1) & 1, p.st));
        if (!alive) break;
        tc_fence_after_sync();
        if (elect_one()) {
          issue_logits(q_base + sq * C::kQStride, k_addr, tmem + kTmS);
          umma_commit(s_full);
        }
        __syncwarp();
        alive = (i > 0 || mbar_wait(v_full, k & 1, p.st)) && mbar_wait(do_full + sd, (j / C::kDoStages) & 1, p.st) &&
                (j == 0 || mbar_wait(dp_empty, (j - 1) & 1, p.st));
        if (!alive) break;
        tc_fence_after_sync();
        if (elect_one()) {
          issue_logits(do_base + sd * C::kDoStride, v_addr, tmem + kTmDp);
          umma_commit(dp_full);
          if (D == 128) {
            umma_commit(do_empty + sd);
            if (i == cur.ntiles - 1) umma_commit(kv_empty + 1);
          }
        }
        __syncwarp();
      }
    }
  } else if (warp == 17) {
    // ===================== dV, dK and dQ products (converged warp, elected lane issues) =====================
    // A warp of its own, because the tensor pipe's queue is shallow: whatever an issuing warp does between two products (waits,
    // commits, ring addresses: 250 clocks of 700 when one warp issued all five) is time in which the pipe runs dry, unless the
    // other warp's products fill it.
    const uint32_t idesc_t = umma_idesc<T>(128, D == 128 ? KT : 2 * KT, true, true);
    const uint32_t k_addr = smem_u32(k_sm), p_addr = smem_u32(p_sm), ds_addr = smem_u32(ds_sm);
    const uint32_t q_base = smem_u32(q_ring), do_base = smem_u32(do_ring);
    // dV^T/dK^T: reduction over the 128 rows, 16 at a time; A = rows MN-major (d as M), B = P or dS tile MN-major
    auto issue_grad = [&](uint32_t a_addr, uint32_t b_addr, uint32_t d_tmem, bool first, uint64_t* bar_rows, uint64_t* bar_tile) {
      if (elect_one()) {
        umma_ss(d_tmem, umma_desc_mnmajor(a_addr, kSpRowPanel), umma_desc_mnmajor(b_addr, kSpPdBytes), idesc_t, !first);
#pragma unroll
        for (int kk = 1; kk < 128 / 16; ++kk)
          umma_ss(d_tmem, umma_desc_mnmajor(a_addr + kk * 2048, kSpRowPanel), umma_desc_mnmajor(b_addr + kk * 2048, kSpPdBytes),
                  idesc_t, true);
        umma_commit(bar_rows);
        umma_commit(bar_tile);
      }
      __syncwarp();
    };
    // dQ^T = K^T dS^T: A = K tile MN-major (d as M over two panels, 16 keys = 2048 bytes; head_dim 64: the K tile and the V tile
    // behind it), B = dS tile K-major (one panel)
    const uint32_t idesc_q = umma_idesc<T>(128, 128, true, false);
    auto issue_dq = [&](int buf, uint32_t ds_addr, uint64_t* bar_tile) {
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk)
          umma_ss(tmem + kTmDq + buf * 128, umma_desc_mnmajor(k_addr + kk * 2048, kSpKvPanel), umma_desc_kmajor(ds_addr + kk * 32), idesc_q, kk > 0);
        umma_commit(dq_full + buf);
        umma_commit(bar_tile);
      }
      __syncwarp();
    };
    auto issue_pair = [&](uint32_t a_addr, uint32_t b_addr, bool first, int stage, int buf) {
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma_ss(tmem + kTmAcc, umma_desc_mnmajor(a_addr + kk * 2048, kSpRowPanel), umma_desc_mnmajor(b_addr + kk * 2048, kSpPdBytes), idesc_t,
                  !first || kk > 0);
        umma_commit(do_empty + stage);
        umma_commit(q_empty + stage);
        umma_commit(p_empty + buf);
        umma_commit(ds_empty + buf);
      }
      __syncwarp();
    };
    int j = 0;
    bool alive = true;
    for (int k = 0; alive; ++k) {
      const SpItem cur = take(k);
      if (cur.ntiles < 0) break;
      for (int i = 0; i < cur.ntiles; ++i, ++j) {
        const int sq = j % C::kQStages, sd = j % C::kDoStages, pd = j % NB;
        // dV^T / dK^T restart from zero with an item: not before the softmax warps have read out the previous item's
        alive = i > 0 || k == 0 || mbar_wait(acc_free, (k - 1) & 1, p.st);
        if constexpr (D == 128) {
          alive = alive && mbar_wait(do_full + sd, (j / C::kDoStages) & 1, p.st) && mbar_wait(p_full, j & 1, p.st);
          if (!alive) break;
          tc_fence_after_sync();
          issue_grad(do_base + sd * C::kDoStride, p_addr, tmem + kTmAcc, i == 0, do_empty + sd, p_empty);
        }
        alive = alive && mbar_wait(ds_full + pd, (j / NB) & 1, p.st) && (j < 2 || mbar_wait(dq_empty + (j & 1), ((j >> 1) - 1) & 1, p.st));
        if (!alive) break;
        tc_fence_after_sync();
        issue_dq(j & 1, ds_addr + pd * 2 * kSpPdBytes, ds_empty + pd);
        // S, dP and dQ of the item's last tile: nothing reads its K tile any more
        if (i == cur.ntiles - 1 && elect_one()) umma_commit(kv_empty);
        __syncwarp();
        if constexpr (D == 128)
          issue_grad(q_base + sq * C::kQStride, ds_addr, tmem + kTmAcc + 64, i == 0, q_empty + sq, ds_empty);
        else  // dS written, P is too (by the same threads, before it): both gradients in one product over the stacked operands
          issue_pair(do_base + sd * C::kDoStride, p_addr + pd * 2 * kSpPdBytes, i == 0, sq, pd);
      }
      if (alive && elect_one()) umma_commit(all_done);
      __syncwarp();
    }
  } else if (warp >= 13) {
    // ===================== dQ drain: lane = d, 128 columns = the rows of the tile =====================
    if (D == 128 || (warp & 3) < 2) {  // head_dim 64: the upper half of the lanes holds dQ^T
      constexpr int SPC = 32 >> LOGG;  // tokens (slots) per chunk of 32 columns
      const uint32_t lane_dq = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kTmDq;
      int gt = 0;
      bool alive = true;
      for (int k = 0; alive; ++k) {
        const SpItem cur = take(k);
        if (cur.ntiles < 0) break;
        {
          const int tok_begin = cur.tok_begin, tok_count = cur.tok_count;
          float* const dst = p.dq32 + (long long)(cur.h * G) * D + (warp & 3) * 32 + lane;
          // lane t holds the id of the tile's t-th token, fetched a tile ahead
          auto tile_tokens = [&](int i) {
            const int ti = i * TPT + lane;
            return (lane < TPT && ti < tok_count) ? __ldg(p.list + tok_begin + ti) : -1;
          };
          int my_n = tile_tokens(0);
          uint32_t ra[32], rb[32];
          bool loaded = false;  // ra holds the tile's first 32 columns
          for (int i = 0; i < cur.ntiles; ++i) {
            const int next_n = tile_tokens(i + 1);
            const int j = gt + i, buf = j & 1;
            const uint32_t lane_base = lane_dq + buf * 128;
            // one reduction per row: the warp's 32 lanes add 32 consecutive floats of the (token, head) row
            auto reduce_chunk = [&](const uint32_t (&r)[32], int c) {
#pragma unroll
              for (int s2 = 0; s2 < SPC; ++s2) {
                const int n = __shfl_sync(0xffffffffu, my_n, c * SPC + s2);
                if (n >= 0) {
                  float* row_dst = dst + (long long)n * p.Hq * D;
#pragma unroll
                  for (int g = 0; g < G; ++g) red_add1(row_dst + g * D, r[s2 * G + g]);
                }
              }
            };
            if (!loaded) {
              if (!mbar_wait(dq_full + buf, (j >> 1) & 1, p.st)) { alive = false; break; }
              tc_fence_after_sync();
              tmem_ld32(lane_base, ra);
              tmem_ld_wait();
            }
            // the next 32 columns are fetched while the reductions of these 32 wait for their turn
            tmem_ld32(lane_base + 32, rb);
            reduce_chunk(ra, 0);
            tmem_ld_wait();
            tmem_ld32(lane_base + 64, ra);
            reduce_chunk(rb, 1);
            tmem_ld_wait();
            tmem_ld32(lane_base + 96, rb);
            reduce_chunk(ra, 2);
            tmem_ld_wait();
            // the rest of the buffer is in registers: the product of the tile after next may overwrite it
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(dq_empty + buf);
            // the next tile's first columns, if its product is done by now (else what is read here is not used)
            loaded = i + 1 < cur.ntiles && mbar_test_warp(dq_full + (buf ^ 1), ((j + 1) >> 1) & 1);
            tc_fence_after_sync();
            tmem_ld32(lane_dq + (buf ^ 1) * 128, ra);
            reduce_chunk(rb, 3);
            tmem_ld_wait();
            my_n = next_n;
          }
          gt += cur.ntiles;
        }
      }
    } else {
      // the queue entries are counted per warp: read them all
      for (int k = 0; take(k).ntiles >= 0; ++k) {
      }
    }
  } else if (warp < 8) {
    // ===================== softmax / dS threads: two threads per row (32 of the 64 key columns each) =====================
    const int half = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const int slot = row >> logG;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t prow0 = smem_u32(p_sm) + row * 128;
    int gt = 0, n_done = 0;
    bool alive = true;
    for (int k = 0; alive; ++k) {
      const SpItem cur = take(k);
      if (cur.ntiles < 0) break;
      {
        const int ntiles = cur.ntiles, tok_begin = cur.tok_begin, tok_count = cur.tok_count, h = cur.h, qs = cur.qs, kpos = cur.kpos,
                  kvalid = cur.kvalid, krow0 = cur.krow0;
        const int head = h * p.G + (row & (p.G - 1));
        // per-row statistics are fetched ahead: the token of tile i+2, (lse, delta) of tile i+1
        auto token_of = [&](int i) { return (i < ntiles && i * TPT + slot < tok_count) ? __ldg(p.list + tok_begin + i * TPT + slot) : -1; };
        auto stats_of = [&](int n) { return n >= 0 ? __ldg(p.ld + (long long)n * p.Hq + head) : make_float2(INFINITY, 0.f); };
        int n_cur = token_of(0), n_next = token_of(1);
        float2 ld_cur = stats_of(n_cur);
        for (int i = 0; i < ntiles && alive; ++i) {
          const int j = gt + i;
          const int pd = j % NB;
          const uint32_t prow = prow0 + pd * 2 * kSpPdBytes, dsrow = prow + kSpPdBytes;
          const int n_next2 = token_of(i + 2);
          const float2 ld_next = stats_of(n_next);
          // keys of this tile the row may see: those at or before its own position
          int lim = n_cur >= 0 ? max(0, min(kvalid, (n_cur - qs) - kpos + 1)) : 0;
          lim -= half * 32;  // relative to this thread's first column
          const float nlse = -ld_cur.x, ndsc = -ld_cur.y * p.sm_scale;

          // ---- P phase ----
          if (!mbar_wait(s_full, j & 1, p.st)) { alive = false; break; }
          tc_fence_after_sync();
          float pf[32];
          {
            uint32_t su[32];
            tmem_ld32(lane_base + kTmS + half * 32, su);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(s_empty);
            // tiles every row of the warp sees in full (all but the block on the diagonal) skip the mask instructions
            if (__all_sync(0xffffffffu, lim >= 32)) {
#pragma unroll
              for (int c2 = 0; c2 < 32; c2 += 2) {
                const float2 x = ffma2(make_float2(__uint_as_float(su[c2]), __uint_as_float(su[c2 + 1])), make_float2(p.scale2, p.scale2),
                                       make_float2(nlse, nlse));
                pf[c2] = fast_exp2(x.x);
                pf[c2 + 1] = fast_exp2(x.y);
              }
            } else {
#pragma unroll
              for (int c2 = 0; c2 < 32; ++c2) pf[c2] = masked_exp2(c2 < lim, fmaf(__uint_as_float(su[c2]), p.scale2, nlse));
            }
            uint32_t pw[16];
#pragma unroll
            for (int c2 = 0; c2 < 16; ++c2) pw[c2] = DT<T>::pack(pf[2 * c2], pf[2 * c2 + 1]);
            if (j >= NB) mbar_wait(p_empty + pd, (j / NB - 1) & 1, p.st);  // dV of the tile that had the P buffer has read it
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(prow + (((half * 4 + c4) ^ (row & 7)) << 4)), "r"(pw[c4 * 4]),
                           "r"(pw[c4 * 4 + 1]), "r"(pw[c4 * 4 + 2]), "r"(pw[c4 * 4 + 3]) : "memory");
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(p_full + pd);

          // ---- dS phase ----
          if (!mbar_wait(dp_full, j & 1, p.st)) { alive = false; break; }
          tc_fence_after_sync();
          {
            uint32_t du[32];
            tmem_ld32(lane_base + kTmDp + half * 32, du);
            tmem_ld_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(dp_empty);
            uint32_t dw[16];
#pragma unroll
            for (int c2 = 0; c2 < 32; c2 += 2) {
              const float2 t2 = ffma2(make_float2(__uint_as_float(du[c2]), __uint_as_float(du[c2 + 1])), make_float2(p.sm_scale, p.sm_scale),
                                      make_float2(ndsc, ndsc));
              const float2 d2 = fmul2(make_float2(pf[c2], pf[c2 + 1]), t2);
              dw[c2 >> 1] = DT<T>::pack(d2.x, d2.y);
            }
            if (j >= NB) mbar_wait(ds_empty + pd, (j / NB - 1) & 1, p.st);  // dK (and dQ) have read the dS buffer
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4)
              asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(dsrow + (((half * 4 + c4) ^ (row & 7)) << 4)), "r"(dw[c4 * 4]),
                           "r"(dw[c4 * 4 + 1]), "r"(dw[c4 * 4 + 2]), "r"(dw[c4 * 4 + 3]) : "memory");
          }
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(ds_full + pd);
          n_cur = n_next;
          n_next = n_next2;
          ld_cur = ld_next;
        }
        if (!alive) break;
        // ---- read out dV and dK of this item: thread (d, half) holds column d for 32 of the 64 keys ----
        if (!mbar_wait(all_done, n_done & 1, p.st)) { alive = false; break; }
        tc_fence_after_sync();
        if constexpr (D == 128) {
          const int d = row;
          uint32_t rv[32], rk[32];
          tmem_ld32(lane_base + kTmAcc + half * 32, rv);
          tmem_ld32(lane_base + kTmAcc + 64 + half * 32, rk);
          tmem_ld_wait();
          // the accumulators are in registers: the next item's dV / dK products may start
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_free);
          float* dstv = p.dv32 + ((size_t)krow0 * p.Hkv + h) * D + d;
          float* dstk = p.dk32 + ((size_t)krow0 * p.Hkv + h) * D + d;
#pragma unroll
          for (int c2 = 0; c2 < 32; ++c2) {
            const int key = half * 32 + c2;
            if (key < kvalid) {
              atomicAdd(dstv + (size_t)key * p.Hkv * D, __uint_as_float(rv[c2]));
              atomicAdd(dstk + (size_t)key * p.Hkv * D, __uint_as_float(rk[c2]));
            }
          }
        } else {  // lanes below 64 hold a column of dV in the left half of the product, lanes above one of dK in the right half
          const bool is_v = (warp & 3) < 2;
          uint32_t r[32];
          tmem_ld32(lane_base + kTmAcc + (is_v ? 0 : 64) + half * 32, r);
          tmem_ld_wait();
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive(acc_free);
          float* dst = (is_v ? p.dv32 : p.dk32) + ((size_t)krow0 * p.Hkv + h) * D + (row & 63);
#pragma unroll
          for (int c2 = 0; c2 < 32; ++c2) {
            const int key = half * 32 + c2;
            if (key < kvalid) atomicAdd(dst + (size_t)key * p.Hkv * D, __uint_as_float(r[c2]));
          }
        }
        gt += ntiles;
        ++n_done;
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 12) tmem_dealloc(tmem, 512);
}

template <typename T, int D>
int launch_sparse_dkdv_tc(const void* q, const void* dout, const void* k, const void* v, const long long* strides, int Nk, dim3 grid,
                          DkdvParams p, cudaStream_t stream) {
  int logG = 0;
  while ((1 << logG) < p.G) ++logG;
  CUtensorMap tmK, tmV;
  int rc = make_tmap_3d(&tmK, DT<T>::kTmapType, k, D, p.Hkv, Nk, strides[3], strides[2], 64, 1, 64);
  if (rc) return rc;
  rc = make_tmap_3d(&tmV, DT<T>::kTmapType, v, D, p.Hkv, Nk, strides[5], strides[4], 64, 1, 64);
  if (rc) return rc;
  const size_t smem = SpCfg<D>::kSmem;
  // a token's rows as TMA boxes; an expanded gradient's strides of 0 are multiples of 16 bytes like any others
  CUtensorMap tmQ, tmDO;
  rc = make_tmap_3d(&tmQ, DT<T>::kTmapType, q, D, p.Hq, Nk, strides[1], strides[0], 64, p.G, 1);
  if (rc) return rc;
  rc = make_tmap_3d(&tmDO, DT<T>::kTmapType, dout, D, p.Hq, Nk, strides[7], strides[6], 64, p.G, 1);
  if (rc) return rc;
  auto launch = [&](auto kern) -> int {
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return cuda_rc(e);
    LaunchScope ls_("sparse_dkdv_tc", stream);
    // persistent CTAs: one per SM (shared memory and the 512 TMEM columns allow no more), each taking work items from a
    // grid-wide counter; grid.x * grid.y on entry is the upper bound of their number
    const int sms = num_sms();
    const unsigned long long bound = (unsigned long long)grid.x * grid.y;   // (list entries) x (tiles per block)
    grid = dim3((unsigned)std::min<unsigned long long>(bound, (unsigned long long)sms), 1, 1);
    kern<<<grid, kSpThreads, smem, stream>>>(tmK, tmV, tmQ, tmDO, p);
    return cuda_rc(cudaGetLastError());
  };
  switch (logG) {
    case 2: return launch(sparse_dkdv_tc_kernel<T, 2, D>);
    case 3: return launch(sparse_dkdv_tc_kernel<T, 3, D>);
    case 4: return launch(sparse_dkdv_tc_kernel<T, 4, D>);
    default: return kUnsupported;
  }
}

#define NSA_INSTANTIATE(T, D) \
  template int launch_sparse_dkdv_tc<T, D>(const void*, const void*, const void*, const void*, const long long*, int, dim3, DkdvParams, cudaStream_t)
NSA_INSTANTIATE(__nv_bfloat16, 64);
NSA_INSTANTIATE(__nv_bfloat16, 128);
NSA_INSTANTIATE(__half, 64);
NSA_INSTANTIATE(__half, 128);
#undef NSA_INSTANTIATE

}  // namespace nsa
