// Forward of dense varlen GQA attention with the strided-causal mask on the 5th-generation tensor
// cores (tcgen05.mma, accumulators in tensor memory).
//
// A work item is two row tiles A and B of 128 rows each; a row tile is (128/G consecutive query tokens) x (G query heads of one
// KV head); B holds the tokens right after A's.  Key tiles of 128 go through SMEM rings shared by both row tiles.  CTAs are
// persistent: one per SM, which takes over items whose own CTA has not started yet (work_steal.cuh), so that the loads and the
// first products of an item run under the last softmax and the output of the one before it.
//   warp 8      : looks up the items and loads with TMA: Q through a ring of 3 row tiles (which the outputs leave through as well),
//                 K and V tiles through rings of 2, K one tile ahead
//   warp 9      : allocates TMEM; issues, per key tile and row tile, S = Q K^T (SMEM x SMEM -> TMEM) and O += P V
//                 (P read from TMEM, V from SMEM MN-major), alternating between the two row tiles: while the softmax
//                 threads of one tile work, the tensor pipe runs the other tile's products
//   warps 0..3  : softmax of tile A, one thread per row (TMEM lane): row maximum, exponentials, P written as 16-bit pairs back
//                 into tensor memory over the logits, where the P V instruction reads its A operand -- P never touches shared
//                 memory.  (Full tiles of rows that already have a reference maximum take a single pass, see the loop.)  A lazily
//                 updated reference maximum is kept: O and l are rescaled only when the row maximum grows by more than 2^8.  At the
//                 end the threads normalise O and write it to the tile's Q buffer, from where a TMA store takes it (row by row to
//                 memory when not all of the tile's tokens belong to the sequence)
//   warps 4..7  : the same for tile B
//   warp 10     : issues the TMA stores and hands the Q buffers back
// The tensor pipe executes one thread's MMAs in issue order, so S(i+1) of a row tile, issued after its P V(i), cannot
// overwrite P(i) before it has been read.
// TMEM columns: [0,128) S/P of A, [128,256) S/P of B, [256,256+D) O of A, [384,384+D) O of B.
//
// What bounds it: a key tile of both row tiles takes 2930 clocks (2048 of products, 1366 of exponentials): softmax of a row tile,
// the hand-over to the issuing warp, its P V and next S, and the hand-over back are a chain.  A CTA of its own per item cost 12 000
// clocks more each, of which set-up, the first loads and the output now run beside the neighbouring items.  64q/4kv, bf16, d 128,
// this kernel alone, a CTA per item -> persistent: window 512 over 32 768 tokens 999 -> 763 us, window 128 694 -> 454; compressed keys
// of 8192 tokens 180 -> 147, of 16 384 451 -> 371, of 32 768 1276 -> 1102; 4096 keys, none masked, 467 -> 454, 8192 1696 -> 1659;
// 8192 tokens, causal, 938 -> 914; 300 sequences of 200 (32q/2kv) 519 -> 476.
// Two threads per row instead of one: 2.05 us a step against 1.7, the exponentials of A and B then coincide.
#include <type_traits>

#include "attn_tile.cuh"
#include "dispatch.h"
#include "host_util.h"
#include "nsa_b200.h"
#include "tc5.cuh"
#include "work_steal.cuh"

namespace nsa {

#ifndef NSA_POLY_EVERY
#define NSA_POLY_EVERY 3
#endif
constexpr int kPolyEvery = NSA_POLY_EVERY;  // one pair of exponentials in kPolyEvery is evaluated as a polynomial

struct DenseFwdTcParams {
  void* o;
  float* lse;  // [Nq, Hq]
  const int* cu_q;
  const int* cu_k;
  long long o_sn, o_sh;
  int B, Hq, Hkv, G, logG;
  int window, stride, causal;
  int left;  // >= 0: sliding window, a query also needs key >= t - left (plain causal mask only); < 0: no lower bound
  float scale2;
  Status st;
};

__device__ __forceinline__ int visible_keys_tc(int t, int Lk, int window, int stride, int causal) {
  if (!causal) return Lk;
  if (t < window - 1) return 0;
  return min(Lk, (t - window + 1) / stride + 1);
}

constexpr int kTcKeyTile = 128;
constexpr int kTcStages = 2;        // K tiles, and V tiles, in flight
constexpr int kTcQBufs = 3;         // row tiles of Q
constexpr int kTcSoftWarps = 8;     // 4 per row tile
constexpr int kTcThreads = (kTcSoftWarps + 3) * 32;

template <typename T, int D>
__global__ void __launch_bounds__(kTcThreads, 1)
dense_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                    const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, DenseFwdTcParams p) {
  constexpr int PANELS = D / 64;
  constexpr int PANEL_BYTES = 128 * 128;            // 128 rows x 128 B
  constexpr int Q_BYTES = 128 * D * 2;              // one row tile
  constexpr int KV_BYTES = kTcKeyTile * D * 2;      // one K or V tile
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* q_sm = smem;                             // row tile t (A and B of the items in turn) sits in buffer t % kTcQBufs
  uint8_t* k_sm = q_sm + kTcQBufs * Q_BYTES;
  uint8_t* v_sm = k_sm + kTcStages * KV_BYTES;
  StealSlot* steal = reinterpret_cast<StealSlot*>(v_sm + kTcStages * KV_BYTES);
  ItemRing* ring = reinterpret_cast<ItemRing*>(steal + 1);
  uint64_t* bars = reinterpret_cast<uint64_t*>(ring + 1);
  uint64_t* q_full = bars;
  uint64_t* q_empty = q_full + kTcQBufs;     // the row tile's output has left
  uint64_t* k_full = q_empty + kTcQBufs;
  uint64_t* k_empty = k_full + kTcStages;
  uint64_t* v_full = k_empty + kTcStages;
  uint64_t* v_empty = v_full + kTcStages;
  uint64_t* s_full = v_empty + kTcStages;    // [2] per row tile
  uint64_t* p_full = s_full + 2;             // [2]
  uint64_t* pv_done = p_full + 2;            // [2]
  // Per Q buffer, not per row tile: a buffer is not filled again before its output was handled, so a phase cannot be overtaken by the
  // next one while the warp that stores the outputs has yet to look at it.
  uint64_t* o_full = pv_done + 2;            // the output is in the Q buffer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_full + kTcQBufs);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (smem_u32(smem) & 1023u) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) p.st.raise(kErrSmemLayout);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kTcQBufs; ++s) {
      mbar_init(q_full + s, 1);
      mbar_init(q_empty + s, 1);
      mbar_init(o_full + s, kTcSoftWarps / 2);
    }
    for (int s = 0; s < kTcStages; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(k_empty + s, 1);
      mbar_init(v_full + s, 1);
      mbar_init(v_empty + s, 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(s_full + s, 1);
      mbar_init(p_full + s, kTcSoftWarps / 2);
      mbar_init(pv_done + s, 1);
    }
    items_init(ring, steal, kTcSoftWarps + 2);
    fence_barrier_init();
  }
  if (warp == kTcSoftWarps + 1) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  const int QT = 128 >> p.logG;  // tokens per row tile

  if (warp == kTcSoftWarps) {
    // ===================== TMA producer: the whole warp looks the items up, one lane issues =====================
    int rt = 0;    // row tiles loaded so far
    int kt = 0;    // key tiles so far
    auto lookup = [&](uint3 blk, AttnItem& w) {
      int b, tile;
      // long rows first
      if (!find_row_tile(p.cu_q, p.B, 8 - p.logG, (int)gridDim.x - 1 - (int)blk.x, b, w.qs, w.Lq, tile)) return false;
      w.head = blk.y;
      w.ksq = __ldg(p.cu_k + b);
      w.Lk = __ldg(p.cu_k + b + 1) - w.ksq;
      w.q0 = tile * 2 * QT;
      const int t_hi = min(w.q0 + 2 * QT, w.Lq) - 1;
      // with a sliding window the first key tiles are invisible to every row of the item: start at tile kt0
      w.kt0 = p.left >= 0 ? max(0, w.q0 - p.left) / kTcKeyTile : 0;
      w.ntiles = max(0, (visible_keys_tc(t_hi, w.Lk, p.window, p.stride, p.causal) + kTcKeyTile - 1) / kTcKeyTile - w.kt0);
      return true;
    };
    produce_items(steal, ring, p.st, lookup, [&](const AttnItem& w) {
      if (w.ntiles == 0) return;
      if (lane == 0) {
        auto load_q = [&](int g) {
          const int t = rt + g, s = t % kTcQBufs;
          if (t >= kTcQBufs) mbar_wait(q_empty + s, ((t / kTcQBufs) - 1) & 1, p.st);
          mbar_expect_tx(q_full + s, Q_BYTES);
#pragma unroll
          for (int pn = 0; pn < PANELS; ++pn)
            tma_load_3d(q_sm + s * Q_BYTES + pn * PANEL_BYTES, &tmQ, q_full + s, pn * 64, w.head * p.G, w.qs + w.q0 + g * QT);
        };
        auto load_kv = [&](uint8_t* sm, const CUtensorMap* tm, uint64_t* full, uint64_t* empty, int i) {
          const int c = kt + i, s = c % kTcStages;
          if (c >= kTcStages) mbar_wait(empty + s, ((c / kTcStages) - 1) & 1, p.st);
          mbar_expect_tx(full + s, KV_BYTES);
#pragma unroll
          for (int pn = 0; pn < PANELS; ++pn)
            tma_load_3d(sm + s * KV_BYTES + pn * PANEL_BYTES, tm, full + s, pn * 64, w.head, w.ksq + (w.kt0 + i) * kTcKeyTile);
        };
        // in the order in which they find room: Q of tile A (an item ahead), the first K tile, Q of tile B
        load_q(0);
        load_kv(k_sm, &tmK, k_full, k_empty, 0);
        load_q(1);
        for (int i = 0; i < w.ntiles; ++i) {
          if (i + 1 < w.ntiles) load_kv(k_sm, &tmK, k_full, k_empty, i + 1);
          load_kv(v_sm, &tmV, v_full, v_empty, i);
        }
      }
      __syncwarp();
      kt += w.ntiles;
      rt += 2;
    });
  } else if (warp == kTcSoftWarps + 1) {
    // ===================== MMA issuer =====================
    // The whole warp runs the control flow converged; one elected lane issues (see tc5.cuh on why).
    const uint32_t idesc_qk = umma_idesc<T>(128, kTcKeyTile, false, false);
    const uint32_t idesc_pv = umma_idesc<T>(128, D, false, true);
    const uint32_t q_base = smem_u32(q_sm), k_base = smem_u32(k_sm), v_base = smem_u32(v_sm);
    // S of row tile g from the Q at q_addr for the key tile in stage st; the second row tile's product releases the K stage
    auto issue_qk = [&](unsigned st, int g, uint32_t q_addr) {
      const uint32_t k_addr = k_base + st * KV_BYTES;
      if (elect_one()) {
        umma_block_ss<D / 16, PANEL_BYTES>(tmem + (uint32_t)(g * 128), q_addr, k_addr, idesc_qk);
        umma_commit(s_full + g);
        if (g == 1) umma_commit(k_empty + st);
      }
      __syncwarp();
    };
    auto issue_pv = [&](unsigned st, int g, bool first) {
      const uint32_t v_addr = v_base + st * KV_BYTES;
      const uint32_t p_tmem = tmem + (uint32_t)(g * 128);  // P overwrote the first 64 columns of the tile's S
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < kTcKeyTile / 16; ++kk)
          umma_ts(tmem + 256 + g * 128, p_tmem + kk * 8, umma_desc_mnmajor(v_addr + kk * 2048, PANEL_BYTES), idesc_pv, !first || kk > 0);
        umma_commit(pv_done + g);
        if (g == 1) umma_commit(v_empty + st);
      }
      __syncwarp();
    };
    // Items without key tiles are passed over.  While products of the present item are still to be issued the next one is only
    // looked for, not waited for: it may depend on the softmax warps getting on with the present one.
    AttnItem w;
    int taken = 0;
    unsigned rt = 0, kt = 0;  // row tiles and key tiles of the items before the present one
    auto next_item = [&](bool wait) {  // 1: w is the next item, 0: there is none left, -1: not known yet
      for (;;) {
        if (!wait && !item_ready(ring, taken)) return -1;
        if (!item_take(ring, taken++, w, p.st)) return 0;
        if (w.ntiles > 0) return 1;
      }
    };
    auto q_tile = [&](unsigned t) { return q_base + t % kTcQBufs * Q_BYTES; };
    // S of tile x of the item that starts at row tile t, for its first key tile c
    auto start = [&](unsigned c, unsigned t, int x) {
      if (x == 0) mbar_wait(k_full + c % kTcStages, (c / kTcStages) & 1, p.st);
      t += x;
      mbar_wait(q_full + t % kTcQBufs, (t / kTcQBufs) & 1, p.st);
      tc_fence_after_sync();
      issue_qk(c % kTcStages, x, q_tile(t));
    };
    int have = next_item(true);
    if (have == 1) {
#pragma unroll 1
      for (int x = 0; x < 2; ++x) start(0, 0, x);
    }
    while (have == 1) {
      const int ntiles = w.ntiles;
      unsigned c = kt;
      const uint32_t q_addr[2] = {q_tile(rt), q_tile(rt + 1)};
      // A product's issue is a link of the chain that bounds a step.  What it needs besides P is waited for in front of P: V of this tile
      // and K of the next one, asked for when the stages of the tile before became free.  (With the waits, the choice of the next
      // item and the addresses between the products a step took 3300 clocks: 32 full key tiles per item 471 us instead of 450.)
      for (int i = 0; i + 1 < ntiles; ++i, ++c) {
        const unsigned n = c + 1;
        mbar_wait(v_full + c % kTcStages, (c / kTcStages) & 1, p.st);
        mbar_wait(k_full + n % kTcStages, (n / kTcStages) & 1, p.st);
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          // P(c) is written (for an item's first tile this also says that O of the item before it has been read)
          mbar_wait(p_full + g, c & 1, p.st);
          tc_fence_after_sync();
          issue_pv(c % kTcStages, g, i == 0);
          issue_qk(n % kTcStages, g, q_addr[g]);
        }
      }
      // The last key tile: the next item's first products take the place of the next tile's.  In as little code as it can be: items of
      // one or two key tiles come by here as often as by the loop above (unrolled, 1024 sequences of 64 tokens 678 us instead of 659).
      have = -1;
      int begun = 0;  // row tiles of the next item whose first product is issued
#pragma unroll 1
      for (int g = 0; g < 2; ++g) {
        mbar_wait(p_full + g, c & 1, p.st);
        if (g == 0) mbar_wait(v_full + c % kTcStages, (c / kTcStages) & 1, p.st);
        tc_fence_after_sync();
        issue_pv(c % kTcStages, g, ntiles == 1);
        if (have < 0) have = next_item(g == 1);
        if (have == 1)
#pragma unroll 1
          for (; begun <= g; ++begun) start(c + 1, rt + 2, begun);
      }
      kt += ntiles;
      rt += 2;
    }
  } else if (warp == kTcSoftWarps + 2) {
    // ===================== output: stores the row tiles that leave through their Q buffers, and gives the buffers back ==========
    AttnItem w;
    int rt = 0;
    for (int taken = 0; item_take(ring, taken, w, p.st); ++taken) {
      if (w.ntiles == 0) continue;
      for (int g = 0; g < 2; ++g, ++rt) {
        const int qb = rt % kTcQBufs;
        mbar_wait(o_full + qb, (rt / kTcQBufs) & 1, p.st);
        if (lane == 0) {
          if (w.q0 + g * QT + QT <= w.Lq) {
#pragma unroll
            for (int pn = 0; pn < PANELS; ++pn)
              tma_store_3d(&tmO, q_sm + qb * Q_BYTES + pn * PANEL_BYTES, pn * 64, w.head * p.G, w.qs + w.q0 + g * QT);
            tma_store_commit();
            tma_store_wait_read();
          }
          mbar_arrive(q_empty + qb);
        }
        __syncwarp();
      }
    }
  } else {
    // ===================== softmax: one thread per row; warps 0..3 row tile A, warps 4..7 row tile B =====================
    const int g = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const uint32_t s_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * 128);
    const uint32_t o_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 256u + (uint32_t)(g * 128);
    int rt = g, kt = 0, taken = 0;  // this warp's row tile, key tiles of the items before the present one, items taken
    AttnItem w;
    while (item_take(ring, taken++, w, p.st)) {
      const int tpos = w.q0 + g * QT + (row >> p.logG);
      const int head = w.head * p.G + (row & (p.G - 1));
      const bool valid = tpos < w.Lq;
      const int nvis = valid ? visible_keys_tc(tpos, w.Lk, p.window, p.stride, p.causal) : 0;
      const int ntiles = w.ntiles;
      float m_ref = -INFINITY, l = 0.f;
      for (int i = 0; i < ntiles; ++i) {
        mbar_wait(s_full + g, (kt + i) & 1, p.st);
        tc_fence_after_sync();
        const int lim = nvis - (w.kt0 + i) * kTcKeyTile;  // columns below lim are visible ...
        const int lo = p.left >= 0 ? tpos - p.left - (w.kt0 + i) * kTcKeyTile : 0;  // ... from column lo on
        // Key tiles that every row of the warp sees in full (all but those on the mask's edge) take a path without the
        // per-element mask instructions.
        const bool full = __all_sync(0xffffffffu, lim >= kTcKeyTile && lo <= 0);
        // Full tiles of rows that already have a reference maximum are tried in ONE pass over the logits: exponentials
        // relative to the current reference, with the maximum of the exponents tracked on the side.  If no row of the
        // warp outgrew its reference by more than 2^8 -- the same test the general form makes -- the packed P is stored
        // and the pass for the maximum was saved; otherwise nothing has been written yet, the logits are intact, and the tile is
        // redone.  Both routes give the same P and the same sums.
        bool done = false;
        if (full && __all_sync(0xffffffffu, m_ref != -INFINITY)) {
          const float nm = -m_ref;
          uint32_t pk[64];
          float2 ls2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            uint32_t su[32];
            tmem_ld32(s_base + c * 32, su);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; ++j) {
              const float2 x = ffma2(make_float2(__uint_as_float(su[2 * j]), __uint_as_float(su[2 * j + 1])), make_float2(p.scale2, p.scale2),
                                     make_float2(nm, nm));
              mx4[j & 3] = fmax3(mx4[j & 3], x.x, x.y);
              // a share of the exponentials runs on the FMA pipe
              const float2 e = j % kPolyEvery == kPolyEvery - 1 ? exp2_poly2(x) : make_float2(fast_exp2(x.x), fast_exp2(x.y));
              ls2[j & 1] = fadd2(ls2[j & 1], e);
              pk[c * 16 + j] = DT<T>::pack(e.x, e.y);
            }
          }
          const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
          if (!__any_sync(0xffffffffu, mx > 8.f)) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t pc[16];
#pragma unroll
              for (int j = 0; j < 16; ++j) pc[j] = pk[c * 16 + j];
              tmem_st16(s_base + c * 16, pc);
            }
            l += (ls2[0].x + ls2[0].y) + (ls2[1].x + ls2[1].y);
            done = true;
          }
        }
        if (!done) {
          // The general form: row maximum of the visible logits (a bit per column), then the exponentials relative to the (possibly
          // raised) reference.
          auto seen = [&](int c) {
            const int hi_c = min(32, max(0, lim - c * 32)), lo_c = min(32, max(0, lo - c * 32));
            return (hi_c < 32 ? (1u << hi_c) - 1u : 0xffffffffu) & ~(lo_c < 32 ? (1u << lo_c) - 1u : 0xffffffffu);
          };
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int c2 = 0; c2 < 2; ++c2) {
            uint32_t su[2][32];
            tmem_ld32(s_base + c2 * 64, su[0]);
            tmem_ld32(s_base + c2 * 64 + 32, su[1]);
            const uint32_t see[2] = {seen(2 * c2), seen(2 * c2 + 1)};
            tmem_ld_wait();
            if (!full) {
#pragma unroll
              for (int j = 0; j < 64; ++j)
                if (!((see[j >> 5] >> (j & 31)) & 1u)) su[j >> 5][j & 31] = __float_as_uint(-INFINITY);
            }
#pragma unroll
            for (int j = 0; j < 64; j += 2)
              mx4[(j >> 1) & 3] = fmax3(mx4[(j >> 1) & 3], __uint_as_float(su[j >> 5][j & 31]), __uint_as_float(su[j >> 5][(j & 31) + 1]));
          }
          const float mt = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * p.scale2;  // (the scale is positive)
          const bool need = mt > m_ref + 8.f;
          float factor = 1.f;
          if (need) {
            factor = (m_ref == -INFINITY) ? 0.f : fast_exp2(m_ref - mt);
            m_ref = mt;
            l *= factor;
          }
          if (i > 0 && __any_sync(0xffffffffu, need)) {
            mbar_wait(pv_done + g, (kt + i - 1) & 1, p.st);  // P V of the previous key tile is complete: O is stable
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < D / 32; ++c) {
              uint32_t r[32];
              tmem_ld32(o_base + c * 32, r);
              tmem_ld_wait();
#pragma unroll
              for (int j = 0; j < 32; j += 2) {
                const float2 y = fmul2(make_float2(__uint_as_float(r[j]), __uint_as_float(r[j + 1])), make_float2(factor, factor));
                r[j] = __float_as_uint(y.x);
                r[j + 1] = __float_as_uint(y.y);
              }
              tmem_st32(o_base + c * 32, r);
            }
            tmem_st_wait();
          }
          // P as 16-bit pairs over the logits: the 32 columns of chunk c become the 16 packed columns [16c, 16c+16), which lie
          // inside the 64 columns already in registers when chunk c is written
          const float nm = (m_ref == -INFINITY) ? 0.f : -m_ref;
          float2 ls2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
#pragma unroll
          for (int c2 = 0; c2 < 2; ++c2) {
            uint32_t su[2][32];
            tmem_ld32(s_base + c2 * 64, su[0]);
            tmem_ld32(s_base + c2 * 64 + 32, su[1]);
            tmem_ld_wait();
#pragma unroll
            for (int c1 = 0; c1 < 2; ++c1) {
              uint32_t pk[16];
              const uint32_t see = seen(2 * c2 + c1);
              auto exps = [&](auto masked_tag) {
                constexpr bool MASKED = decltype(masked_tag)::value;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                  const float2 x = ffma2(make_float2(__uint_as_float(su[c1][2 * j]), __uint_as_float(su[c1][2 * j + 1])),
                                         make_float2(p.scale2, p.scale2), make_float2(nm, nm));
                  float2 e;
                  if (MASKED)
                    e = make_float2(masked_exp2((see >> (2 * j)) & 1u, x.x), masked_exp2((see >> (2 * j + 1)) & 1u, x.y));
                  else if (j % kPolyEvery == kPolyEvery - 1)
                    e = exp2_poly2(x);
                  else
                    e = make_float2(fast_exp2(x.x), fast_exp2(x.y));
                  ls2[j & 1] = fadd2(ls2[j & 1], e);
                  pk[j] = DT<T>::pack(e.x, e.y);
                }
              };
              if (full) exps(std::false_type{}); else exps(std::true_type{});
              tmem_st16(s_base + c2 * 32 + c1 * 16, pk);
            }
          }
          l += (ls2[0].x + ls2[0].y) + (ls2[1].x + ls2[1].y);
        }
        tmem_st_wait();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_full + g);
      }
      // ---- epilogue: O / l ----
      const float inv = l > 0.f ? 1.f / l : 0.f;
      if (valid) p.lse[(long long)(w.qs + tpos) * p.Hq + head] = l > 0.f ? m_ref + log2f(l) : -INFINITY;
      // A row tile whose tokens all belong to the sequence leaves through its own Q buffer (free since its last S product, in the
      // swizzled panel layout) and one TMA store per panel; otherwise row by row.
      const bool staged = ntiles > 0 && w.q0 + g * QT + QT <= w.Lq;
      const int qb = rt % kTcQBufs;
      if (ntiles > 0) {
        mbar_wait(pv_done + g, (kt + ntiles - 1) & 1, p.st);
        tc_fence_after_sync();
      }
      T* orow = static_cast<T*>(p.o) + (long long)(w.qs + tpos) * p.o_sn + (long long)head * p.o_sh;
      const uint32_t stage = smem_u32(q_sm + qb * Q_BYTES) + row * 128;
      uint32_t r[D / 32][32];
      if (ntiles > 0) {
#pragma unroll
        for (int c = 0; c < D / 32; ++c) tmem_ld32(o_base + c * 32, r[c]);
        tmem_ld_wait();
        tc_fence_before_sync();
      } else {
#pragma unroll
        for (int c = 0; c < D / 32; ++c)
#pragma unroll
          for (int j = 0; j < 32; ++j) r[c][j] = 0u;
      }
#pragma unroll
      for (int ci = 0; ci < D / 8; ++ci) {  // 16-byte chunks of the row
        const uint32_t* x = r[ci >> 2] + (ci & 3) * 8;
        uint4 out;
        out.x = DT<T>::pack(__uint_as_float(x[0]) * inv, __uint_as_float(x[1]) * inv);
        out.y = DT<T>::pack(__uint_as_float(x[2]) * inv, __uint_as_float(x[3]) * inv);
        out.z = DT<T>::pack(__uint_as_float(x[4]) * inv, __uint_as_float(x[5]) * inv);
        out.w = DT<T>::pack(__uint_as_float(x[6]) * inv, __uint_as_float(x[7]) * inv);
        if (staged) {
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(stage + (ci >> 3) * PANEL_BYTES + (((ci & 7) ^ (row & 7)) << 4)),
                       "r"(out.x), "r"(out.y), "r"(out.z), "r"(out.w) : "memory");
        } else if (valid) {
          *reinterpret_cast<uint4*>(orow + ci * 8) = out;
        }
      }
      if (ntiles > 0) {
        if (staged) fence_proxy_async();  // the TMA engine reads the tile through the async proxy
        __syncwarp();
        if (lane == 0) mbar_arrive(o_full + qb);
      }
      kt += ntiles;
      if (ntiles > 0) rt += 2;
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kTcSoftWarps + 1) tmem_dealloc(tmem, 512);
}

template <typename T, int D>
static int launch_dense_fwd_tc(const void* q, const void* k, const void* v, const long long* S, int Nq, int Nk, DenseFwdTcParams p, cudaStream_t stream) {
  // S: q_n q_h k_n k_h v_n v_h o_n o_h
  CUtensorMap tmQ, tmK, tmV;
  const int QT = 128 / p.G;
  int rc = make_tmap_3d(&tmQ, DT<T>::kTmapType, q, D, p.Hq, Nq, S[1], S[0], 64, p.G, QT);
  if (rc) return rc;
  rc = make_tmap_3d(&tmK, DT<T>::kTmapType, k, D, p.Hkv, Nk, S[3], S[2], 64, 1, kTcKeyTile);
  if (rc) return rc;
  rc = make_tmap_3d(&tmV, DT<T>::kTmapType, v, D, p.Hkv, Nk, S[5], S[4], 64, 1, kTcKeyTile);
  if (rc) return rc;
  CUtensorMap tmO;
  rc = make_tmap_3d(&tmO, DT<T>::kTmapType, p.o, D, p.Hq, Nq, p.o_sh, p.o_sn, 64, p.G, QT);
  if (rc) return rc;
  const size_t smem = (kTcQBufs + 2 * kTcStages) * 128 * D * 2 + sizeof(StealSlot) + sizeof(ItemRing) + 24 * sizeof(uint64_t);
  auto kern = dense_fwd_tc_kernel<T, D>;
  cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return cuda_rc(e);
  const dim3 grid((unsigned)row_tile_slots(Nq, p.B, 8 - p.logG), p.Hkv);
  { LaunchScope ls_("dense_fwd_tc", stream); kern<<<grid, kTcThreads, smem, stream>>>(tmQ, tmK, tmV, tmO, p); }
  return cuda_rc(cudaGetLastError());
}

// entry used by nsa_varlen_attn_fwd (dense_fwd.cu)
int varlen_attn_fwd_tc(const void* q, const void* k, const void* v, const int* cu_q, const int* cu_k, void* o, float* lse,
                       int total_q, int total_k, int batch, int Hq, int Hkv, int head_dim, int causal,
                       int window, int stride, int left, const long long* strides, float sm_scale, int dtype, cudaStream_t stream) {
  DenseFwdTcParams p;
  p.o = o; p.lse = lse; p.cu_q = cu_q; p.cu_k = cu_k;
  p.o_sn = strides[6]; p.o_sh = strides[7];
  p.B = batch; p.Hq = Hq; p.Hkv = Hkv; p.G = Hq / Hkv;
  p.logG = 0;
  while ((1 << p.logG) < p.G) ++p.logG;
  p.window = window; p.stride = stride; p.causal = causal; p.left = left;
  p.scale2 = sm_scale * kLog2e;
  p.st.word = status_word();
  return NSA_DISPATCH_T_D(dtype, head_dim, launch_dense_fwd_tc, q, k, v, strides, total_q, total_k, p, stream);
}

}  // namespace nsa
