// Forward of the selected-block attention where neighbouring tokens share most of their blocks (tcgen05).
//
// sparse_fwd.cu gives every (token, KV head) pair a warp that fetches its selected 64-key tiles privately: 32 KB through the
// L2-to-SM path per (token, block), at that path's limit (73 bytes per clock and SM), whatever the number of query heads in the
// group.  But in a sequence of a few thousand tokens a handful of neighbours together touch nearly every block, and with small
// groups the private tile serves four rows or one.  Here a CTA takes two row tiles of 128 rows (2 x 128 / G consecutive tokens),
// forms the UNION of their selections and walks it like dense attention: two 64-key tiles of the union make a 128-key step, a
// row that did not select one of them gets its exponentials biased by -inf, a warp none of whose rows selected it skips them.
// A tile is fetched once per 256 rows; what bounds the kernel is the softmax (two reads of the logits, 16 exponentials per clock;
// about 2100 clocks per 64-key tile of the union at head_dim 128 against 1024 of products).  The logits come in 64 columns a load, and
// those of the first tile stay in registers between the two passes: three waits for tensor memory per step instead of eight (32q/8kv,
// 7097 tokens, top-16: 316 -> 292 us; 64q/4kv, ragged 16 K: 882 -> 863).  Which tokens gain follows from their
// position in the sequence (union_limit below, with the measurements): this kernel takes the tokens before the limit in every
// sequence and sparse_fwd.cu those behind it.
//
// The result is no less exact than the private walk's.  The reference maximum of a row is its running maximum, so that the largest
// probability is an exact 1 (raised only when outgrown by 2^8, as in dense_fwd_tc.cu, it costs 1.8 % of the error against 64 bits:
// 32q/8kv bf16 2.120e-3 against 2.083e-3), all exponentials come from the exponential unit (one pair in three as a cubic would put
// 7.5e-5 into the fp32 row sum and the lse), and the output is divided by the sum of the ROUNDED probabilities, those the product
// with V saw: with 128 keys per update instead of 64 fewer of them are exact, which alone would leave 2.087e-3; so it is 2.072e-3.
// The lse comes from the unrounded sum.
//   warp 8      : TMA producer: Q of both row tiles, then K and V tiles of the union (ring of 2 each)
//   warp 9      : tensor memory, MMA issue (as in dense_fwd_tc.cu: S of a row tile, then P V, alternating between the row tiles)
//   warps 0..7  : softmax, one thread per row (0..3 row tile A, 4..7 row tile B)
// TMEM columns: [0,128) S/P of A, [128,256) S/P of B, [256,256+D) O of A, [384,384+D) O of B.
#include <algorithm>
#include <cmath>
#include <type_traits>

#include "attn_tile.cuh"
#include "dispatch.h"
#include "host_util.h"
#include "nsa_b200.h"
#include "sparse_fwd.h"
#include "tc5.cuh"

namespace nsa {
namespace {

constexpr int kUnKeys = 128;        // keys per step: two 64-key tiles of the union
constexpr int kUnStages = 2;        // K tiles, and V tiles, in flight
constexpr int kUnMaskWords = 4096;  // 32-bit words of selection masks per CTA
constexpr int kUnMaxTokens = 256;   // tokens of a CTA (groups of one)
constexpr int kUnMaxBlocks = 2048;  // blocks, and 64-key tiles of the union

template <typename T, int D>
__global__ void __launch_bounds__(320, 1)
sparse_fwd_union_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmK,
                        const __grid_constant__ CUtensorMap tmV, const __grid_constant__ CUtensorMap tmO, SparseFwdParams p, int logG,
                        int limit) {
  constexpr int PANELS = D / 64;
  constexpr int PANEL_BYTES = 128 * 128;       // 128 rows x 128 B
  constexpr int HALF_PANEL = 64 * 128;
  constexpr int Q_BYTES = 128 * D * 2;         // one row tile
  constexpr int KV_BYTES = kUnKeys * D * 2;    // one K or V step
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* q_sm = smem;                        // [2] row tiles
  uint8_t* k_sm = q_sm + 2 * Q_BYTES;
  uint8_t* v_sm = k_sm + kUnStages * KV_BYTES;
  uint64_t* bars = reinterpret_cast<uint64_t*>(v_sm + kUnStages * KV_BYTES);
  uint64_t* q_full = bars;                     // [2]
  uint64_t* k_full = bars + 2;
  uint64_t* k_empty = k_full + kUnStages;
  uint64_t* v_full = k_empty + kUnStages;
  uint64_t* v_empty = v_full + kUnStages;
  uint64_t* s_full = v_empty + kUnStages;      // [2] per row tile
  uint64_t* p_full = s_full + 2;               // [2]
  uint64_t* pv_done = p_full + 2;              // [2]
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(pv_done + 2);
  int* list_n = reinterpret_cast<int*>(tmem_slot + 1);
  unsigned* twice = reinterpret_cast<unsigned*>(tmem_slot + 4);              // [kUnMaxTokens / 32]: tokens that gave a block twice
  unsigned* mask = twice + kUnMaxTokens / 32;                                // [blocks][mw]: which tokens of the CTA selected a block
  uint16_t* list = reinterpret_cast<uint16_t*>(mask + kUnMaskWords);         // 64-key tiles of the union, ascending

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (smem_u32(smem) & 1023u) {  // the swizzled operand tiles need a 1024-byte aligned base
    if (threadIdx.x == 0) p.st.raise(kErrSmemLayout);
    return;
  }
  const int h = blockIdx.y;
  const int QT = 128 >> logG;                  // tokens per row tile
  // The CTA's row tiles: those before the limit of all sequences are counted through, so that the grid need not know any length
  // (it has room for tokens / (2 QT) + sequences of them); the last ones, with the most blocks, start first.
  int b = 0, qs = 0, L = 0, q0 = -1;
  {
    int want = gridDim.x - 1 - blockIdx.x;
    for (int b0 = 0; b0 < p.B && q0 < 0; b0 += 32) {
      const int mine = b0 + lane;
      int start = 0, len = 0;
      if (mine < p.B) {
        start = __ldg(p.cu_seqlens + mine);
        len = __ldg(p.cu_seqlens + mine + 1) - start;
      }
      const int tiles = (min(max(len, 0), limit) + 2 * QT - 1) / (2 * QT);
      int incl = tiles;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int up = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += up;
      }
      const unsigned hit = __ballot_sync(0xffffffffu, incl > want);
      const int src = hit ? __ffs(hit) - 1 : 31;
      const int before = __shfl_sync(0xffffffffu, incl - tiles, src);
      if (hit) {
        b = b0 + src;
        qs = __shfl_sync(0xffffffffu, start, src);
        L = __shfl_sync(0xffffffffu, len, src);
        q0 = (want - before) * 2 * QT;
      } else {
        want -= __shfl_sync(0xffffffffu, incl, 31);
      }
    }
  }
  if (q0 < 0) return;
  const int t_hi = min(q0 + 2 * QT, L) - 1;    // the limit is a multiple of 2 * QT: no row tile straddles it
  const int BS = p.block_size, nsub = BS / 64;
  const int nblk = t_hi / BS + 1, mw = (2 * QT + 31) / 32;

  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(q_full + s, 1);
      mbar_init(s_full + s, 1);
      mbar_init(p_full + s, 4);
      mbar_init(pv_done + s, 1);
    }
    for (int s = 0; s < kUnStages; ++s) {
      mbar_init(k_full + s, 1);
      mbar_init(k_empty + s, 1);
      mbar_init(v_full + s, 1);
      mbar_init(v_empty + s, 1);
    }
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  for (int i = threadIdx.x; i < nblk * mw; i += 320) mask[i] = 0u;
  if (threadIdx.x < kUnMaxTokens / 32) twice[threadIdx.x] = 0u;
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);
  if (warp == 8 && lane == 0) {
#pragma unroll
    for (int g = 0; g < 2; ++g) {
      mbar_expect_tx(q_full + g, Q_BYTES);
#pragma unroll
      for (int pn = 0; pn < PANELS; ++pn)
        tma_load_3d(q_sm + g * Q_BYTES + pn * PANEL_BYTES, &tmQ, q_full + g, pn * 64, h * p.G, qs + q0 + g * QT);
    }
  }
  // ---- the union: a mask of the CTA's tokens per block, then the blocks that have one, cut into 64-key tiles ----
  for (int i = threadIdx.x; i < 2 * QT * p.T; i += 320) {
    const int tt = i / p.T, j = i - tt * p.T;
    if (q0 + tt < L) {
      const int idx = __ldg(p.topk_idx + h * p.t_sh + (long long)(qs + q0 + tt) * p.t_sn + j * p.t_sk);
      if (idx >= 0 && idx <= (q0 + tt) / BS) {
        const unsigned bit = 1u << (tt & 31);
        if (atomicOr(mask + idx * mw + (tt >> 5), bit) & bit) atomicOr(twice + (tt >> 5), bit);
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    int n = 0;
    for (int base = 0; base < nblk * nsub; base += 32) {
      const int sub = base + lane;
      unsigned any = 0u;
      if (sub < nblk * nsub && sub * 64 <= t_hi)
        for (int w = 0; w < mw; ++w) any |= mask[(sub / nsub) * mw + w];
      const unsigned live = __ballot_sync(0xffffffffu, any != 0u);
      if (any) list[n + __popc(live & ((1u << lane) - 1u))] = (uint16_t)sub;
      n += __popc(live);
    }
    if (lane == 0) *list_n = n;
  }
  __syncthreads();
  const int nlist = *reinterpret_cast<volatile int*>(list_n);
  const int ntiles = (nlist + 1) / 2;

  if (warp == 8) {
    // ===================== TMA producer =====================
    if (lane == 0 && ntiles > 0) {
      auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int i) {
        mbar_expect_tx(bar, KV_BYTES);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          // an odd last tile is loaded twice: the second copy is masked, but has to be finite
          const int row = qs + list[min(2 * i + hf, nlist - 1)] * 64;
#pragma unroll
          for (int pn = 0; pn < PANELS; ++pn) tma_load_3d(dst + pn * PANEL_BYTES + hf * HALF_PANEL, tm, bar, pn * 64, h, row);
        }
      };
      for (int i = 0; i <= ntiles; ++i) {  // K runs one tile ahead of V
        if (i < ntiles) {
          const int s = i % kUnStages;
          if (i >= kUnStages) mbar_wait(k_empty + s, ((i / kUnStages) - 1) & 1, p.st);
          load(k_sm + s * KV_BYTES, &tmK, k_full + s, i);
        }
        if (i >= 1) {
          const int j = i - 1, s = j % kUnStages;
          if (j >= kUnStages) mbar_wait(v_empty + s, ((j / kUnStages) - 1) & 1, p.st);
          load(v_sm + s * KV_BYTES, &tmV, v_full + s, j);
        }
      }
    }
  } else if (warp == 9) {
    // ===================== MMA issuer: the whole warp runs the control flow, one elected lane issues =====================
    if (ntiles == 0) {  // nothing selected: the Q tiles still have to land before the CTA may leave
      mbar_wait(q_full, 0, p.st);
      mbar_wait(q_full + 1, 0, p.st);
    } else {
      const uint32_t idesc_qk = umma_idesc<T>(128, kUnKeys, false, false);
      const uint32_t idesc_pv = umma_idesc<T>(128, D, false, true);
      const uint32_t q_addr = smem_u32(q_sm);
      auto issue_qk = [&](int i, int g) {
        const uint32_t k_addr = smem_u32(k_sm + (i % kUnStages) * KV_BYTES);
        if (elect_one()) {
          umma_block_ss<D / 16, PANEL_BYTES>(tmem + (uint32_t)(g * 128), q_addr + g * Q_BYTES, k_addr, idesc_qk);
          if (g == 1) umma_commit(k_empty + (i % kUnStages));
          umma_commit(s_full + g);
        }
        __syncwarp();
      };
      auto issue_pv = [&](int i, int g) {
        const uint32_t v_addr = smem_u32(v_sm + (i % kUnStages) * KV_BYTES);
        const uint32_t p_tmem = tmem + (uint32_t)(g * 128);  // P overwrote the first 64 columns of the tile's S
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kUnKeys / 16; ++kk)
            umma_ts(tmem + 256 + g * 128, p_tmem + kk * 8, umma_desc_mnmajor(v_addr + kk * 2048, PANEL_BYTES), idesc_pv, i > 0 || kk > 0);
          if (g == 1) umma_commit(v_empty + (i % kUnStages));
          umma_commit(pv_done + g);
        }
        __syncwarp();
      };
      mbar_wait(k_full, 0, p.st);
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        mbar_wait(q_full + g, 0, p.st);
        tc_fence_after_sync();
        issue_qk(0, g);
      }
      for (int i = 0; i < ntiles; ++i) {
#pragma unroll
        for (int g = 0; g < 2; ++g) {
          mbar_wait(p_full + g, i & 1, p.st);
          if (g == 0) mbar_wait(v_full + (i % kUnStages), (i / kUnStages) & 1, p.st);
          tc_fence_after_sync();
          issue_pv(i, g);
          if (i + 1 < ntiles) {
            if (g == 0) {
              mbar_wait(k_full + ((i + 1) % kUnStages), ((i + 1) / kUnStages) & 1, p.st);
              tc_fence_after_sync();
            }
            issue_qk(i + 1, g);
          }
        }
      }
    }
  } else {
    // ===================== softmax: one thread per row =====================
    const int g = warp >> 2;
    const int row = (warp & 3) * 32 + lane;
    const int tt = g * QT + (row >> logG), tpos = q0 + tt;
    const int head = h * p.G + (row & (p.G - 1));
    const bool valid = tpos < L;
    const unsigned* my_mask = mask + (tt >> 5);
    const uint32_t s_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(g * 128);
    const uint32_t o_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + 256u + (uint32_t)(g * 128);
    float m_ref = -INFINITY, l = 0.f, l_rounded = 0.f;
    for (int i = 0; i < ntiles; ++i) {
      // visible keys of the step's two tiles: 0 where the row's token did not select the block (or sees none of the tile)
      int lim[2];
#pragma unroll
      for (int hf = 0; hf < 2; ++hf) {
        const int e = 2 * i + hf;
        lim[hf] = 0;
        if (e < nlist && valid) {
          const int sub = list[e];
          if ((my_mask[(sub / nsub) * mw] >> (tt & 31)) & 1u) lim[hf] = max(0, min(64, tpos - sub * 64 + 1));
        }
      }
      const bool any0 = __any_sync(0xffffffffu, lim[0] > 0), any1 = __any_sync(0xffffffffu, lim[1] > 0);
      // every row takes a tile whole or not at all: no mask per element, the rows that do not take it are biased by -inf
      const bool whole = __all_sync(0xffffffffu, (lim[0] & 63) == 0 && (lim[1] & 63) == 0);
      mbar_wait(s_full + g, i & 1, p.st);
      tc_fence_after_sync();
      const bool any[2] = {any0, any1};  // some row of the warp takes the tile
      auto load64 = [&](int hf, uint32_t (&su)[2][32]) {
        tmem_ld32(s_base + hf * 64, su[0]);
        tmem_ld32(s_base + hf * 64 + 32, su[1]);
        tmem_ld_wait();
      };
      // ---- pass 1: row maximum of the raw logits (the scale is positive); the first tile's stay in registers ----
      float mh[2] = {-INFINITY, -INFINITY};
      uint32_t su[2][32];
      auto pass1 = [&](auto masked_tag) {
        constexpr bool MASKED = decltype(masked_tag)::value;
#pragma unroll
        for (int hf = 1; hf >= 0; --hf) {
          if (!any[hf]) continue;
          load64(hf, su);
          float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
          for (int j = 0; j < 64; j += 2) {
            const float v0 = (!MASKED || j < lim[hf]) ? __uint_as_float(su[j >> 5][j & 31]) : -INFINITY;
            const float v1 = (!MASKED || j + 1 < lim[hf]) ? __uint_as_float(su[j >> 5][(j & 31) + 1]) : -INFINITY;
            mx4[(j >> 1) & 3] = fmax3(mx4[(j >> 1) & 3], v0, v1);
          }
          mh[hf] = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3]));
        }
      };
      if (whole) pass1(std::false_type{}); else pass1(std::true_type{});
      const float mt = fmaxf(lim[0] > 0 ? mh[0] : -INFINITY, lim[1] > 0 ? mh[1] : -INFINITY) * p.scale2;
      const bool need = mt > m_ref;
      float factor = 1.f;
      if (need) {
        factor = (m_ref == -INFINITY) ? 0.f : fast_exp2(m_ref - mt);
        m_ref = mt;
        l *= factor;
        l_rounded *= factor;
      }
      if (i > 0 && __any_sync(0xffffffffu, need)) {
        mbar_wait(pv_done + g, (i - 1) & 1, p.st);  // P V of the previous step is complete: O is stable
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
      // ---- pass 2: P = exp2(S * scale - m_ref) as 16-bit pairs over the logits (chunk c's 16 packed columns lie inside the first
      // tile's logits, which are in registers) ----
      const float nm = (m_ref == -INFINITY) ? 0.f : -m_ref;
      float2 ls2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)}, lr2[2] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      auto pass2 = [&](auto masked_tag) {
        constexpr bool MASKED = decltype(masked_tag)::value;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
          if (hf == 1 && any[1]) load64(1, su);
          const float bias = lim[hf] > 0 ? nm : -INFINITY;
#pragma unroll
          for (int c = 0; c < 2; ++c) {
            uint32_t pk[16];
            if (!any[hf]) {
#pragma unroll
              for (int j = 0; j < 16; ++j) pk[j] = 0u;
            } else {
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                const float2 x = ffma2(make_float2(__uint_as_float(su[c][2 * j]), __uint_as_float(su[c][2 * j + 1])),
                                       make_float2(p.scale2, p.scale2), make_float2(bias, bias));
                const float p0 = MASKED ? masked_exp2(c * 32 + 2 * j < lim[hf], x.x) : fast_exp2(x.x);
                const float p1 = MASKED ? masked_exp2(c * 32 + 2 * j + 1 < lim[hf], x.y) : fast_exp2(x.y);
                ls2[j & 1] = fadd2(ls2[j & 1], make_float2(p0, p1));
                pk[j] = DT<T>::pack(p0, p1);
                lr2[j & 1] = fadd2(lr2[j & 1], DT<T>::unpack(pk[j]));
              }
            }
            tmem_st16(s_base + hf * 32 + c * 16, pk);
          }
        }
      };
      if (whole) pass2(std::false_type{}); else pass2(std::true_type{});
      tmem_st_wait();
      l += (ls2[0].x + ls2[0].y) + (ls2[1].x + ls2[1].y);
      l_rounded += (lr2[0].x + lr2[0].y) + (lr2[1].x + lr2[1].y);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full + g);
    }
    // ---- epilogue: O / l ----
    if (ntiles > 0) {
      mbar_wait(pv_done + g, (ntiles - 1) & 1, p.st);
      tc_fence_after_sync();
    }
    const float inv = l_rounded > 0.f ? 1.f / l_rounded : 0.f;
    // A row tile whose tokens all belong to the sequence leaves through shared memory (its own Q buffer, free since its
    // last S product, in the swizzled panel layout) and one TMA store per panel; otherwise row by row.
    const bool staged = ntiles > 0 && q0 + g * QT + QT <= L;
    float probe = l;  // becomes NaN with any output of the row
    T* orow = static_cast<T*>(p.o) + (long long)(qs + tpos) * p.o_sn + (long long)head * p.o_sh;
#pragma unroll
    for (int c = 0; c < D / 32; ++c) {
      uint32_t r[32];
      if (ntiles > 0) {
        tmem_ld32(o_base + c * 32, r);
        tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 32; ++j) r[j] = 0u;
      }
#pragma unroll
      for (int j = 0; j < 32; j += 2) probe = fmaf(0.f, __uint_as_float(r[j]) + __uint_as_float(r[j + 1]), probe);
      if (staged) {
        const uint32_t stage = smem_u32(q_sm + g * Q_BYTES);
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          const int ci = c * 4 + q4;  // 16-byte chunk of the row
          const uint32_t off = (ci >> 3) * PANEL_BYTES + row * 128 + (((ci & 7) ^ (row & 7)) << 4);
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(stage + off),
                       "r"(DT<T>::pack(__uint_as_float(r[q4 * 8 + 0]) * inv, __uint_as_float(r[q4 * 8 + 1]) * inv)),
                       "r"(DT<T>::pack(__uint_as_float(r[q4 * 8 + 2]) * inv, __uint_as_float(r[q4 * 8 + 3]) * inv)),
                       "r"(DT<T>::pack(__uint_as_float(r[q4 * 8 + 4]) * inv, __uint_as_float(r[q4 * 8 + 5]) * inv)),
                       "r"(DT<T>::pack(__uint_as_float(r[q4 * 8 + 6]) * inv, __uint_as_float(r[q4 * 8 + 7]) * inv)) : "memory");
        }
      } else if (valid) {
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          uint4 out;
          out.x = DT<T>::pack(__uint_as_float(r[q4 * 8 + 0]) * inv, __uint_as_float(r[q4 * 8 + 1]) * inv);
          out.y = DT<T>::pack(__uint_as_float(r[q4 * 8 + 2]) * inv, __uint_as_float(r[q4 * 8 + 3]) * inv);
          out.z = DT<T>::pack(__uint_as_float(r[q4 * 8 + 4]) * inv, __uint_as_float(r[q4 * 8 + 5]) * inv);
          out.w = DT<T>::pack(__uint_as_float(r[q4 * 8 + 6]) * inv, __uint_as_float(r[q4 * 8 + 7]) * inv);
          *reinterpret_cast<uint4*>(orow + c * 32 + q4 * 8) = out;
        }
      }
    }
    // one row of the pair not finite, or a block given twice (it counts twice; a mask holds it once): the pair's first lse says so,
    // and sparse_fwd.cu does the pair again after this kernel
    const bool again = isnan(probe) || ((twice[tt >> 5] >> (tt & 31)) & 1u);
    const unsigned bad = __ballot_sync(0xffffffffu, valid && again);
    const unsigned pair_rows = ((1u << p.G) - 1u) << (lane & ~(p.G - 1));  // G <= 16
    const bool redo = (bad & pair_rows) != 0u && (row & (p.G - 1)) == 0;
    if (valid) p.lse[(long long)(qs + tpos) * p.Hq + head] = redo ? __int_as_float(0x7fffffff) : l > 0.f ? m_ref + log2f(l) : -INFINITY;
    if (staged) {
      fence_proxy_async();  // the TMA engine reads the tile through the async proxy
      asm volatile("bar.sync %0, 128;\n" ::"r"(1 + g) : "memory");
      if ((warp & 3) == 0 && lane == 0) {
#pragma unroll
        for (int pn = 0; pn < PANELS; ++pn) tma_store_3d(&tmO, q_sm + g * Q_BYTES + pn * PANEL_BYTES, pn * 64, h * p.G, qs + q0 + g * QT);
        tma_store_commit();
        tma_store_wait_read();
      }
    }
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}


// Tokens of a sequence before which the union of a CTA's selections is cheaper than a private walk per token.  Taking a token's
// T - 3 free choices as uniform over the nb blocks before it (neighbours that agree more only make the union smaller), 2 QT tokens
// touch U = 3 + nb (1 - (1 - (T - 3) / nb)^(2 QT)) of them; the union wins while U * (clocks per union tile) < 2 QT * T * (clocks per
// private tile).  Measured with such selections, all tokens private / all in unions / split by this rule, us:
//   32q/2kv d128 top-8   1024 tokens: 43 / 38 / 38    4096: 148 / 153 / 144    8192: 285 / 372 / 286
//   64q/4kv d128 top-16  1024: 96 / 54 / 54   4096: 455 / 341 / 341   8192: 930 / 999 / 859   16384: 1884 / 2822 / 1830
//   32q/8kv d128 top-16  1024: 162 / 44 / 42  4096: 857 / 238 / 228   8192: 1774 / 648 / 638  16384: 3619 / 2159 / 2158
//   16q/2kv d64  top-8   1024: 31 / 34 / 34   4096: 90 / 83 / 89      8192: 172 / 222 / 175
//   32q/2kv d64  top-8   1024: 31 / 34 / 34   4096: 92 / 130 / 104    8192: 178 / 312 / 185
// From the increments between the lengths: about 2100 clocks per union tile (64 keys, both row tiles) against 530 per private one at
// head_dim 128.  The rule counts 1850 there: the second kernel's start and its last wave count against a division that leaves it few
// tokens.  At head_dim 64 it counts 1950 against 370 for groups of 8 and 16 alike, which gives groups of 16 too many tokens to the unions
// (the last line).
int union_limit(int G, int T, int block_size, int head_dim) {
  const double union_clocks = head_dim == 128 ? 1850. : 1950., private_clocks = head_dim == 128 ? 530. : 370.;
  const int tokens = 2 * (128 / G), nsub = block_size / 64, mw = (tokens + 31) / 32;
  const double free_choices = std::max(0, T - 3);
  int most = std::min(kUnMaxBlocks / nsub, kUnMaskWords / mw);
  int lo = 0;  // largest number of blocks for which the union wins, by bisection
  while (lo < most) {
    const int nb = (lo + most + 1) / 2;
    const double u = nb <= T ? nb : 3. + nb * (1. - std::pow(1. - free_choices / nb, tokens));
    if (u * union_clocks < (double)tokens * T * private_clocks) lo = nb; else most = nb - 1;
  }
  return (int)((long long)lo * block_size / tokens * tokens);
}

template <typename T, int D>
int launch_union(const void* q, const void* k, const void* v, const long long* S, SparseFwdParams p, int limit, cudaStream_t stream) {
  // S: q_n q_h k_n k_h v_n v_h o_n o_h
  const int QT = 128 / p.G;
  CUtensorMap tmQ, tmK, tmV, tmO;
  int rc = make_tmap_3d(&tmQ, DT<T>::kTmapType, q, D, p.Hq, p.N, S[1], S[0], 64, p.G, QT);
  if (rc) return rc;
  rc = make_tmap_3d(&tmK, DT<T>::kTmapType, k, D, p.Hkv, p.N, S[3], S[2], 64, 1, 64);
  if (rc) return rc;
  rc = make_tmap_3d(&tmV, DT<T>::kTmapType, v, D, p.Hkv, p.N, S[5], S[4], 64, 1, 64);
  if (rc) return rc;
  rc = make_tmap_3d(&tmO, DT<T>::kTmapType, p.o, D, p.Hq, p.N, p.o_sh, p.o_sn, 64, p.G, QT);
  if (rc) return rc;
  int logG = 0;
  while ((1 << logG) < p.G) ++logG;
  const size_t smem = 2 * 128 * D * 2 + 2 * kUnStages * kUnKeys * D * 2 + 32 * sizeof(uint64_t) + kUnMaskWords * 4 + kUnMaxBlocks * 2;
  auto kern = sparse_fwd_union_kernel<T, D>;
  const cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return cuda_rc(e);
  const long long per_seq = (std::min(p.N, limit) + 2 * QT - 1) / (2 * QT);
  const long long ctas = std::min((long long)p.N / (2 * QT) + p.B, per_seq * p.B);
  LaunchScope ls_("sparse_fwd_union", stream);
  kern<<<dim3((unsigned)ctas, p.Hkv), 320, smem, stream>>>(tmQ, tmK, tmV, tmO, p, logG, limit);
  return cuda_rc(cudaGetLastError());
}

}  // namespace

int sparse_fwd_union_limit(int G, int T, int block_size, int head_dim) {
  return (G & (G - 1)) ? 0 : union_limit(G, T, block_size, head_dim);
}

int sparse_fwd_union(const void* q, const void* k, const void* v, const long long* strides, SparseFwdParams p, int limit, int head_dim,
                     int dtype, cudaStream_t stream) {
  return NSA_DISPATCH_T_D(dtype, head_dim, launch_union, q, k, v, strides, p, limit, stream);
}

}  // namespace nsa
