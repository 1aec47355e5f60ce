// dQ, dK and dV of dense strided-causal attention in one pass on the 5th-generation tensor cores (head_dim 128): five products per
// tile where a dQ pass and a dK/dV pass form seven, since each has to form the logits and dP for itself.
//
// CTA = one tile of 128 keys (K and V tiles resident in SMEM) x a stream of row tiles; a row tile is
// 128 rows = (128/G consecutive tokens) x (G query heads of the KV group).  The KEYS are the M dimension:
//     S^T  = K  Q^T          [128 keys x 128 rows]   A = K tile (SMEM, K-major),    B = Q  rows (SMEM, K-major)
//     dP^T = V  dO^T         [128 keys x 128 rows]   A = V tile (SMEM, K-major),    B = dO rows (SMEM, K-major)
//     dV  += P^T  dO         [128 keys x 128 d]      A = P^T  (TMEM, 16-bit),       B = dO rows (SMEM, MN-major)
//     dQ^T = K^T dS          [128 d    x 128 rows]   A = K tile (SMEM, MN-major),   B = dS [keys][rows] (SMEM, MN-major)
//     dK  += dS^T Q          [128 keys x 128 d]      A = dS [keys][rows] (SMEM, K-major),  B = Q rows (SMEM, MN-major)
// P^T is written over the logits in TMEM; dS goes to shared memory, where both products that need it read it.  dP is then of no use
// any more and dQ^T takes its TMEM columns: the drain warps read three quarters of it into registers at once, so that the next dP
// waits for a quarter of the reductions and not for all of them.  dQ^T has d on the lanes: a warp's reduction covers one 128-byte
// line of a (token, head) row, as in sparse_dkdv_tc.cu.
//   warps 0..7   : two threads per key (64 of the 128 row columns each): P phase, dS phase; at the end dV and dK to global memory
//   warp 8       : TMA producer (Q and dO rings of two tiles) and the per-row table (lse, delta)
//   warp 9       : S and dP products;  warp 10 : dV, dQ and dK products (two warps: see sparse_dkdv_tc.cu);  warp 11 : idle
//   warps 12..15 : dQ drain, warp w the lanes (= d) of quarter w % 4
// What bounds it (8192 tokens, 64q/4kv, causal; clocks of a row tile): the softmax threads, whose P phase takes 1800 clocks and dS
// phase 1800 because their shared-memory accesses queue behind the drain warps' reductions (1450 and 1150 without those, and 3300 a
// tile), and waits of 500 for each of S and dP: 4650 a tile.  The two passes it replaces take 3.2-3.5 ms there, this one 2.7-3.1
// (both move with the clock under the power cap), and its launches around it 0.2 ms more; where it is taken: attn_bwd.cu.
// TMEM columns: dV [0,128)  dK [128,256)  S^T / P^T [256,384)  dP^T / dQ^T [384,512).
#include "dense_bwd_tile.cuh"
#include "host_util.h"

namespace nsa {
namespace {
constexpr int kStages = 2;
constexpr int kPanel = 128 * 128;   // [128][64] 16-bit elements
constexpr int kTile = 2 * kPanel;   // [128][128]
constexpr int kThreads = 16 * 32;
constexpr int kColDv = 0, kColDk = 128, kColS = 256, kColDp = 384;
constexpr size_t kSmem = (size_t)(2 + 2 * kStages + 1) * kTile + 4 * 128 * sizeof(float) + 28 * sizeof(uint64_t) + 16;
}  // namespace

template <typename T, int LOGG>
__global__ void __launch_bounds__(kThreads, 1)
dense_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmQ, const __grid_constant__ CUtensorMap tmDO,
                    const __grid_constant__ CUtensorMap tmK, const __grid_constant__ CUtensorMap tmV, DkdvParams p) {
  constexpr int KT = 128, D = 128, logG = LOGG, G = 1 << LOGG;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* k_sm = smem;
  uint8_t* v_sm = k_sm + kTile;
  uint8_t* q_ring = v_sm + kTile;
  uint8_t* do_ring = q_ring + kStages * kTile;
  uint8_t* ds_sm = do_ring + kStages * kTile;                        // [128 keys][128 rows]
  float* nlse_sh = reinterpret_cast<float*>(ds_sm + kTile);          // [2][128]  -lse (base 2)
  float* dsc_sh = nlse_sh + 2 * 128;                                 // [2][128]  delta * sm_scale
  uint64_t* kv_full = reinterpret_cast<uint64_t*>(dsc_sh + 2 * 128);
  uint64_t* q_full = kv_full + 1;           // [kStages] each
  uint64_t* q_empty = q_full + kStages;
  uint64_t* do_full = q_empty + kStages;
  uint64_t* do_empty = do_full + kStages;
  uint64_t* meta_full = do_empty + kStages;  // [2]
  uint64_t* meta_empty = meta_full + 2;      // [2]
  uint64_t* s_full = meta_empty + 2;
  uint64_t* s_empty = s_full + 1;            // P^T has been read by dV: the columns are free for the next logits
  uint64_t* dp_full = s_empty + 1;
  uint64_t* p_full = dp_full + 1;
  uint64_t* ds_full = p_full + 1;
  uint64_t* ds_empty = ds_full + 1;
  uint64_t* dq_full = ds_empty + 1;
  uint64_t* dq_empty = dq_full + 1;
  uint64_t* all_done = dq_empty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(all_done + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int TPT = 128 >> logG;  // tokens per row tile

  // the swizzled operand tiles need a 1024-byte aligned base
  if (smem_u32(smem) & 1023u) {
    if (threadIdx.x == 0) p.st.raise(kErrSmemLayout);
    return;
  }

  // ---- which key tile, which tokens ----
  const int b = blockIdx.z / p.Hkv;
  const int h = blockIdx.z % p.Hkv;
  const int qs = __ldg(p.cu_q + b);
  const int Lq = __ldg(p.cu_q + b + 1) - qs;
  const int ks0 = __ldg(p.cu_k + b), Lk = __ldg(p.cu_k + b + 1) - ks0;
  const int kpos = blockIdx.x * KT;  // key tiles vary fastest: CTAs that run together share a token chunk in L2
  if (kpos >= Lk) return;
  const int krow0 = ks0 + kpos;
  const int kvalid = min(KT, Lk - kpos);
  const int t_first = p.causal ? kpos * p.stride + p.window - 1 : 0;
  const int c_lo = blockIdx.y * p.chunk;
  const int tok_begin = max(c_lo, t_first);
  const int tok_end = min(c_lo + p.chunk, Lq);
  if (tok_end <= tok_begin) return;
  const int ntiles = (tok_end - tok_begin + TPT - 1) / TPT;

  if (threadIdx.x == 0) {
    mbar_init(kv_full, 1);
    for (int s = 0; s < kStages; ++s) {
      mbar_init(q_full + s, 1);
      mbar_init(q_empty + s, 1);
      mbar_init(do_full + s, 1);
      mbar_init(do_empty + s, 2);  // read by dP and dV, which come from two warps
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(meta_full + s, 1);
      mbar_init(meta_empty + s, 8);
    }
    mbar_init(s_full, 1);
    mbar_init(s_empty, 1);
    mbar_init(dp_full, 1);
    mbar_init(p_full, 8);
    mbar_init(ds_full, 8);
    mbar_init(ds_empty, 1);
    mbar_init(dq_full, 1);
    mbar_init(dq_empty, 4);
    mbar_init(all_done, 1);
    fence_barrier_init();
  }
  if (warp == 9) {
    tmem_alloc(tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot);

  if (warp == 8) {
    // ===================== producer =====================
    if (lane == 0) {
      mbar_expect_tx(kv_full, 2 * kTile);
#pragma unroll
      for (int pn = 0; pn < 2; ++pn) {
        tma_load_3d(k_sm + pn * kPanel, &tmK, kv_full, pn * 64, h, krow0);
        tma_load_3d(v_sm + pn * kPanel, &tmV, kv_full, pn * 64, h, krow0);
      }
    }
    for (int i = 0; i < ntiles; ++i) {
      const int tok0 = tok_begin + i * TPT;
      const int s = i % kStages;
      const uint32_t before = ((i / kStages) - 1) & 1;
      if (lane == 0) {
        if (i >= kStages) mbar_wait(q_empty + s, before, p.st);
        mbar_expect_tx(q_full + s, kTile);
#pragma unroll
        for (int pn = 0; pn < 2; ++pn) tma_load_3d(q_ring + s * kTile + pn * kPanel, &tmQ, q_full + s, pn * 64, h * p.G, qs + tok0);
      }
      {
        const int m = i & 1;
        if (i >= 2) mbar_wait(meta_empty + m, ((i >> 1) - 1) & 1, p.st);
        fill_row_table(nlse_sh + m * 128, dsc_sh + m * 128, p, logG, h, qs, tok0, tok_end, lane);
        __syncwarp();
        if (lane == 0) mbar_arrive(meta_full + m);
      }
      if (lane == 0) {
        if (i >= kStages) mbar_wait(do_empty + s, before, p.st);
        mbar_expect_tx(do_full + s, kTile);
#pragma unroll
        for (int pn = 0; pn < 2; ++pn) tma_load_3d(do_ring + s * kTile + pn * kPanel, &tmDO, do_full + s, pn * 64, h * p.G, qs + tok0);
      }
      __syncwarp();
    }
  } else if (warp == 9) {
    // ===================== S and dP products (converged warp, elected lane issues) =====================
    const uint32_t idesc = umma_idesc<T>(128, 128, false, false);
    const uint32_t k_addr = smem_u32(k_sm), v_addr = smem_u32(v_sm), q_base = smem_u32(q_ring), do_base = smem_u32(do_ring);
    bool alive = mbar_wait(kv_full, 0, p.st);
    for (int i = 0; i < ntiles && alive; ++i) {
      const int s = i % kStages;
      const uint32_t now = (i / kStages) & 1;
      if (!mbar_wait(q_full + s, now, p.st) || (i > 0 && !mbar_wait(s_empty, (i - 1) & 1, p.st))) break;
      tc_fence_after_sync();
      if (elect_one()) {
        umma_block_ss<D / 16, kPanel>(tmem + kColS, k_addr, q_base + s * kTile, idesc);
        umma_commit(s_full);
      }
      __syncwarp();
      alive = mbar_wait(do_full + s, now, p.st) && (i == 0 || mbar_wait(dq_empty, (i - 1) & 1, p.st));
      if (!alive) break;
      tc_fence_after_sync();
      if (elect_one()) {
        umma_block_ss<D / 16, kPanel>(tmem + kColDp, v_addr, do_base + s * kTile, idesc);
        umma_commit(dp_full);
        umma_commit(do_empty + s);
      }
      __syncwarp();
    }
  } else if (warp == 10) {
    // ===================== dV, dQ and dK products =====================
    const uint32_t idesc_v = umma_idesc<T>(128, D, false, true);
    const uint32_t idesc_q = umma_idesc<T>(D, 128, true, true);
    const uint32_t k_addr = smem_u32(k_sm), ds_addr = smem_u32(ds_sm), q_base = smem_u32(q_ring), do_base = smem_u32(do_ring);
    bool alive = true;
    for (int i = 0; i < ntiles; ++i) {
      const int s = i % kStages;
      alive = mbar_wait(do_full + s, (i / kStages) & 1, p.st) && mbar_wait(p_full, i & 1, p.st);
      if (!alive) break;
      tc_fence_after_sync();
      if (elect_one()) {
        umma_block_ts<128 / 16, kPanel>(tmem + kColDv, tmem + kColS, do_base + s * kTile, idesc_v, i > 0);
        umma_commit(s_empty);
        umma_commit(do_empty + s);
      }
      __syncwarp();
      alive = mbar_wait(ds_full, i & 1, p.st);  // dP has been read, too: dQ takes its columns
      if (!alive) break;
      tc_fence_after_sync();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < KT / 16; ++kk)
          umma_ss(tmem + kColDp, umma_desc_mnmajor(k_addr + kk * 2048, kPanel), umma_desc_mnmajor(ds_addr + kk * 2048, kPanel), idesc_q, kk > 0);
        umma_commit(dq_full);
      }
      __syncwarp();
      if (elect_one()) {
#pragma unroll
        for (int kk = 0; kk < 128 / 16; ++kk)
          umma_ss(tmem + kColDk, umma_desc_kmajor(ds_addr + (kk >> 2) * kPanel + (kk & 3) * 32),
                  umma_desc_mnmajor(q_base + s * kTile + kk * 2048, kPanel), idesc_v, i > 0 || kk > 0);
        umma_commit(ds_empty);
        umma_commit(q_empty + s);
      }
      __syncwarp();
    }
    if (elect_one()) umma_commit(all_done);
    __syncwarp();
  } else if (warp >= 12) {
    // ===================== dQ drain: lane = d, 128 columns = the rows of the tile =====================
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16) + kColDp;
    // 32 rows from row r0 of the tile on, tokens at `tile`; the warp's 32 lanes add 32 consecutive floats of each.  A token's rows are
    // at constant offsets from its pointer: an address register that is moved on from one reduction to the next has to wait until the
    // reduction has left its queue to be read (60 clocks a row against 26).
    auto reduce_chunk = [&](const uint32_t (&x)[32], float* tile, int r0, int nrows) {
#pragma unroll
      for (int t = 0; t < (32 >> LOGG); ++t) {
        float* dst = tile + (long long)((r0 >> LOGG) + t) * p.Hq * D;
        if (r0 + t * G < nrows) {
#pragma unroll
          for (int g = 0; g < G; ++g) red_add1(dst + g * D, x[t * G + g]);
        }
      }
    };
    for (int i = 0; i < ntiles; ++i) {
      const int tok0 = tok_begin + i * TPT;
      const int nrows = min(TPT, tok_end - tok0) << logG;
      float* tile = p.dq32 + ((long long)(qs + tok0) * p.Hq + h * p.G) * D + (warp & 3) * 32 + lane;
      if (!mbar_wait(dq_full, i & 1, p.st)) break;
      tc_fence_after_sync();
      uint32_t x0[32], x1[32], x2[32];
      tmem_ld32(lane_base, x0);
      tmem_ld32(lane_base + 32, x1);
      tmem_ld32(lane_base + 64, x2);
      tmem_ld_wait();
      reduce_chunk(x0, tile, 0, nrows);
      tmem_ld32(lane_base + 96, x0);
      tmem_ld_wait();
      // the tile is in registers: the next tile's dP may have the columns
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(dq_empty);
      reduce_chunk(x1, tile, 32, nrows);
      reduce_chunk(x2, tile, 64, nrows);
      reduce_chunk(x0, tile, 96, nrows);
    }
  } else if (warp < 8) {
    // ===================== softmax / dS threads: thread = (key, half of the row columns) =====================
    const int half = warp >> 2;
    const int key = (warp & 3) * 32 + lane;
    const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    const uint32_t ds_row = smem_u32(ds_sm) + half * kPanel + key * 128;
    // first in-sequence token position that sees this key
    const int thr = p.causal ? (kpos + key) * p.stride + p.window - 1 : 0;
    const bool key_ok = key < kvalid;
    for (int i = 0; i < ntiles; ++i) {
      const int ms = i & 1;
      const int tok0 = tok_begin + i * TPT;
      // visible columns of this thread: [clo, chi) in tile columns, shifted to the thread's own 64
      const int clo = max(0, thr - tok0) << logG;
      const int chi = key_ok ? (min(TPT, tok_end - tok0) << logG) : 0;
      const int clo_rel = clo - half * 64;
      const unsigned span = chi > clo ? (unsigned)(chi - clo) : 0u;
      // tiles every key of the warp sees in full (all but those on the mask's edge) skip the mask instructions
      const bool full = __all_sync(0xffffffffu, clo == 0 && chi == 128);

      mbar_wait(meta_full + ms, (i >> 1) & 1, p.st);
      mbar_wait(s_full, i & 1, p.st);
      tc_fence_after_sync();
      float pf[64];
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t su[1][32];
        tmem_ld32(lane_base + kColS + half * 64 + c * 32, su[0]);
        tmem_ld_wait();
        uint32_t pk[16];
        probabilities<T, 1>(su, nlse_sh + ms * 128 + half * 64 + c * 32, p.scale2, full, clo_rel - c * 32, span, pf + c * 32, pk);
        tmem_st16(lane_base + kColS + half * 64 + c * 16, pk);  // over logits of this thread's that are in registers by now
      }
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(p_full);

      mbar_wait(dp_full, i & 1, p.st);
      tc_fence_after_sync();
      if (i > 0) mbar_wait(ds_empty, (i - 1) & 1, p.st);  // dQ and dK of the tile before have read the dS tile
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t du[1][32];
        tmem_ld32(lane_base + kColDp + half * 64 + c * 32, du[0]);
        tmem_ld_wait();
        uint32_t pk[16];
        ds_columns<T, 1>(du, dsc_sh + ms * 128 + half * 64 + c * 32, p.sm_scale, pf + c * 32, pk);
#pragma unroll
        for (int c4 = 0; c4 < 4; ++c4)
          asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};\n" ::"r"(ds_row + (((c * 4 + c4) ^ (key & 7)) << 4)), "r"(pk[c4 * 4]),
                       "r"(pk[c4 * 4 + 1]), "r"(pk[c4 * 4 + 2]), "r"(pk[c4 * 4 + 3]) : "memory");
      }
      fence_proxy_async();  // the tensor pipe reads the tile through the async proxy
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(ds_full);
        mbar_arrive(meta_empty + ms);
      }
    }
    // ---- read-out ----
    mbar_wait(all_done, 0, p.st);
    tc_fence_after_sync();
    static_assert(kColDk == kColDv + 128);
    add_key_rows<D>(p, lane_base + kColDv, (size_t)(krow0 + key) * p.Hkv + h, half, key_ok);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 9) tmem_dealloc(tmem, 512);
}

template <typename T>
int launch_dense_bwd_tc(const void* q, const void* dout, const void* k, const void* v, const long long* strides, int Nq, int Nk, int max_q,
                        int max_k, int batch, DkdvParams p, cudaStream_t stream) {
  constexpr int D = 128;
  int logG = 0;
  while ((1 << logG) < p.G) ++logG;
  const int TPT = 128 >> logG;
  CUtensorMap tmQ, tmDO, tmK, tmV;
  int rc = make_tmap_3d(&tmQ, DT<T>::kTmapType, q, D, p.Hq, Nq, strides[1], strides[0], 64, p.G, TPT);
  if (rc) return rc;
  rc = make_tmap_3d(&tmDO, DT<T>::kTmapType, dout, D, p.Hq, Nq, strides[7], strides[6], 64, p.G, TPT);
  if (rc) return rc;
  rc = make_tmap_3d(&tmK, DT<T>::kTmapType, k, D, p.Hkv, Nk, strides[3], strides[2], 64, 1, 128);
  if (rc) return rc;
  rc = make_tmap_3d(&tmV, DT<T>::kTmapType, v, D, p.Hkv, Nk, strides[5], strides[4], 64, 1, 128);
  if (rc) return rc;
  const dim3 grid((max_k + 127) / 128, (max_q + p.chunk - 1) / p.chunk, batch * p.Hkv);
  auto launch = [&](auto kern) -> int {
    cudaError_t e = allow_smem(kern, kSmem);
    if (e != cudaSuccess) return cuda_rc(e);
    { LaunchScope ls_("dense_bwd_tc", stream); kern<<<grid, kThreads, kSmem, stream>>>(tmQ, tmDO, tmK, tmV, p); }
    return cuda_rc(cudaGetLastError());
  };
  switch (logG) {
    case 0: return launch(dense_bwd_tc_kernel<T, 0>);
    case 1: return launch(dense_bwd_tc_kernel<T, 1>);
    case 2: return launch(dense_bwd_tc_kernel<T, 2>);
    case 3: return launch(dense_bwd_tc_kernel<T, 3>);
    case 4: return launch(dense_bwd_tc_kernel<T, 4>);
    default: return kUnsupported;
  }
}

#define NSA_INSTANTIATE(T)                                                                                                               \
  template int launch_dense_bwd_tc<T>(const void*, const void*, const void*, const void*, const long long*, int, int, int, int, int, DkdvParams, \
                                      cudaStream_t)
NSA_INSTANTIATE(__nv_bfloat16);
NSA_INSTANTIATE(__half);
#undef NSA_INSTANTIATE

}  // namespace nsa
