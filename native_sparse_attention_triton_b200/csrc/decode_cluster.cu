// Single-token attention with one thread-block CLUSTER per (sequence, KV head): the three decode operators for small and
// medium batches, and the whole decode step of a layer in one launch.
//
// What bounds these kernels is not bytes but the chain of dependent steps: at batch 4 a step reads 8 MB (1.2 us of HBM) while
// the split-KV kernel of decode.cu took 36 us for dense decode over 8256 rows, 23 us for compressed decode with selection and
// 14 us for the selected blocks, and five more kernels (staging, pooling, rotation, append, gated sum) 16 us -- tiles walked in
// sequence by one warp, partial results through global memory and merged by a single warp, and a launch's latency each time.
// Here
//   * the keys of a pair are dealt out in sub-tiles of 32 rows to the S * NW warps of its cluster (S CTAs), so that a warp has
//     one sub-tile where the batch is small; rows come in by cp.async (no tensor map to build, fetch or wait for; rows beyond
//     the sequence are zero-filled, so nothing stale is multiplied);
//   * partial results meet in shared memory: the warps' inside the CTA, the CTAs' through distributed shared memory, every
//     CTA writing its slice of the output -- no scratch in global memory, no counters, no last finisher;
//   * compressed attention keeps its logits in shared memory, turns them into key scores in the CTA that computed them, and
//     one warp of rank 0 folds and selects;
//   * everything a decode step does is local to a (sequence, KV head) pair -- staging, pooling, rotation of the new rows,
//     appending them, the three branches, the gated sum -- so the step is this one kernel with a cluster barrier between its
//     parts.  The length counters, shared by the heads of a sequence, are advanced by the last of its clusters to have read
//     them.
// Measured (8 pairs of 8256 rows): dense 13 us, compressed with selection 8.5, selected blocks 7; a whole step 18 us (34 k clocks:
// counters, angles and rotation 3 k, staging and append 1 k -- 4 k where a window completes --, compressed and window branches 4 k,
// their merge and weights 4 k, key scores and output slices 3 k, selection 2-4 k, list and selected blocks 5 k, merge, weights and
// output 5 k, six cluster barriers of about 1 k each).
#include "attn_tile.cuh"
#include "cluster.cuh"
#include "decode_cluster.h"
#include "dispatch.h"
#include "host_util.h"
#include "nsa_b200.h"
#include "topk_select.cuh"

#include <atomic>

namespace nsa {
namespace {

constexpr int kSub = 32;           // keys per sub-tile
constexpr int kMaxSelTiles = 64;   // selected 64-key tiles per query
constexpr int kMaxList = 2 * kMaxSelTiles;
constexpr int kMaxCluster = 16;

enum Mode { kDense = 0, kSparse = 1, kCompressed = 2, kStep = 3 };

struct Cache {
  void* base;
  long long s2, sb, sn, sh;  // key / value planes (step only), sequence, row, head
  int* len;
  int rows;
};

struct Params {
  const void* q;
  const void* k;  // operators: the cache; step: the new token's key and value rows
  const void* v;
  void* o;
  const int* seqlens;
  const int* cmp_seqlens;
  const int* topk_idx;  // sparse: in
  int* topk_out_idx;    // compressed: out, or nullptr
  long long q_sb, q_sh, o_sb, o_sh, k_sb, k_sn, k_sh, v_sb, v_sn, v_sh, t_sh, t_sb, t_sk;
  int B, Hkv, G, T, block_size, cache_len, S;
  int window, stride, topk_out, init_blocks, local_blocks, lc_pad, nb_pad, slots;  // slots: logits sub-tiles per CTA
  float scale2;
  // step
  const void* gate;
  long long g_sb, g_sh;
  Cache sel, cmp, stage, win;
  int* ticket;  // [B] zero between steps
  const void* w[2];
  const void* pe;        // [Hkv, window, D] position embedding of the keys' windows (pooling), or nullptr
  const float* partial;  // linear compression: [window][B][2][Hkv][D] per-tap products, or nullptr
  const float* inv_freq;
  float rope_scaling;
  Status st;
};

template <int D, int NW>
struct Layout {
  static constexpr int kTile = kSub * D * 2;               // K or V sub-tile
  static constexpr int kWarpBuf = 2 * kTile;
  static constexpr int kOStride = D + 8;                   // floats per row of a warp's partial output (in its tile buffers)
  static_assert(16 * kOStride * 4 <= kWarpBuf, "a warp's partial output lives in its tile buffers");
  static constexpr int kPart = NW * kWarpBuf;              // float [2][16][D]: the CTA's partial outputs
  static constexpr int kMlw = kPart + 2 * 16 * D * 4;      // float2 [NW][16]: (max, sum) of every warp
  static constexpr int kMlc = kMlw + NW * 16 * 8;          // float2 [2][16]: of the CTA
  static constexpr int kWts = kMlc + 2 * 16 * 8;           // float [2][kMaxCluster][16]: weight of every CTA's partial output
  static constexpr int kLse = kWts + 2 * kMaxCluster * 16 * 4;  // float [16]
  static constexpr int kList = kLse + 64;                  // int [kMaxList + kMaxSelTiles]: sub-tile rows; selected blocks
  static constexpr int kQ = (kList + (kMaxList + kMaxSelTiles) * 4 + 127) / 128 * 128;  // step: [16][kQLd] rotated query, 16-bit
  static constexpr int kQLd = D + 8;                       // elements per row of the rotated query: fragment loads hit 32 banks
  static constexpr int kTrig = kQ + 16 * kQLd * 2;         // step: float [4][D / 2] cos / sin of the two positions
  static constexpr int kVar = kTrig + 4 * (D / 2) * 4;     // logits [G][slots * 32], key scores [lc_pad], block scores [nb_pad]
};

template <typename T, int D>
__device__ __forceinline__ void load_sub(uint32_t dst, const T* base, long long sn, int row0, int lim) {
  constexpr int CH = D / 8, RPI = 32 / CH;
  const int c = lane_id() % CH, r_in = lane_id() / CH;
  const T* src = base + (long long)row0 * sn + c * 8;
#pragma unroll
  for (int it = 0; it < kSub / RPI; ++it) {
    const int r = r_in + it * RPI;
    const bool ok = r < lim;
    cp_async16(swz_addr<kSub>(dst, r, c), src + (long long)(ok ? r : 0) * sn, ok);
  }
}

// One online-softmax step over a [16 x 32] logit tile (base-2 domain); lim: leading visible keys.  scaled() sees the scaled,
// masked logits.
template <int NT_O, typename Scaled>
__device__ __forceinline__ void softmax_step32(float (&s)[4][4], int lim, float scale2, float (&m)[2], float (&l)[2],
                                               float (&o)[NT_O][4], Scaled scaled) {
  const int c0 = (lane_id() & 3) * 2;
  float mx[2] = {-INFINITY, -INFINITY};
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float v = (j * 8 + c0 + (e & 1) < lim) ? s[j][e] * scale2 : -INFINITY;
      s[j][e] = v;
      mx[e >> 1] = fmaxf(mx[e >> 1], v);
    }
  scaled(s);
  float corr[2], ref[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    const float mn = fmaxf(m[r], quad_max(mx[r]));
    ref[r] = mn == -INFINITY ? 0.f : mn;
    corr[r] = fast_exp2(m[r] - ref[r]);
    m[r] = mn;
  }
  float sum[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 4; ++j)
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      s[j][e] = fast_exp2(s[j][e] - ref[e >> 1]);
      sum[e >> 1] += s[j][e];
    }
#pragma unroll
  for (int r = 0; r < 2; ++r) l[r] = l[r] * corr[r] + quad_sum(sum[r]);
#pragma unroll
  for (int j = 0; j < NT_O; ++j) {
    o[j][0] *= corr[0]; o[j][1] *= corr[0]; o[j][2] *= corr[1]; o[j][3] *= corr[1];
  }
}

// This warp's share of a branch: sub-tiles first, first + step, ... below n of the rows whose K and V start at kb / vb.
// sub_at(i, row, lim): first row and number of visible rows of sub-tile i.  logits(i, s): the scaled logits of sub-tile i.
// Leaves the warp's partial output in its buffer and (max, sum) in mlw.
template <typename T, int D, int NW, typename SubAt, typename Logits>
__device__ __forceinline__ void attend(uint8_t* smem, const uint32_t (&qf)[D / 16][4], const T* kb, const T* vb, long long k_sn,
                                       long long v_sn, int first, int step, int n, float scale2, SubAt sub_at, Logits logits) {
  using L = Layout<D, NW>;
  const int warp = threadIdx.x >> 5, lane = lane_id();
  uint8_t* buf = smem + warp * L::kWarpBuf;
  const uint32_t kbuf = smem_u32(buf), vbuf = kbuf + L::kTile;
  float o[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j) o[j][0] = o[j][1] = o[j][2] = o[j][3] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};
  if (first < n) {
    int row, lim;
    sub_at(first, row, lim);
    load_sub<T, D>(kbuf, kb, k_sn, row, lim);
    cp_async_commit();
    load_sub<T, D>(vbuf, vb, v_sn, row, lim);
    cp_async_commit();
    for (int i = first; i < n; i += step) {
      sub_at(i, row, lim);
      int nrow = 0, nlim = 0;
      if (i + step < n) sub_at(i + step, nrow, nlim);
      cp_async_wait<1>();
      __syncwarp();
      float s[4][4];
#pragma unroll
      for (int j = 0; j < 4; ++j) s[j][0] = s[j][1] = s[j][2] = s[j][3] = 0.f;
      mma_nk<T, 4, D / 16, kSub>(s, qf, kbuf, 0, 0);
      __syncwarp();
      if (nlim > 0) load_sub<T, D>(kbuf, kb, k_sn, nrow, nlim);
      cp_async_commit();
      softmax_step32<D / 8>(s, lim, scale2, m, l, o, [&](const float (&sc)[4][4]) { logits(i, sc); });
      uint32_t pf[2][4];
      acc_to_a_frags<T, 2>(pf, s);
      cp_async_wait<1>();
      __syncwarp();
      mma_kn<T, D / 8, 2, kSub>(o, pf, vbuf, 0, 0);
      __syncwarp();
      if (nlim > 0) load_sub<T, D>(vbuf, vb, v_sn, nrow, nlim);
      cp_async_commit();
    }
  }
  cp_async_wait<0>();
  __syncwarp();
  const int r0 = lane >> 2, c0 = (lane & 3) * 2;
  float* po = reinterpret_cast<float*>(buf);
#pragma unroll
  for (int j = 0; j < D / 8; ++j) {
    *reinterpret_cast<float2*>(po + r0 * L::kOStride + j * 8 + c0) = make_float2(o[j][0], o[j][1]);
    *reinterpret_cast<float2*>(po + (r0 + 8) * L::kOStride + j * 8 + c0) = make_float2(o[j][2], o[j][3]);
  }
  if ((lane & 3) == 0) {
    float2* mlw = reinterpret_cast<float2*>(smem + L::kMlw) + warp * 16;
    mlw[r0] = make_float2(m[0], l[0]);
    mlw[r0 + 8] = make_float2(m[1], l[1]);
  }
}

// Threads t of nt (a multiple of 16) merge the partial outputs of warps [w0, w0 + nw) into branch `br` of this CTA.
template <int D, int NW>
__device__ __forceinline__ void cta_merge(uint8_t* smem, int br, int w0, int nw, int t, int nt) {
  using L = Layout<D, NW>;
  const int tpr = nt / 16, row = t / tpr, c = t % tpr;
  const float2* mlw = reinterpret_cast<const float2*>(smem + L::kMlw) + w0 * 16 + row;
  float mx = -INFINITY;
  for (int w = 0; w < nw; ++w) mx = fmaxf(mx, mlw[w * 16].x);
  float sum = 0.f;
  for (int w = 0; w < nw; ++w)
    if (mlw[w * 16].y != 0.f) sum += mlw[w * 16].y * fast_exp2(mlw[w * 16].x - mx);
  float* part = reinterpret_cast<float*>(smem + L::kPart) + (br * 16 + row) * D;
  for (int v = c; v < D / 4; v += tpr) {
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int w = 0; w < nw; ++w) {
      const float mw = mlw[w * 16].x;
      if (mlw[w * 16].y == 0.f) continue;  // saw no key (a NaN row has a NaN here)
      const float wt = fast_exp2(mw - mx);
      const float4 x = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(smem + (w0 + w) * L::kWarpBuf) + row * L::kOStride + v * 4);
      acc.x += x.x * wt; acc.y += x.y * wt; acc.z += x.z * wt; acc.w += x.w * wt;
    }
    *reinterpret_cast<float4*>(part + v * 4) = acc;
  }
  if (c == 0) reinterpret_cast<float2*>(smem + L::kMlc)[br * 16 + row] = make_float2(mx, sum);
}

// After a cluster barrier: the weight of every CTA's partial output (divided by the row's denominator), for `branches` branches;
// branch 0 also leaves its base-2 log-sum-exp (+inf for a row without a key).  Followed by __syncthreads.
template <int D, int NW>
__device__ __forceinline__ void cluster_weights(uint8_t* smem, int S, int branches) {
  using L = Layout<D, NW>;
  // S lanes per row (S is a power of two): one load each, then shuffles
  for (int t = threadIdx.x; t < 16 * branches * S; t += NW * 32) {
    const int s = t & (S - 1), row = t / S;  // row: branch * 16 + row
    const float2 ml = ld_peer2(peer_addr(reinterpret_cast<const float2*>(smem + L::kMlc) + row, s));
    float mx = ml.x;
    for (int o = S >> 1; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float w = ml.y == 0.f ? 0.f : fast_exp2(ml.x - mx);
    float sum = ml.y * w;
    for (int o = S >> 1; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    w *= sum > 0.f ? 1.f / sum : 0.f;
    reinterpret_cast<float*>(smem + L::kWts)[((row >> 4) * kMaxCluster + s) * 16 + (row & 15)] = w;
    if (s == 0 && row < 16) reinterpret_cast<float*>(smem + L::kLse)[row] = sum > 0.f ? mx + log2f(sum) : INFINITY;
  }
}

// The CTA's k-th group of four outputs of branch `br`: vector index v of [16][D / 4].
template <int D, int NW>
__device__ __forceinline__ float4 cluster_gather(uint8_t* smem, int S, int br, int v) {
  using L = Layout<D, NW>;
  const float* part = reinterpret_cast<const float*>(smem + L::kPart) + br * 16 * D + v * 4;
  const float* wts = reinterpret_cast<const float*>(smem + L::kWts) + br * kMaxCluster * 16 + v / (D / 4);
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
  for (int s = 0; s < S; ++s) {
    const float w = wts[s * 16];
    const float4 x = ld_peer4(peer_addr(part, s));
    acc.x += x.x * w; acc.y += x.y * w; acc.z += x.z * w; acc.w += x.w * w;
  }
  return acc;
}

template <typename T>
__device__ __forceinline__ float round16(float x) { return DT<T>::to_float(DT<T>::from_float(x)); }

template <typename T, int D>
__device__ __forceinline__ T* cache_ptr(const Cache& c, int kv, int b, long long row, int h) {
  return static_cast<T*>(c.base) + kv * c.s2 + b * c.sb + row * c.sn + h * c.sh;
}

// cos and sin of inv_freq * pos, scaled and rounded to the storage type, for the D / 2 frequencies (as in rope.cu)
template <typename T, int D>
__device__ __forceinline__ void trig_table(float* cs, float* sn, const float* inv_freq, int pos, float scaling, int t) {
  float s, c;
  sincosf(__ldg(inv_freq + t) * (float)pos, &s, &c);
  cs[t] = round16<T>(c * scaling);
  sn[t] = round16<T>(s * scaling);
}

template <typename T, int D, int NW, int MODE>
__global__ void __launch_bounds__(NW * 32, NW == 4 ? 2 : 1) decode_cluster_kernel(const __grid_constant__ Params p) {
  using L = Layout<D, NW>;
  constexpr int NT = NW * 32;
  constexpr int NV = 16 * D / 4;             // vectors of four outputs of a pair
  constexpr int VPT = (NV + NT - 1) / NT;
  constexpr int NC = MODE == kStep ? NW / 2 : NW;  // warps of the compressed branch (step: the other half attends the window)
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = p.S;
  const uint32_t rank = cluster_rank();
  const int pair = blockIdx.x / S;
  const int h = pair % p.Hkv, b = pair / p.Hkv;
  float* logit_sm = reinterpret_cast<float*>(smem + L::kVar);
  const int logit_ld = p.slots * kSub;
  float* keysc = logit_sm + p.G * logit_ld;
  float* bsc = keysc + p.lc_pad;
  int* list = reinterpret_cast<int*>(smem + L::kList);
  int* sel = list + kMaxList;

  // ---- lengths, and for a step everything that happens to the new token before attention ----
  int len, cmp_rows = 0, win_rows = 0;
  uint32_t qf[D / 16][4];
  if constexpr (MODE == kStep) {
    const int ls = __ldcg(p.sel.len + b), lc = __ldcg(p.cmp.len + b), lw = __ldcg(p.win.len + b), lst = __ldcg(p.stage.len + b);
    const bool shift = lst == p.window;                      // a full staging buffer was compressed in the step before
    const int kept = shift ? lst - p.stride : lst;
    const bool full = kept + 1 == p.window;                  // ... and this token completes the next window
    const bool has_cmp = full && lc < p.cmp.rows;
    len = min(ls + 1, p.sel.rows);
    cmp_rows = lc + (has_cmp ? 1 : 0);
    win_rows = min(lw + 1, p.win.rows);
    float* trig = reinterpret_cast<float*>(smem + L::kTrig);
    // the query elements are on their way while the counters arrive and the angles are computed
    constexpr int QPT = 16 * (D / 2) / NT;
    T qx1[QPT], qx2[QPT];
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const int g = (tid + u * NT) / (D / 2), j = (tid + u * NT) % (D / 2);
      const T* src = static_cast<const T*>(p.q) + b * p.q_sb + (long long)(h * p.G + min(g, p.G - 1)) * p.q_sh;
      qx1[u] = src[j];
      qx2[u] = src[j + D / 2];
    }
    if (tid < D / 2) trig_table<T, D>(trig, trig + D / 2, p.inv_freq, ls, p.rope_scaling, tid);
    else if (tid >= 64 && tid < 64 + D / 2 && rank == 0 && full)
      trig_table<T, D>(trig + D, trig + 3 * D / 2, p.inv_freq, lc * p.stride, p.rope_scaling, tid - 64);
    __syncthreads();
    // rotated query: 16 rows of D in shared memory (rows beyond the group are zero); every CTA makes its own copy
    T* qs = reinterpret_cast<T*>(smem + L::kQ);
#pragma unroll
    for (int u = 0; u < QPT; ++u) {
      const int g = (tid + u * NT) / (D / 2), j = (tid + u * NT) % (D / 2);
      float y1 = 0.f, y2 = 0.f;
      if (g < p.G) {
        const float x1 = DT<T>::to_float(qx1[u]), x2 = DT<T>::to_float(qx2[u]);
        y1 = fmaf(x1, trig[j], -x2 * trig[D / 2 + j]);
        y2 = fmaf(x2, trig[j], x1 * trig[D / 2 + j]);
      }
      qs[g * L::kQLd + j] = DT<T>::from_float(y1);
      qs[g * L::kQLd + j + D / 2] = DT<T>::from_float(y2);
    }
    if (rank == 0) {
      // one thread per pair of columns (j, j + D / 2) of the key or value: it owns them in every row it touches
      if (tid < D) {
        const int kv = tid / (D / 2), j = tid % (D / 2);
        const T* src = kv ? static_cast<const T*>(p.v) + b * p.v_sb + h * p.v_sh : static_cast<const T*>(p.k) + b * p.k_sb + h * p.k_sh;
        const T n1 = src[j], n2 = src[j + D / 2];
        // staging buffer: drop the first `stride` rows if it was full, append the new row, pool it if that completes a window
        const T* w = static_cast<const T*>(p.w[kv]);
        const bool weighted = w != nullptr && p.partial == nullptr;
        const bool pool = full && !p.partial;
        // (the position embedding's sum is kept apart and rounded, as the operators do)
        const T* pe = kv == 0 && pool && p.pe ? static_cast<const T*>(p.pe) + (long long)h * p.window * D + j : nullptr;
        float a1 = 0.f, a2 = 0.f, e1 = 0.f, e2 = 0.f;
        if (shift || full) {
          // Sixteen rows at a time, every load of them before the first store: a store to the buffer in between holds back the
          // loads behind it, and 32 weights fetched one by one were 10 of the 30 us of a step that completes a window.
          const int off = shift ? p.stride : 0;
          const int n_rows = pe ? p.window : kept;
          for (int r0 = 0; r0 < n_rows; r0 += 16) {
            T x1[16], x2[16], z1[16], z2[16], wr[16];
#pragma unroll
            for (int u = 0; u < 16; ++u) {
              const int r = min(r0 + u, n_rows - 1), rk = max(min(r, kept - 1), 0);
              const T* row = cache_ptr<T, D>(p.stage, kv, b, rk + off, h);
              x1[u] = row[j];
              x2[u] = row[j + D / 2];
              wr[u] = pool && weighted ? w[h * p.window + r] : DT<T>::from_float(1.f);
              z1[u] = z2[u] = DT<T>::from_float(0.f);
              if (pe) {
                z1[u] = pe[r * D];
                z2[u] = pe[r * D + D / 2];
              }
            }
#pragma unroll
            for (int u = 0; u < 16; ++u) {
              const float wv = DT<T>::to_float(wr[u]);
              if (r0 + u < kept) {
                if (shift) {
                  T* row = cache_ptr<T, D>(p.stage, kv, b, r0 + u, h);
                  row[j] = x1[u];
                  row[j + D / 2] = x2[u];
                }
                a1 += wv * DT<T>::to_float(x1[u]);
                a2 += wv * DT<T>::to_float(x2[u]);
              }
              if (r0 + u < n_rows) {
                e1 += wv * DT<T>::to_float(z1[u]);
                e2 += wv * DT<T>::to_float(z2[u]);
              }
            }
          }
        }
        {
          T* row = cache_ptr<T, D>(p.stage, kv, b, kept, h);
          row[j] = n1;
          row[j + D / 2] = n2;
        }
        if (full) {
          if (p.partial) {  // linear compression: the taps' products, summed in order
            const long long tap = (long long)p.B * 2 * p.Hkv * D;
            const float* pt = p.partial + (((long long)b * 2 + kv) * p.Hkv + h) * D;
            a1 = a2 = 0.f;
#pragma unroll 8
            for (int r = 0; r < p.window; ++r) {
              a1 += __ldcg(pt + r * tap + j);
              a2 += __ldcg(pt + r * tap + j + D / 2);
            }
          } else {
            const float wv = weighted ? DT<T>::to_float(w[h * p.window + kept]) : 1.f;
            a1 += wv * DT<T>::to_float(n1);
            a2 += wv * DT<T>::to_float(n2);
            if (!weighted) {
              const float inv = 1.f / (float)p.window;
              a1 *= inv;
              a2 *= inv;
              e1 /= (float)p.window;
              e2 /= (float)p.window;
            }
          }
          if (pe) {
            a1 = round16<T>(a1) + round16<T>(e1);
            a2 = round16<T>(a2) + round16<T>(e2);
          }
          a1 = round16<T>(a1);
          a2 = round16<T>(a2);
          if (has_cmp) {
            T* row = cache_ptr<T, D>(p.cmp, kv, b, lc, h);
            if (kv == 0) {
              const float c = trig[D + j], s = trig[3 * D / 2 + j];
              row[j] = DT<T>::from_float(fmaf(a1, c, -a2 * s));
              row[j + D / 2] = DT<T>::from_float(fmaf(a2, c, a1 * s));
            } else {
              row[j] = DT<T>::from_float(a1);
              row[j + D / 2] = DT<T>::from_float(a2);
            }
          }
        }
        // the new row (key rotated) goes to the selected-block cache and the ring
        T y1 = n1, y2 = n2;
        if (kv == 0) {
          const float x1 = DT<T>::to_float(n1), x2 = DT<T>::to_float(n2);
          y1 = DT<T>::from_float(fmaf(x1, trig[j], -x2 * trig[D / 2 + j]));
          y2 = DT<T>::from_float(fmaf(x2, trig[j], x1 * trig[D / 2 + j]));
        }
        if (ls < p.sel.rows) {
          T* row = cache_ptr<T, D>(p.sel, kv, b, ls, h);
          row[j] = y1;
          row[j + D / 2] = y2;
        }
        T* row = cache_ptr<T, D>(p.win, kv, b, lw % p.win.rows, h);
        row[j] = y1;
        row[j + D / 2] = y2;
      }
    }
    cluster_barrier();
    if (rank == 0 && tid == 0) {
      // the last of the sequence's clusters to have read its counters advances them
      __threadfence();
      if (atomicInc(reinterpret_cast<unsigned*>(p.ticket + b), (unsigned)(p.Hkv - 1)) == (unsigned)(p.Hkv - 1)) {
        if (full) {
          if (has_cmp) p.cmp.len[b] = lc + 1; else p.st.raise(kErrBadIndex);
        }
        if (ls < p.sel.rows) p.sel.len[b] = ls + 1; else p.st.raise(kErrBadIndex);
        p.win.len[b] = lw + 1;
        p.stage.len[b] = kept + 1;
      }
    }
    {
      const T* q0 = qs;
      const int r = lane >> 2, c = (lane & 3) * 2;
#pragma unroll
      for (int kk = 0; kk < D / 16; ++kk) {
        qf[kk][0] = *reinterpret_cast<const uint32_t*>(q0 + r * L::kQLd + kk * 16 + c);
        qf[kk][1] = *reinterpret_cast<const uint32_t*>(q0 + (r + 8) * L::kQLd + kk * 16 + c);
        qf[kk][2] = *reinterpret_cast<const uint32_t*>(q0 + r * L::kQLd + kk * 16 + c + 8);
        qf[kk][3] = *reinterpret_cast<const uint32_t*>(q0 + (r + 8) * L::kQLd + kk * 16 + c + 8);
      }
    }
  } else {
    len = __ldg(p.seqlens + b);
    if constexpr (MODE == kCompressed) cmp_rows = min(__ldg(p.cmp_seqlens + b), p.cache_len);
    const T* qbase = static_cast<const T*>(p.q) + b * p.q_sb + (long long)h * p.G * p.q_sh;
    load_a_frags_global<T, D / 16>(qf, [&](int r) -> const T* { return r < p.G ? qbase + r * p.q_sh : nullptr; });
  }

  // ---- which four-output vectors this thread finishes ----
  const int nv = NV / S, v0 = rank * nv;
  auto plain_rows = [](int rows) {
    return [rows](int i, int& row, int& lim) {
      row = i * kSub;
      lim = min(kSub, rows - row);
    };
  };
  auto no_logits = [](int, const float (&)[4][4]) {};
  // output rows of the pair
  T* obase = static_cast<T*>(p.o) + b * p.o_sb + (long long)h * p.G * p.o_sh;
  auto store4 = [&](int v, float4 x) {
    const int g = v / (D / 4), c = v % (D / 4);
    if (g < p.G) {
      uint2 u;
      u.x = DT<T>::pack(x.x, x.y);
      u.y = DT<T>::pack(x.z, x.w);
      *reinterpret_cast<uint2*>(obase + g * p.o_sh + c * 4) = u;
    }
  };
  float4 cmp4[VPT], win4[VPT];

  // ---- compressed branch (and, in a step, the window branch on the other half of the warps) ----
  if constexpr (MODE == kCompressed || MODE == kStep) {
    const int n_cmp = (cmp_rows + kSub - 1) / kSub;
    const bool on_cmp = warp < NC;
    if (on_cmp) {
      const T* kb = MODE == kStep ? cache_ptr<T, D>(p.cmp, 0, b, 0, h) : static_cast<const T*>(p.k) + b * p.k_sb + h * p.k_sh;
      const T* vb = MODE == kStep ? cache_ptr<T, D>(p.cmp, 1, b, 0, h) : static_cast<const T*>(p.v) + b * p.v_sb + h * p.v_sh;
      const int first = rank * NC + warp, step = NC * S;
      const int r0 = lane >> 2, c0 = (lane & 3) * 2;
      attend<T, D, NW>(smem, qf, kb, vb, MODE == kStep ? p.cmp.sn : p.k_sn, MODE == kStep ? p.cmp.sn : p.v_sn, first, step, n_cmp, p.scale2,
                       plain_rows(cmp_rows), [&](int i, const float (&sc)[4][4]) {
                         float* dst = logit_sm + ((i - first) / step * NC + warp) * kSub;
#pragma unroll
                         for (int j = 0; j < 4; ++j) {
                           if (r0 < p.G) *reinterpret_cast<float2*>(dst + r0 * logit_ld + j * 8 + c0) = make_float2(sc[j][0], sc[j][1]);
                           if (r0 + 8 < p.G) *reinterpret_cast<float2*>(dst + (r0 + 8) * logit_ld + j * 8 + c0) = make_float2(sc[j][2], sc[j][3]);
                         }
                       });
    } else if constexpr (MODE == kStep) {
      attend<T, D, NW>(smem, qf, cache_ptr<T, D>(p.win, 0, b, 0, h), cache_ptr<T, D>(p.win, 1, b, 0, h), p.win.sn, p.win.sn,
                       rank * NC + warp - NC, NC * S, (win_rows + kSub - 1) / kSub, p.scale2, plain_rows(win_rows), no_logits);
    }
    __syncthreads();
    if constexpr (MODE == kStep) {
      if (tid < NT / 2) cta_merge<D, NW>(smem, 0, 0, NC, tid, NT / 2);
      else cta_merge<D, NW>(smem, 1, NC, NC, tid - NT / 2, NT / 2);
    } else {
      cta_merge<D, NW>(smem, 0, 0, NW, tid, NT);
    }
    cluster_barrier();
    cluster_weights<D, NW>(smem, S, MODE == kStep ? 2 : 1);
    __syncthreads();
    if (MODE == kStep || p.topk_out_idx) {
      // key scores of this CTA's sub-tiles, to rank 0
      const float* lse = reinterpret_cast<const float*>(smem + L::kLse);
      const uint32_t dst = peer_addr(keysc, 0);
      for (int i = tid; i < logit_ld; i += NT) {
        const int slot = i / kSub;
        const int key = ((slot / NC) * (NC * S) + rank * NC + slot % NC) * kSub + i % kSub;
        if (key < cmp_rows) {
          float v = 0.f;
          for (int g = 0; g < p.G; ++g) v += fast_exp2(logit_sm[g * logit_ld + i] - lse[g]);
          st_peer(dst + key * 4, v);
        }
      }
    }
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      const int i = tid + k * NT;
      if (i < nv) {
        cmp4[k] = cluster_gather<D, NW>(smem, S, 0, v0 + i);
        if constexpr (MODE == kStep) win4[k] = cluster_gather<D, NW>(smem, S, 1, v0 + i);
        else store4(v0 + i, cmp4[k]);
      }
    }
    cluster_barrier();
    if (rank == 0 && (MODE == kStep || p.topk_out_idx)) {
      const int a = p.window / p.stride, c = p.block_size / p.stride;
      const int bq = (len - 1) / p.block_size;
      for (int bb = tid; bb <= bq && bb < p.nb_pad; bb += NT) {
        float acc = 0.f;
        for (int o2 = 0; o2 <= a + c - 2; ++o2) {
          const int key = bb * c - (a - 1) + o2;
          if (key >= 0 && key < cmp_rows) acc += (float)fold_weight(o2, a, c) * keysc[key];
        }
        bsc[bb] = acc;
      }
      __syncthreads();
      if (warp == 0) {
        if constexpr (MODE == kStep) warp_select_topk<false>(bsc, min(bq, p.nb_pad - 1), p.topk_out, p.init_blocks, p.local_blocks, sel, 1);
        else warp_select_topk<false>(bsc, min(bq, p.nb_pad - 1), p.topk_out, p.init_blocks, p.local_blocks,
                              p.topk_out_idx + h * p.t_sh + (long long)b * p.t_sb, p.t_sk);
      }
    }
    if constexpr (MODE == kCompressed) return;
    cluster_barrier();
  }

  // ---- selected blocks / every row ----
  int n = 0;
  if constexpr (MODE == kSparse || MODE == kStep) {
    // sub-tiles of the selected blocks, in the order of the selection
    const int rows = MODE == kStep ? len : min(len, p.cache_len);
    if (warp == 0) {
      const int BS = p.block_size, nsub = BS / kSub;
      const int bq = rows > 0 ? (len - 1) / BS : -1;
      const int T_in = MODE == kStep ? p.topk_out : p.T;
      const int* tptr = MODE == kStep ? nullptr : p.topk_idx + h * p.t_sh + (long long)b * p.t_sb;
      for (int base = 0; base < T_in; base += 32) {
        const int j = base + lane;
        int idx = -1;
        if (j < T_in) {
          if constexpr (MODE == kStep) idx = ld_peer_i(peer_addr(sel + j, 0));
          else idx = __ldg(tptr + j * p.t_sk);
        }
        const bool valid = idx >= 0 && idx <= bq && idx * BS < rows;
        const int cnt = valid ? min(nsub, (rows - 1 - idx * BS) / kSub + 1) : 0;
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int t = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += t;
        }
        for (int s = 0; s < cnt; ++s) {
          const int pos = n + incl - cnt + s;
          if (pos < kMaxList) list[pos] = idx * BS + s * kSub;
        }
        n += __shfl_sync(0xffffffffu, incl, 31);
      }
      if (n > kMaxList) {
        if (lane == 0) p.st.raise(kErrBadIndex);
        n = kMaxList;
      }
      if (lane == 0) reinterpret_cast<int*>(smem + L::kLse)[0] = n;
    }
    __syncthreads();
    n = reinterpret_cast<const int*>(smem + L::kLse)[0];
    const T* kb = MODE == kStep ? cache_ptr<T, D>(p.sel, 0, b, 0, h) : static_cast<const T*>(p.k) + b * p.k_sb + h * p.k_sh;
    const T* vb = MODE == kStep ? cache_ptr<T, D>(p.sel, 1, b, 0, h) : static_cast<const T*>(p.v) + b * p.v_sb + h * p.v_sh;
    attend<T, D, NW>(smem, qf, kb, vb, MODE == kStep ? p.sel.sn : p.k_sn, MODE == kStep ? p.sel.sn : p.v_sn, rank * NW + warp, NW * S, n,
                     p.scale2, [&](int i, int& row, int& lim) {
                       row = list[i];
                       lim = min(kSub, rows - row);
                     }, no_logits);
  } else {
    const int rows = min(len, p.cache_len);
    n = (rows + kSub - 1) / kSub;
    attend<T, D, NW>(smem, qf, static_cast<const T*>(p.k) + b * p.k_sb + h * p.k_sh, static_cast<const T*>(p.v) + b * p.v_sb + h * p.v_sh,
                     p.k_sn, p.v_sn, rank * NW + warp, NW * S, n, p.scale2, plain_rows(rows), no_logits);
  }
  __syncthreads();
  cta_merge<D, NW>(smem, 0, 0, NW, tid, NT);
  cluster_barrier();
  cluster_weights<D, NW>(smem, S, 1);
  __syncthreads();
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const int i = tid + k * NT;
    if (i < nv) {
      const int v = v0 + i, g = v / (D / 4);
      float4 x = cluster_gather<D, NW>(smem, S, 0, v);
      if constexpr (MODE == kStep) {
        if (g < p.G) {
          // gated sum; the branch outputs are rounded to the storage type first, as when each is an operator's result
          const T* gp = static_cast<const T*>(p.gate) + b * p.g_sb + (long long)(h * p.G + g) * p.g_sh;
          const float g0 = DT<T>::to_float(gp[0]), g1 = DT<T>::to_float(gp[1]), g2 = DT<T>::to_float(gp[2]);
          auto mix = [&](float c, float s, float w) { return fmaf(g2, round16<T>(w), fmaf(g1, round16<T>(s), g0 * round16<T>(c))); };
          x = make_float4(mix(cmp4[k].x, x.x, win4[k].x), mix(cmp4[k].y, x.y, win4[k].y), mix(cmp4[k].z, x.z, win4[k].z),
                          mix(cmp4[k].w, x.w, win4[k].w));
        }
      }
      store4(v, x);
    }
  }
  cluster_barrier();  // no CTA leaves while its shared memory is being read
}

// ---- linear compression of the windows a decode step completes ----
// One CTA per (tap, KV head, key or value): the products of the tap's row with its [D x D] weight slice, for every sequence
// whose window is completed by the new token.  Most steps complete none, and the CTA leaves after reading the counters.
struct LinearTapParams {
  const void* x[2];  // the new token's key and value rows [B, Hkv, D]
  long long x_sb[2], x_sh[2];
  const void* w[2];  // [Hkv, window * D, D]
  const void* pe;    // [Hkv, window, D] added to the keys' rows, or nullptr
  Cache stage;
  float* partial;    // [window][B][2][Hkv][D]
  int B, Hkv, window, stride;
};

template <typename T, int D>
__global__ void __launch_bounds__(256) linear_tap_kernel(LinearTapParams p) {
  constexpr int CH = D / 8, RG = 256 / CH;  // 16-byte column groups; row groups
  const int tap = blockIdx.x, h = blockIdx.y, kv = blockIdx.z;
  __shared__ float xs[D];
  __shared__ float red[RG][D];
  const int c = threadIdx.x % CH, rg = threadIdx.x / CH;
  const T* w = static_cast<const T*>(p.w[kv]) + ((size_t)h * p.window + tap) * D * D;
  for (int b = 0; b < p.B; ++b) {
    const int lst = __ldg(p.stage.len + b);
    const bool shift = lst == p.window;
    const int kept = shift ? lst - p.stride : lst;
    if (kept + 1 != p.window) continue;
    if (threadIdx.x < D) {
      const T* src = tap == kept ? static_cast<const T*>(p.x[kv]) + b * p.x_sb[kv] + h * p.x_sh[kv]
                                 : cache_ptr<T, D>(p.stage, kv, b, tap + (shift ? p.stride : 0), h);
      float x = DT<T>::to_float(src[threadIdx.x]);
      if (kv == 0 && p.pe) x += DT<T>::to_float(static_cast<const T*>(p.pe)[((size_t)h * p.window + tap) * D + threadIdx.x]);
      xs[threadIdx.x] = x;
    }
    __syncthreads();
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int r = rg; r < D; r += RG) {
      const uint4 v = __ldg(reinterpret_cast<const uint4*>(w + (size_t)r * D + c * 8));
      const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = DT<T>::unpack(u[e]);
        acc[2 * e] = fmaf(xs[r], f.x, acc[2 * e]);
        acc[2 * e + 1] = fmaf(xs[r], f.y, acc[2 * e + 1]);
      }
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) red[rg][c * 8 + e] = acc[e];
    __syncthreads();
    if (threadIdx.x < D) {
      float sum = 0.f;
#pragma unroll
      for (int g = 0; g < RG; ++g) sum += red[g][threadIdx.x];
      p.partial[((((size_t)tap * p.B + b) * 2 + kv) * p.Hkv + h) * D + threadIdx.x] = sum;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------------------------------------------------- launching
constexpr size_t kSmemLimit = 227 * 1024;

// CTAs per cluster: a power of two, doubled while a warp still has more than one sub-tile to walk and the machine has room (one
// CTA of eight warps or two of four per SM, by shared memory).
int cluster_size(long long pairs, int subtiles, int warps, int most) {
  const int room = num_sms() * (8 / warps);
  int s = 1;
  while (s < most && s * warps < subtiles && pairs * s * 2 <= room) s <<= 1;
  return s;
}

template <typename T, int D, int NW, int MODE>
size_t smem_bytes(const Params& p) {
  const size_t var = MODE == kCompressed || MODE == kStep ? (size_t)p.G * p.slots * kSub + p.lc_pad + p.nb_pad : 0;
  return Layout<D, NW>::kVar + var * sizeof(float);
}

void cluster_config(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, const Params& p, int threads, size_t smem, cudaStream_t stream) {
  cfg = {};
  cfg.gridDim = dim3((unsigned)(p.B * p.Hkv * p.S));
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  attr.id = cudaLaunchAttributeClusterDimension;
  attr.val.clusterDim.x = (unsigned)p.S;
  attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
}

// Clusters of 16 CTAs are opt-in and need a GPC with 16 SMs to spare: how many run at a time is asked once per device.
template <typename T, int D, int NW>
int clusters_of_16(size_t smem) {
  static std::atomic<int> known[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev >= 64) return 0;
  int f = known[dev].load(std::memory_order_acquire);
  if (f == 0) {
    auto kern = decode_cluster_kernel<T, D, NW, kDense>;
    f = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess && allow_smem(kern, smem) == cudaSuccess) {
      Params p{};
      p.B = 8; p.Hkv = 1; p.S = 16;
      cudaLaunchConfig_t cfg;
      cudaLaunchAttribute attr;
      cluster_config(cfg, attr, p, NW * 32, smem, nullptr);
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) == cudaSuccess && n > 0) f = 1 + n;
    }
    (void)cudaGetLastError();
    known[dev].store(f, std::memory_order_release);
  }
  return f - 1;
}

template <typename T, int D, int NW, int MODE>
int launch(const Params& p, const char* name, cudaStream_t stream) {
  auto kern = decode_cluster_kernel<T, D, NW, MODE>;
  const size_t smem = smem_bytes<T, D, NW, MODE>(p);
  if (smem > kSmemLimit) return kUnsupported;
  const cudaError_t e = allow_smem(kern, smem);
  if (e != cudaSuccess) return cuda_rc(e);
  cudaLaunchConfig_t cfg;
  cudaLaunchAttribute attr;
  cluster_config(cfg, attr, p, NW * 32, smem, stream);
  LaunchScope ls_(name, stream);
  return cuda_rc(cudaLaunchKernelEx(&cfg, kern, p));
}

// logits sub-tiles a CTA keeps: its warps' share of the longest compressed row
void set_logit_slots(Params& p, int max_rows, int warps) {
  const int subtiles = (max_rows + kSub - 1) / kSub;
  p.slots = (subtiles + warps * p.S - 1) / (warps * p.S) * warps;
  p.lc_pad = subtiles * kSub;
}

Params op_params(const DecodeOpArgs& a) {
  Params p{};
  const long long* s = a.strides;
  p.q = a.q; p.k = a.k; p.v = a.v; p.o = a.o;
  p.seqlens = a.seqlens; p.cmp_seqlens = a.cmp_seqlens; p.topk_idx = a.topk_idx; p.topk_out_idx = a.topk_out_idx;
  p.q_sb = s[0]; p.q_sh = s[1]; p.k_sb = s[2]; p.k_sn = s[3]; p.k_sh = s[4]; p.v_sb = s[5]; p.v_sn = s[6]; p.v_sh = s[7];
  p.o_sb = s[8]; p.o_sh = s[9]; p.t_sh = s[10]; p.t_sb = s[11]; p.t_sk = s[12];
  p.B = a.batch; p.Hkv = a.num_kv_heads; p.G = a.num_q_heads / a.num_kv_heads; p.T = a.topk; p.block_size = a.block_size;
  p.cache_len = a.cache_len;
  p.window = a.kernel_size; p.stride = a.kernel_stride; p.init_blocks = a.init_blocks; p.local_blocks = a.local_blocks;
  p.scale2 = a.sm_scale * kLog2e;
  p.st.word = status_word();
  return p;
}

// Four warps per CTA, two CTAs per SM: with few sub-tiles a smaller merge, with many pairs one CTA's set-up and merge under the
// other's loads (selected blocks, 304 pairs of 16 blocks: 33.7 us against 38.0 with eight warps).  Eight warps only where a few
// pairs have long rows and even clusters of 16 leave a warp several sub-tiles (8 pairs of 8256 rows: 13.4 us against 16.0).
template <typename T, int D>
int run_dense(Params p, cudaStream_t stream) {
  const long long pairs = (long long)p.B * p.Hkv;
  const int subtiles = (p.cache_len + kSub - 1) / kSub;
  p.S = cluster_size(pairs, subtiles, 8, 16);
  if (p.S == 16 && clusters_of_16<T, D, 8>(smem_bytes<T, D, 8, kDense>(p)) >= pairs) return launch<T, D, 8, kDense>(p, "decode_attn", stream);
  p.S = cluster_size(pairs, subtiles, 4, 8);
  // long rows are cut further, down to 16 sub-tiles per warp, until there are some four CTAs per place: lengths differ, and the
  // longest rows otherwise finish alone (304 pairs of 1 to 8192 rows: 120 us in one piece, 112 in two)
  while (p.S < 8 && subtiles / (p.S * 4) >= 16 && pairs * p.S < 8ll * num_sms()) p.S <<= 1;
  return launch<T, D, 4, kDense>(p, "decode_attn", stream);
}
template <typename T, int D>
int run_sparse(Params p, cudaStream_t stream) {
  p.S = cluster_size((long long)p.B * p.Hkv, p.T * (p.block_size / kSub), 4, 8);
  return launch<T, D, 4, kSparse>(p, "decode_attn_sparse", stream);
}
template <typename T, int D>
int run_compressed(Params p, cudaStream_t stream) {
  p.S = cluster_size((long long)p.B * p.Hkv, (p.cache_len + kSub - 1) / kSub, 4, 8);
  set_logit_slots(p, p.cache_len, 4);
  return launch<T, D, 4, kCompressed>(p, "decode_attn_compressed", stream);
}

// CTAs per cluster and logits per CTA of a step; kUnsupported where they do not fit into shared memory
constexpr int kStepWarps = 8;
template <typename T, int D>
int plan_step(Params* plan) {
  Params& p = *plan;
  const int half = kStepWarps / 2;
  // sub-tiles of the longest branch per warp that serves it
  int subtiles = (p.cmp.rows + kSub - 1) / kSub;
  const int win = (p.win.rows + kSub - 1) / kSub, sel = (p.topk_out * (p.block_size / kSub) + 1) / 2;
  if (win > subtiles) subtiles = win;
  if (sel > subtiles) subtiles = sel;
  p.S = cluster_size((long long)p.B * p.Hkv, subtiles, half, 8);
  set_logit_slots(p, p.cmp.rows, half);
  return smem_bytes<T, D, kStepWarps, kStep>(p) > kSmemLimit ? kUnsupported : kOk;
}

template <typename T, int D>
int run_step(Params p, cudaStream_t stream) {
  const int rc = plan_step<T, D>(&p);
  return rc ? rc : launch<T, D, kStepWarps, kStep>(p, "decode_step", stream);
}

// The sizes of a step, checked
int step_sizes(Params& p, int batch, int num_q_heads, int num_kv_heads, int kernel_size, int kernel_stride, int block_size, int topk,
               int init_blocks, int local_blocks, int sparse_rows, int compress_rows, int sliding_rows) {
  if (batch <= 0 || num_kv_heads <= 0 || num_q_heads % num_kv_heads) return kInvalid;
  if (num_q_heads / num_kv_heads > 16) return kUnsupported;
  if (kernel_size <= 0 || kernel_stride <= 0 || kernel_size % kernel_stride || block_size <= 0 || block_size % kernel_stride || topk < 1) return kInvalid;
  if (topk < init_blocks + local_blocks || sparse_rows <= 0 || compress_rows <= 0 || sliding_rows <= 0) return kInvalid;
  if (block_size % kSub) return kUnsupported;
  p.B = batch; p.Hkv = num_kv_heads; p.G = num_q_heads / num_kv_heads; p.block_size = block_size; p.window = kernel_size;
  p.stride = kernel_stride; p.init_blocks = init_blocks; p.local_blocks = local_blocks;
  p.sel.rows = sparse_rows; p.cmp.rows = compress_rows; p.stage.rows = kernel_size; p.win.rows = sliding_rows;
  const int max_blocks = (sparse_rows + block_size - 1) / block_size;
  p.topk_out = topk < max_blocks ? topk : max_blocks;
  p.nb_pad = (max_blocks + 31) & ~31;
  if ((long long)p.topk_out * block_size > (long long)kMaxSelTiles * 64 || p.topk_out > kMaxSelTiles) return kUnsupported;
  return kOk;
}

template <typename T, int D>
int run_taps(LinearTapParams p, cudaStream_t stream) {
  LaunchScope ls_("linear_taps", stream);
  linear_tap_kernel<T, D><<<dim3(p.window, p.Hkv, 2), 256, 0, stream>>>(p);
  return cuda_rc(cudaGetLastError());
}

bool cache_ok(const Cache& c) {
  return c.base && c.len && aligned16(c.base) && c.rows > 0 && ((c.s2 | c.sb | c.sn | c.sh) % 8) == 0;
}
Cache make_cache(void* base, int* len, const long long* s, int rows) { return Cache{base, s[0], s[1], s[2], s[3], len, rows}; }

}  // namespace

int decode_cluster_dense(const DecodeOpArgs& a, cudaStream_t stream) {
  return NSA_DISPATCH_T_D(a.dtype, a.head_dim, run_dense, op_params(a), stream);
}
int decode_cluster_sparse(const DecodeOpArgs& a, cudaStream_t stream) {
  return NSA_DISPATCH_T_D(a.dtype, a.head_dim, run_sparse, op_params(a), stream);
}
int decode_cluster_compressed(const DecodeOpArgs& a, cudaStream_t stream) {
  Params p = op_params(a);
  p.topk_out = a.topk < a.max_blocks ? a.topk : a.max_blocks;
  p.nb_pad = (a.max_blocks + 31) & ~31;
  return NSA_DISPATCH_T_D(a.dtype, a.head_dim, run_compressed, p, stream);
}

}  // namespace nsa

extern "C" int nsa_decode_step_supported(int batch, int num_q_heads, int num_kv_heads, int head_dim, int kernel_size, int kernel_stride,
                                         int block_size, int topk, int init_blocks, int local_blocks, int sparse_rows, int compress_rows,
                                         int sliding_rows, int dtype) {
  using namespace nsa;
  Params p{};
  const int rc = step_sizes(p, batch, num_q_heads, num_kv_heads, kernel_size, kernel_stride, block_size, topk, init_blocks, local_blocks,
                            sparse_rows, compress_rows, sliding_rows);
  if (rc) return rc;
  return NSA_DISPATCH_T_D(dtype, head_dim, plan_step, &p);
}

// strides: q_b q_h | k_b k_h | v_b v_h | gate_b gate_h | out_b out_h | then (kv, sequence, row, head) of the selected-block,
// compressed, staging and window caches: 26 entries, elements
extern "C" int nsa_decode_step(const void* q, const void* k, const void* v, const void* gate, void* out, void* sparse_cache, int* sparse_len,
                               void* compress_cache, int* compress_len, void* stage_cache, int* stage_len, void* sliding_cache,
                               int* sliding_len, int* ticket, const void* w_k, const void* w_v, const void* pe, const float* linear_taps,
                               const float* inv_freq, float attention_scaling, int batch, int num_q_heads, int num_kv_heads, int head_dim,
                               int kernel_size, int kernel_stride, int block_size, int topk, int init_blocks, int local_blocks,
                               int sparse_rows, int compress_rows, int sliding_rows, const long long* strides, float sm_scale, int dtype,
                               void* stream) {
  using namespace nsa;
  if (!q || !k || !v || !gate || !out || !ticket || !inv_freq || !strides) return kInvalid;
  Params p{};
  const int rc = step_sizes(p, batch, num_q_heads, num_kv_heads, kernel_size, kernel_stride, block_size, topk, init_blocks, local_blocks,
                            sparse_rows, compress_rows, sliding_rows);
  if (rc) return rc;
  for (int i = 0; i < 6; ++i)
    if (strides[i] % 8) return kInvalid;
  if (strides[8] % 8 || strides[9] % 8 || !aligned16(q) || !aligned16(k) || !aligned16(v) || !aligned16(out)) return kInvalid;
  p.q = q; p.k = k; p.v = v; p.gate = gate; p.o = out;
  p.q_sb = strides[0]; p.q_sh = strides[1]; p.k_sb = strides[2]; p.k_sh = strides[3]; p.v_sb = strides[4]; p.v_sh = strides[5];
  p.g_sb = strides[6]; p.g_sh = strides[7]; p.o_sb = strides[8]; p.o_sh = strides[9];
  p.sel = make_cache(sparse_cache, sparse_len, strides + 10, sparse_rows);
  p.cmp = make_cache(compress_cache, compress_len, strides + 14, compress_rows);
  p.stage = make_cache(stage_cache, stage_len, strides + 18, kernel_size);
  p.win = make_cache(sliding_cache, sliding_len, strides + 22, sliding_rows);
  if (!cache_ok(p.sel) || !cache_ok(p.cmp) || !cache_ok(p.stage) || !cache_ok(p.win)) return kInvalid;
  p.ticket = ticket; p.w[0] = w_k; p.w[1] = w_v; p.pe = linear_taps ? nullptr : pe; p.partial = linear_taps; p.inv_freq = inv_freq;
  p.rope_scaling = attention_scaling;
  p.scale2 = sm_scale * kLog2e;
  p.st.word = status_word();
  return NSA_DISPATCH_T_D(dtype, head_dim, run_step, p, static_cast<cudaStream_t>(stream));
}

// strides: k_b k_h | v_b v_h | (kv, sequence, row, head) of the staging cache
extern "C" int nsa_linear_decode_taps(const void* k, const void* v, const void* w_k, const void* w_v, const void* pe,
                                      const void* stage_cache, const int* stage_len, float* taps, int batch, int num_kv_heads, int head_dim, int kernel_size,
                                      int kernel_stride, const long long* strides, int dtype, void* stream) {
  using namespace nsa;
  if (!k || !v || !w_k || !w_v || !stage_cache || !stage_len || !taps || !strides || batch <= 0 || num_kv_heads <= 0) return kInvalid;
  if (kernel_size <= 0 || kernel_stride <= 0 || kernel_size % kernel_stride || !aligned16(w_k) || !aligned16(w_v)) return kInvalid;
  LinearTapParams p;
  p.x[0] = k; p.x[1] = v; p.w[0] = w_k; p.w[1] = w_v; p.pe = pe;
  p.x_sb[0] = strides[0]; p.x_sh[0] = strides[1]; p.x_sb[1] = strides[2]; p.x_sh[1] = strides[3];
  p.stage = make_cache(const_cast<void*>(stage_cache), const_cast<int*>(stage_len), strides + 4, kernel_size);
  if (!cache_ok(p.stage)) return kInvalid;
  p.partial = taps; p.B = batch; p.Hkv = num_kv_heads; p.window = kernel_size; p.stride = kernel_stride;
  return NSA_DISPATCH_T_D(dtype, head_dim, run_taps, p, static_cast<cudaStream_t>(stream));
}
