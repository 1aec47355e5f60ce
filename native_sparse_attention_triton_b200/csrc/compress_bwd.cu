// Backward of the compression operators (deterministic: no floating-point atomics).
//
// Linear compression  y = Xwin W + bias(pe, W):
//   dbias[h,n]   = sum_m dy[m,h,n]
//   dW[h,(k,d),n] = sum_m x[s+m*stride+k,h,d] dy[m,h,n] + pe[h,k,d] dbias[h,n]     one CTA per (tap k, head):
//                   a [d x d] tile accumulated over all windows with mma (A = x rows read transposed)
//   dpe[h,(k,d)] = sum_n dbias[h,n] W[h,(k,d),n]
//   dx[t]        = sum_{i < ks/stride} dy[t/stride - i] W_{t%stride + i*stride}^T   grouped by j = t % stride so
//                   that every group is a plain GEMM with the taps on the reduction dimension (overlap-add
//                   happens in registers, not through atomics)
// Pooling:
//   dx[t] = sum_i w[h, j + i*stride] dy[t/stride - i],  dw[h,k] = sum_m <x[s+m*stride+k,h,:], dy[m,h,:]> + <pe[h,k,:], dbias[h,:]>,
//   dpe[h,k,:] = w[h,k] dbias[h,:]
#include "attn_tile.cuh"
#include "cluster.cuh"
#include "dispatch.h"
#include "host_util.h"
#include "nsa_b200.h"
#include "pool_bwd_stream.h"

namespace nsa {

// dbias[c] = sum_m dy[m, c] over the M rows of H * D columns (fp32), in a fixed order (deterministic).  A cluster of eight CTAs
// takes 32 columns, an eighth of the rows each; a thread sums every 64th row of its CTA's eighth with eight 16-byte loads in
// flight, the CTA's 64 partial sums are added in its shared memory, and rank 0 reads and adds the eight CTAs' behind a cluster
// barrier: a CTA whose share of the rows is empty gets there long before the others have started.
constexpr int kColsumCluster = 8;
template <typename T>
__global__ void __cluster_dims__(kColsumCluster, 1, 1) __launch_bounds__(256)
colsum_kernel(const T* __restrict__ dy, float* __restrict__ dbias, int M, int C) {
  __shared__ float red[64][33];
  __shared__ float sum[32];
  const uint32_t rank = cluster_rank();
  const int c4 = threadIdx.x & 3, rl = threadIdx.x >> 2;
  const int col = blockIdx.y * 32 + c4 * 8;
  const int per = (M + kColsumCluster - 1) / kColsumCluster;
  const int m_end = min(M, (int)(rank + 1) * per);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  for (int m = rank * per + rl; m < m_end; m += 512) {
    uint4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      v[u] = m + 64 * u < m_end ? __ldg(reinterpret_cast<const uint4*>(dy + (size_t)(m + 64 * u) * C + col)) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t w[4] = {v[u].x, v[u].y, v[u].z, v[u].w};
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const float2 f = DT<T>::unpack(w[e]);
        acc[2 * e] += f.x;
        acc[2 * e + 1] += f.y;
      }
    }
  }
#pragma unroll
  for (int e = 0; e < 8; ++e) red[rl][c4 * 8 + e] = acc[e];
  __syncthreads();
  if (threadIdx.x < 32) {
    float s = 0.f;
#pragma unroll 8
    for (int r = 0; r < 64; ++r) s += red[r][threadIdx.x];
    sum[threadIdx.x] = s;
  }
  cluster_barrier();
  if (rank == 0 && threadIdx.x < 32) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < kColsumCluster; ++r) s += ld_peer(peer_addr(sum + threadIdx.x, r));
    dbias[blockIdx.y * 32 + threadIdx.x] = s;
  }
  cluster_barrier();  // no CTA leaves while its shared memory is being read
}

template <typename T>
static void launch_colsum(const void* dy, float* dbias, int M, int H, int D, cudaStream_t stream) {
  LaunchScope ls_("colsum", stream);
  colsum_kernel<T><<<dim3(kColsumCluster, H * D / 32), 256, 0, stream>>>(static_cast<const T*>(dy), dbias, M, H * D);
}

// dpe[h, r] = sum_n dbias[h, n] * W[h, r, n]: D / 8 lanes per row of W, 16 bytes each
template <typename T, int D>
__global__ void __launch_bounds__(256) linear_dpe_kernel(const float* __restrict__ dbias, const T* __restrict__ w, T* __restrict__ dpe, int H, int R) {
  constexpr int CH = D / 8;
  const long long row = ((long long)blockIdx.x * 256 + threadIdx.x) / CH;
  const int c = threadIdx.x % CH;
  const bool live = row < (long long)H * R;
  float acc = 0.f;
  if (live) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(w + (size_t)row * D + c * 8));
    const float4 b0 = __ldg(reinterpret_cast<const float4*>(dbias + (row / R) * D + c * 8)), b1 = __ldg(reinterpret_cast<const float4*>(dbias + (row / R) * D + c * 8) + 1);
    const float2 f0 = DT<T>::unpack(v.x), f1 = DT<T>::unpack(v.y), f2 = DT<T>::unpack(v.z), f3 = DT<T>::unpack(v.w);
    acc = b0.x * f0.x + b0.y * f0.y + b0.z * f1.x + b0.w * f1.y + b1.x * f2.x + b1.y * f2.y + b1.z * f3.x + b1.w * f3.y;
  }
#pragma unroll
  for (int off = CH / 2; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (live && c == 0) dpe[row] = DT<T>::from_float(acc);
}

struct LinBwdParams {
  const void* x;
  const void* w;
  const void* pe;
  const void* dy;   // [M, H, D] contiguous
  const float* dbias;
  void* dx;         // [N, H, D] contiguous
  void* dw;         // [H, ks*D, D] contiguous
  const int* cu;
  const int* ycu;
  long long x_sn, x_sh;
  int B, H, ks, stride;
};

// ---- dW: one CTA per (tap, head) ----
template <typename T, int D>
__global__ void __launch_bounds__(D * 2) linear_dw_kernel(LinBwdParams p) {
  constexpr int MT = 64;
  constexpr int TILE = MT * D * 2;
  constexpr int CH = D / 8;
  constexpr int NTHREADS = D * 2;  // D/16 warps, 16 output rows (d) each
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5, l = threadIdx.x & 31;
  const int k = blockIdx.x, h = blockIdx.y;
  const T* x = static_cast<const T*>(p.x);
  const T* dy = static_cast<const T*>(p.dy);

  // flattened list of (sequence, m-tile): walk sequences on the fly
  int b = 0, m0 = 0;
  auto advance_to_valid = [&]() {
    while (b < p.B && m0 >= __ldg(p.ycu + b + 1) - __ldg(p.ycu + b)) { ++b; m0 = 0; }
  };
  auto load_stage = [&](int bb, int mm0, int stg) {
    const uint32_t xa = smem_u32(smem + stg * 2 * TILE);
    const uint32_t ya = xa + TILE;
    const int s0 = __ldg(p.cu + bb), y0 = __ldg(p.ycu + bb), Mb = __ldg(p.ycu + bb + 1) - y0;
    for (int i = threadIdx.x; i < MT * CH; i += NTHREADS) {
      const int r = i / CH, c = i % CH;
      const bool ok = (mm0 + r) < Mb;
      const T* xs = x + (long long)(s0 + (ok ? (mm0 + r) * p.stride + k : 0)) * p.x_sn + (long long)h * p.x_sh + c * 8;
      cp_async16(swz_addr<MT>(xa, r, c), xs, ok);
      const T* ys = dy + ((size_t)(y0 + (ok ? mm0 + r : 0)) * p.H + h) * D + c * 8;
      cp_async16(swz_addr<MT>(ya, r, c), ys, ok);
    }
    cp_async_commit();
  };

  float acc[D / 8][4];
#pragma unroll
  for (int j = 0; j < D / 8; ++j) acc[j][0] = acc[j][1] = acc[j][2] = acc[j][3] = 0.f;

  advance_to_valid();
  int stg = 0;
  if (b < p.B) load_stage(b, m0, 0);
  while (b < p.B) {
    int nb = b, nm0 = m0 + MT;
    {  // next tile
      int sb = b, sm0 = m0;
      b = nb; m0 = nm0;
      advance_to_valid();
      nb = b; nm0 = m0;
      b = sb; m0 = sm0;
    }
    if (nb < p.B) {
      load_stage(nb, nm0, stg ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const uint32_t xa = smem_u32(smem + stg * 2 * TILE);
    // A[dd][m] = X[m][dd] read transposed; this warp's rows are dd = 16*warp .. 16*warp+15
#pragma unroll
    for (int kk = 0; kk < MT / 16; ++kk) {
      uint32_t a[1][4];
      ldmatrix_x4_trans(a[0], swz_addr<MT>(xa, kk * 16 + (l & 7) + ((l >> 4) << 3), 2 * warp + ((l >> 3) & 1)));
      mma_kn<T, D / 8, 1, MT>(acc, a, xa + TILE, kk * 16, 0);
    }
    __syncthreads();
    b = nb; m0 = nm0; stg ^= 1;
  }

  // epilogue: + pe[h,k,dd] * dbias[h,n], store dW[h, k*D + dd, n]
  const int r0 = l >> 2, c0 = (l & 3) * 2;
  float pe0 = 0.f, pe1 = 0.f;
  if (p.pe) {
    const T* pe = static_cast<const T*>(p.pe) + ((size_t)h * p.ks + k) * D + warp * 16;
    pe0 = DT<T>::to_float(pe[r0]);
    pe1 = DT<T>::to_float(pe[r0 + 8]);
  }
  T* dw = static_cast<T*>(p.dw) + ((size_t)h * p.ks + k) * D * D + (size_t)warp * 16 * D;
#pragma unroll
  for (int j = 0; j < D / 8; ++j) {
    const int n = j * 8 + c0;
    float b0 = 0.f, b1 = 0.f;
    if (p.pe) { b0 = p.dbias[h * D + n]; b1 = p.dbias[h * D + n + 1]; }
    *reinterpret_cast<uint32_t*>(dw + (size_t)r0 * D + n) = DT<T>::pack(acc[j][0] + pe0 * b0, acc[j][1] + pe0 * b1);
    *reinterpret_cast<uint32_t*>(dw + (size_t)(r0 + 8) * D + n) = DT<T>::pack(acc[j][2] + pe1 * b0, acc[j][3] + pe1 * b1);
  }
}

// ---- dx: CTA = (tile of 64 stride-chunks, phase j, sequence x head) ----
template <typename T, int D>
__global__ void __launch_bounds__(128) linear_dx_kernel(LinBwdParams p) {
  constexpr int CT = 64;
  constexpr int W_BYTES = D * D * 2;
  constexpr int CH = D / 8;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  const int warp = threadIdx.x >> 5;
  const int j = blockIdx.y;
  const int b = blockIdx.z / p.H, h = blockIdx.z % p.H;
  const int s0 = __ldg(p.cu + b), L = __ldg(p.cu + b + 1) - s0;
  const int y0 = __ldg(p.ycu + b), Mb = __ldg(p.ycu + b + 1) - y0;
  const int c_base = blockIdx.x * CT;
  if (c_base * p.stride + j >= L) return;
  const int a = p.ks / p.stride;
  const T* w = static_cast<const T*>(p.w) + (size_t)h * p.ks * D * D;
  const T* dy = static_cast<const T*>(p.dy);

  float acc[D / 8][4];
#pragma unroll
  for (int jj = 0; jj < D / 8; ++jj) acc[jj][0] = acc[jj][1] = acc[jj][2] = acc[jj][3] = 0.f;

  for (int i = 0; i < a; ++i) {
    // W_{j + i*stride}: [dd rows][nn contiguous] -> B operand with n = dd, k = nn
    const T* wk = w + (size_t)(j + i * p.stride) * D * D;
    const uint32_t wb = smem_u32(smem);
    __syncthreads();  // previous tap's reads are done
    for (int t = threadIdx.x; t < D * CH; t += 128) {
      const int r = t / CH, c = t % CH;
      cp_async16(swz_addr<D>(wb, r, c), wk + (size_t)r * D + c * 8, true);
    }
    cp_async_commit();
    // A rows: dy[c - i] for c = c_base + 16*warp + r
    uint32_t af[D / 16][4];
    load_a_frags_global<T, D / 16>(af, [&](int r) -> const T* {
      const int m = c_base + warp * 16 + r - i;
      return (m >= 0 && m < Mb) ? dy + ((size_t)(y0 + m) * p.H + h) * D : nullptr;
    });
    cp_async_wait<0>();
    __syncthreads();
    mma_nk<T, D / 8, D / 16, D>(acc, af, wb, 0, 0);
  }
  __syncthreads();
  T* stage = reinterpret_cast<T*>(smem + warp * (16 * (D + 8) * 2));
  T* dx = static_cast<T*>(p.dx);
  const float one[2] = {1.f, 1.f};
  store_rows_staged<T, D>(acc, one, stage, [&](int r) -> T* {
    const int t = (c_base + warp * 16 + r) * p.stride + j;
    return t < L ? dx + ((size_t)(s0 + t) * p.H + h) * D : nullptr;
  });
}

// ------------------------------------------------------------------------------------------------
// pooling backward
// ------------------------------------------------------------------------------------------------
struct PoolBwdParams {
  const void* x;
  const void* w;   // [H, ks] or nullptr
  const void* pe;  // [H, ks, D] or nullptr
  const void* dy;
  const float* dbias;
  void* dx;
  void* dw;   // [H, ks] or nullptr
  void* dpe;  // [H, ks, D] or nullptr
  const int* cu;
  const int* ycu;
  long long x_sn, x_sh;
  int N, B, H, D, ks, stride;
};

template <typename T>
__global__ void __launch_bounds__(256) pool_dx_kernel(PoolBwdParams p) {
  const int CH = p.D / 8;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)p.N * p.H * CH) return;
  const int c = idx % CH;
  const int h = (idx / CH) % p.H;
  const int n = idx / ((long long)CH * p.H);
  const int b = find_sequence(p.cu, p.B, n);
  const int t = n - __ldg(p.cu + b);
  const int y0 = __ldg(p.ycu + b), Mb = __ldg(p.ycu + b + 1) - y0;
  const int j = t % p.stride, cq = t / p.stride, a = p.ks / p.stride;
  const T* dy = static_cast<const T*>(p.dy);
  const T* w = p.w ? static_cast<const T*>(p.w) + h * p.ks : nullptr;
  float acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int i = 0; i < a; ++i) {
    const int m = cq - i;
    if (m < 0 || m >= Mb) continue;
    const float wv = w ? DT<T>::to_float(w[j + i * p.stride]) : 1.f / (float)p.ks;
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(dy + ((size_t)(y0 + m) * p.H + h) * p.D + c * 8));
    const uint32_t u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float2 f = DT<T>::unpack(u[e]);
      acc[2 * e] += wv * f.x;
      acc[2 * e + 1] += wv * f.y;
    }
  }
  uint4 out;
  out.x = DT<T>::pack(acc[0], acc[1]);
  out.y = DT<T>::pack(acc[2], acc[3]);
  out.z = DT<T>::pack(acc[4], acc[5]);
  out.w = DT<T>::pack(acc[6], acc[7]);
  *reinterpret_cast<uint4*>(static_cast<T*>(p.dx) + ((size_t)n * p.H + h) * p.D + c * 8) = out;
}

// dw[h,k] (one CTA per (h,k)) and dpe[h,k,:]
template <typename T>
__global__ void __launch_bounds__(256) pool_dw_kernel(PoolBwdParams p) {
  __shared__ float red[8];
  const int h = blockIdx.x, k = blockIdx.y;
  const int CH = p.D / 8;
  const T* x = static_cast<const T*>(p.x);
  const T* dy = static_cast<const T*>(p.dy);
  float acc = 0.f;
  if (p.dw) {
    for (int b = 0; b < p.B; ++b) {
      const int s0 = __ldg(p.cu + b), y0 = __ldg(p.ycu + b), Mb = __ldg(p.ycu + b + 1) - y0;
      for (int i = threadIdx.x; i < Mb * CH; i += blockDim.x) {
        const int m = i / CH, c = i % CH;
        const uint4 xv = __ldg(reinterpret_cast<const uint4*>(x + (long long)(s0 + m * p.stride + k) * p.x_sn + (long long)h * p.x_sh + c * 8));
        const uint4 yv = __ldg(reinterpret_cast<const uint4*>(dy + ((size_t)(y0 + m) * p.H + h) * p.D + c * 8));
        const uint32_t xu[4] = {xv.x, xv.y, xv.z, xv.w}, yu[4] = {yv.x, yv.y, yv.z, yv.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float2 a = DT<T>::unpack(xu[e]), bb = DT<T>::unpack(yu[e]);
          acc += a.x * bb.x + a.y * bb.y;
        }
      }
    }
    if (p.pe)
      for (int n = threadIdx.x; n < p.D; n += blockDim.x)
        acc += DT<T>::to_float(static_cast<const T*>(p.pe)[((size_t)h * p.ks + k) * p.D + n]) * p.dbias[h * p.D + n];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      float tot = 0.f;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += red[i];
      static_cast<T*>(p.dw)[h * p.ks + k] = DT<T>::from_float(tot);
    }
  }
  if (p.dpe) {
    const float wv = p.w ? DT<T>::to_float(static_cast<const T*>(p.w)[h * p.ks + k]) : 1.f / (float)p.ks;
    for (int n = threadIdx.x; n < p.D; n += blockDim.x)
      static_cast<T*>(p.dpe)[((size_t)h * p.ks + k) * p.D + n] = DT<T>::from_float(wv * p.dbias[h * p.D + n]);
  }
}

// dw[h,k] and dpe[h,k,:] from the streaming pass's partial rows, summed in their order (deterministic).  Every CTA sums its head's
// rows of dy's column sums for itself: 74 KB out of L2 for 144 rows, against a launch of its own (pool_bwd_stream_sums on how many).
template <typename T>
__global__ void __launch_bounds__(256) pool_dw_finish_kernel(PoolBwdParams p, const float* __restrict__ partial, PoolBwdRows rows) {
  constexpr int D = 128;
  __shared__ float red[8];
  __shared__ float part[8][D];
  __shared__ float dbias[D];
  const int h = blockIdx.x, k = blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (p.pe && rows.bias) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 6
    for (int r = warp; r < rows.ctas; r += 8)
#pragma unroll
      for (int e = 0; e < 4; ++e) s[e] += __ldg(rows.bias + ((size_t)r * p.H + h) * D + e * 32 + lane);
#pragma unroll
    for (int e = 0; e < 4; ++e) part[warp][e * 32 + lane] = s[e];
    __syncthreads();
    if (threadIdx.x < D) {
      float t = 0.f;
#pragma unroll
      for (int r = 0; r < 8; ++r) t += part[r][threadIdx.x];
      dbias[threadIdx.x] = t;
    }
  } else if (p.pe && threadIdx.x < D) {
    dbias[threadIdx.x] = p.dbias[h * D + threadIdx.x];
  }
  __syncthreads();
  if (p.dw) {
    float acc = 0.f;
    for (int s = threadIdx.x; s < rows.slots; s += blockDim.x) acc += partial[((size_t)s * p.H + h) * p.ks + k];
    if (p.pe && threadIdx.x < D)
      acc += DT<T>::to_float(static_cast<const T*>(p.pe)[((size_t)h * p.ks + k) * D + threadIdx.x]) * dbias[threadIdx.x];
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
      float tot = 0.f;
      for (int i = 0; i < (int)(blockDim.x >> 5); ++i) tot += red[i];
      static_cast<T*>(p.dw)[h * p.ks + k] = DT<T>::from_float(tot);
    }
  }
  if (p.dpe && threadIdx.x < D) {
    const float wv = p.w ? DT<T>::to_float(static_cast<const T*>(p.w)[h * p.ks + k]) : 1.f / (float)p.ks;
    static_cast<T*>(p.dpe)[((size_t)h * p.ks + k) * D + threadIdx.x] = DT<T>::from_float(wv * dbias[threadIdx.x]);
  }
}

template <typename T, int D>
static int run_linear_bwd(LinBwdParams p, void* dpe, float* dbias, int total_y, int max_len, cudaStream_t stream) {
  if (p.pe) {
    launch_colsum<T>(p.dy, dbias, total_y, p.H, D, stream);
    p.dbias = dbias;
    const long long lanes = (long long)p.H * p.ks * D * (D / 8);
    LaunchScope ls_("linear_dpe", stream);
    linear_dpe_kernel<T, D><<<(unsigned)((lanes + 255) / 256), 256, 0, stream>>>(dbias, static_cast<const T*>(p.w), static_cast<T*>(dpe), p.H, p.ks * D);
  }
  {
    const size_t smem = 1024 + 4 * 64 * D * 2;
    auto kern = linear_dw_kernel<T, D>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return cuda_rc(e);
    { LaunchScope ls_("linear_dw", stream); kern<<<dim3(p.ks, p.H), D * 2, smem, stream>>>(p); }
  }
  {
    const size_t smem = 1024 + D * D * 2;
    auto kern = linear_dx_kernel<T, D>;
    cudaError_t e = allow_smem(kern, smem);
    if (e != cudaSuccess) return cuda_rc(e);
    const int chunks = (max_len + p.stride - 1) / p.stride;
    { LaunchScope ls_("linear_dx", stream); kern<<<dim3((chunks + 63) / 64, p.stride, p.B * p.H), 128, smem, stream>>>(p); }
  }
  return cuda_rc(cudaGetLastError());
}

template <typename T, int D>
static int run_pool_bwd(PoolBwdParams p, float* dbias, float* partial, long long partial_floats, int total_y, int max_seqlen,
                        int dtype, cudaStream_t stream) {
  // long inputs: one streaming pass writes dx and the partial rows of dw (weighted pooling) and of dy's column sums (with pe)
  const long long need = pool_bwd_stream_partial_floats(p.H, D, p.N, p.B, max_seqlen, p.ks, p.stride);
  const bool room = partial && partial_floats >= need;
  const bool bias_rows = p.pe && room && need > 0 && pool_bwd_stream_sums(p.H, D, p.N, p.B, max_seqlen, p.stride);
  bool summed = false;
  if (total_y > 0 && need > 0 && (!p.dw || room)) {
    if (p.pe && !bias_rows) {
      launch_colsum<T>(p.dy, dbias, total_y, p.H, D, stream);
      p.dbias = dbias;
      summed = true;
    }
    PoolBwdRows rows;
    const int rc = pool_bwd_stream(p.x, p.dw ? p.w : nullptr, p.dy, p.dx, room ? partial : nullptr, bias_rows, &rows, p.cu, p.ycu, p.B,
                                   p.N, max_seqlen, p.H, D, p.ks, p.stride, p.x_sn, p.x_sh, dtype, stream);
    if (rc != kInvalid && rc != kUnsupported) {
      if (rc) return rc;
      if (p.dw || p.dpe) {
        LaunchScope ls_("pool_dw_finish", stream);
        pool_dw_finish_kernel<T><<<dim3(p.H, p.ks), 256, 0, stream>>>(p, partial, rows);
      }
      return cuda_rc(cudaGetLastError());
    }
  }
  if (p.pe && !summed) {
    launch_colsum<T>(p.dy, dbias, total_y, p.H, D, stream);
    p.dbias = dbias;
  }
  const long long total = (long long)p.N * p.H * (D / 8);
  { LaunchScope ls_("pool_dx", stream); pool_dx_kernel<T><<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(p); }
  if (p.dw || p.dpe) { LaunchScope ls_("pool_dw", stream); pool_dw_kernel<T><<<dim3(p.H, p.ks), 256, 0, stream>>>(p); }
  return cuda_rc(cudaGetLastError());
}

}  // namespace nsa

extern "C" int nsa_linear_compress_bwd(const void* x, const void* w, const void* pe, const void* dy, const int* cu_seqlens,
                                       const int* y_cu_seqlens, void* dx, void* dw, void* dpe, float* dbias_scratch,
                                       int total_len, int batch, int total_y, int max_seqlen, int num_heads, int head_dim,
                                       int kernel_size, int kernel_stride, long long x_stride_n, long long x_stride_h,
                                       int dtype, void* stream) {
  using namespace nsa;
  if (!x || !w || !cu_seqlens || !y_cu_seqlens || !dx || !dw || batch <= 0 || num_heads <= 0 || total_len <= 0) return kInvalid;
  if (pe && (!dpe || !dbias_scratch)) return kInvalid;
  if (kernel_size <= 0 || kernel_stride <= 0 || kernel_size % kernel_stride || max_seqlen <= 0) return kInvalid;
  if (total_y > 0 && !dy) return kInvalid;
  if ((x_stride_n | x_stride_h) % 8 || !aligned16(x) || !aligned16(w) || !aligned16(dx) || !aligned16(dw) || !aligned16(dy)) return kInvalid;
  LinBwdParams p;
  p.x = x; p.w = w; p.pe = pe; p.dy = dy; p.dbias = nullptr; p.dx = dx; p.dw = dw; p.cu = cu_seqlens; p.ycu = y_cu_seqlens;
  p.x_sn = x_stride_n; p.x_sh = x_stride_h; p.B = batch; p.H = num_heads; p.ks = kernel_size; p.stride = kernel_stride;
  return NSA_DISPATCH_T_D(dtype, head_dim, run_linear_bwd, p, dpe, dbias_scratch, total_y, max_seqlen,
                          static_cast<cudaStream_t>(stream));
}

extern "C" long long nsa_pool_compress_bwd_workspace_floats(int total_len, int batch, int max_seqlen, int num_heads, int head_dim,
                                                           int kernel_size, int kernel_stride) {
  if (total_len <= 0 || batch <= 0 || num_heads <= 0 || head_dim <= 0 || kernel_size <= 0 || kernel_stride <= 0) return 0;
  return (long long)num_heads * head_dim +
         nsa::pool_bwd_stream_partial_floats(num_heads, head_dim, total_len, batch, max_seqlen, kernel_size, kernel_stride);
}

extern "C" int nsa_pool_compress_bwd(const void* x, const void* w, const void* pe, const void* dy, const int* cu_seqlens,
                                     const int* y_cu_seqlens, void* dx, void* dw, void* dpe, float* workspace,
                                     long long workspace_floats, int total_len, int batch, int total_y, int max_seqlen,
                                     int num_heads, int head_dim, int kernel_size, int kernel_stride, long long x_stride_n,
                                     long long x_stride_h, int dtype, void* stream) {
  using namespace nsa;
  if (!x || !cu_seqlens || !y_cu_seqlens || !dx || batch <= 0 || num_heads <= 0 || total_len <= 0 || max_seqlen <= 0) return kInvalid;
  // workspace: [H, d] column sums of dy (needed iff pe), then the partial rows of the streaming pass (optional: without them weighted
  // pooling runs on the per-thread kernels)
  const long long dbias_floats = (long long)num_heads * head_dim;
  float* dbias_scratch = workspace && workspace_floats >= dbias_floats ? workspace : nullptr;
  float* partial = workspace && workspace_floats > dbias_floats ? workspace + dbias_floats : nullptr;
  const long long partial_floats = partial ? workspace_floats - dbias_floats : 0;
  if (pe && (!dpe || !dbias_scratch)) return kInvalid;
  if (w && !dw) return kInvalid;
  if (kernel_size <= 0 || kernel_stride <= 0 || kernel_size % kernel_stride) return kInvalid;
  if (total_y > 0 && !dy) return kInvalid;
  if ((x_stride_n | x_stride_h) % 8 || !aligned16(x) || !aligned16(dx) || !aligned16(dy)) return kInvalid;
  PoolBwdParams p;
  p.x = x; p.w = w; p.pe = pe; p.dy = dy; p.dbias = nullptr; p.dx = dx; p.dw = w ? dw : nullptr; p.dpe = pe ? dpe : nullptr;
  p.cu = cu_seqlens; p.ycu = y_cu_seqlens; p.x_sn = x_stride_n; p.x_sh = x_stride_h;
  p.N = total_len; p.B = batch; p.H = num_heads; p.D = head_dim; p.ks = kernel_size; p.stride = kernel_stride;
  return NSA_DISPATCH_T_D(dtype, head_dim, run_pool_bwd, p, dbias_scratch, partial, partial_floats, total_y, max_seqlen, dtype,
                          static_cast<cudaStream_t>(stream));
}
