// Pooling compression backward as chunk streams (pool_bwd_stream.cu): dx and the per-tap partial sums of dw in one pass.
#pragma once
#include <cuda_runtime.h>

namespace nsa {

bool pool_bwd_stream_eligible(int num_heads, int head_dim, int total_len, int kernel_size, int kernel_stride);

// fp32 words of workspace the streaming pass needs for its partial rows (0 when it does not run)
long long pool_bwd_stream_partial_floats(int num_heads, int head_dim, int total_len, int batch, int max_seqlen,
                                         int kernel_size, int kernel_stride);

// Whether the pass can sum dy's columns as well; else they are better left to a pass of their own
bool pool_bwd_stream_sums(int num_heads, int head_dim, int total_len, int batch, int max_seqlen, int kernel_stride);

struct PoolBwdRows {
  int slots = 0;                // partial rows of dw, [slots][H][ks] at the workspace's start
  int ctas = 0;                 // partial rows of the column sums of dy, [ctas][H][128] at `bias`
  const float* bias = nullptr;
};

// dx [total_len, H, 128] contiguous <- dy, w;  when w != nullptr also partial rows of dw (fp32) <- x, dy, and with `bias` partial rows
// of the column sums of dy, all in `partial` (pool_bwd_stream_partial_floats), to be summed in their order by the caller.  *rows says
// how many there are.
int pool_bwd_stream(const void* x, const void* w, const void* dy, void* dx, float* partial, bool bias, PoolBwdRows* rows, const int* cu,
                    const int* ycu, int batch, int total_len, int max_seqlen, int num_heads, int head_dim, int kernel_size,
                    int kernel_stride, long long x_sn, long long x_sh, int dtype, cudaStream_t stream);

}  // namespace nsa
