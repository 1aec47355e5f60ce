// Cluster-per-pair decode kernels (decode_cluster.cu), called by the entry points in decode.cu where their rule says so.
#pragma once
#include <cuda_runtime.h>

namespace nsa {

struct DecodeOpArgs {
  const void *q, *k, *v;
  void* o;
  const int *seqlens, *cmp_seqlens, *topk_idx;
  int* topk_out_idx;
  int batch, cache_len, num_q_heads, num_kv_heads, head_dim, dtype;
  int topk, block_size, kernel_size, kernel_stride, init_blocks, local_blocks, max_blocks;
  const long long* strides;  // q_b q_h | k_b k_n k_h | v_b v_n v_h | o_b o_h | idx_h idx_b idx_k
  float sm_scale;
};

// Return kUnsupported when the split-KV kernel of decode.cu is the better (or the only) one for the shape.
int decode_cluster_dense(const DecodeOpArgs& a, cudaStream_t stream);
int decode_cluster_sparse(const DecodeOpArgs& a, cudaStream_t stream);
int decode_cluster_compressed(const DecodeOpArgs& a, cudaStream_t stream);

}  // namespace nsa
