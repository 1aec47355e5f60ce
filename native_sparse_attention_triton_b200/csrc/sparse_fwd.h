// Parameter block shared by the two kernels of the selected-block forward.
#pragma once
#include <cuda_runtime.h>

#include "common.cuh"

namespace nsa {

struct SparseFwdParams {
  const void* q;
  void* o;
  float* lse;  // [N, Hq], base-2 log-sum-exp of the scaled logits
  const int* topk_idx;
  const int* cu_seqlens;
  long long q_sn, q_sh, o_sn, o_sh;
  long long t_sh, t_sn, t_sk;
  int N, B, Hq, Hkv, G, T, block_size;
  int first;   // in-sequence position of the first token sparse_fwd.cu takes; the union kernel takes those before it, and leaves
               // a NaN in the first lse of a (token, KV head) pair whose result is not finite or whose selection has a block twice,
               // which sparse_fwd.cu then redoes
  int span;    // tokens a warp of sparse_fwd.cu looks at per round (1 or 32)
  float scale2;
  Status st;
};

// The union kernel (sparse_fwd_union_tc.cu): the number of leading tokens of every sequence it is the better kernel for (a multiple
// of its CTA's tokens; 0: none), and its launch over the tokens before `limit`.  strides: q_n q_h k_n k_h v_n v_h o_n o_h.
// Its grid follows from the token count and the batch alone, so that nothing depends on a length known on the host.
int sparse_fwd_union_limit(int G, int T, int block_size, int head_dim);
int sparse_fwd_union(const void* q, const void* k, const void* v, const long long* strides, SparseFwdParams p, int limit, int head_dim,
                     int dtype, cudaStream_t stream);

}  // namespace nsa
