// What the two dense backward passes with the keys as the M dimension have in common (dense_dkdv_tc.cu, dense_bwd_tc.cu): the table of
// row statistics, the probabilities and dS of a key's row columns, and the adding of a key's dV and dK rows.
#pragma once
#include "attn_bwd.h"
#include "tc5.cuh"

namespace nsa {

__device__ __forceinline__ void red_add_v4(float* dst, const uint32_t* v) {
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};\n" ::"l"(dst), "f"(__uint_as_float(v[0])), "f"(__uint_as_float(v[1])),
               "f"(__uint_as_float(v[2])), "f"(__uint_as_float(v[3])) : "memory");
}

// -lse (base 2) and delta * sm_scale of a tile's 128 rows, four a lane; rows past the last token have probability 0.
__device__ __forceinline__ void fill_row_table(float* nlse, float* dsc, const DkdvParams& p, int logG, int h, int qs, int tok0, int tok_end, int lane) {
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int r = lane + 32 * j;
    const int tok = tok0 + (r >> logG);
    float2 ldv = make_float2(INFINITY, 0.f);
    if (tok < tok_end) ldv = __ldg(p.ld + (long long)(qs + tok) * p.Hq + h * p.G + (r & (p.G - 1)));
    nlse[r] = -ldv.x;
    dsc[r] = ldv.y * p.sm_scale;
  }
}

// pf = exp2(s * scale2 + nlse) of C times 32 row columns, and their 16-bit pairs.  `full`: all columns are visible; else those in
// [clo, clo + span), counted from the first.
template <typename T, int C>
__device__ __forceinline__ void probabilities(const uint32_t (&s)[C][32], const float* nlse, float scale2, bool full, int clo, unsigned span, float* pf,
                                              uint32_t* pk) {
  const float4* nl4 = reinterpret_cast<const float4*>(nlse);
  auto x = [&](int j) { return __uint_as_float(s[j >> 5][j & 31]); };
  if (full) {
    const float2 sc2 = make_float2(scale2, scale2);
#pragma unroll
    for (int j4 = 0; j4 < 8 * C; ++j4) {
      const float4 nl = nl4[j4];
      const int j = 4 * j4;
      const float2 x01 = ffma2(make_float2(x(j), x(j + 1)), sc2, make_float2(nl.x, nl.y));
      const float2 x23 = ffma2(make_float2(x(j + 2), x(j + 3)), sc2, make_float2(nl.z, nl.w));
      pf[j + 0] = fast_exp2(x01.x);
      pf[j + 1] = fast_exp2(x01.y);
      pf[j + 2] = fast_exp2(x23.x);
      pf[j + 3] = fast_exp2(x23.y);
    }
  } else {
#pragma unroll
    for (int j4 = 0; j4 < 8 * C; ++j4) {
      const float4 nl = nl4[j4];
      const int j = 4 * j4;
      pf[j + 0] = masked_exp2((unsigned)(j + 0 - clo) < span, fmaf(x(j + 0), scale2, nl.x));
      pf[j + 1] = masked_exp2((unsigned)(j + 1 - clo) < span, fmaf(x(j + 1), scale2, nl.y));
      pf[j + 2] = masked_exp2((unsigned)(j + 2 - clo) < span, fmaf(x(j + 2), scale2, nl.z));
      pf[j + 3] = masked_exp2((unsigned)(j + 3 - clo) < span, fmaf(x(j + 3), scale2, nl.w));
    }
  }
#pragma unroll
  for (int j = 0; j < 16 * C; ++j) pk[j] = DT<T>::pack(pf[2 * j], pf[2 * j + 1]);
}

// 16-bit pairs of dS = P (dP - delta) scale of C times 32 row columns.
template <typename T, int C>
__device__ __forceinline__ void ds_columns(const uint32_t (&dp)[C][32], const float* dsc, float sm_scale, const float* pf, uint32_t* pk) {
  const float4* dl4 = reinterpret_cast<const float4*>(dsc);
  const float2 sm2 = make_float2(sm_scale, sm_scale);
  auto x = [&](int j) { return __uint_as_float(dp[j >> 5][j & 31]); };
#pragma unroll
  for (int j4 = 0; j4 < 8 * C; ++j4) {
    const float4 dl = dl4[j4];
    const int j = 4 * j4;
    const float2 t01 = ffma2(make_float2(x(j), x(j + 1)), sm2, make_float2(-dl.x, -dl.y));
    const float2 t23 = ffma2(make_float2(x(j + 2), x(j + 3)), sm2, make_float2(-dl.z, -dl.w));
    const float2 d01 = fmul2(make_float2(pf[j], pf[j + 1]), t01);
    const float2 d23 = fmul2(make_float2(pf[j + 2], pf[j + 3]), t23);
    pk[2 * j4] = DT<T>::pack(d01.x, d01.y);
    pk[2 * j4 + 1] = DT<T>::pack(d23.x, d23.y);
  }
}

// Thread (key, half) adds half of the d columns of its key's dV row, then dK row; `acc` = its lanes of the dV accumulator, dK 128
// columns on.  `row` = (key row * KV heads + KV head).
template <int D>
__device__ __forceinline__ void add_key_rows(const DkdvParams& p, uint32_t acc, size_t row, int half, bool key_ok) {
#pragma unroll
  for (int which = 0; which < 2; ++which) {
    float* dst = (which == 0 ? p.dv32 : p.dk32) + row * D + half * (D / 2);
#pragma unroll
    for (int c = 0; c < D / 64; ++c) {
      uint32_t r[32];
      tmem_ld32(acc + which * 128 + half * (D / 2) + c * 32, r);
      tmem_ld_wait();
      if (key_ok) {
#pragma unroll
        for (int j = 0; j < 32; j += 4) red_add_v4(dst + c * 32 + j, r + j);
      }
    }
  }
}

}  // namespace nsa
