// The per-query terms of the tensor-core backward, as the main kernel wants them, from LSE and delta of one padded query row.
#pragma once

#include <cuda_bf16.h>
#include <stdint.h>

namespace sntl {

// Whether the per-query terms (LSE, delta) are folded into the S^T and dP^T products as one extra contraction step (see
// kAugBytes in attn_bwd_tc_kernel).  That trades shared-memory loads and arithmetic in the compute warps for 2 x 65 tensor-pipe
// cycles per step on the two chains of products: a clear gain at head_dim 64, where the compute warps set the pace
// (-11 % kernel time), a loss at 128, where the chains do (+3 %).
__host__ __device__ constexpr bool bwd_folds_row_terms(int D) { return D == 64; }

// Where they go: [B][Hq][Sq_pad] records of 16 bytes (head_dim 64) or fp32 columns (128); see tc_backward_workspace_bytes.
struct RowTerms {
    void *lse, *delta;
    float inv_scale;
};
__host__ inline RowTerms row_terms_of(void* base, long long rows_padded, int D, float scale)
{
    if (bwd_folds_row_terms(D)) return RowTerms{(uint4*)base + rows_padded, base, 1.0f / scale};
    return RowTerms{(float*)base + rows_padded, base, 1.0f / scale};   // the plain-column form takes the head of the same region
}

// r: padded row; live: the row exists; lse: natural log, -inf for a row without visible keys; delta = rowsum(dO o O).
// Rows that contribute nothing get a term that makes P = 0.
template <int D>
__device__ __forceinline__ void store_row_terms(const RowTerms& t, long long r, bool live, float lse, float delta)
{
    if constexpr (bwd_folds_row_terms(D)) {
        // value -> three bf16 (hi, mid, lo) whose sum is the fp32 value exactly (3 x 8 significant bits), as the first
        // three slots of a record
        auto split = [](float x) {
            const __nv_bfloat16 hi = __float2bfloat16_rn(x);
            const float r1 = x - __bfloat162float(hi);
            const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
            const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
            return make_uint4((uint32_t)__bfloat16_as_ushort(hi) | ((uint32_t)__bfloat16_as_ushort(mid) << 16),
                              (uint32_t)__bfloat16_as_ushort(lo), 0u, 0u);
        };
        constexpr float kMasked = -1.0e30f;   // times scale*log2(e) still far below the exponent range: P = 0, and finite
        static_cast<uint4*>(t.lse)[r] = split(!live || lse == -INFINITY ? kMasked : -lse * t.inv_scale);
        static_cast<uint4*>(t.delta)[r] = live ? split(-delta) : make_uint4(0u, 0u, 0u, 0u);
    } else {
        static_cast<float*>(t.lse)[r] = !live || lse == -INFINITY ? -INFINITY : -lse * 1.4426950408889634f;
        static_cast<float*>(t.delta)[r] = live ? -delta : 0.0f;
    }
}

}  // namespace sntl
