// Pieces of the online softmax on one row of S per thread: 64 columns in the forward kernels, 128 in the KV-cache kernel.
#pragma once

#include "sm100_ptx.cuh"

namespace sntl {

// Row maximum with eight independent chains (a single 128-long dependent chain costs ~600 cycles) of three-input maxima: half
// the instructions of a two-input reduction.
struct RowMax {
    float m[8];
    template <int N> __device__ __forceinline__ void start(const uint32_t (&s)[N])
    {
#pragma unroll
        for (int c = 0; c < 8; ++c) m[c] = __uint_as_float(s[c]);
    }
    // step i of N / 2 - 4: two more columns
    template <int N> __device__ __forceinline__ void step(const uint32_t (&s)[N], int i)
    {
        m[i & 7] = ptx::fmax3(m[i & 7], __uint_as_float(s[8 + 2 * i]), __uint_as_float(s[9 + 2 * i]));
    }
    __device__ __forceinline__ float value() const
    {
        return ptx::fmax3(ptx::fmax3(m[0], m[1], m[2]), ptx::fmax3(m[3], m[4], m[5]), fmaxf(m[6], m[7]));
    }
};
template <int N> __device__ __forceinline__ float row_max(const uint32_t (&s)[N])
{
    RowMax r;
    r.start(s);
#pragma unroll
    for (int i = 0; i < N / 2 - 4; ++i) r.step(s, i);
    return r.value();
}

// Half a row: P = exp2(s * scale + shift) as packed bf16 in pk, and the sum of the fp32 values added to sum (two pairs of partial
// sums).
template <int kHalf>
__device__ __forceinline__ void exp_half(const uint32_t (&s)[128], float scale, float shift, uint32_t (&pk)[32], float2 (&sum)[2])
{
    const float2 sc = make_float2(scale, scale), sh = make_float2(shift, shift);
#pragma unroll
    for (int c = 0; c < 32; ++c) {
        const float2 x = ptx::ffma2(make_float2(__uint_as_float(s[kHalf * 64 + 2 * c]), __uint_as_float(s[kHalf * 64 + 2 * c + 1])), sc, sh);
        const float p0 = ptx::ex2(x.x), p1 = ptx::ex2(x.y);
        sum[c & 1] = ptx::fadd2(sum[c & 1], make_float2(p0, p1));
        pk[c] = ptx::pack_bf16(p0, p1);
    }
}

// The same for a row of 64 columns.  kMax: the row's maximum is taken on the way, in the issue slots that the special-function unit
// leaves free.
template <bool kMax>
__device__ __forceinline__ void exp_row(const uint32_t (&s)[64], float scale, float shift, uint32_t (&pk)[32], float2 (&sum)[2], RowMax& mx)
{
    const float2 sc = make_float2(scale, scale), sh = make_float2(shift, shift);
    if (kMax) mx.start(s);
#pragma unroll
    for (int c = 0; c < 32; ++c) {
        const float2 x = ptx::ffma2(make_float2(__uint_as_float(s[2 * c]), __uint_as_float(s[2 * c + 1])), sc, sh);
        const float p0 = ptx::ex2(x.x), p1 = ptx::ex2(x.y);
        if (kMax && c < 28) mx.step(s, c);
        sum[c & 1] = ptx::fadd2(sum[c & 1], make_float2(p0, p1));
        pk[c] = ptx::pack_bf16(p0, p1);
    }
}

}  // namespace sntl
