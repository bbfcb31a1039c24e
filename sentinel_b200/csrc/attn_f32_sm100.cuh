// Exact-fp32 products on the tensor cores: building blocks of attn_f32_fwd_sm100.cu and attn_f32_bwd_sm100.cu.
//
// An fp32 value is the exact sum of three bf16 values, x = h + m + l (8 + 8 + 8 significant bits; each is the rounding of what the
// ones before leave).  A product of two matrices is taken as six bf16 products over these parts, hh, hm, mh, mm, hl, lh; what is
// left out is below 2^-26 of a term.  The tensor core adds in fp32 and cuts off below 2^-24 of the largest addend, towards zero, so
//   * the small parts are added first: an accumulator is large only in the last few steps (the hh part);
//   * every product starts from zero and is at most 128 terms long; longer sums are made of such products in registers, rounded
//     to nearest.
// Measured against 64-bit sums, normal operands: 64 terms 7.9e-8 relative (a chain of fp32 FMAs 1.5e-7, two chains 1.1e-7), 128
// terms 1.2e-7 (2.1e-7, 1.5e-7).
//
// The parts of a value that is not finite, or so small that l underflows, do not add up to it, and weight 0 times them is not 0;
// large values could overflow where the FMA kernels do not.  A block that meets such a value (Check) leaves its results alone and
// marks itself, and the FMA kernels, launched behind with the marks, compute the marked blocks.
#pragma once

#include "common.cuh"
#include "sm100_ptx.cuh"

namespace sntl {
namespace f32tc {

constexpr int kDim = 64;                 // features of a tile (head_dim filled up with zeros)
constexpr int kRowBytes = kDim * 2;      // a row of one part: 128 bytes, 128-byte swizzle
constexpr int kOwnRows = 128;            // rows of a block: the TMEM lanes
constexpr int kFetchRows = 64;           // rows that are staged at a time
// warps 0-7 sums, 8-13 stage, 14 issues the products, 15 idle; the first two warpgroups take registers from the others
constexpr int kSumThreads = 256, kStageThreads = 192, kThreads = 512, kIssueWarp = 14, kSumRegs = 160, kOtherRegs = 96;
static_assert(kSumThreads * kSumRegs + (kThreads - kSumThreads) * kOtherRegs <= kThreads * 128, "what the block is launched with");
constexpr float kLargest = 1073741824.0f;                 // 2^30: products of two such, summed, stay far from overflow
constexpr float kLargestWeight = 1.152921504606847e18f;   // 2^60, for what the kernels compute themselves

// rows [.., S) of a slab of D features with element strides ss, sd
struct Rows {
    const float* base;
    long long ss, sd;
    int S, D;
    bool vec;       // sd == 1, D % 4 == 0 and every row on a 16-byte boundary
};

// What a thread has seen of the values that it staged.
struct Check {
    uint32_t lost = 0;       // low halves of the last remainders: not zero where the parts do not add up (or the value is inf or NaN)
    float largest = 0.f;
    __device__ __forceinline__ bool odd() const { return (lost & 0xffffu) != 0 || !(largest < kLargest); }
};

__device__ __forceinline__ float2 unpack2(uint32_t w) { return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u)); }

// two values -> their parts, packed
__device__ __forceinline__ void split2(float2 x, uint32_t& h, uint32_t& m, uint32_t& l, uint32_t& lost)
{
    const float2 minus = make_float2(-1.f, -1.f);
    h = ptx::pack_bf16(x.x, x.y);
    const float2 r = ffma2(unpack2(h), minus, x);
    m = ptx::pack_bf16(r.x, r.y);
    const float2 t = ffma2(unpack2(m), minus, r);
    const uint32_t a = __float_as_uint(t.x), b = __float_as_uint(t.y);
    l = __byte_perm(a, b, 0x7632);       // exact: at most eight bits are left
    lost |= a | b;
}

// eight features of a row, from feature d
__device__ __forceinline__ void load8(float (&x)[8], const Rows& m, int row, int d)
{
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = 0.f;
    if (row >= m.S || d >= m.D) return;
    const float* p = m.base + row * m.ss + d * m.sd;
    if (m.vec) {
        const float4 a = __ldg(reinterpret_cast<const float4*>(p));
        x[0] = a.x; x[1] = a.y; x[2] = a.z; x[3] = a.w;
        if (d + 4 < m.D) {
            const float4 b = __ldg(reinterpret_cast<const float4*>(p + 4));
            x[4] = b.x; x[5] = b.y; x[6] = b.z; x[7] = b.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (d + i < m.D) x[i] = __ldg(p + i * m.sd);
    }
}

// kFetchRows rows on their way from global memory to shared memory, in the registers of kStageThreads threads numbered t: loaded ahead
// of the wait for the place that they go to.  A unit is eight features of a row, numbered along the contiguous direction of the
// source so that a warp's loads coalesce.
struct Fetch {
    static constexpr int kUnits = kFetchRows * 8, kPer = (kUnits + kStageThreads - 1) / kStageThreads;
    float x[kPer][8];

    static __device__ __forceinline__ bool unit(int k, int t, bool rows_contiguous, int& r, int& c)
    {
        const int u = k * kStageThreads + t;
        r = rows_contiguous ? u % kFetchRows : u >> 3;
        c = rows_contiguous ? u / kFetchRows : u & 7;
        return kUnits % kStageThreads == 0 || k + 1 < kPer || u < kUnits;
    }
    __device__ __forceinline__ void load(const Rows& m, int row0, int t)
    {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            int r, c;
            if (unit(k, t, m.sd != 1, r, c)) load8(x[k], m, row0 + r, c * 8);
        }
    }
    // -> the three parts, `pitch` bytes apart, each kFetchRows x 128 bytes.  (The 16-byte stores of eight lanes fall into different
    // banks in either order of the units: rows are swizzled.)
    __device__ __forceinline__ void put(uint8_t* dst, int pitch, bool rows_contiguous, int t, Check& check) const
    {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            int r, c;
            if (!unit(k, t, rows_contiguous, r, c)) continue;
            uint4 h, m, l;
            split2(make_float2(x[k][0], x[k][1]), h.x, m.x, l.x, check.lost);
            split2(make_float2(x[k][2], x[k][3]), h.y, m.y, l.y, check.lost);
            split2(make_float2(x[k][4], x[k][5]), h.z, m.z, l.z, check.lost);
            split2(make_float2(x[k][6], x[k][7]), h.w, m.w, l.w, check.lost);
            uint8_t* at = dst + r * kRowBytes + ((c ^ (r & 7)) << 4);
            *reinterpret_cast<uint4*>(at) = h;
            *reinterpret_cast<uint4*>(at + pitch) = m;
            *reinterpret_cast<uint4*>(at + 2 * pitch) = l;
#pragma unroll
            for (int i = 0; i < 8; i += 2) check.largest = ptx::fmax3(check.largest, fabsf(x[k][i]), fabsf(x[k][i + 1]));
        }
    }
    // sums of products with the same units of `other`, to part[row * 9 + unit]
    __device__ __forceinline__ void dots(bool rows_contiguous, int t, const Fetch& other, float* part) const
    {
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            int r, c;
            if (!unit(k, t, rows_contiguous, r, c)) continue;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) sum = fmaf(x[k][i], other.x[k][i], sum);
            part[r * 9 + c] = sum;
        }
    }
};

// exp(x) = 2^t (1 + x - t ln 2) with t = x / ln 2 rounded: t ln 2 in two parts, the correction is below |x| 2^-24.  ex2.approx is low by
// 5e-8 on average for arguments below -1 (2e-8 between -1/2 and 0), which the correction gives back: 4.0e-8 relative (rms), as
// expf; 6.4e-8 without.  kHidden gives 0.
constexpr float kHidden = -1e30f;
__device__ __forceinline__ float2 exp_pair(float2 x)
{
    const float2 t = ptx::fmul2(x, make_float2(1.44269504f, 1.44269504f));
    float2 e = ffma2(t, make_float2(-0.693147182f, -0.693147182f), x);
    e = ptx::fadd2(ffma2(t, make_float2(1.90465421e-9f, 1.90465421e-9f), e), make_float2(5e-8f, 5e-8f));
    const float2 p = make_float2(ptx::ex2(t.x), ptx::ex2(t.y));
    return ffma2(p, e, p);
}

// bit i: whether i < n
__device__ __forceinline__ uint32_t bits_below(int n) { return n <= 0 ? 0u : n >= 32 ? 0xffffffffu : (1u << n) - 1u; }

// Which of the 32 keys from key0 on the query at position pos sees (keys below `end` exist for it)
__device__ __forceinline__ uint32_t keys_seen(const AttnShape& s, int pos, int end, int key0)
{
    uint32_t seen = bits_below(end - key0);
    if (s.window > 0) seen &= ~bits_below(pos - s.window + 1 - key0) | bits_below(s.global_tokens - key0);
    return seen;
}
// Which of the 32 queries from position pos0 on see the key
__device__ __forceinline__ uint32_t queries_seeing(const AttnShape& s, int key, int pos0)
{
    uint32_t seen = key < s.Skv ? 0xffffffffu : 0u;
    if (s.causal) seen &= ~bits_below(key - pos0);
    if (s.window > 0 && key >= s.global_tokens) seen &= bits_below(key + s.window - pos0);
    return seen;
}

// The six products in the order of their size, smallest first: parts (a, b).  kSwap: with the parts of a and b exchanged, so that a
// transposed product adds the same terms in the same order.
template <bool kSwap = false, typename F> __device__ __forceinline__ void six(F&& f)
{
    f(kSwap ? 2 : 0, kSwap ? 0 : 2, 0u);
    f(kSwap ? 0 : 2, kSwap ? 2 : 0, 1u);
    f(1, 1, 1u);
    f(kSwap ? 1 : 0, kSwap ? 0 : 1, 1u);
    f(kSwap ? 0 : 1, kSwap ? 1 : 0, 1u);
    f(0, 0, 1u);
}

// kN columns of the parts of kN pairs of values, part p at taddr + p * kPitch; what is left in x is the last part.
template <int kN, int kPitch> __device__ __forceinline__ void put_parts(uint32_t taddr, float2 (&x)[kN])
{
    const float2 minus = make_float2(-1.f, -1.f);
    uint32_t w[kN];
#pragma unroll
    for (int p = 0; p < 3; ++p) {
#pragma unroll
        for (int i = 0; i < kN; ++i) {
            if (p < 2) {
                w[i] = ptx::pack_bf16(x[i].x, x[i].y);
                x[i] = ffma2(unpack2(w[i]), minus, x[i]);
            } else {
                w[i] = __byte_perm(__float_as_uint(x[i].x), __float_as_uint(x[i].y), 0x7632);
            }
        }
        if constexpr (kN == 32) ptx::tmem_st32(taddr + p * kPitch, w);
        else ptx::tmem_st16(taddr + p * kPitch, w);
    }
}

// Whether the call has the work that the blocks' set-up and their chains of tiles are worth: visible pairs x features.  Below, the FMA
// kernels' small tiles and their split of the keys over clusters are faster (B4 H8 S128 D64 forward 12.1 us against 13.3, S256 D32
// 16.7 against 15.2).
inline bool enough_work(const AttnShape& s)
{
    const double per_row = s.causal ? s.Skv - 0.5 * s.Sq : s.Skv;
    return s.Sq >= 64 && (double)s.B * s.Hq * s.Sq * per_row * s.D >= 32.0 * 128 * 128 * 64;
}

// Scales that keep the scores of values below kLargest, and those that stand for hidden pairs, apart from each other and in range
inline bool scale_supported(float scale) { return scale >= 1.0f / 65536 && scale <= 65536.0f; }

// 32 features of a row times f, from feature d0 on, to global memory
__device__ __forceinline__ void store_row(float* base, const Rows& m, int row, int d0, const float2 (&y)[16], float f)
{
    if (row >= m.S) return;
    float* p = base + row * m.ss + d0 * m.sd;
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = (i & 1 ? y[i / 2].y : y[i / 2].x) * f;
    if (m.vec) {
#pragma unroll
        for (int i = 0; i < 32; i += 4)
            if (d0 + i < m.D) *reinterpret_cast<float4*>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (d0 + i < m.D) p[i * m.sd] = x[i];
    }
}

}  // namespace f32tc
}  // namespace sntl
