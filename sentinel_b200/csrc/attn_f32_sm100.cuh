// Exact-fp32 products on the tensor cores: building blocks of attn_f32_fwd_sm100.cu and attn_f32_bwd_sm100.cu.
//
// An fp32 value is the exact sum of three bf16 values, x = h + m + l (8 + 8 + 8 significant bits; each is the rounding of what the
// ones before leave).  A product of two matrices is taken as six bf16 products over these parts, hh, hm, mh, mm, hl, lh; what is
// left out is at most 2^-24 of a term, 2^-27 rms (operands between 1 and 1.03: 2^-26).  The tensor core adds in fp32 and cuts off below 2^-24 of the largest addend, towards zero, so
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

#include "block_queue.cuh"
#include "common.cuh"
#include "sm100_ptx.cuh"

namespace sntl {
namespace f32tc {

constexpr int kDim = 64;                 // features of a tile (head_dim filled up with zeros)
constexpr int kRowBytes = kDim * 2;      // a row of one part: 128 bytes, 128-byte swizzle
constexpr int kOwnRows = 128;            // rows of a block: the TMEM lanes
constexpr int kFetchRows = 64;           // rows that are staged at a time
// warps 0-7 sums, 8-13 stage, 14 issues the products, 15 idle; the first two warpgroups take registers from the others
constexpr int kSumThreads = 256, kStageThreads = 192, kThreads = 512, kIssueWarp = 14;
// (128 registers a thread at launch.  A spill in the staging loop is read from L2: next to the streamed rows local memory does not stay in
// L1.  The split between the groups is the one that spills least: 28 bytes in the forward, 96 and 100 in the backward; more on either side
// of it.)
__host__ __device__ constexpr int other_regs(int sum_regs) { return (kThreads * 128 - kSumThreads * sum_regs) / (kThreads - kSumThreads) / 8 * 8; }
constexpr float kLargest = 1073741824.0f;                 // 2^30: products of two such, summed, stay far from overflow
// The kernels compute weights and dS times kUp: parts add up to a value from 2^-110 on (below, the last ones have no room in bf16), and so
// they do for all of these from 2^-134 on; the results are divided again, which costs no bits.  (Weights below 2^-126, which fp32
// holds with fewer bits anyway, are 0: ex2.)
constexpr float kUp = 16777216.0f, kDown = 1.0f / kUp;    // 2^24
constexpr float kLargestWeight = 7.555786372591432e22f;   // 2^76 = kUp 2^52, for these
constexpr float kLargestDelta = 1.152921504606847e18f;    // 2^60

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

// Rows that are to be staged: the address of the first, and how many there are from it on (the others read as zero).
struct Source {
    const float* at;
    int left;
};

// A staging thread's share of a half tile: units of eight features of a row, numbered along the contiguous direction of the tensors so
// that a warp's loads coalesce.  (kStageThreads is a multiple of the 8 units of a row and of kFetchRows: from one unit of a thread to
// its next either the row or the features change, by a constant.)
// kVec: all rows lie on 16-byte boundaries with features side by side, head_dim a multiple of 4.
template <bool kVec> struct Share {
    static constexpr int kUnits = kFetchRows * 8, kPer = (kUnits + kStageThreads - 1) / kStageThreads;
    static_assert(kStageThreads % kFetchRows == 0 && kStageThreads % 64 == 0, "");
    int t, row0, chunk0, off0, step, sd, D;
    bool rows_contiguous;        // (feature-major matrices)

    __device__ __forceinline__ Share(int t_, int ss, int sd_, int D_) : t(t_), sd(sd_), D(D_), rows_contiguous(sd_ != 1)
    {
        row0 = matrix() ? t % kFetchRows : t >> 3;
        chunk0 = matrix() ? t / kFetchRows : t & 7;
        off0 = row0 * ss + chunk0 * 8 * sd;
        step = kStageThreads / 8 * (matrix() ? sd : ss);
    }
    __device__ __forceinline__ bool matrix() const { return !kVec && rows_contiguous; }
    __device__ __forceinline__ bool valid(int k) const { return k + 1 < kPer || t < kUnits - (kPer - 1) * kStageThreads; }
    __device__ __forceinline__ int row(int k) const { return matrix() ? row0 : row0 + k * (kStageThreads / 8); }
    __device__ __forceinline__ int chunk(int k) const { return matrix() ? chunk0 + k * (kStageThreads / kFetchRows) : chunk0; }
    // where the unit goes inside a part: rows of 128 bytes, 128-byte swizzle (the rows of a thread's units differ by multiples of 8)
    __device__ __forceinline__ int place(int k) const
    {
        return matrix() ? row0 * kRowBytes + ((chunk(k) ^ (row0 & 7)) << 4)
                        : row0 * kRowBytes + ((chunk0 ^ (row0 & 7)) << 4) + k * (kStageThreads / 8) * kRowBytes;
    }
};

// Loads of rows that pass once: they go first when L1 (28 KB beside this shared memory) is full, not what the other warps have there.
// x stays what it is where `in` is false.  (Predicated, into place: behind a branch the compiler copies the values where the paths
// meet, and the copy waits for the load; the staging warps then spent two thirds of their time on the latency of L2.)
__device__ __forceinline__ void load_once4(float* x, const float* p, bool in)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %5, 0;\n\t@p ld.global.nc.L1::evict_first.v4.f32 {%0, %1, %2, %3}, [%4];\n\t}"
                 : "+f"(x[0]), "+f"(x[1]), "+f"(x[2]), "+f"(x[3]) : "l"(p), "r"((uint32_t)in));
}
__device__ __forceinline__ void load_once(float& x, const float* p, bool in)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p ld.global.nc.L1::evict_first.f32 %0, [%1];\n\t}" : "+f"(x) : "l"(p), "r"((uint32_t)in));
}

// Half a tile on its way from global memory to shared memory, in registers: loaded ahead of the wait for the place that it goes to.
template <bool kVec> struct Fetch {
    using Share = f32tc::Share<kVec>;
    float x[Share::kPer][8];

    __device__ __forceinline__ void load(const Source& m, const Share& w)
    {
#pragma unroll
        for (int k = 0; k < Share::kPer; ++k) {
#pragma unroll
            for (int i = 0; i < 8; ++i) x[k][i] = 0.f;
            int sd = w.sd;
            if (!kVec) asm volatile("" : "+r"(sd));      // (or its multiples, 64 bits each, would be kept in registers)
            const int d = w.chunk(k) * 8;
            const bool in = w.valid(k) && w.row(k) < m.left;
            const float* p = m.at + w.off0 + k * w.step;
            if constexpr (kVec) {
                load_once4(x[k], p, in && d < w.D);
                load_once4(x[k] + 4, p + 4, in && d + 4 < w.D);
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i, p += sd) load_once(x[k][i], p, in && d + i < w.D);
            }
        }
    }
    // -> the three parts, `pitch` bytes apart, each kFetchRows x 128 bytes.  (The 16-byte stores of eight lanes fall into different
    // banks in either order of the units: rows are swizzled.)
    __device__ __forceinline__ void put(uint8_t* dst, int pitch, const Share& w, Check& check) const
    {
#pragma unroll
        for (int k = 0; k < Share::kPer; ++k) {
            if (!w.valid(k)) continue;
            uint4 h, m, l;
            split2(make_float2(x[k][0], x[k][1]), h.x, m.x, l.x, check.lost);
            split2(make_float2(x[k][2], x[k][3]), h.y, m.y, l.y, check.lost);
            split2(make_float2(x[k][4], x[k][5]), h.z, m.z, l.z, check.lost);
            split2(make_float2(x[k][6], x[k][7]), h.w, m.w, l.w, check.lost);
            uint8_t* at = dst + w.place(k);
            *reinterpret_cast<uint4*>(at) = h;
            *reinterpret_cast<uint4*>(at + pitch) = m;
            *reinterpret_cast<uint4*>(at + 2 * pitch) = l;
#pragma unroll
            for (int i = 0; i < 8; i += 2) check.largest = ptx::fmax3(check.largest, fabsf(x[k][i]), fabsf(x[k][i + 1]));
        }
    }
    // sums of products with the same units of `other`, to part[row * 9 + unit]
    __device__ __forceinline__ void dots(const Share& w, const Fetch& other, float* part) const
    {
#pragma unroll
        for (int k = 0; k < Share::kPer; ++k) {
            if (!w.valid(k)) continue;
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) sum = fmaf(x[k][i], other.x[k][i], sum);
            part[w.row(k) * 9 + w.chunk(k)] = sum;
        }
    }
};

// exp(x) = 2^t (1 + x - t ln 2) with t = x / ln 2 rounded: t ln 2 in two parts, the correction is below |x| 2^-24.  ex2.approx is low by
// 5e-8 on average for arguments below -1 (2e-8 between -1/2 and 0), which the correction gives back: 4.0e-8 relative (rms), as
// expf; 6.4e-8 without.  kHidden gives 0.
constexpr float kHidden = -1e30f;
template <bool kTimesUp = false> __device__ __forceinline__ float2 exp_pair(float2 x)
{
    const float2 t = ptx::fmul2(x, make_float2(1.44269504f, 1.44269504f));
    float2 e = ffma2(t, make_float2(-0.693147182f, -0.693147182f), x);
    e = ptx::fadd2(ffma2(t, make_float2(1.90465421e-9f, 1.90465421e-9f), e), make_float2(5e-8f, 5e-8f));
    float2 p = make_float2(ptx::ex2(t.x), ptx::ex2(t.y));
    if (kTimesUp) p = ptx::fmul2(p, make_float2(kUp, kUp));
    return ffma2(p, e, p);
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

// kN columns of each of the parts of kN pairs of values, part p at taddr + p * kPitch; what is left in x is the last part.
template <int kN, int kPitch> __device__ __forceinline__ void put_parts(uint32_t taddr, float2 (&x)[kN])
{
    constexpr int kC = kN == 16 ? 16 : 8;      // (as registers allow)
    const float2 minus = make_float2(-1.f, -1.f);
#pragma unroll
    for (int c = 0; c < kN; c += kC) {
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            uint32_t w[kC];
#pragma unroll
            for (int i = 0; i < kC; ++i) {
                float2& y = x[c + i];
                if (p < 2) {
                    w[i] = ptx::pack_bf16(y.x, y.y);
                    y = ffma2(unpack2(w[i]), minus, y);
                } else {
                    w[i] = __byte_perm(__float_as_uint(y.x), __float_as_uint(y.y), 0x7632);
                }
            }
            if constexpr (kC == 8) ptx::tmem_st8(taddr + p * kPitch + c, w);
            else ptx::tmem_st16(taddr + p * kPitch + c, w);
        }
    }
}

using Queue = BlockQueue<kIssueWarp + 1>;      // every warp but the idle one
// Which block (u + 1) of the last four was found odd
struct OddBlocks {
    volatile int number[4];
    __device__ __forceinline__ void set(int u) { number[u & 3] = u + 1; }
    __device__ __forceinline__ bool get(int u) const { return number[u & 3] == u + 1; }
};

// A lower bound for what is worth the blocks' set-up: pairs x features, in tiles of 128 x 128 x 64.  Measured, FMA -> here: forward B4 H8 S128
// D64 (16 tiles) 12.1 -> 13.3 us, B2 H2 S512 D64 (32) 22.5 -> 21.5, B4 H8 S256 D32 (32) 16.7 -> 15.1; backward B8 H12 S64 D64 (12) 26 ->
// 29, B4 H8 S128 D64 (16) 25 -> 20, B1 H8 S256 D64 (16) 36 -> 28.  Above it the estimates of attn_f32_route.cu decide.
constexpr int kForwardTiles = 32, kBackwardTiles = 16;
inline bool enough_work(const AttnShape& s, int tiles)
{
    const double per_row = s.causal ? s.Skv - 0.5 * s.Sq : s.Skv;
    return s.Sq >= 64 && (double)s.B * s.Hq * s.Sq * per_row * s.D >= tiles * (128.0 * 128 * 64);
}

// Scales that keep the scores of values below kLargest, and those that stand for hidden pairs, apart from each other and in range
inline bool scale_supported(float scale) { return scale >= 1.0f / 65536 && scale <= 65536.0f; }

// One pair of strides for all tensors, and offsets inside a tile that fit 32 bits
inline bool strides_supported(const SimtArgs& a)
{
    return a.vq.ss == a.vkv.ss && a.vq.sd == a.vkv.sd && a.vq.ss <= (1 << 24) && a.vq.sd <= (1 << 24);
}

// 32 features of row `row` times f, from feature d0 on, to a slab of S rows with strides ss, sd (vec: stores of four features)
__device__ __forceinline__ void store_row(float* base, long long ss, long long sd, int S, int D, bool vec, int row, int d0, const float2 (&y)[16], float f)
{
    if (row >= S) return;
    float* p = base + row * ss + d0 * sd;
    float x[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) x[i] = (i & 1 ? y[i / 2].y : y[i / 2].x) * f;
    if (vec) {
#pragma unroll
        for (int i = 0; i < 32; i += 4)
            if (d0 + i < D) *reinterpret_cast<float4*>(p + i) = make_float4(x[i], x[i + 1], x[i + 2], x[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
            if (d0 + i < D) p[i * sd] = x[i];
    }
}

}  // namespace f32tc
}  // namespace sntl
