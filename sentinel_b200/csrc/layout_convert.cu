// HBM-bound staging kernels: the reference's fp32 feature-major matrices <-> bf16 token-major tensors,
// plain dtype casts, LSE re-indexing, and the log-sum-exp merge of two partial attention results.
//
// Feature-major ("SENTINEL") addressing follows sentinel/NeuralNet/Cuda/CudaFlashAttention.cu:129-131:
// element (b,h,s,d) lives at (h*D + d)*stride_columns + column_start + b*S + s.
#include "common.cuh"
#include "row_terms.cuh"

namespace sntl {
namespace {

// 32x32 transposing tile: reads are contiguous along tokens (source rows), writes along d (destination rows).
__global__ void sentinel_to_bhsd_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int H, int S, int D,
                                        int stride_columns, int column_start)
{
    __shared__ float tile[32][33];
    const int bh = blockIdx.z, b = bh / H, h = bh % H;
    const int s0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        const int d = d0 + r, s = s0 + tx;
        tile[r][tx] = (d < D && s < S) ? src[(long long)(h * D + d) * stride_columns + column_start + (long long)b * S + s] : 0.0f;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int s = s0 + r, d = d0 + tx;
        if (s < S && d < D) dst[((long long)bh * S + s) * D + d] = __float2bfloat16_rn(tile[tx][r]);
    }
}

__global__ void bhsd_to_sentinel_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, int H, int S, int D,
                                        int stride_columns, int column_start)
{
    __shared__ float tile[32][33];
    const int bh = blockIdx.z, b = bh / H, h = bh % H;
    const int s0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int r = ty; r < 32; r += 8) {
        const int s = s0 + r, d = d0 + tx;
        tile[r][tx] = (s < S && d < D) ? __bfloat162float(src[((long long)bh * S + s) * D + d]) : 0.0f;
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int d = d0 + r, s = s0 + tx;
        if (d < D && s < S) dst[(long long)(h * D + d) * stride_columns + column_start + (long long)b * S + s] = tile[tx][r];
    }
}

// Rotary position embedding fused into the two transposes above: what the reference does as separate passes
// (rotaryRotateInPlace / rotaryRotateInverseInPlace over the fp32 matrices, sentinel/NeuralNet/Cuda/CudaOps.cu:362-399,
// then the flash kernel's per-load conversion) becomes part of the one read + one write of the relayout.
// Pairs are interleaved, (2i, 2i+1), angle table entry [position][i] (RotaryEmbedding.cpp:19-27, :38-59); the two members
// of a pair are neighbouring d, i.e. neighbouring lanes of the token-major side, so the partner comes from a shuffle.
// Products and sums are rounded separately (no FMA contraction), which is what the reference's host code computes.
template <bool kInverse>
__device__ __forceinline__ float rotate_lane(float mine, int d, float c, float sn)
{
    const float other = __shfl_xor_sync(0xffffffffu, mine, 1);
    const float even = (d & 1) ? other : mine, odd = (d & 1) ? mine : other;
    if (!kInverse)   // even' = e*cos - o*sin ; odd' = e*sin + o*cos
        return (d & 1) ? __fadd_rn(__fmul_rn(even, sn), __fmul_rn(odd, c)) : __fsub_rn(__fmul_rn(even, c), __fmul_rn(odd, sn));
    // inverse (transpose of the rotation): even' = e*cos + o*sin ; odd' = -e*sin + o*cos
    return (d & 1) ? __fadd_rn(__fmul_rn(-even, sn), __fmul_rn(odd, c)) : __fadd_rn(__fmul_rn(even, c), __fmul_rn(odd, sn));
}

__global__ void rope_pack_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int H, int S, int D,
                                 int stride_columns, int column_start, const float* __restrict__ cos_t,
                                 const float* __restrict__ sin_t, int position_offset)
{
    __shared__ float tile[32][33];
    const int bh = blockIdx.z, b = bh / H, h = bh % H;
    const int s0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
    for (int r = ty; r < 32; r += 8) {
        const int d = d0 + r, s = s0 + tx;
        tile[r][tx] = (d < D && s < S) ? src[(long long)(h * D + d) * stride_columns + column_start + (long long)b * S + s] : 0.0f;
    }
    __syncthreads();
    const int pairs = D >> 1;
    for (int r = ty; r < 32; r += 8) {
        const int s = s0 + r, d = d0 + tx;       // D is even and d0 a multiple of 32: a pair never straddles tiles
        const bool live = s < S && d < D;
        const long long ti = (long long)(position_offset + s) * pairs + (d >> 1);
        const float c = live ? cos_t[ti] : 1.0f, sn = live ? sin_t[ti] : 0.0f;
        const float v = rotate_lane<false>(tile[tx][r], d, c, sn);
        if (live) dst[((long long)bh * S + s) * D + d] = __float2bfloat16_rn(v);
    }
}

template <bool kInverse>
__global__ void rope_unpack_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, int H, int S, int D,
                                   int stride_columns, int column_start, const float* __restrict__ cos_t,
                                   const float* __restrict__ sin_t, int position_offset)
{
    __shared__ float tile[32][33];
    const int bh = blockIdx.z, b = bh / H, h = bh % H;
    const int s0 = blockIdx.x * 32, d0 = blockIdx.y * 32;
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int pairs = D >> 1;
    for (int r = ty; r < 32; r += 8) {
        const int s = s0 + r, d = d0 + tx;
        const bool live = s < S && d < D;
        const float x = live ? __bfloat162float(src[((long long)bh * S + s) * D + d]) : 0.0f;
        const long long ti = (long long)(position_offset + s) * pairs + (d >> 1);
        const float c = live ? cos_t[ti] : 1.0f, sn = live ? sin_t[ti] : 0.0f;
        tile[r][tx] = rotate_lane<kInverse>(x, d, c, sn);
    }
    __syncthreads();
    for (int r = ty; r < 32; r += 8) {
        const int d = d0 + r, s = s0 + tx;
        if (d < D && s < S) dst[(long long)(h * D + d) * stride_columns + column_start + (long long)b * S + s] = tile[tx][r];
    }
}

// Head sizes that are multiples of 64 (the tensor-core kernels' sizes) take the kernels below: a rotation pair lives in one thread.
// kRot: 0 no rotation, 1 forward, 2 inverse.
template <int kRot>
__device__ __forceinline__ void rotate_pair(float& even, float& odd, float c, float sn)
{
    if (kRot == 0) return;
    const float e = even, o = odd;
    if (kRot == 1) {
        even = __fsub_rn(__fmul_rn(e, c), __fmul_rn(o, sn));
        odd = __fadd_rn(__fmul_rn(e, sn), __fmul_rn(o, c));
    } else {
        even = __fadd_rn(__fmul_rn(e, c), __fmul_rn(o, sn));
        odd = __fadd_rn(__fmul_rn(-e, sn), __fmul_rn(o, c));
    }
}

// Tiles of kTok tokens x DT = 64 features: on the bf16 side a thread moves eight consecutive features of one token, on the fp32
// side runs of kTok tokens of one feature.  (A tile covering a whole 128-feature head makes the bf16 side one contiguous block,
// but its shared memory leaves too few CTAs per SM: 35 % slower.)  The angle tables come as float4 (four pairs).
constexpr int kTok = 128;
constexpr int kHeadsPerCta = 8;   // heads one CTA converts in turn, at most
constexpr int kHeadsPerCtaScalar = 4;   // in the scalar form, which has one tile at a time

// lane maps (see above): fp32 side -> (first of four tokens, feature); bf16 side -> (token, 8-feature unit)
template <int DT> struct PackMap {
    static constexpr int kQuads = kTok * DT / 4 / 256;        // float4 accesses per thread on the fp32 side
    static constexpr int kUnits = kTok * (DT / 8) / 256;      // 16-byte units per thread on the bf16 side
    static constexpr int kUnitGroups = DT / 32;
    __device__ static void quad(int r, int& s4, int& d)
    {
        const int idx = r * 256 + threadIdx.x, rest = idx >> 5;
        s4 = (rest & 3) * 32 + (idx & 7) * 4;
        d = (rest >> 2) * 4 + ((idx >> 3) & 3);
    }
    __device__ static void unit(int r, int& sl, int& u)
    {
        const int idx = r * 256 + threadIdx.x, rest = idx >> 5;
        sl = (rest / kUnitGroups) * 8 + ((idx >> 2) & 7);
        u = (rest % kUnitGroups) * 4 + (idx & 3);
    }
};

// The angles depend on the token and the feature pair only: a thread fetches those of its (token, unit) slots once
// and keeps them in registers for all the heads its CTA converts.
template <int kRot, int DT>
__device__ __forceinline__ void load_angles(float4* cs, float4* sn, const float* __restrict__ cos_t, const float* __restrict__ sin_t,
                                            int s0, int d0, int S, int pairs, int position_offset)
{
    if (kRot == 0) return;
#pragma unroll
    for (int r = 0; r < PackMap<DT>::kUnits; ++r) {
        int sl, u;
        PackMap<DT>::unit(r, sl, u);
        const int s = min(s0 + sl, S - 1);
        const long long ti = (long long)(position_offset + s) * pairs + (d0 >> 1) + 4 * u;   // a multiple of 4: 16-byte aligned
        cs[r] = __ldg(reinterpret_cast<const float4*>(cos_t + ti));
        sn[r] = __ldg(reinterpret_cast<const float4*>(sin_t + ti));
    }
}

// eight features of one token, rotated and stored as bf16
template <int kRot>
__device__ __forceinline__ void store_unit(__nv_bfloat16* dst, float (&x)[8], const float4& cs, const float4& sn)
{
    if (kRot != 0) {
        rotate_pair<kRot>(x[0], x[1], cs.x, sn.x);
        rotate_pair<kRot>(x[2], x[3], cs.y, sn.y);
        rotate_pair<kRot>(x[4], x[5], cs.z, sn.z);
        rotate_pair<kRot>(x[6], x[7], cs.w, sn.w);
    }
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const __nv_bfloat162 y = __floats2bfloat162_rn(x[2 * i], x[2 * i + 1]);
        w[i] = *reinterpret_cast<const uint32_t*>(&y);
    }
    *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Scalar form, for windows whose first column, length or row pitch is not a multiple of four elements: 4-byte accesses on the
// fp32 side, one tile at a time, so that the loads in flight (16 a thread) and the CTAs beside each other (four heads each, not eight)
// have to hide the latency.  Four tensors of B3 Hq12 Hkv12 S6997 D128: 485 us with 4 loads in flight, 419 with 16 (588 with 4 and six
// heads).
template <int kRot, int DT>
__global__ void __launch_bounds__(256, 4) pack64_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int H, int S, int D,
                                                     int stride_columns, int column_start, const float* __restrict__ cos_t,
                                                     const float* __restrict__ sin_t, int position_offset, int heads_per_cta)
{
    using M = PackMap<DT>;
    extern __shared__ float tile_raw[];
    wait_for_stream();
    float (*tile)[DT + 1] = reinterpret_cast<float (*)[DT + 1]>(tile_raw);   // [token][feature]
    const int groups = (H + heads_per_cta - 1) / heads_per_cta;
    const int b = blockIdx.z / groups, h_first = (blockIdx.z % groups) * heads_per_cta;
    const int s0 = blockIdx.x * kTok, d0 = blockIdx.y * DT;
    float4 cs[M::kUnits], sn[M::kUnits];
    load_angles<kRot, DT>(cs, sn, cos_t, sin_t, s0, d0, S, D >> 1, position_offset);
    for (int h = h_first; h < min(H, h_first + heads_per_cta); ++h) {
        const float* base = src + (long long)(h * D + d0) * stride_columns + column_start + (long long)b * S + s0;
#pragma unroll 16
        for (int r = 0; r < kTok * DT / 256; ++r) {
            const int idx = r * 256 + threadIdx.x, d = idx / kTok, sl = idx % kTok;
            tile[sl][d] = (s0 + sl < S) ? base[(long long)d * stride_columns + sl] : 0.0f;
        }
        __syncthreads();
        __nv_bfloat16* out = dst + ((long long)(b * H + h) * S + s0) * D + d0;
#pragma unroll
        for (int r = 0; r < M::kUnits; ++r) {
            int sl, u;
            M::unit(r, sl, u);
            if (s0 + sl >= S) continue;
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = tile[sl][8 * u + i];
            store_unit<kRot>(out + (long long)sl * D + 8 * u, x, cs[r], sn[r]);
        }
        __syncthreads();      // the tile is refilled for the next head
    }
}

template <int kRot, int DT>
__global__ void __launch_bounds__(256, 4) unpack64_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, int H, int S, int D,
                                                       int stride_columns, int column_start, const float* __restrict__ cos_t,
                                                       const float* __restrict__ sin_t, int position_offset, int heads_per_cta)
{
    using M = PackMap<DT>;
    extern __shared__ float tile_raw[];
    wait_for_stream();
    float (*tile)[DT + 1] = reinterpret_cast<float (*)[DT + 1]>(tile_raw);
    const int groups = (H + heads_per_cta - 1) / heads_per_cta;
    const int b = blockIdx.z / groups, h_first = (blockIdx.z % groups) * heads_per_cta;
    const int s0 = blockIdx.x * kTok, d0 = blockIdx.y * DT;
    float4 cs[M::kUnits], sn[M::kUnits];
    load_angles<kRot, DT>(cs, sn, cos_t, sin_t, s0, d0, S, D >> 1, position_offset);
    for (int h = h_first; h < min(H, h_first + heads_per_cta); ++h) {
        const __nv_bfloat16* in = src + ((long long)(b * H + h) * S + s0) * D + d0;
        uint4 win[M::kUnits];
#pragma unroll
        for (int r = 0; r < M::kUnits; ++r) {      // all loads first
            int sl, u;
            M::unit(r, sl, u);
            win[r] = (s0 + sl < S) ? __ldg(reinterpret_cast<const uint4*>(in + (long long)sl * D + 8 * u)) : make_uint4(0, 0, 0, 0);
        }
#pragma unroll
        for (int r = 0; r < M::kUnits; ++r) {
            int sl, u;
            M::unit(r, sl, u);
            const uint32_t ws[4] = {win[r].x, win[r].y, win[r].z, win[r].w};
            float x[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                x[2 * i] = __uint_as_float(ws[i] << 16);
                x[2 * i + 1] = __uint_as_float(ws[i] & 0xffff0000u);
            }
            if (kRot != 0) {      // (rows past the end are zeros and stay zeros under the rotation)
                rotate_pair<kRot>(x[0], x[1], cs[r].x, sn[r].x);
                rotate_pair<kRot>(x[2], x[3], cs[r].y, sn[r].y);
                rotate_pair<kRot>(x[4], x[5], cs[r].z, sn[r].z);
                rotate_pair<kRot>(x[6], x[7], cs[r].w, sn[r].w);
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) tile[sl][8 * u + i] = x[i];
        }
        __syncthreads();
        float* base = dst + (long long)(h * D + d0) * stride_columns + column_start + (long long)b * S + s0;
#pragma unroll 16
        for (int r = 0; r < kTok * DT / 256; ++r) {
            const int idx = r * 256 + threadIdx.x, d = idx / kTok, sl = idx % kTok;
            if (s0 + sl < S) base[(long long)d * stride_columns + sl] = tile[sl][d];
        }
        __syncthreads();      // the tile is refilled for the next head
    }
}

// The usual form: every global access 16 bytes, and the next head's tile on its way into shared memory (asynchronous copies, two
// buffers) while this one is converted.  Bound by HBM: 6 bytes per element; B2 H28 S8192 D128 (352 MB): rotated 95 us with the
// tile loaded, converted and stored in turn, 62 us here (0.87 of the copy rate), plain 63 and 60.  The tile lies in shared memory as it came; its 16-byte units are XOR-permuted
// by row so that the reads across the grain (eight tokens x four units, or eight quads of tokens x four pairs) hit all banks.
template <int kRot, int DT>
__global__ void __launch_bounds__(256, 3) pack64_pipe_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, int H, int S, int D,
                                                          int stride_columns, int column_start, const float* __restrict__ cos_t,
                                                          const float* __restrict__ sin_t, int position_offset, int heads_per_cta)
{
    using M = PackMap<DT>;
    extern __shared__ float tile_raw[];            // [2][feature][128 tokens], token quad q of feature d at quad q ^ (d >> 3) * 2
    wait_for_stream();
    const int groups = (H + heads_per_cta - 1) / heads_per_cta;
    const int b = blockIdx.z / groups, h_first = (blockIdx.z % groups) * heads_per_cta, h_end = min(H, h_first + heads_per_cta);
    const int s0 = blockIdx.x * kTok, d0 = blockIdx.y * DT;
    auto fetch = [&](int h, float* tile) {
        const float* base = src + (long long)(h * D + d0) * stride_columns + column_start + (long long)b * S + s0;
#pragma unroll
        for (int r = 0; r < M::kQuads; ++r) {
            const int d = r * 8 + (threadIdx.x >> 5), q = threadIdx.x & 31;      // a warp: the 512 bytes of one feature
            if (s0 + 4 * q < S) copy16(tile + d * kTok + ((q ^ ((d >> 3) << 1)) << 2), base + (long long)d * stride_columns + 4 * q);
        }
        copies_commit();
    };
    fetch(h_first, tile_raw);
    float4 cs[M::kUnits], sn[M::kUnits];
    load_angles<kRot, DT>(cs, sn, cos_t, sin_t, s0, d0, S, D >> 1, position_offset);
    for (int h = h_first; h < h_end; ++h) {
        const float* tile = tile_raw + ((h - h_first) & 1) * (DT * kTok);
        if (h + 1 < h_end) {
            fetch(h + 1, tile_raw + ((h + 1 - h_first) & 1) * (DT * kTok));
            copies_left<1>();
        } else copies_left<0>();
        __syncthreads();
        __nv_bfloat16* out = dst + ((long long)(b * H + h) * S + s0) * D + d0;
#pragma unroll
        for (int r = 0; r < M::kUnits; ++r) {
            int sl, u;
            M::unit(r, sl, u);
            if (s0 + sl >= S) continue;
            const float* p = tile + 8 * u * kTok + (((sl >> 2) ^ (u << 1)) << 2) + (sl & 3);
            float x[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) x[i] = p[i * kTok];
            store_unit<kRot>(out + (long long)sl * D + 8 * u, x, cs[r], sn[r]);
        }
        __syncthreads();
    }
}

template <int kRot, int DT>
__global__ void __launch_bounds__(256, 4) unpack64_pipe_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, int H, int S, int D,
                                                            int stride_columns, int column_start, const float* __restrict__ cos_t,
                                                            const float* __restrict__ sin_t, int position_offset, int heads_per_cta)
{
    static_assert(DT == 64, "eight 16-byte units per token");
    constexpr int kWords = DT / 2, kItems = kTok / 4 * kWords / 256;   // an item: four tokens of one feature pair
    extern __shared__ float tile_raw[];
    uint32_t* tiles = reinterpret_cast<uint32_t*>(tile_raw);           // [2][token][32 pairs], unit c of token t at c ^ (t >> 2 & 7)
    wait_for_stream();
    const int groups = (H + heads_per_cta - 1) / heads_per_cta;
    const int b = blockIdx.z / groups, h_first = (blockIdx.z % groups) * heads_per_cta, h_end = min(H, h_first + heads_per_cta);
    const int s0 = blockIdx.x * kTok, d0 = blockIdx.y * DT;
    auto fetch = [&](int h, uint32_t* tile) {
        const __nv_bfloat16* in = src + ((long long)(b * H + h) * S + s0) * D + d0;
#pragma unroll
        for (int r = 0; r < kTok * 8 / 256; ++r) {
            const int t = r * 32 + (threadIdx.x >> 3), c = threadIdx.x & 7;
            if (s0 + t < S) copy16(tile + t * kWords + ((c ^ ((t >> 2) & 7)) << 2), in + (long long)t * D + 8 * c);
        }
        copies_commit();
    };
    fetch(h_first, tiles);
    const int q8 = threadIdx.x & 7, p4 = (threadIdx.x >> 3) & 3, warp = threadIdx.x >> 5;
    auto item = [&](int r, int& quad, int& pair) {
        const int rest = r * 8 + warp;
        quad = (rest & 3) * 8 + q8;
        pair = (rest >> 2) * 4 + p4;
    };
    float cs[kItems][4], sn[kItems][4];
    if (kRot != 0) {
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            int quad, pair;
            item(r, quad, pair);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const long long ti = (long long)(position_offset + min(s0 + 4 * quad + k, S - 1)) * (D >> 1) + (d0 >> 1) + pair;
                cs[r][k] = __ldg(cos_t + ti);
                sn[r][k] = __ldg(sin_t + ti);
            }
        }
    }
    for (int h = h_first; h < h_end; ++h) {
        const uint32_t* tile = tiles + ((h - h_first) & 1) * (kTok * kWords);
        if (h + 1 < h_end) {
            fetch(h + 1, tiles + ((h + 1 - h_first) & 1) * (kTok * kWords));
            copies_left<1>();
        } else copies_left<0>();
        __syncthreads();
        float* base = dst + (long long)(h * D + d0) * stride_columns + column_start + (long long)b * S + s0;
#pragma unroll
        for (int r = 0; r < kItems; ++r) {
            int quad, pair;
            item(r, quad, pair);
            if (s0 + 4 * quad >= S) continue;
            const uint32_t* p = tile + 4 * quad * kWords + (((pair >> 2) ^ q8) << 2) + p4;
            float e[4], o[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t w = p[k * kWords];
                e[k] = __uint_as_float(w << 16);
                o[k] = __uint_as_float(w & 0xffff0000u);
                if (kRot != 0) rotate_pair<kRot>(e[k], o[k], cs[r][k], sn[r][k]);
            }
            float* out = base + (long long)(2 * pair) * stride_columns + 4 * quad;
            *reinterpret_cast<float4*>(out) = make_float4(e[0], e[1], e[2], e[3]);
            *reinterpret_cast<float4*>(out + stride_columns) = make_float4(o[0], o[1], o[2], o[3]);
        }
        __syncthreads();
    }
}

// One tile column of 64 features per blockIdx.y.  A CTA converts several heads in turn: the angles cost it one fetch and the
// pipeline runs; fewer heads where the grid would leave SMs without CTAs.
template <typename Kernel, typename Src, typename Dst>
cudaError_t launch_convert64(Kernel kernel, size_t smem, std::atomic<unsigned long long>& configured, const Src* src, Dst* dst, int B, int H, int S,
                             int D, int stride_columns, int column_start, const float* cos_t, const float* sin_t, int position_offset, int max_heads,
                             cudaStream_t st)
{
    const cudaError_t e = ensure_dynamic_smem(kernel, smem, configured);
    if (e != cudaSuccess) return e;
    const long long tiles = (long long)((S + kTok - 1) / kTok) * (D / 64) * B, want = (4LL * sm_count() + tiles - 1) / tiles;
    int groups = (int)(want < H ? want : H);
    if (groups * max_heads < H) groups = (H + max_heads - 1) / max_heads;
    const int per = (H + groups - 1) / groups;
    const dim3 grid((S + kTok - 1) / kTok, D / 64, B * ((H + per - 1) / per));
    return launch_kernel(kernel, grid, 256, smem, st, 1, src, dst, H, S, D, stride_columns, column_start, cos_t, sin_t, position_offset, per);
}
#define SNTL_CONVERT(KERNEL, ROT, SMEM, HEADS)                                                                                                   \
    do {                                                                                                                                  \
        static std::atomic<unsigned long long> configured{0};                                                                             \
        return launch_convert64(KERNEL<ROT, 64>, SMEM, configured, src, dst, B, H, S, D, stride_columns, column_start, cos_t, sin_t,      \
                                position_offset, HEADS, st);                                                                              \
    } while (0)

constexpr size_t kTileBytes = (size_t)kTok * 65 * sizeof(float);

cudaError_t launch_pack64(bool rot, bool vec, const float* src, __nv_bfloat16* dst, int B, int H, int S, int D, int stride_columns,
                          int column_start, const float* cos_t, const float* sin_t, int position_offset, cudaStream_t st)
{
    constexpr size_t pipe = 2 * kTok * 64 * sizeof(float);
    if (vec && rot) SNTL_CONVERT(pack64_pipe_kernel, 1, pipe, kHeadsPerCta);
    if (vec) SNTL_CONVERT(pack64_pipe_kernel, 0, pipe, kHeadsPerCta);
    if (rot) SNTL_CONVERT(pack64_kernel, 1, kTileBytes, kHeadsPerCtaScalar);
    SNTL_CONVERT(pack64_kernel, 0, kTileBytes, kHeadsPerCtaScalar);
}
cudaError_t launch_unpack64(int rot, bool vec, const __nv_bfloat16* src, float* dst, int B, int H, int S, int D, int stride_columns,
                            int column_start, const float* cos_t, const float* sin_t, int position_offset, cudaStream_t st)
{
    constexpr size_t pipe = 2 * kTok * 64 * sizeof(__nv_bfloat16);
    if (vec && rot == 2) SNTL_CONVERT(unpack64_pipe_kernel, 2, pipe, kHeadsPerCta);
    if (vec && rot == 1) SNTL_CONVERT(unpack64_pipe_kernel, 1, pipe, kHeadsPerCta);
    if (vec) SNTL_CONVERT(unpack64_pipe_kernel, 0, pipe, kHeadsPerCta);
    if (rot == 2) SNTL_CONVERT(unpack64_kernel, 2, kTileBytes, kHeadsPerCtaScalar);
    if (rot == 1) SNTL_CONVERT(unpack64_kernel, 1, kTileBytes, kHeadsPerCtaScalar);
    SNTL_CONVERT(unpack64_kernel, 0, kTileBytes, kHeadsPerCtaScalar);
}
#undef SNTL_CONVERT

// ---- everything a tensor-core call needs from feature-major matrices (see MatrixStage) ----
// One launch instead of one per tensor: on the sizes of a training microstep (16 MB a matrix) a conversion takes as long as the
// gaps between launches, and O needs no bf16 copy at all -- the backward only wants rowsum(dO o O), which the terms role takes
// from the matrices (dO rounded to bf16 as the products see it).  Blocks by role: per-query terms, conversions (128 tokens x 64
// features of one head each, the tile of pack64_kernel), zeroing of the dQ accumulator (64 KB each).
// Call with B2 H32 S1024 D64 matrices, forward + backward: 17 launches, 227 us -> 5 launches, 115 us (with the results stored
// as matrices by the kernels that compute them).
struct StagePlan {
    MatrixStage m;
    int first_pack, first_zero, pack_end[4];   // block ranges: [0, first_pack) terms, then job by job, then zeroing
    int Hq, S, S_pad, stride_columns, column_start;
    long long rows_padded;
    RowTerms terms;
};
constexpr size_t kZeroBytes = 64 * 1024;

template <bool kVec, int D>
__global__ void __launch_bounds__(256, 4) stage_matrices_kernel(const __grid_constant__ StagePlan p)
{
    extern __shared__ float tile_raw[];
    wait_for_stream();
    if ((int)blockIdx.x < p.first_pack) {
        // one padded query row per thread: consecutive threads read consecutive tokens of each feature
        const long long r = (long long)blockIdx.x * 256 + threadIdx.x;
        if (r >= p.rows_padded) return;
        const int bh = (int)(r / p.S_pad), s = (int)(r - (long long)bh * p.S_pad), b = bh / p.Hq, h = bh - b * p.Hq;
        const bool live = s < p.S;
        float acc = 0.f, lse = 0.f;
        if (live) {
            const long long col = p.column_start + (long long)b * p.S + s;
            const float* o = p.m.o_mat + (long long)h * D * p.stride_columns + col;
            const float* g = p.m.do_mat + (long long)h * D * p.stride_columns + col;
#pragma unroll 16
            for (int d = 0; d < D; ++d)
                acc = fmaf(__ldg(o + (long long)d * p.stride_columns), __bfloat162float(__float2bfloat16_rn(__ldg(g + (long long)d * p.stride_columns))), acc);
            lse = p.m.lse_mat[(long long)h * p.stride_columns + col];
        }
        store_row_terms<D>(p.terms, r, live, lse, acc);
    } else if ((int)blockIdx.x < p.first_zero) {
        using M = PackMap<64>;
        float (*tile)[65] = reinterpret_cast<float (*)[65]>(tile_raw);   // [token][feature]
        int job = 0;
        while ((int)blockIdx.x >= p.pack_end[job]) ++job;
        const int H = p.m.heads[job], n_tok = (p.S + kTok - 1) / kTok;
        int i = blockIdx.x - (job ? p.pack_end[job - 1] : p.first_pack);
        const int s0 = i % n_tok * kTok;
        i /= n_tok;
        const int d0 = i % (D / 64) * 64, bh = i / (D / 64), b = bh / H, h = bh - b * H;
        const float* base = p.m.src[job] + (long long)(h * D + d0) * p.stride_columns + p.column_start + (long long)b * p.S + s0;
        if (kVec) {
            float4 x[M::kQuads];
#pragma unroll
            for (int r = 0; r < M::kQuads; ++r) {
                int s4, d;
                M::quad(r, s4, d);
                x[r] = (s0 + s4 < p.S) ? __ldg(reinterpret_cast<const float4*>(base + (long long)d * p.stride_columns + s4))
                                       : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int r = 0; r < M::kQuads; ++r) {
                int s4, d;
                M::quad(r, s4, d);
                tile[s4][d] = x[r].x; tile[s4 + 1][d] = x[r].y; tile[s4 + 2][d] = x[r].z; tile[s4 + 3][d] = x[r].w;
            }
        } else {
#pragma unroll 8
            for (int r = 0; r < kTok * 64 / 256; ++r) {
                const int idx = r * 256 + threadIdx.x, d = idx / kTok, sl = idx % kTok;
                tile[sl][d] = (s0 + sl < p.S) ? __ldg(base + (long long)d * p.stride_columns + sl) : 0.0f;
            }
        }
        __syncthreads();
        __nv_bfloat16* out = p.m.dst[job] + ((long long)bh * p.S + s0) * D + d0;
#pragma unroll
        for (int r = 0; r < M::kUnits; ++r) {
            int sl, u;
            M::unit(r, sl, u);
            if (s0 + sl >= p.S) continue;
            uint32_t w[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const __nv_bfloat162 y = __floats2bfloat162_rn(tile[sl][8 * u + 2 * k], tile[sl][8 * u + 2 * k + 1]);
                w[k] = *reinterpret_cast<const uint32_t*>(&y);
            }
            *reinterpret_cast<uint4*>(out + (long long)sl * D + 8 * u) = make_uint4(w[0], w[1], w[2], w[3]);
        }
    } else {
        float4* z = reinterpret_cast<float4*>(reinterpret_cast<char*>(p.m.dq_accum) + (size_t)(blockIdx.x - p.first_zero) * kZeroBytes);
        const size_t left = p.m.accum_bytes - (size_t)(blockIdx.x - p.first_zero) * kZeroBytes;
        const int n = (int)((left < kZeroBytes ? left : kZeroBytes) / 16);
        for (int i = threadIdx.x; i < n; i += 256) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
}

template <bool kVec, int D>
cudaError_t launch_stage(const StagePlan& p, unsigned blocks, cudaStream_t st)
{
    constexpr size_t smem = (size_t)kTok * 65 * sizeof(float);
    static std::atomic<unsigned long long> configured{0};
    const cudaError_t e = ensure_dynamic_smem(stage_matrices_kernel<kVec, D>, smem, configured);
    if (e != cudaSuccess) return e;
    return launch_kernel(stage_matrices_kernel<kVec, D>, blocks, 256, smem, st, 1, p);
}

__global__ void f32_to_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = __float2bfloat16_rn(src[i]);
}
__global__ void bf16_to_f32_kernel(const __nv_bfloat16* __restrict__ src, float* __restrict__ dst, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = __bfloat162float(src[i]);
}

template <typename T> __device__ __forceinline__ float ldf(const T* p);
template <> __device__ __forceinline__ float ldf<float>(const float* p) { return *p; }
template <> __device__ __forceinline__ float ldf<__nv_bfloat16>(const __nv_bfloat16* p) { return __bfloat162float(*p); }
template <typename T> __device__ __forceinline__ void stf(T* p, float x);
template <> __device__ __forceinline__ void stf<float>(float* p, float x) { *p = x; }
template <> __device__ __forceinline__ void stf<__nv_bfloat16>(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }

// One warp per row: (o_acc, lse_acc) <- the softmax-weighted combination with (o_part, lse_part).
template <typename T, typename P>
__global__ void merge_kernel(long long rows, int D, T* __restrict__ o_acc, float* __restrict__ lse_acc,
                             const P* __restrict__ o_part, const float* __restrict__ lse_part)
{
    const int lane = threadIdx.x & 31;
    const long long row = blockIdx.x * (long long)(blockDim.x >> 5) + (threadIdx.x >> 5);
    if (row >= rows) return;
    const float la = lse_acc[row], lb = lse_part[row];
    const float m = fmaxf(la, lb);
    if (m == -INFINITY) return;  // both empty: keep zeros / -inf
    const float wa = expf(la - m), wb = expf(lb - m);
    const float inv = 1.0f / (wa + wb);
    for (int d = lane; d < D; d += 32) {
        const float x = ldf(o_acc + row * D + d) * wa + ldf(o_part + row * D + d) * wb;
        stf(o_acc + row * D + d, x * inv);
    }
    if (lane == 0) lse_acc[row] = m + logf(wa + wb);
}

template <typename P>
__global__ void accumulate_kernel(float* __restrict__ acc, const P* __restrict__ part, size_t n)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        acc[i] += ldf(part + i);
}

inline int blocks_for(size_t n, int threads)
{
    size_t b = (n + threads - 1) / threads;
    return (int)(b > 148 * 16 ? 148 * 16 : (b ? b : 1));
}

}  // namespace

static cudaError_t sentinel_to_bhsd_bf16(const float* src, __nv_bfloat16* dst, int B, int H, int S, int D, int stride_columns,
                                  int column_start, cudaStream_t st)
{
    dim3 grid((S + 31) / 32, (D + 31) / 32, B * H), block(32, 8);
    sentinel_to_bhsd_kernel<<<grid, block, 0, st>>>(src, dst, H, S, D, stride_columns, column_start);
    count_launch();
    return cudaGetLastError();
}

static cudaError_t bhsd_bf16_to_sentinel(const __nv_bfloat16* src, float* dst, int B, int H, int S, int D, int stride_columns,
                                  int column_start, cudaStream_t st)
{
    dim3 grid((S + 31) / 32, (D + 31) / 32, B * H), block(32, 8);
    bhsd_to_sentinel_kernel<<<grid, block, 0, st>>>(src, dst, H, S, D, stride_columns, column_start);
    count_launch();
    return cudaGetLastError();
}

// the fp32 side can be accessed 16 bytes at a time when every row of the window starts on a 16-byte boundary
static bool f32_rows_aligned(const void* p, int S, int stride_columns, int column_start)
{
    return ((uintptr_t)p & 15u) == 0 && stride_columns % 4 == 0 && column_start % 4 == 0 && S % 4 == 0;
}
static bool tables_aligned(const float* cos_t, const float* sin_t) { return (((uintptr_t)cos_t | (uintptr_t)sin_t) & 15u) == 0; }

cudaError_t rope_pack_bf16(const float* src, __nv_bfloat16* dst, int B, int H, int S, int D, int stride_columns,
                           int column_start, const float* cos_t, const float* sin_t, int position_offset, cudaStream_t st)
{
    if (D % 64 == 0) {
        // the bf16 side and the angle tables are accessed 16 bytes at a time (as are all bf16 tensors of the tensor-core kernels)
        if (((uintptr_t)dst & 15u) != 0 || (cos_t && !tables_aligned(cos_t, sin_t))) return cudaErrorMisalignedAddress;
        return launch_pack64(cos_t != nullptr, f32_rows_aligned(src, S, stride_columns, column_start), src, dst, B, H, S, D, stride_columns,
                             column_start, cos_t, sin_t, position_offset, st);
    }
    if (!cos_t) return sentinel_to_bhsd_bf16(src, dst, B, H, S, D, stride_columns, column_start, st);
    dim3 grid((S + 31) / 32, (D + 31) / 32, B * H), block(32, 8);
    rope_pack_kernel<<<grid, block, 0, st>>>(src, dst, H, S, D, stride_columns, column_start, cos_t, sin_t, position_offset);
    count_launch();
    return cudaGetLastError();
}

cudaError_t rope_unpack_f32(const __nv_bfloat16* src, float* dst, int B, int H, int S, int D, int stride_columns,
                            int column_start, const float* cos_t, const float* sin_t, int position_offset, bool inverse,
                            cudaStream_t st)
{
    if (D % 64 == 0) {
        if (((uintptr_t)src & 15u) != 0 || (cos_t && !tables_aligned(cos_t, sin_t))) return cudaErrorMisalignedAddress;
        return launch_unpack64(!cos_t ? 0 : (inverse ? 2 : 1), f32_rows_aligned(dst, S, stride_columns, column_start), src, dst, B, H, S, D,
                               stride_columns, column_start, cos_t, sin_t, position_offset, st);
    }
    if (!cos_t) return bhsd_bf16_to_sentinel(src, dst, B, H, S, D, stride_columns, column_start, st);
    dim3 grid((S + 31) / 32, (D + 31) / 32, B * H), block(32, 8);
    if (inverse)
        rope_unpack_kernel<true><<<grid, block, 0, st>>>(src, dst, H, S, D, stride_columns, column_start, cos_t, sin_t, position_offset);
    else
        rope_unpack_kernel<false><<<grid, block, 0, st>>>(src, dst, H, S, D, stride_columns, column_start, cos_t, sin_t, position_offset);
    count_launch();
    return cudaGetLastError();
}

cudaError_t stage_matrices(const MatrixStage& m, int B, int Hq, int S, int D, int stride_columns, int column_start, float scale, cudaStream_t st)
{
    // the bf16 tensors, the row terms and the accumulator are written 16 bytes at a time
    if (!aligned(16, m.dst[0], m.dst[1], m.dst[2], m.dst[3], m.row_terms, m.dq_accum)) return cudaErrorMisalignedAddress;
    StagePlan p{};
    p.m = m;
    p.Hq = Hq; p.S = S; p.S_pad = (S + 127) / 128 * 128;
    p.stride_columns = stride_columns; p.column_start = column_start;
    p.rows_padded = (long long)B * Hq * p.S_pad;
    long long blocks = 0;
    if (m.o_mat) {
        p.terms = row_terms_of(m.row_terms, p.rows_padded, D, scale);
        blocks = (p.rows_padded + 255) / 256;
    }
    p.first_pack = (int)blocks;
    bool vec = true;
    for (int j = 0; j < 4; ++j) {
        if (j < m.n) {
            blocks += (long long)((S + kTok - 1) / kTok) * (D / 64) * B * m.heads[j];
            vec = vec && f32_rows_aligned(m.src[j], S, stride_columns, column_start);
        }
        if (blocks > 0x3fffffffLL) return cudaErrorInvalidConfiguration;
        p.pack_end[j] = (int)blocks;
    }
    p.first_zero = (int)blocks;
    blocks += (long long)((m.accum_bytes + kZeroBytes - 1) / kZeroBytes);
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    if (D == 64) return vec ? launch_stage<true, 64>(p, (unsigned)blocks, st) : launch_stage<false, 64>(p, (unsigned)blocks, st);
    return vec ? launch_stage<true, 128>(p, (unsigned)blocks, st) : launch_stage<false, 128>(p, (unsigned)blocks, st);
}

cudaError_t f32_to_bf16(const float* src, __nv_bfloat16* dst, size_t n, cudaStream_t st)
{
    f32_to_bf16_kernel<<<blocks_for(n, 256), 256, 0, st>>>(src, dst, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t bf16_to_f32(const __nv_bfloat16* src, float* dst, size_t n, cudaStream_t st)
{
    bf16_to_f32_kernel<<<blocks_for(n, 256), 256, 0, st>>>(src, dst, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t accumulate_f32(int part_dtype, float* acc, const void* part, size_t n, cudaStream_t st)
{
    if (n == 0) return cudaSuccess;
    if (part_dtype == SNTL_DTYPE_BF16)
        accumulate_kernel<<<blocks_for(n, 256), 256, 0, st>>>(acc, (const __nv_bfloat16*)part, n);
    else
        accumulate_kernel<<<blocks_for(n, 256), 256, 0, st>>>(acc, (const float*)part, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t merge_partials(int acc_dtype, int part_dtype, long long rows, int D, void* o_acc, float* lse_acc,
                           const void* o_part, const float* lse_part, cudaStream_t st)
{
    const int warps = 8;
    const long long blocks = (rows + warps - 1) / warps;
    if (blocks <= 0) return cudaSuccess;
    const unsigned g = (unsigned)blocks;
    const bool ab = acc_dtype == SNTL_DTYPE_BF16, pb = part_dtype == SNTL_DTYPE_BF16;
    if (ab && pb)
        merge_kernel<<<g, warps * 32, 0, st>>>(rows, D, (__nv_bfloat16*)o_acc, lse_acc, (const __nv_bfloat16*)o_part, lse_part);
    else if (!ab && pb)
        merge_kernel<<<g, warps * 32, 0, st>>>(rows, D, (float*)o_acc, lse_acc, (const __nv_bfloat16*)o_part, lse_part);
    else if (ab && !pb)
        merge_kernel<<<g, warps * 32, 0, st>>>(rows, D, (__nv_bfloat16*)o_acc, lse_acc, (const float*)o_part, lse_part);
    else
        merge_kernel<<<g, warps * 32, 0, st>>>(rows, D, (float*)o_acc, lse_acc, (const float*)o_part, lse_part);
    count_launch();
    return cudaGetLastError();
}

}  // namespace sntl
