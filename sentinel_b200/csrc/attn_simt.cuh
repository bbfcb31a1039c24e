// Building blocks of the exact-fp32 kernels (attn_simt_fwd.cu, attn_simt_bwd.cu): staging of a tile into shared memory, the
// two register-tiled products, and the store of a tile.
//
// A CTA is 128 threads, thread = (tx, ty) = (tid % 16, tid / 16).  It owns 8*TM rows (queries in the forward and for dQ,
// keys for dK/dV): thread ty owns rows ty + 8*i, i < TM.  The other side is visited in tiles of 16*TN rows, of which thread tx
// owns rows tx + 16*j in the score products.  Tiles lie in shared memory as [row][feature] with a pitch of DP + 4 floats (an
// odd number of 16-byte units, so rows eight apart or neighbouring rows fall into different banks), DP = head_dim rounded up
// to a compiled size and filled with zeros.
//   scores   acc[i][j] += sum_d A[ty + 8i][d] * B[tx + 16j][d]     16-byte loads along d: TM + TN loads per 4*TM*TN FMAs
//   outputs  acc[i][c] += sum_k W[k][ty + 8i] * B[k][c]            W (probabilities) is stored [k][ty*TM + i]: the order in which
//                                                                  the thread that owns the rows reads them back
// W is written and read by the 16 threads of one ty, which are half a warp: no CTA barrier between the two products.
// A hidden (query, key) pair has weight 0, which adds nothing unless the other factor is not finite (0 * inf).  Tiles that the mask
// cuts through are looked at for that, V while it is staged and the backward's operands by their scores; where a value is not
// finite the products leave the hidden pairs out one by one (outputs_visible).
#pragma once

#include "common.cuh"

#include <math.h>

namespace sntl {
namespace simt {

constexpr int kThreads = 128;

template <typename T> struct Elem;
template <> struct Elem<float> {
    static __device__ __forceinline__ float4 load4(const float* p) { return __ldg(reinterpret_cast<const float4*>(p)); }
    static __device__ __forceinline__ float load(const float* p) { return __ldg(p); }
    static __device__ __forceinline__ void store4(float* p, float4 x) { *reinterpret_cast<float4*>(p) = x; }
    static __device__ __forceinline__ void store(float* p, float x) { *p = x; }
};
template <> struct Elem<__nv_bfloat16> {
    static __device__ __forceinline__ float4 load4(const __nv_bfloat16* p)
    {
        const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
        return make_float4(__uint_as_float(w.x << 16), __uint_as_float(w.x & 0xffff0000u), __uint_as_float(w.y << 16),
                           __uint_as_float(w.y & 0xffff0000u));
    }
    static __device__ __forceinline__ float load(const __nv_bfloat16* p) { return __bfloat162float(*p); }
    static __device__ __forceinline__ void store4(__nv_bfloat16* p, float4 x)
    {
        __nv_bfloat162 a = __floats2bfloat162_rn(x.x, x.y), b = __floats2bfloat162_rn(x.z, x.w);
        *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<uint32_t*>(&a), *reinterpret_cast<uint32_t*>(&b));
    }
    static __device__ __forceinline__ void store(__nv_bfloat16* p, float x) { *p = __float2bfloat16_rn(x); }
};

// Rows [row0, row0 + ROWS) of a [S][D] slab with element strides ss, sd; rows past S and features past D read as zero.
struct Slab {
    long long ss, sd;
    int S, D;
    bool vec;   // sd == 1 and every row can be read four elements at a time
};

// four consecutive features of one row
template <typename T>
__device__ __forceinline__ float4 load_unit(const T* base, const Slab& m, int row, int d)
{
    if (row >= m.S || d >= m.D) return make_float4(0.f, 0.f, 0.f, 0.f);
    const T* p = base + row * m.ss + d * m.sd;
    if (m.vec) return Elem<T>::load4(p);
    float4 x = make_float4(Elem<T>::load(p), 0.f, 0.f, 0.f);
    if (d + 1 < m.D) x.y = Elem<T>::load(p + m.sd);
    if (d + 2 < m.D) x.z = Elem<T>::load(p + 2 * m.sd);
    if (d + 3 < m.D) x.w = Elem<T>::load(p + 3 * m.sd);
    return x;
}

// unit u of a tile -> (row, first feature): along the contiguous direction of the source, so that a warp's loads coalesce
template <int DP, int ROWS>
__device__ __forceinline__ void unit_of(int u, bool rows_contiguous, int& r, int& d)
{
    if (!rows_contiguous) { r = u / (DP / 4); d = (u - r * (DP / 4)) * 4; }   // token-major: features are contiguous
    else { d = (u / ROWS) * 4; r = u % ROWS; }                                // feature-major: tokens are
}

// 0, or NaN once a value was not finite
__device__ __forceinline__ float zero_if_finite(float z, const float4& x)
{
    return fmaf(x.x, 0.f, fmaf(x.y, 0.f, fmaf(x.z, 0.f, fmaf(x.w, 0.f, z))));
}

// Returns zero_if_finite of what this thread has staged.
template <typename T, int DP, int ROWS>
__device__ __forceinline__ float stage(float* dst, const T* base, const Slab& m, int row0)
{
    float z = 0.f;
    constexpr int kUnits = ROWS * DP / 4, kPer = (kUnits + kThreads - 1) / kThreads, kBatch = kPer < 4 ? kPer : 4;
#pragma unroll
    for (int k0 = 0; k0 < kPer; k0 += kBatch) {
        float4 x[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = (k0 + k) * kThreads + (int)threadIdx.x;
            int r, d;
            unit_of<DP, ROWS>(u, m.sd != 1, r, d);
            if (u < kUnits) x[k] = load_unit(base, m, row0 + r, d);
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = (k0 + k) * kThreads + (int)threadIdx.x;
            int r, d;
            unit_of<DP, ROWS>(u, m.sd != 1, r, d);
            if (u < kUnits) {
                *reinterpret_cast<float4*>(dst + r * (DP + 4) + d) = x[k];
                z = zero_if_finite(z, x[k]);
            }
        }
    }
    return z;
}

// dO rows as above and, for delta = rowsum(dO o O), one partial sum per 16-byte unit: part[row][unit]
template <typename T, int DP, int ROWS>
__device__ __forceinline__ void stage_with_delta(float* dst, float* part, const T* dout, const T* o, const Slab& m, int row0)
{
    constexpr int kUnits = ROWS * DP / 4, kPer = (kUnits + kThreads - 1) / kThreads, kBatch = kPer < 2 ? kPer : 2;
#pragma unroll
    for (int k0 = 0; k0 < kPer; k0 += kBatch) {
        float4 x[kBatch], y[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = (k0 + k) * kThreads + (int)threadIdx.x;
            int r, d;
            unit_of<DP, ROWS>(u, m.sd != 1, r, d);
            if (u < kUnits) {
                x[k] = load_unit(dout, m, row0 + r, d);
                y[k] = load_unit(o, m, row0 + r, d);
            }
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            const int u = (k0 + k) * kThreads + (int)threadIdx.x;
            int r, d;
            unit_of<DP, ROWS>(u, m.sd != 1, r, d);
            if (u < kUnits) {
                *reinterpret_cast<float4*>(dst + r * (DP + 4) + d) = x[k];
                part[r * (DP / 4 + 1) + d / 4] = fmaf(x[k].x, y[k].x, fmaf(x[k].y, y[k].y, fmaf(x[k].z, y[k].z, x[k].w * y[k].w)));
            }
        }
    }
}
template <int DP>
__device__ __forceinline__ float delta_of(const float* part, int r)
{
    float s = 0.f;
#pragma unroll
    for (int c = 0; c < DP / 4; ++c) s += part[r * (DP / 4 + 1) + c];
    return s;
}

// The products below use nothing but packed FMAs (ffma2): three-operand scalar ones stall in dispatch on their register reads (forward
// B8 H12 S512 D64: 129 us with them, the FMA pipes 45 % busy).
// (the two halves of an accumulator take the even and the odd features)
template <int TM, int TN, int DP>
__device__ __forceinline__ void scores(float (&out)[TM][TN], const float* A, const float* B)
{
    constexpr int P = DP + 4;
    const float* a0 = A + (threadIdx.x >> 4) * P;
    const float* b0 = B + (threadIdx.x & 15) * P;
    float2 acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);
#pragma unroll 4
    for (int d = 0; d < DP; d += 4) {
        float4 b[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) b[j] = *reinterpret_cast<const float4*>(b0 + j * 16 * P + d);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const float4 a = *reinterpret_cast<const float4*>(a0 + i * 8 * P + d);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = ffma2(make_float2(a.x, a.y), make_float2(b[j].x, b[j].y), acc[i][j]);
#pragma unroll
            for (int j = 0; j < TN; ++j) acc[i][j] = ffma2(make_float2(a.z, a.w), make_float2(b[j].z, b[j].w), acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) out[i][j] = acc[i][j].x + acc[i][j].y;
}

// Whether one of the warp's scores (all scores of a row are not finite if one of its values is not) or of the terms of their columns
// (in shared memory, or null) is not finite.
template <int TM, int TN>
__device__ __forceinline__ bool not_finite(const float (&a)[TM][TN], const float (&b)[TM][TN], const float* terms)
{
    float z = 0.f, y = 0.f;     // (two chains: one would be 2 * TM * TN long)
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        if (terms) z = fmaf(terms[(threadIdx.x & 15) + 16 * j], 0.f, z);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            z = fmaf(a[i][j], 0.f, z);
            y = fmaf(b[i][j], 0.f, y);
        }
    }
    return __any_sync(0xffffffffu, z + y != 0.f);
}

// columns of the outputs a thread owns: NV vectors of VW, starting at tx*VW + 16*VW*c
template <int DP> struct OutMap {
    static constexpr int VW = DP % 64 == 0 ? 4 : DP % 32 == 0 ? 2 : 1;
    static constexpr int NV = DP / (16 * VW);
    static constexpr int N = VW * NV;
    static __device__ __forceinline__ int col(int n) { return (n / VW) * 16 * VW + (int)(threadIdx.x & 15) * VW + n % VW; }
};

template <int V> __device__ __forceinline__ void load_vec(float* x, const float* p)
{
    if constexpr (V % 4 == 0) {
#pragma unroll
        for (int i = 0; i < V; i += 4) {
            const float4 t = *reinterpret_cast<const float4*>(p + i);
            x[i] = t.x; x[i + 1] = t.y; x[i + 2] = t.z; x[i + 3] = t.w;
        }
    } else if constexpr (V == 2) {
        const float2 t = *reinterpret_cast<const float2*>(p);
        x[0] = t.x; x[1] = t.y;
    } else {
        x[0] = *p;
    }
}

// W: [K][8*TM + 4], B: [K][DP + 4].  acc[i] holds rows 2i and 2i + 1 of the thread: their weights are neighbours in W.
template <int TM, int DP, int K>
__device__ __forceinline__ void outputs(float2 (&acc)[TM / 2][OutMap<DP>::N], const float* W, const float* B)
{
    using M = OutMap<DP>;
    const float* w0 = W + (threadIdx.x >> 4) * TM;
    const float* b0 = B + (threadIdx.x & 15) * M::VW;
#pragma unroll 4
    for (int k = 0; k < K; ++k) {
        float w[TM], b[M::N];
        load_vec<TM>(w, w0 + k * (8 * TM + 4));
#pragma unroll
        for (int c = 0; c < M::NV; ++c) load_vec<M::VW>(b + c * M::VW, b0 + k * (DP + 4) + c * 16 * M::VW);
#pragma unroll
        for (int n = 0; n < M::N; ++n)
#pragma unroll
            for (int i = 0; i < TM / 2; ++i) acc[i][n] = ffma2(make_float2(w[2 * i], w[2 * i + 1]), make_float2(b[n], b[n]), acc[i][n]);
    }
}
// The same for a tile that holds values that are not finite and pairs that are hidden: visible(i, k), of the thread's row ty + 8*i.
template <int TM, int DP, int K, typename F>
__device__ __forceinline__ void outputs_visible(float2 (&acc)[TM / 2][OutMap<DP>::N], const float* W, const float* B, F&& visible)
{
    using M = OutMap<DP>;
#pragma unroll 1
    for (int k = 0; k < K; ++k) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            if (!visible(i, k)) continue;
            const float w = W[k * (8 * TM + 4) + (threadIdx.x >> 4) * TM + i];
#pragma unroll
            for (int n = 0; n < M::N; ++n) {
                float& a = i & 1 ? acc[i / 2][n].y : acc[i / 2][n].x;
                a = fmaf(w, B[k * (DP + 4) + M::col(n)], a);
            }
        }
    }
}
template <int TM, int N> __device__ __forceinline__ void clear(float2 (&acc)[TM][N])
{
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int n = 0; n < N; ++n) acc[i][n] = make_float2(0.f, 0.f);
}
template <int TM> __device__ __forceinline__ void put_weights(float* W, int k, const float (&w)[TM])
{
    float* p = W + k * (8 * TM + 4) + (threadIdx.x >> 4) * TM;
    if constexpr (TM % 4 == 0) {
#pragma unroll
        for (int i = 0; i < TM; i += 4) *reinterpret_cast<float4*>(p + i) = make_float4(w[i], w[i + 1], w[i + 2], w[i + 3]);
    } else {
#pragma unroll
        for (int i = 0; i < TM; i += 2) *reinterpret_cast<float2*>(p + i) = make_float2(w[i], w[i + 1]);
    }
}

// The CTA's 8*TM rows of outputs, through `buf` ([8*TM][DP + 4], free of readers) so that stores coalesce in either layout.
template <typename T, int TM, int DP>
__device__ __forceinline__ void store_rows(T* base, const Slab& m, int row0, const float2 (&acc)[TM / 2][OutMap<DP>::N], float* buf)
{
    using M = OutMap<DP>;
    const int ty = threadIdx.x >> 4;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int n = 0; n < M::N; ++n) buf[(ty + 8 * i) * (DP + 4) + M::col(n)] = i & 1 ? acc[i / 2][n].y : acc[i / 2][n].x;
    __syncthreads();
    constexpr int kUnits = 8 * TM * DP / 4;
    for (int u = threadIdx.x; u < kUnits; u += kThreads) {
        int r, d;
        unit_of<DP, 8 * TM>(u, m.sd != 1, r, d);
        const int row = row0 + r;
        if (row >= m.S || d >= m.D) continue;
        const float4 x = *reinterpret_cast<const float4*>(buf + r * (DP + 4) + d);
        T* p = base + row * m.ss + d * m.sd;
        if (m.vec) { Elem<T>::store4(p, x); continue; }
        Elem<T>::store(p, x.x);
        if (d + 1 < m.D) Elem<T>::store(p + m.sd, x.y);
        if (d + 2 < m.D) Elem<T>::store(p + 2 * m.sd, x.z);
        if (d + 3 < m.D) Elem<T>::store(p + 3 * m.sd, x.w);
    }
}

__device__ __forceinline__ int visible_keys(const AttnShape& s, int query)
{
    if (!s.causal) return s.Skv;
    const int n = query + (s.Skv - s.Sq) + 1;
    return n < 0 ? 0 : (n > s.Skv ? s.Skv : n);
}

}  // namespace simt
}  // namespace sntl
