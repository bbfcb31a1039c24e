// Exact-fp32 forward for a handful of query rows per KV head: decode, and short continuations of a cache.
//
// Bound by latency: K and V are read once (a few MB), and what counts is how many of those bytes are in flight.  The rows of
// one (batch, KV head) -- query heads of the group times new tokens, at most 8 -- are served by a cluster of up to eight CTAs,
// each with a contiguous piece of the keys.  A CTA copies 128 keys of K and of V into shared memory with two groups of
// asynchronous 16-byte copies, scores one key per thread, and accumulates P V with the lanes along the features while every
// warp takes a quarter of the keys.  Partial (m, l, O) merge through distributed shared memory: one launch, no scratch.
// 1 token x 777 keys x 12 heads, head_dim 64: 165 us with one warp per row, 11.7 us through the 16-row tiles of
// attn_simt_fwd.cu (15 of 16 rows empty), 5.1 us here (6.4 when the merge went through distributed shared memory once per peer and a
// score was one chain of FMAs; 2000 keys x 4 sequences 11.9 -> 11.1, 100 keys 4.6 -> 4.0, 2 x 2048 keys of head_dim 128 14.1 -> 12.6).
#include "attn_simt.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace sntl {
using namespace simt;
namespace {

constexpr int kChunk = kThreads;   // keys per pass: one per thread
constexpr int kWarps = kThreads / 32;
constexpr int kMaxSplit = 8;       // CTAs of a cluster

template <int DP, int R> struct DecodeSmem {
    static constexpr int P = DP + 4;
    static constexpr int k = 0, v = k + kChunk * P, q = v + kChunk * P, p = q + R * DP, red = p + R * kChunk;   // red: [warp][m, l][R]
    static constexpr int out = k, ml = red + kWarps * 2 * R;                                                    // out: [R][DP] of the CTA
    static constexpr size_t bytes = (ml + 2 * R) * sizeof(float);
    static_assert(kWarps * R * DP <= kChunk * P, "the warps' partial outputs reuse the K buffer");
};

// rows [k0, k0 + n) of K or V
template <int DP>
__device__ __forceinline__ void stage_async(float* dst, const float* base, long long ss, int k0, int n)
{
    constexpr int kUnits = DP / 4;
#pragma unroll 4
    for (int u = threadIdx.x; u < kChunk * kUnits; u += kThreads) {
        const int r = u / kUnits, d = (u % kUnits) * 4;
        if (r < n) copy16(dst + r * (DP + 4) + d, base + (k0 + r) * ss + d);
    }
    copies_commit();
}

template <int DP, int R>
__global__ void __launch_bounds__(kThreads) simt_decode_kernel(const SimtArgs a, int n_split)
{
    using L = DecodeSmem<DP, R>;
    constexpr int kCols = DP / 32;                            // features per lane in the P V product
    extern __shared__ __align__(16) float smem[];
    wait_for_stream();
    const AttnShape& s = a.s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slab = blockIdx.x / n_split, rank = blockIdx.x - slab * n_split;
    const int b = slab / s.Hkv, hk = slab - b * s.Hkv, group = s.Hq / s.Hkv, rows = group * s.Sq;
    const int first_pos = s.Skv - s.Sq;                       // position of the first new token
    const float* kb = (const float*)a.k + b * a.vkv.sb + hk * a.vkv.sh;
    const float* vb = (const float*)a.v + b * a.vkv.sb + hk * a.vkv.sh;
    const int per = (s.Skv + n_split - 1) / n_split, k_begin = rank * per, k_end = min(s.Skv, k_begin + per);
    // row r of the slab: query head hk * group + r / Sq, new token r % Sq
    auto row_offset = [&](int r) { return b * a.vq.sb + (long long)(hk * group + r / s.Sq) * a.vq.sh + (long long)(r % s.Sq) * a.vq.ss; };

    float m[R], l[R], acc[R][kCols];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        m[r] = -INFINITY;
        l[r] = 0.f;
#pragma unroll
        for (int c = 0; c < kCols; ++c) acc[r][c] = 0.f;
    }
    bool q_staged = false;
    for (int k0 = k_begin; k0 < k_end; k0 += kChunk) {
        const int n = min(kChunk, k_end - k0);
        if (s.window > 0 && k0 >= s.global_tokens && k0 + n - 1 < first_pos - s.window + 1) continue;   // hidden from every row
        stage_async<DP>(smem + L::k, kb, a.vkv.ss, k0, n);
        stage_async<DP>(smem + L::v, vb, a.vkv.ss, k0, n);
        if (!q_staged) {
            q_staged = true;
            for (int u = threadIdx.x; u < R * DP; u += kThreads) {
                const int r = u / DP, d = u % DP;
                smem[L::q + u] = r < rows ? ((const float*)a.q)[row_offset(r) + d] : 0.f;
            }
        }
        copies_left<1>();
        __syncthreads();
        // ---- one key per thread ----
        const int key = k0 + (int)threadIdx.x;
        float sc[R];
        bool visible[R];
#pragma unroll
        for (int r = 0; r < R; ++r) sc[r] = 0.f;
        if ((int)threadIdx.x < n) {
            const float* kr = smem + L::k + threadIdx.x * L::P;
            float part[R][4] = {};       // four chains of FMAs instead of one
#pragma unroll 8
            for (int d = 0; d < DP; d += 4) {
                const float4 x = *reinterpret_cast<const float4*>(kr + d);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float4 y = *reinterpret_cast<const float4*>(smem + L::q + r * DP + d);
                    part[r][0] = fmaf(x.x, y.x, part[r][0]);
                    part[r][1] = fmaf(x.y, y.y, part[r][1]);
                    part[r][2] = fmaf(x.z, y.z, part[r][2]);
                    part[r][3] = fmaf(x.w, y.w, part[r][3]);
                }
            }
#pragma unroll
            for (int r = 0; r < R; ++r) sc[r] = (part[r][0] + part[r][1]) + (part[r][2] + part[r][3]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int pos = first_pos + r % s.Sq;
            visible[r] = (int)threadIdx.x < n && r < rows && key <= pos && window_allows(s, pos, key);
            sc[r] = visible[r] ? sc[r] * s.scale : -INFINITY;
            float mx = sc[r];
#pragma unroll
            for (int x = 16; x > 0; x >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            if (lane == 0) smem[L::red + warp * 2 * R + r] = mx;
        }
        __syncthreads();
        float corr[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            float mx = m[r];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) mx = fmaxf(mx, smem[L::red + w * 2 * R + r]);
            const float ref = mx == -INFINITY ? 0.f : mx;
            corr[r] = expf(m[r] - ref);
            m[r] = mx;
            const float p = expf(sc[r] - ref);
            smem[L::p + r * kChunk + threadIdx.x] = visible[r] ? p : -1.f;   // hidden: V is left out below, whatever it holds (rows past
                                                                             // the last: never stored)
            float sum = p;
#pragma unroll
            for (int x = 16; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            if (lane == 0) smem[L::red + warp * 2 * R + R + r] = sum;
        }
        copies_left<0>();
        __syncthreads();
        // ---- P V: warp w takes keys [32 w, 32 w + 32) of the pass, lanes along the features ----
#pragma unroll
        for (int r = 0; r < R; ++r) {
            l[r] *= corr[r];
#pragma unroll
            for (int w = 0; w < kWarps; ++w) l[r] += smem[L::red + w * 2 * R + R + r];
#pragma unroll
            for (int c = 0; c < kCols; ++c) acc[r][c] *= corr[r];
        }
        const int j_end = min(n, warp * 32 + 32);
#pragma unroll 8
        for (int j = warp * 32; j < j_end; ++j) {
            float v[kCols];
            load_vec<kCols>(v, smem + L::v + j * L::P + lane * kCols);
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const float p = smem[L::p + r * kChunk + j];
#pragma unroll
                for (int c = 0; c < kCols; ++c) acc[r][c] = p < 0.f ? acc[r][c] : fmaf(p, v[c], acc[r][c]);
            }
        }
        __syncthreads();                                      // the buffers are refilled
    }
    // ---- the warps' partial outputs, then the cluster's ----
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int c = 0; c < kCols; ++c) smem[L::k + (warp * R + r) * DP + lane * kCols + c] = acc[r][c];
    if (threadIdx.x == 0)
#pragma unroll
        for (int r = 0; r < R; ++r) {
            smem[L::ml + r] = m[r];
            smem[L::ml + R + r] = l[r];
        }
    __syncthreads();
    for (int u = threadIdx.x; u < R * DP; u += kThreads) {    // (each thread adds into the slot of warp 0 that it alone reads)
        float x = smem[L::out + u];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) x += smem[L::k + w * R * DP + u];
        smem[L::out + u] = x;
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int u = rank * kThreads + threadIdx.x; u < rows * DP; u += n_split * kThreads) {
        const int r = u / DP, d = u % DP;
        // every peer's values are asked for before the first is used: one trip through distributed shared memory, not one per peer
        float pm[kMaxSplit], pl[kMaxSplit], po[kMaxSplit];
#pragma unroll
        for (int p = 0; p < kMaxSplit; ++p)
            if (p < n_split) {
                const float* peer = cluster.map_shared_rank(smem, p);
                pm[p] = peer[L::ml + r];
                pl[p] = peer[L::ml + R + r];
                po[p] = peer[L::out + u];
            }
        float mx = -INFINITY, sum = 0.f, x = 0.f;
#pragma unroll
        for (int p = 0; p < kMaxSplit; ++p)
            if (p < n_split) mx = fmaxf(mx, pm[p]);
#pragma unroll
        for (int p = 0; p < kMaxSplit; ++p)
            if (p < n_split && mx > -INFINITY) {
                const float w = expf(pm[p] - mx);
                sum = fmaf(w, pl[p], sum);
                x = fmaf(w, po[p], x);
            }
        ((float*)a.o_out)[row_offset(r) + d] = sum > 0.f ? x / sum : 0.f;
        if (d == 0)
            a.lse_out[b * a.vlse.sb + (hk * group + r / s.Sq) * a.vlse.sh + (long long)(r % s.Sq) * a.vlse.ss] =
                sum > 0.f ? mx + logf(sum) : -INFINITY;
    }
    cluster.sync();                                           // no CTA leaves while another reads its shared memory
}

template <int DP, int R>
cudaError_t launch(const SimtArgs& a, cudaStream_t st)
{
    using L = DecodeSmem<DP, R>;
    auto kernel = simt_decode_kernel<DP, R>;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(kernel, L::bytes, configured);
    if (e != cudaSuccess) return e;
    // split the keys while CTAs are fewer than about three per SM and a piece keeps at least half a pass of keys
    const long long slabs = (long long)a.s.B * a.s.Hkv;
    int split = 1;
    while (split < kMaxSplit && slabs * split * 2 <= 3 * sm_count() && a.s.Skv >= split * kChunk) split *= 2;
    return launch_kernel(kernel, (unsigned)(slabs * split), kThreads, L::bytes, st, split, a, split);
}

template <int DP>
cudaError_t dispatch(const SimtArgs& a, cudaStream_t st)
{
    const int rows = a.s.Hq / a.s.Hkv * a.s.Sq;
    if (rows == 1) return launch<DP, 1>(a, st);
    if (rows == 2) return launch<DP, 2>(a, st);
    if (rows <= 4) return launch<DP, 4>(a, st);
    return launch<DP, 8>(a, st);
}

}  // namespace

// fp32 rows that are contiguous and 16-byte aligned, a head size that fills the lanes, and few enough rows for one key per
// thread to beat the 16-row tiles
bool simt_decode_supported(const SimtArgs& a)
{
    const long long slabs = (long long)a.s.B * a.s.Hkv;
    return !a.is_bf16 && a.s.causal && a.vec_q && a.vec_kv && (a.s.D == 32 || a.s.D == 64 || a.s.D == 128) &&
           a.s.Sq <= 8 && a.s.Hq / a.s.Hkv * (long long)a.s.Sq <= 8 && a.s.Skv > 2 * a.s.Sq && slabs * 8 <= 0x7fffffffLL;
}

cudaError_t simt_decode(const SimtArgs& a, cudaStream_t st)
{
    if (a.s.D == 32) return dispatch<32>(a, st);
    if (a.s.D == 64) return dispatch<64>(a, st);
    return dispatch<128>(a, st);
}

}  // namespace sntl
