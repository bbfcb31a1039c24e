// Exact-fp32 forward: O and LSE of a tile of 8*TM query rows per CTA, keys in tiles of 16*TN with an online softmax
// (same math as sentinel/NeuralNet/Layers/CausalSelfAttention.cpp:232-254, tiled like
// sentinel/NeuralNet/Cuda/CudaFlashAttention.cu:337-438).
//
// With only_odd it computes the blocks that the split products on the tensor cores leave (attn_f32_fwd_sm100.cu), and alone the calls
// that are too small for those, head_dim above 64 and bf16 tensors without a tensor-core kernel.
//
// Bound by the fp32 FMA pipes: 2*D FMAs per visible (query, key) pair.  B8 H12 S512 D64: 118 us, 1000 us with one warp per
// row.  Small grids (few heads, few
// new tokens behind a long cache) take smaller query tiles first and then a cluster of up to eight CTAs per query tile, each
// with every eighth key tile; their partial (m, l, O) are merged through distributed shared memory, without scratch or a
// second launch.
#include "attn_simt.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace sntl {
using namespace simt;
namespace {

template <int TM, int TN, int DP> struct FwdSmem {
    static constexpr int kRows = 8 * TM, kKeys = 16 * TN, P = DP + 4;
    static constexpr int q = 0, k = q + kRows * P, v = k + kKeys * P, w = v + kKeys * P, ml = w + kKeys * (kRows + 4);
    static constexpr size_t bytes = (ml + 2 * kRows) * sizeof(float);
};

// kSplit: gridDim.x counts clusters of `n_split` CTAs that share one query tile
template <typename T, int TM, int TN, int DP, bool kSplit>
__global__ void __launch_bounds__(kThreads, DP <= 64 ? 3 : 2) simt_fwd_kernel(const SimtArgs a, int n_qt, int n_split)
{
    using L = FwdSmem<TM, TN, DP>;
    using M = OutMap<DP>;
    extern __shared__ __align__(16) float smem[];
    wait_for_stream();
    const AttnShape& s = a.s;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int tile = kSplit ? blockIdx.x / n_split : blockIdx.x, rank = kSplit ? blockIdx.x - tile * n_split : 0;
    const int slabs = s.B * s.Hq, bh = tile % slabs, b = bh / s.Hq, h = bh - b * s.Hq, hk = h / (s.Hq / s.Hkv);
    const int qt = n_qt - 1 - tile / slabs;                   // longest query tiles first
    const int row0 = qt * L::kRows;
    // (every row carries the mark, and only its tile's CTA or cluster overwrites it, after all of that have looked)
    if (a.only_odd && __float_as_uint(a.lse_out[b * a.vlse.sb + h * a.vlse.sh + (long long)row0 * a.vlse.ss]) != kOddLse) return;
    const T* kb = (const T*)a.k + b * a.vkv.sb + hk * a.vkv.sh;
    const T* vb = (const T*)a.v + b * a.vkv.sb + hk * a.vkv.sh;
    const Slab mq{a.vq.ss, a.vq.sd, s.Sq, s.D, a.vec_q}, mk{a.vkv.ss, a.vkv.sd, s.Skv, s.D, a.vec_kv};
    stage<T, DP, L::kRows>(smem + L::q, (const T*)a.q + b * a.vq.sb + h * a.vq.sh, mq, row0);

    const int shift = s.causal ? s.Skv - s.Sq : 0;            // query row r sits at position r + shift (new tokens after a KV cache)
    const int n_keys = visible_keys(s, min(row0 + L::kRows, s.Sq) - 1);   // keys any row of the tile can see
    float m[TM], l[TM];
    float2 o[TM / 2][M::N];
    clear(o);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
    for (int k0 = rank * L::kKeys; k0 < n_keys; k0 += (kSplit ? n_split : 1) * L::kKeys) {
        // tiles between the global tokens and the window of the first row are visible to no row
        if (s.window > 0 && k0 >= s.global_tokens && k0 + L::kKeys - 1 < row0 + shift - s.window + 1) continue;
        __syncthreads();
        stage<T, DP, L::kKeys>(smem + L::k, kb, mk, k0);
        const float z = stage<T, DP, L::kKeys>(smem + L::v, vb, mk, k0);
        const bool cut = k0 + L::kKeys > visible_keys(s, row0) || s.window > 0;   // some (row, key) pair may be hidden
        bool odd = false;                                     // ... and V holds values that are not finite
        if (cut) odd = __syncthreads_or(z != 0.f);
        else __syncthreads();
        float sc[TM][TN];
        scores<TM, TN, DP>(sc, smem + L::q, smem + L::k);
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int row = row0 + ty + 8 * i, n_row = cut ? visible_keys(s, row) : 0;
            float mx = m[i];
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int key = k0 + tx + 16 * j;
                sc[i][j] = (cut && (key >= n_row || !window_allows(s, row + shift, key))) ? -INFINITY : sc[i][j] * s.scale;
                mx = fmaxf(mx, sc[i][j]);
            }
#pragma unroll
            for (int x = 1; x < 16; x <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, x));
            const float ref = mx == -INFINITY ? 0.f : mx;     // nothing visible yet: every weight is 0
            const float corr = expf(m[i] - ref);
            m[i] = mx;
            l[i] *= corr;
#pragma unroll
            for (int n = 0; n < M::N; ++n) (i & 1 ? o[i / 2][n].y : o[i / 2][n].x) *= corr;
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                sc[i][j] = expf(sc[i][j] - ref);
                l[i] += sc[i][j];
            }
        }
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            float w[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) w[i] = sc[i][j];
            put_weights<TM>(smem + L::w, tx + 16 * j, w);
        }
        __syncwarp();
        if (!odd) {
            outputs<TM, DP, L::kKeys>(o, smem + L::w, smem + L::v);
        } else {
            outputs_visible<TM, DP, L::kKeys>(o, smem + L::w, smem + L::v, [&](int i, int k) {
                const int row = row0 + ty + 8 * i, key = k0 + k;
                return key < visible_keys(s, row) && window_allows(s, row + shift, key);
            });
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int x = 1; x < 16; x <<= 1) l[i] += __shfl_xor_sync(0xffffffffu, l[i], x);

    T* ob = (T*)a.o_out + b * a.vq.sb + h * a.vq.sh;
    float* lse = a.lse_out + b * a.vlse.sb + h * a.vlse.sh;
    if constexpr (!kSplit) {
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
#pragma unroll
            for (int n = 0; n < M::N; ++n) (i & 1 ? o[i / 2][n].y : o[i / 2][n].x) *= inv;
            const int row = row0 + ty + 8 * i;
            if (tx == 0 && row < s.Sq) lse[(long long)row * a.vlse.ss] = l[i] > 0.f ? m[i] + logf(l[i]) : -INFINITY;
        }
        __syncthreads();                                      // the Q tile has been read for the last time
        store_rows<T, TM, DP>(ob, mq, row0, o, smem + L::q);
    } else {
        cg::cluster_group cluster = cg::this_cluster();
        __syncthreads();
#pragma unroll
        for (int i = 0; i < TM; ++i) {
#pragma unroll
            for (int n = 0; n < M::N; ++n) smem[L::q + (ty + 8 * i) * L::P + M::col(n)] = i & 1 ? o[i / 2][n].y : o[i / 2][n].x;
            if (tx == 0) {
                smem[L::ml + ty + 8 * i] = m[i];
                smem[L::ml + L::kRows + ty + 8 * i] = l[i];
            }
        }
        cluster.sync();
        // the rows of the tile are dealt to the CTAs of the cluster; 16-byte units of a row to its threads
        constexpr int kUnits = DP / 4;
        const int rows_mine = (L::kRows - rank + n_split - 1) / n_split;
        for (int u = threadIdx.x; u < rows_mine * kUnits; u += kThreads) {
            const int r = rank + (u / kUnits) * n_split, d = (u % kUnits) * 4, row = row0 + r;
            if (row >= s.Sq || d >= s.D) continue;
            float mx = -INFINITY, sum = 0.f;
            for (int p = 0; p < n_split; ++p) mx = fmaxf(mx, cluster.map_shared_rank(smem, p)[L::ml + r]);
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
            for (int p = 0; p < n_split && mx > -INFINITY; ++p) {
                const float* peer = cluster.map_shared_rank(smem, p);
                const float w = expf(peer[L::ml + r] - mx);
                const float4 y = *reinterpret_cast<const float4*>(peer + L::q + r * L::P + d);
                sum = fmaf(w, peer[L::ml + L::kRows + r], sum);
                x = make_float4(fmaf(w, y.x, x.x), fmaf(w, y.y, x.y), fmaf(w, y.z, x.z), fmaf(w, y.w, x.w));
            }
            const float inv = sum > 0.f ? 1.f / sum : 0.f;
            const float out[4] = {x.x * inv, x.y * inv, x.z * inv, x.w * inv};
            for (int i = 0; i < 4 && d + i < s.D; ++i) Elem<T>::store(ob + row * mq.ss + (d + i) * mq.sd, out[i]);
            if (d == 0) lse[(long long)row * a.vlse.ss] = sum > 0.f ? mx + logf(sum) : -INFINITY;
        }
        cluster.sync();                                       // no CTA leaves while another reads its shared memory
    }
}

template <typename T, int TM, int TN, int DP, bool kSplit>
cudaError_t launch(const SimtArgs& a, int n_qt, int n_split, cudaStream_t st)
{
    constexpr size_t smem = FwdSmem<TM, TN, DP>::bytes;
    auto kernel = simt_fwd_kernel<T, TM, TN, DP, kSplit>;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(kernel, smem, configured);
    if (e != cudaSuccess) return e;
    const long long ctas = (long long)n_qt * a.s.B * a.s.Hq * n_split;
    if (ctas > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    return launch_kernel(kernel, (unsigned)ctas, kThreads, smem, st, kSplit ? n_split : 1, a, n_qt, n_split);
}

template <typename T, int DP>
cudaError_t dispatch(const SimtArgs& a, cudaStream_t st)
{
    constexpr int TN = DP <= 64 ? 4 : 2, kTop = DP <= 64 ? 8 : 4;
    const SimtTiles t = simt_forward_tiles(a.s);
    const int n_qt = (a.s.Sq + t.rows - 1) / t.rows;
    if (kTop == 8 && t.rows == 64) return launch<T, kTop, TN, DP, false>(a, n_qt, 1, st);
    if (t.rows == 32) return launch<T, 4, TN, DP, false>(a, n_qt, 1, st);
    return t.split > 1 ? launch<T, 2, TN, DP, true>(a, n_qt, t.split, st) : launch<T, 2, TN, DP, false>(a, n_qt, 1, st);
}

template <typename T>
cudaError_t dispatch_dim(const SimtArgs& a, cudaStream_t st)
{
    if (a.s.D <= 16) return dispatch<T, 16>(a, st);
    if (a.s.D <= 32) return dispatch<T, 32>(a, st);
    if (a.s.D <= 64) return dispatch<T, 64>(a, st);
    if (a.s.D <= 96) return dispatch<T, 96>(a, st);
    if (a.s.D <= 128) return dispatch<T, 128>(a, st);
    return dispatch<T, 256>(a, st);
}

}  // namespace

// Tile height: 64 rows keep the FMA pipes busiest, but a grid that does not give every SM a CTA or two loses more than the
// smaller tiles cost.  After the smallest tile, the keys are split as well.
SimtTiles simt_forward_tiles(const AttnShape& s)
{
    const bool tall = s.D <= 64;
    const long long slabs = (long long)s.B * s.Hq;
    auto tiles = [&](int rows) { return (s.Sq + rows - 1) / rows; };
    const int sms = sm_count(), keys = tall ? 64 : 32;
    if (tall && tiles(64) * slabs >= 2 * sms) return SimtTiles{64, 1};
    if (tiles(32) * slabs >= 2 * sms) return SimtTiles{32, 1};
    const long long ctas = tiles(16) * slabs;
    const int key_tiles = (s.Skv + keys - 1) / keys;
    int split = 1;
    while (split < 8 && ctas * split * 2 <= 3 * sms && split * 2 <= key_tiles) split *= 2;
    return SimtTiles{16, split};
}

cudaError_t simt_forward(const SimtArgs& a, cudaStream_t st)
{
    if (!a.only_odd && simt_decode_supported(a)) return simt_decode(a, st);
    return a.is_bf16 ? dispatch_dim<__nv_bfloat16>(a, st) : dispatch_dim<float>(a, st);
}

}  // namespace sntl
