// Exact-fp32 backward: one launch whose CTAs have one of two roles.
//   dK/dV   8*TM key rows of one (batch, KV head); visits the query tiles that see them, for every query head of the group:
//           S^T, dP^T, then dV += P^T dO and dK += dS^T Q.  One owner per element: deterministic, no atomics.
//   dQ      8*TM query rows of one (batch, head); visits the key tiles they see: S, dP, then dQ += dS K.
// (sentinel/NeuralNet/Layers/CausalSelfAttention.cpp:333-352.)  Both recompute P from the saved log-sum-exp and take
// delta = rowsum(dO o O) from the O rows that are read along with dO: 1/64 of a tile's FMAs instead of a launch of its own.
// Seven products where a backward with dQ reductions needs five, but dQ stays reproducible without scratch.
//
// With odd_marks it computes the blocks that the split products on the tensor cores leave (attn_f32_bwd_sm100.cu), and alone the calls
// that are too small for those, head_dim above 64 and bf16 tensors without a tensor-core kernel.
//
// Bound by the fp32 FMA pipes (B8 H12 S512 D64: 404 us against 195 us of packed FMAs at the 112 lanes per clock that they
// reach in isolation; staging and exponentials are 10 % each, the rest is shared-memory latency at eight warps per SM; 2740 us
// with one warp per row).  Twice the warps with half the rows each take as long: they load twice as much per FMA.  The dK/dV CTAs come first: they are the longer ones (four products per pair against three,
// times the heads of the group).
#include "attn_simt.cuh"

namespace sntl {
using namespace simt;
namespace {

template <int TM, int TN, int DP> struct BwdSmem {
    static constexpr int kRows = 8 * TM, kLoop = 16 * TN, P = DP + 4;
    // own rows (K, V or Q, dO), loop rows (Q, dO or K, V), P and dS weights, partial sums of delta, per-row terms
    static constexpr int own0 = 0, own1 = own0 + kRows * P, in0 = own1 + kRows * P, in1 = in0 + kLoop * P;
    static constexpr int w0 = in1 + kLoop * P, w1 = w0 + kLoop * (kRows + 4);
    static constexpr int kDeltaRows = kRows > kLoop ? kRows : kLoop;
    static constexpr int part = w1 + kLoop * (kRows + 4), lse = part + kDeltaRows * (DP / 4 + 1), delta = lse + kDeltaRows;
    static constexpr size_t bytes = (delta + kDeltaRows) * sizeof(float);
};

// outputs_visible as a function of its own, with the sums handed over in memory: inlined, it costs the kernel registers where it never
// runs (B8 H12 S512 D64 410 us without it, 447 inlined, 412 so).
template <int TM, int DP, int K, typename F>
__device__ __noinline__ void outputs_visible_call(float2* sums, const float* W, const float* B, F visible)
{
    using M = OutMap<DP>;
    for (int i = 0; i < TM; ++i)
        for (int n = 0; n < M::N; ++n) {
            float2& sum = sums[i / 2 * M::N + n];
            float a = i & 1 ? sum.y : sum.x;
            for (int k = 0; k < K; ++k)
                if (visible(i, k)) a = fmaf(W[k * (8 * TM + 4) + (threadIdx.x >> 4) * TM + i], B[k * (DP + 4) + M::col(n)], a);
            (i & 1 ? sum.y : sum.x) = a;
        }
}
template <int TM, int DP, int K, typename F>
__device__ __forceinline__ void outputs_visible_apart(float2 (&acc)[TM / 2][OutMap<DP>::N], const float* W, const float* B, F visible)
{
    constexpr int N = OutMap<DP>::N;
    float2 sums[TM / 2 * N];
#pragma unroll
    for (int i = 0; i < TM / 2 * N; ++i) sums[i] = acc[i / N][i % N];
    outputs_visible_call<TM, DP, K>(sums, W, B, visible);
#pragma unroll
    for (int i = 0; i < TM / 2 * N; ++i) acc[i / N][i % N] = sums[i];
}

template <typename T, int TM, int TN, int DP>
__device__ __forceinline__ void dkv_role(const SimtArgs& a, int tile, float* smem)
{
    using L = BwdSmem<TM, TN, DP>;
    using M = OutMap<DP>;
    const AttnShape& s = a.s;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4, group = s.Hq / s.Hkv;
    const int slabs = s.B * s.Hkv, slab = tile % slabs, b = slab / s.Hkv, hk = slab - b * s.Hkv;
    const int key0 = (tile / slabs) * L::kRows;               // causal: the first key tiles are seen by the most queries
    const Slab mq{a.vq.ss, a.vq.sd, s.Sq, s.D, a.vec_q}, mk{a.vkv.ss, a.vkv.sd, s.Skv, s.D, a.vec_kv};
    const long long kvoff = b * a.vkv.sb + hk * a.vkv.sh;
    stage<T, DP, L::kRows>(smem + L::own0, (const T*)a.k + kvoff, mk, key0);
    stage<T, DP, L::kRows>(smem + L::own1, (const T*)a.v + kvoff, mk, key0);
    float2 dk[TM / 2][M::N], dv[TM / 2][M::N];
    clear(dk);
    clear(dv);

    const int shift = s.Skv - s.Sq;                           // first query that sees key j: j - shift
    const int q_first = s.causal ? max(0, key0 - shift) / L::kLoop * L::kLoop : 0;
    for (int g = 0; g < group; ++g) {
        const int h = hk * group + g;
        const long long qoff = b * a.vq.sb + h * a.vq.sh;
        for (int q0 = q_first; q0 < s.Sq; q0 += L::kLoop) {
            // past the window of the last key (and no key is global): no later query sees these keys
            if (s.window > 0 && key0 >= s.global_tokens && q0 + shift > key0 + L::kRows - 1 + s.window - 1) break;
            __syncthreads();
            stage<T, DP, L::kLoop>(smem + L::in0, (const T*)a.q + qoff, mq, q0);
            stage_with_delta<T, DP, L::kLoop>(smem + L::in1, smem + L::part, (const T*)a.dout + qoff, (const T*)a.o + qoff, mq, q0);
            if (threadIdx.x < L::kLoop) {
                const int r = q0 + threadIdx.x;
                smem[L::lse + threadIdx.x] = r < s.Sq ? a.lse[b * a.vlse.sb + h * a.vlse.sh + (long long)r * a.vlse.ss] : -INFINITY;
            }
            __syncthreads();
            if (threadIdx.x < L::kLoop) smem[L::delta + threadIdx.x] = delta_of<DP>(smem + L::part, threadIdx.x);
            float p[TM][TN], ds[TM][TN];
            scores<TM, TN, DP>(p, smem + L::own0, smem + L::in0);
            scores<TM, TN, DP>(ds, smem + L::own1, smem + L::in1);
            __syncthreads();
            // every (query, key) pair of the tile is visible: no masks
            const bool cut = (s.causal && q0 + shift < key0 + L::kRows - 1) || s.window > 0 || key0 + L::kRows > s.Skv;
            const bool odd = cut && not_finite(p, ds, smem + L::delta);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const int q = q0 + tx + 16 * j;
                const float lse = smem[L::lse + tx + 16 * j], delta = smem[L::delta + tx + 16 * j];
                float wp[TM], ws[TM];
#pragma unroll
                for (int i = 0; i < TM; ++i) {
                    const int key = key0 + ty + 8 * i;
                    const bool vis = lse > -INFINITY && (!cut || ((!s.causal || key <= q + shift) && window_allows(s, q + shift, key)));
                    wp[i] = vis ? expf(fmaf(p[i][j], s.scale, -lse)) : 0.f;
                    ws[i] = wp[i] * (ds[i][j] - delta) * s.scale;
                }
                put_weights<TM>(smem + L::w0, tx + 16 * j, wp);
                put_weights<TM>(smem + L::w1, tx + 16 * j, ws);
            }
            __syncwarp();
            if (!odd) {
                outputs<TM, DP, L::kLoop>(dv, smem + L::w0, smem + L::in1);
                outputs<TM, DP, L::kLoop>(dk, smem + L::w1, smem + L::in0);
            } else {
                auto visible = [=](int i, int k) {
                    const int key = key0 + ty + 8 * i, q = q0 + k;
                    return q < s.Sq && (!s.causal || key <= q + shift) && window_allows(s, q + shift, key);
                };
                outputs_visible_apart<TM, DP, L::kLoop>(dv, smem + L::w0, smem + L::in1, visible);
                outputs_visible_apart<TM, DP, L::kLoop>(dk, smem + L::w1, smem + L::in0, visible);
            }
        }
    }
    __syncthreads();
    store_rows<T, TM, DP>((T*)a.dk + kvoff, mk, key0, dk, smem + L::own0);
    store_rows<T, TM, DP>((T*)a.dv + kvoff, mk, key0, dv, smem + L::own1);
}

template <typename T, int TM, int TN, int DP>
__device__ __forceinline__ void dq_role(const SimtArgs& a, int tile, int n_qt, float* smem)
{
    using L = BwdSmem<TM, TN, DP>;
    using M = OutMap<DP>;
    const AttnShape& s = a.s;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int slabs = s.B * s.Hq, bh = tile % slabs, b = bh / s.Hq, h = bh - b * s.Hq, hk = h / (s.Hq / s.Hkv);
    const int row0 = (n_qt - 1 - tile / slabs) * L::kRows;    // longest query tiles first
    const Slab mq{a.vq.ss, a.vq.sd, s.Sq, s.D, a.vec_q}, mk{a.vkv.ss, a.vkv.sd, s.Skv, s.D, a.vec_kv};
    const long long qoff = b * a.vq.sb + h * a.vq.sh;
    const T* kb = (const T*)a.k + b * a.vkv.sb + hk * a.vkv.sh;
    const T* vb = (const T*)a.v + b * a.vkv.sb + hk * a.vkv.sh;
    stage<T, DP, L::kRows>(smem + L::own0, (const T*)a.q + qoff, mq, row0);
    stage_with_delta<T, DP, L::kRows>(smem + L::own1, smem + L::part, (const T*)a.dout + qoff, (const T*)a.o + qoff, mq, row0);
    __syncthreads();
    float lse[TM], delta[TM];
    float2 dq[TM / 2][M::N];
    clear(dq);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int row = row0 + ty + 8 * i;
        lse[i] = row < s.Sq ? a.lse[b * a.vlse.sb + h * a.vlse.sh + (long long)row * a.vlse.ss] : -INFINITY;
        delta[i] = delta_of<DP>(smem + L::part, ty + 8 * i);
    }
    const int shift = s.causal ? s.Skv - s.Sq : 0;
    const int n_keys = visible_keys(s, min(row0 + L::kRows, s.Sq) - 1);
    for (int k0 = 0; k0 < n_keys; k0 += L::kLoop) {
        // tiles between the global tokens and the window of the first row are visible to no row
        if (s.window > 0 && k0 >= s.global_tokens && k0 + L::kLoop - 1 < row0 + shift - s.window + 1) continue;
        __syncthreads();
        stage<T, DP, L::kLoop>(smem + L::in0, kb, mk, k0);
        stage<T, DP, L::kLoop>(smem + L::in1, vb, mk, k0);
        __syncthreads();
        float p[TM][TN], ds[TM][TN];
        scores<TM, TN, DP>(p, smem + L::own0, smem + L::in0);
        scores<TM, TN, DP>(ds, smem + L::own1, smem + L::in1);
        const bool cut = k0 + L::kLoop > visible_keys(s, row0) || s.window > 0, odd = cut && not_finite(p, ds, nullptr);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int key = k0 + tx + 16 * j;
            float w[TM];
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const int row = row0 + ty + 8 * i;
                const bool vis = lse[i] > -INFINITY && (!cut || (key < visible_keys(s, row) && window_allows(s, row + shift, key)));
                const float x = vis ? expf(fmaf(p[i][j], s.scale, -lse[i])) : 0.f;
                w[i] = x * (ds[i][j] - delta[i]) * s.scale;
            }
            put_weights<TM>(smem + L::w0, tx + 16 * j, w);
        }
        __syncwarp();
        if (!odd) {
            outputs<TM, DP, L::kLoop>(dq, smem + L::w0, smem + L::in0);
        } else {
            outputs_visible_apart<TM, DP, L::kLoop>(dq, smem + L::w0, smem + L::in0, [=](int i, int k) {
                const int row = row0 + ty + 8 * i, key = k0 + k;
                return key < visible_keys(s, row) && window_allows(s, row + shift, key);
            });
        }
    }
    __syncthreads();
    store_rows<T, TM, DP>((T*)a.dq + qoff, mq, row0, dq, smem + L::own0);
}

// CTAs beside each other that shared memory allows and registers can follow without spilling (left to the compiler, 16-row tiles at
// head_dim 128 take 254 registers and run two beside each other: B4 H8 S256 119 -> 143 us)
template <int TM, int DP> constexpr int kMinCtas = TM == 2 ? (DP == 16 ? 4 : DP <= 128 ? 3 : 1) : TM == 4 && (DP <= 32 || DP == 96) ? 3 : 1;

template <typename T, int TM, int TN, int DP>
__global__ void __launch_bounds__(kThreads, kMinCtas<TM, DP>) simt_bwd_kernel(const SimtArgs a, int n_dkv, int n_qt)
{
    extern __shared__ __align__(16) float smem[];
    wait_for_stream();
    if (a.odd_marks) {      // (here and not in the roles, whose loops it would cost registers: B1 Hq8 Hkv2 S512 D128 465 us, as without marks, and 470)
        const AttnShape& s = a.s;
        const bool dkv = (int)blockIdx.x < n_dkv;
        const int slabs = s.B * (dkv ? s.Hkv : s.Hq), tile = dkv ? blockIdx.x : blockIdx.x - n_dkv;
        const int row0 = (dkv ? tile / slabs : n_qt - 1 - tile / slabs) * 8 * TM, first = dkv ? 0 : (s.Skv + 127) / 128 * (s.B * s.Hkv);
        if (a.odd_marks[first + row0 / 128 * slabs + tile % slabs] == 0) return;
    }
    if ((int)blockIdx.x < n_dkv) dkv_role<T, TM, TN, DP>(a, blockIdx.x, smem);
    else dq_role<T, TM, TN, DP>(a, blockIdx.x - n_dkv, n_qt, smem);
}

template <typename T, int TM, int TN, int DP>
cudaError_t launch(const SimtArgs& a, cudaStream_t st)
{
    using L = BwdSmem<TM, TN, DP>;
    auto kernel = simt_bwd_kernel<T, TM, TN, DP>;
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(kernel, L::bytes, configured);
    if (e != cudaSuccess) return e;
    const int n_qt = (a.s.Sq + L::kRows - 1) / L::kRows, n_kt = (a.s.Skv + L::kRows - 1) / L::kRows;
    const long long n_dkv = (long long)n_kt * a.s.B * a.s.Hkv, n_dq = (long long)n_qt * a.s.B * a.s.Hq;
    if (n_dkv + n_dq > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    return launch_kernel(kernel, (unsigned)(n_dkv + n_dq), kThreads, L::bytes, st, 1, a, (int)n_dkv, n_qt);
}

template <typename T, int DP>
cudaError_t dispatch(const SimtArgs& a, cudaStream_t st)
{
    constexpr int TN = DP <= 64 ? 4 : 2, kTop = DP <= 64 ? 8 : 4;
    const int rows = simt_backward_rows(a.s);
    if (kTop == 8 && rows == 64) return launch<T, kTop, TN, DP>(a, st);
    return rows == 32 ? launch<T, 4, TN, DP>(a, st) : launch<T, 2, TN, DP>(a, st);
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

// Tile height as in the forward: the largest whose grid still gives every SM its two resident CTAs.
int simt_backward_rows(const AttnShape& s)
{
    auto ctas = [&](int rows) { return ((s.Sq + rows - 1) / rows * (long long)s.Hq + (s.Skv + rows - 1) / rows * (long long)s.Hkv) * s.B; };
    const int sms = sm_count();
    if (s.D <= 64 && ctas(64) >= 4 * sms) return 64;
    return ctas(32) >= 4 * sms ? 32 : 16;
}

cudaError_t simt_backward(const SimtArgs& a, cudaStream_t st)
{
    return a.is_bf16 ? dispatch_dim<__nv_bfloat16>(a, st) : dispatch_dim<float>(a, st);
}

}  // namespace sntl
