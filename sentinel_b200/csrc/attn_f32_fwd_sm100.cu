// Exact-fp32 forward on the tensor cores (attn_f32_sm100.cuh says how): 128 query rows of one (batch, head) per CTA, keys in tiles of
// 128 with an online softmax, head_dim up to 64.
//
//   warps 0-7   sums: thread = one query row and half the columns (64 keys of a tile, 32 features of O).  Scores from TMEM, weights as
//               three bf16 parts back to TMEM, and the product of the tile before into O, which stays in registers.
//   warps 8-13  stage: fp32 rows of Q, K, V (either layout) -> parts in shared memory.
//   warp 14     issues the products.
//
// S = Q K^T takes six products of 64 terms into one accumulator.  For P V the parts of V lie beside each other as 192 columns:
// P_h meets all of them, P_m two, P_l one; a step of 16 keys costs 222 cycles instead of 360 for six products of 64 columns, and the
// three column groups (hh | hm, mh | hl, mm, lh) are accumulators of their own.
// A CTA takes over blocks (BlockQueue).  B8 H12 S512 D64: 42 us; 48 with a block per CTA, whose set-up and first loads then cost as much as
// two of its tiles; 118 with the FMA kernels.  What bounds it is the staging warps' rate (a tile of K or V: 4300 cycles), then the
// products (3300 per pair of tiles).
// TMEM: S [0, 128), parts of P [128, 320), P V [320, 512).
#include "attn_f32_sm100.cuh"

namespace sntl {
using namespace f32tc;
using namespace ptx;
namespace {

constexpr int kKeys = 128, kTileBytes = kOwnRows * kRowBytes, kParts = 3 * kTileBytes;
constexpr uint32_t kColS = 0, kColP = 128, kColO = 320;
constexpr int kSumRegs = 144;

struct Bars {
    Queue queue;
    uint64_t q_free, k_full[2], k_free[2], v_full[2], v_free[2], s_full, s_free, p_full, o_full, pair[4];   // (V: its two halves)
    uint32_t tmem_base, abort_flag;
    OddBlocks odd;
};
struct Smem {
    static constexpr int q = 0, k = kParts, v = 3 * kParts, exchange = 4 * kParts, bars = exchange + 2 * 2 * kOwnRows * 4;
    static constexpr int bytes = bars + (int)sizeof(Bars) + 1024;
};
static_assert(Smem::bytes <= 227 * 1024, "");

// A row's two threads exchange a value, for the n-th time.  (A barrier in memory: its wait is bounded.)
__device__ __forceinline__ bool other_half(Bars* bars, float* exchange, int n, int half, int row, float x, float& y)
{
    float* at = exchange + (n & 1) * 2 * kOwnRows + row;
    at[half * kOwnRows] = x;
    mbar_arrive(&bars->pair[row >> 5]);
    const bool ok = mbar_wait_warp(&bars->pair[row >> 5], n & 1, &bars->abort_flag, 9);
    y = at[(half ^ 1) * kOwnRows];
    return ok;
}

struct Block {
    int b, h, hk, row0, shift, n_keys;

    __device__ __forceinline__ Block(const AttnShape& s, int block, int n_qt)
    {
        const int slabs = s.B * s.Hq, bh = block % slabs;
        b = bh / s.Hq;
        h = bh - b * s.Hq;
        hk = h / (s.Hq / s.Hkv);
        row0 = (n_qt - 1 - block / slabs) * kOwnRows;        // longest query tiles first
        shift = s.causal ? s.Skv - s.Sq : 0;                 // query row r sits at position r + shift
        n_keys = s.causal ? min(min(row0 + kOwnRows, s.Sq) + shift, s.Skv) : s.Skv;
    }
    // k0, or the first key tile after it that some row sees (those between the global tokens and the window of the first row: none)
    __device__ __forceinline__ int tile(const AttnShape& s, int k0) const
    {
        while (s.window > 0 && k0 < n_keys && k0 >= s.global_tokens && k0 + kKeys - 1 < row0 + shift - s.window + 1) k0 += kKeys;
        return k0;
    }
};

template <bool kVec> __global__ void __launch_bounds__(kThreads, 1) f32_fwd_kernel(const SimtArgs a, int n_qt)
{
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + (1024 - (smem_u32(raw) & 1023)) % 1024;
    Bars* bars = reinterpret_cast<Bars*>(smem + Smem::bars);
    float* exchange = reinterpret_cast<float*>(smem + Smem::exchange);
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        bars->queue.init();
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->k_full[i], kStageThreads);
            mbar_init(&bars->k_free[i], 1);
            mbar_init(&bars->v_full[i], kStageThreads);
            mbar_init(&bars->v_free[i], 1);
        }
        mbar_init(&bars->q_free, 1);
        mbar_init(&bars->s_full, 1);
        mbar_init(&bars->s_free, kSumThreads);
        mbar_init(&bars->p_full, kSumThreads);
        mbar_init(&bars->o_full, 2);      // the product, and what the issuing warp has seen of the staging warps
        for (int i = 0; i < 4; ++i) {
            mbar_init(&bars->pair[i], 64);
            bars->odd.number[i] = 0;
        }
        bars->abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == kIssueWarp) {
        tmem_alloc(&bars->tmem_base, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    volatile uint32_t* abort_flag = &bars->abort_flag;
    wait_for_stream();

    // Counters of key tiles run on over the blocks: c for this block's tile.
    const AttnShape& s = a.s;
    if (warp < 8) {
        setmaxnreg_inc<kSumRegs>();
        const int half = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(warp & 3) << 21);
        const float2 scale = make_float2(s.scale, s.scale);
        int c = 0, exchanges = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(s, block, n_qt);
            const int row = w.row0 + r, n_row = s.causal ? min(row + w.shift + 1, s.Skv) : s.Skv;
            const int n_first = s.causal ? min(w.row0 + w.shift + 1, s.Skv) : s.Skv;
            // Largest score before scaling (kHidden: no key seen yet).  It is subtracted before scaling: the largest weight is 1 whatever the
            // size of the scores.  (Subtracted afterwards, with one FMA, it left exp of the rounding error of the scaled score, half a unit in
            // its last place: infinity or 0 from 2^31 on.)
            float top = kHidden, l = 0.f, corr = 1.f;
            float2 o[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = make_float2(0.f, 0.f);
            auto add_product = [&]() {      // O so far is relative to the reference before the last one
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    uint32_t g[3][8];
#pragma unroll
                    for (int p = 0; p < 3; ++p) tmem_ld8(lanes + kColO + p * 64 + half * 32 + x * 8, g[p]);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        auto pair = [&](int p) { return make_float2(__uint_as_float(g[p][2 * i]), __uint_as_float(g[p][2 * i + 1])); };
                        o[x * 4 + i] = ffma2(o[x * 4 + i], make_float2(corr, corr), fadd2(pair(0), fadd2(pair(1), pair(2))));
                    }
                }
            };
            bool ok = true, started = false;
            for (int k0 = w.tile(s, 0); k0 < w.n_keys; k0 = w.tile(s, k0 + kKeys), ++c, started = true) {
                if (!(ok = mbar_wait_warp(&bars->s_full, c & 1, abort_flag, 1))) break;
                tc_fence_after();
                float2 x[32];
                tmem_ld32(lanes + kColS + half * 64, reinterpret_cast<uint32_t*>(x));
                tmem_ld32(lanes + kColS + half * 64 + 32, reinterpret_cast<uint32_t*>(x) + 32);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(&bars->s_free);
                if (k0 + kKeys > n_first || s.window > 0) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        const uint32_t seen = keys_seen(s, row + w.shift, n_row, k0 + half * 64 + j * 32);
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            float2& y = x[j * 16 + i];
                            if (!(seen & (1u << (2 * i)))) y.x = kHidden;
                            if (!(seen & (2u << (2 * i)))) y.y = kHidden;
                        }
                    }
                }
                float mx[2] = {top, top};
#pragma unroll
                for (int i = 0; i < 32; ++i) mx[i & 1] = fmax3(mx[i & 1], x[i].x, x[i].y);
                float other;
                if (!(ok = other_half(bars, exchange, exchanges++, half, r, fmaxf(mx[0], mx[1]), other))) break;
                const float before = top;
                top = fmax3(mx[0], mx[1], other);
                const float sub = top <= 0.5f * kHidden ? 0.f : -top;
                const float next_corr = exp_pair(make_float2((before - top) * s.scale, 0.f)).x;
                float2 sum[4] = {};
#pragma unroll
                for (int i = 0; i < 32; ++i) {
                    x[i] = exp_pair<true>(fmul2(fadd2(x[i], make_float2(sub, sub)), scale));
                    sum[i % 4] = fadd2(sum[i % 4], x[i]);
                }
                const float2 all = fadd2(fadd2(sum[0], sum[1]), fadd2(sum[2], sum[3]));
                l = fmaf(l, next_corr, all.x + all.y);
                if (started) {
                    if (!(ok = mbar_wait_warp(&bars->o_full, (c - 1) & 1, abort_flag, 2))) break;
                    tc_fence_after();
                    add_product();
                }
                corr = next_corr;
                put_parts<32, 64>(lanes + kColP + half * 32, x);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&bars->p_full);
            }
            if (!ok || !mbar_wait_warp(&bars->o_full, (c - 1) & 1, abort_flag, 2)) break;
            tc_fence_after();
            add_product();
            tc_fence_before();
            float other;
            if (!other_half(bars, exchange, exchanges++, half, r, l, other)) break;
            l += other;
            // A block with odd values is left to the FMA kernels, which find the mark in its LSE rows.
            const bool odd = bars->odd.get(u);
            if (!odd)
                store_row((float*)a.o_out + w.b * a.vq.sb + w.h * a.vq.sh, a.vq.ss, a.vq.sd, s.Sq, s.D, a.vec_q, row, half * 32, o, l > 0.f ? 1.f / l : 0.f);
            if (half == 0 && row < s.Sq)
                a.lse_out[w.b * a.vlse.sb + w.h * a.vlse.sh + (long long)row * a.vlse.ss] =
                    odd ? __uint_as_float(kOddLse) : l > 0.f ? fmaf(top, s.scale, logf(l * kDown)) : -INFINITY;
        }
    } else if (warp < kIssueWarp) {
        setmaxnreg_dec<other_regs(kSumRegs)>();
        const int t = threadIdx.x - kSumThreads;
        const Share<kVec> share(t, (int)a.vq.ss, (int)a.vq.sd, s.D);
        int c_k = 0, c_v = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(s, block, n_qt);
            const float* q = (const float*)a.q + w.b * a.vq.sb + w.h * a.vq.sh;
            const float* k = (const float*)a.k + w.b * a.vkv.sb + w.hk * a.vkv.sh;
            const float* v = (const float*)a.v + w.b * a.vkv.sb + w.hk * a.vkv.sh;
            Check check;
            // Q, K_0, K_1, V_0, K_2, V_1, ...: half tiles, of which one is on its way while the one before is split.  (One loop for all
            // of them: unrolled for each, the code of a block's first tiles took longer to fetch than the tiles.)
            int kind = 0, k_at = w.tile(s, 0), v_at = k_at;       // kind: 0 Q, 1 K, 2 V
            bool first_k = true, ok = true;
            auto half_tile = [&](int i) {
                const int row = (kind == 0 ? w.row0 : kind == 1 ? k_at : v_at) + i * kFetchRows;
                return Source{(kind == 0 ? q : kind == 1 ? k : v) + row * a.vq.ss, (kind == 0 ? s.Sq : s.Skv) - row};
            };
            Fetch<kVec> x, y;
            x.load(half_tile(0), share);
            while (true) {
                y.load(half_tile(1), share);
                // the places that the two halves go to, free once the products that read them have run
                uint64_t* free0 = kind == 0 ? &bars->q_free : kind == 1 ? &bars->k_free[c_k & 1] : &bars->v_free[0];
                const int count = kind == 0 ? u : kind == 1 ? c_k >> 1 : c_v;
                uint8_t* dst = smem + (kind == 0 ? Smem::q : kind == 1 ? Smem::k + (c_k & 1) * kParts : Smem::v);
                if (count > 0 && !(ok = mbar_wait_warp(free0, (count - 1) & 1, abort_flag, 3))) break;
                x.put(dst, kTileBytes, share, check);
                const bool is_v = kind == 2;
                uint64_t* full = is_v ? &bars->v_full[1] : kind == 1 ? &bars->k_full[c_k & 1] : nullptr;
                if (is_v) {
                    fence_proxy_async_smem();
                    mbar_arrive(&bars->v_full[0]);
                }
                // the next one: K is one tile ahead of V
                if (kind == 1) { k_at = w.tile(s, k_at + kKeys); ++c_k; }
                if (kind == 2) { v_at = w.tile(s, v_at + kKeys); ++c_v; }
                const bool to_v = kind == 1 && !first_k;
                if (kind == 1) first_k = false;
                kind = to_v || k_at >= w.n_keys ? 2 : 1;
                const bool more = kind == 1 || v_at < w.n_keys;
                if (more) x.load(half_tile(0), share);
                if (!more && t == 0) ok = bars->queue.ask(u + 1, abort_flag);
                __syncwarp();
                if (is_v && count > 0 && !(ok = __all_sync(0xffffffffu, ok) && mbar_wait_warp(&bars->v_free[1], (count - 1) & 1, abort_flag, 4))) break;
                y.put(dst + kFetchRows * kRowBytes, kTileBytes, share, check);
                if (!more && check.odd()) bars->odd.set(u);
                if (full) {
                    fence_proxy_async_smem();
                    mbar_arrive(full);
                }
                if (!more) break;
            }
            if (!__all_sync(0xffffffffu, ok)) break;
        }
    } else if (warp > kIssueWarp) {
        setmaxnreg_dec<other_regs(kSumRegs)>();
    } else {
        setmaxnreg_dec<other_regs(kSumRegs)>();
        constexpr uint32_t idesc_s = make_idesc(128, kKeys, false, false);
        const uint64_t dq = make_sdesc(smem_u32(smem + Smem::q), 16, 1024), dk = make_sdesc(smem_u32(smem + Smem::k), 16, 1024);
        const uint64_t dv = make_sdesc(smem_u32(smem + Smem::v), kTileBytes, 1024);      // 192 columns: the parts one after the other
        int c = 0;
        // the scores of tile number n, `last` of its block: once its K is there and the scores before have been read
        auto scores = [&](int n, bool last) {
            const int st = n & 1;
            if (!mbar_wait_warp(&bars->k_full[st], (n >> 1) & 1, abort_flag, 5)) return false;
            if (n > 0 && !mbar_wait_warp(&bars->s_free, (n - 1) & 1, abort_flag, 6)) return false;
            tc_fence_after();
            six([&](int pa, int pb, uint32_t add) {
                mma_ss_4<2, 2>(tmem + kColS, sdesc_advance(dq, pa * kTileBytes), sdesc_advance(dk, st * kParts + pb * kTileBytes), idesc_s, add);
            });
            tc_commit_p(&bars->s_full);
            tc_commit_p(&bars->k_free[st]);
            if (last) tc_commit_p(&bars->q_free);
            return true;
        };
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(s, block, n_qt);
            int k0 = w.tile(s, 0);
            bool ok = scores(c, w.tile(s, k0 + kKeys) >= w.n_keys);
            for (; ok && k0 < w.n_keys; ++c) {
                k0 = w.tile(s, k0 + kKeys);
                if (k0 < w.n_keys && !(ok = scores(c + 1, w.tile(s, k0 + kKeys) >= w.n_keys))) break;
                if (!(ok = mbar_wait_warp(&bars->p_full, c & 1, abort_flag, 8))) break;
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    if (!(ok = mbar_wait_warp(&bars->v_full[i], c & 1, abort_flag, 7))) break;
                    tc_fence_after();
#pragma unroll
                    for (int p = 0; p < 3; ++p)      // part p of P with the first 3 - p parts of V, into the last 3 - p column groups
                        mma_ts_4<8, 128>(tmem + kColO + 64 * p, tmem + kColP + 64 * p + 32 * i, sdesc_advance(dv, i * 4 * 2048),
                                         make_idesc(128, 64 * (3 - p), false, true), i > 0 || p > 0);
                    tc_commit_p(&bars->v_free[i]);
                }
                if (!ok) break;
                tc_commit_p(&bars->o_full);
                if (lane == 0) mbar_arrive(&bars->o_full);
            }
            if (!ok) break;
        }
    }
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);      // a wait gave up: products and answers in flight end before the block does
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kIssueWarp) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

}  // namespace

bool f32_tc_forward_supported(const SimtArgs& a)
{
    const AttnShape& s = a.s;
    return !a.is_bf16 && s.D <= kDim && strides_supported(a) && scale_supported(s.scale) && enough_work(s, kForwardTiles) &&
           (long long)s.B * s.Hq * ((s.Sq + kOwnRows - 1) / kOwnRows) <= 0x7fffffffLL && f32_tc_forward_pays(s);
}

template <bool kVec> static cudaError_t launch(const SimtArgs& a, cudaStream_t st)
{
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(f32_fwd_kernel<kVec>, Smem::bytes, configured);
    if (e != cudaSuccess) return e;
    const int n_qt = (a.s.Sq + kOwnRows - 1) / kOwnRows;
    return launch_kernel(f32_fwd_kernel<kVec>, (unsigned)(n_qt * a.s.B * a.s.Hq), kThreads, Smem::bytes, st, 1, a, n_qt);
}

cudaError_t f32_tc_forward(const SimtArgs& a, cudaStream_t st) { return a.vec_q && a.vec_kv ? launch<true>(a, st) : launch<false>(a, st); }

cudaError_t read_and_clear_f32_fwd_status(uint32_t* word)
{
    uint32_t w = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&w, g_device_status, sizeof(w));
    if (e != cudaSuccess) return e;
    if (w != 0 && (e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(zero))) != cudaSuccess) return e;
    *word = w;
    return cudaSuccess;
}

}  // namespace sntl
