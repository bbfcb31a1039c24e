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
// TMEM: S [0, 128), parts of P [128, 320), P V [320, 512).
#include "attn_f32_sm100.cuh"

namespace sntl {
using namespace f32tc;
using namespace ptx;
namespace {

constexpr int kKeys = 128, kTileBytes = kOwnRows * kRowBytes, kParts = 3 * kTileBytes;
constexpr uint32_t kColS = 0, kColP = 128, kColO = 320;

struct Bars {
    uint64_t k_full[2], k_free[2], v_full, v_free, s_full, s_free, p_full, o_full, pair[4];
    uint32_t tmem_base, abort_flag, odd;
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

__global__ void __launch_bounds__(kThreads, 1) f32_fwd_kernel(const SimtArgs a, int n_qt)
{
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + (1024 - (smem_u32(raw) & 1023)) % 1024;
    Bars* bars = reinterpret_cast<Bars*>(smem + Smem::bars);
    float* exchange = reinterpret_cast<float*>(smem + Smem::exchange);
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->k_full[i], kStageThreads);
            mbar_init(&bars->k_free[i], 1);
        }
        mbar_init(&bars->v_full, kStageThreads);
        mbar_init(&bars->v_free, 1);
        mbar_init(&bars->s_full, 1);
        mbar_init(&bars->s_free, kSumThreads);
        mbar_init(&bars->p_full, kSumThreads);
        mbar_init(&bars->o_full, 1);
        for (int i = 0; i < 4; ++i) mbar_init(&bars->pair[i], 64);
        bars->abort_flag = 0;
        bars->odd = 0;
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

    const AttnShape& s = a.s;
    const int slabs = s.B * s.Hq, bh = blockIdx.x % slabs, b = bh / s.Hq, h = bh - b * s.Hq, hk = h / (s.Hq / s.Hkv);
    const int row0 = (n_qt - 1 - (int)blockIdx.x / slabs) * kOwnRows;      // longest query tiles first
    const int shift = s.causal ? s.Skv - s.Sq : 0;                         // query row r sits at position r + shift
    const int n_keys = s.causal ? min(min(row0 + kOwnRows, s.Sq) + shift, s.Skv) : s.Skv;
    const Rows mq{(const float*)a.q + b * a.vq.sb + h * a.vq.sh, a.vq.ss, a.vq.sd, s.Sq, s.D, a.vec_q};
    // tiles between the global tokens and the window of the first row are visible to no row
    auto next_tile = [&](int k0) {
        while (s.window > 0 && k0 < n_keys && k0 >= s.global_tokens && k0 + kKeys - 1 < row0 + shift - s.window + 1) k0 += kKeys;
        return k0;
    };

    if (warp < 8) {
        setmaxnreg_inc<kSumRegs>();
        const int half = warp >> 2, r = (warp & 3) * 32 + lane, row = row0 + r, n_row = s.causal ? min(row + shift + 1, s.Skv) : s.Skv;
        const int n_first = s.causal ? min(row0 + shift + 1, s.Skv) : s.Skv;
        const uint32_t lanes = tmem + ((uint32_t)(warp & 3) << 21);
        const float2 scale = make_float2(s.scale, s.scale);
        // largest score before scaling; what weights are relative to: that times scale (kHidden: no key seen yet)
        float top = kHidden, ref = kHidden, l = 0.f, corr = 1.f;
        float2 o[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) o[i] = make_float2(0.f, 0.f);
        auto add_product = [&]() {      // O so far is relative to the reference before the last one
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t g[3][16];
#pragma unroll
                for (int p = 0; p < 3; ++p) tmem_ld16(lanes + kColO + p * 64 + half * 32 + c * 16, g[p]);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    auto pair = [&](int p) { return make_float2(__uint_as_float(g[p][2 * i]), __uint_as_float(g[p][2 * i + 1])); };
                    o[c * 8 + i] = ffma2(o[c * 8 + i], make_float2(corr, corr), fadd2(pair(0), fadd2(pair(1), pair(2))));
                }
            }
        };
        int n = 0;
        bool ok = true;
        for (int k0 = next_tile(0); k0 < n_keys; k0 = next_tile(k0 + kKeys), ++n) {
            if (!(ok = mbar_wait_warp(&bars->s_full, n & 1, abort_flag, 1))) break;
            tc_fence_after();
            float2 x[32];
            tmem_ld32(lanes + kColS + half * 64, reinterpret_cast<uint32_t*>(x));
            tmem_ld32(lanes + kColS + half * 64 + 32, reinterpret_cast<uint32_t*>(x) + 32);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(&bars->s_free);
            if (k0 + kKeys > n_first || s.window > 0) {
#pragma unroll
                for (int w = 0; w < 2; ++w) {
                    const uint32_t seen = keys_seen(s, row + shift, n_row, k0 + half * 64 + w * 32);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        float2& y = x[w * 16 + i];
                        if (!(seen & (1u << (2 * i)))) y.x = kHidden;
                        if (!(seen & (2u << (2 * i)))) y.y = kHidden;
                    }
                }
            }
            float mx[2] = {top, top};
#pragma unroll
            for (int i = 0; i < 32; ++i) mx[i & 1] = fmax3(mx[i & 1], x[i].x, x[i].y);
            float other;
            if (!(ok = other_half(bars, exchange, n, half, r, fmaxf(mx[0], mx[1]), other))) break;
            top = fmax3(mx[0], mx[1], other);
            const bool none = top <= 0.5f * kHidden;
            const float next_ref = none ? kHidden : top * s.scale, sub = none ? 0.f : -next_ref;
            const float next_corr = exp_pair(make_float2(ref - next_ref, 0.f)).x;
            ref = next_ref;
            float2 sum[4] = {};
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                x[i] = exp_pair(ffma2(x[i], scale, make_float2(sub, sub)));
                sum[i % 4] = fadd2(sum[i % 4], x[i]);
            }
            const float2 all = fadd2(fadd2(sum[0], sum[1]), fadd2(sum[2], sum[3]));
            l = fmaf(l, next_corr, all.x + all.y);
            if (n > 0) {
                if (!(ok = mbar_wait_warp(&bars->o_full, (n - 1) & 1, abort_flag, 2))) break;
                tc_fence_after();
                add_product();
            }
            corr = next_corr;
            put_parts<32, 64>(lanes + kColP + half * 32, x);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&bars->p_full);
        }
        if (ok && n > 0 && mbar_wait_warp(&bars->o_full, (n - 1) & 1, abort_flag, 2)) {
            tc_fence_after();
            add_product();
            float other;
            other_half(bars, exchange, n, half, r, l, other);
            l += other;
        }
        __syncthreads();
        // A block with odd values is left to the FMA kernels, which find the mark in its LSE rows.
        const bool odd = bars->odd != 0;
        if (!odd) store_row((float*)a.o_out + b * a.vq.sb + h * a.vq.sh, mq, row, half * 32, o, l > 0.f ? 1.f / l : 0.f);
        if (half == 0 && row < s.Sq)
            a.lse_out[b * a.vlse.sb + h * a.vlse.sh + (long long)row * a.vlse.ss] =
                odd ? __uint_as_float(kOddLse) : l > 0.f ? ref + logf(l) : -INFINITY;
    } else if (warp < kIssueWarp) {
        setmaxnreg_dec<kOtherRegs>();
        const int t = threadIdx.x - kSumThreads;
        const Rows mk{(const float*)a.k + b * a.vkv.sb + hk * a.vkv.sh, a.vkv.ss, a.vkv.sd, s.Skv, s.D, a.vec_kv};
        const Rows mv{(const float*)a.v + b * a.vkv.sb + hk * a.vkv.sh, a.vkv.ss, a.vkv.sd, s.Skv, s.D, a.vec_kv};
        const bool tokens = mq.sd != 1;
        Check check;
        // Q, K_0, K_1, V_0, K_2, V_1, ...: half tiles, of which one is on its way while the one before is split.  (One loop for all of
        // them: unrolled for each, the code of a block's first tiles took longer to fetch than the tiles.)
        int kind = 0, k_n = 0, v_n = 0, k_at = next_tile(0), v_at = k_at;       // kind: 0 Q, 1 K, 2 V
        auto rows = [&]() { return kind == 0 ? mq : kind == 1 ? mk : mv; };
        auto first_row = [&]() { return kind == 0 ? row0 : kind == 1 ? k_at : v_at; };
        Fetch x, y;
        x.load(rows(), first_row(), t);
        while (true) {
            y.load(rows(), first_row() + kFetchRows, t);
            if (kind == 1 && k_n > 1 && !mbar_wait_warp(&bars->k_free[k_n & 1], ((k_n >> 1) - 1) & 1, abort_flag, 3)) break;
            if (kind == 2 && v_n > 0 && !mbar_wait_warp(&bars->v_free, (v_n - 1) & 1, abort_flag, 4)) break;
            uint8_t* dst = smem + (kind == 0 ? Smem::q : kind == 1 ? Smem::k + (k_n & 1) * kParts : Smem::v);
            uint64_t* full = kind == 1 ? &bars->k_full[k_n & 1] : &bars->v_full;
            const bool arrive = kind != 0;
            x.put(dst, kTileBytes, tokens, t, check);
            // the next one: K is one tile ahead of V
            if (kind == 1) { k_at = next_tile(k_at + kKeys); ++k_n; }
            if (kind == 2) { v_at = next_tile(v_at + kKeys); ++v_n; }
            kind = kind == 1 && k_n > 1 ? 2 : 1;
            if (kind == 1 && k_at >= n_keys) kind = 2;
            const bool more = kind == 1 || v_at < n_keys;
            if (more) x.load(rows(), first_row(), t);
            y.put(dst + kFetchRows * kRowBytes, kTileBytes, tokens, t, check);
            if (arrive) {
                fence_proxy_async_smem();
                mbar_arrive(full);
            }
            if (!more) break;
        }
        if (check.odd()) bars->odd = 1;
        __syncthreads();
    } else if (warp > kIssueWarp) {
        setmaxnreg_dec<kOtherRegs>();
        __syncthreads();
    } else {
        setmaxnreg_dec<kOtherRegs>();
        constexpr uint32_t idesc_s = make_idesc(128, kKeys, false, false);
        const uint64_t dq = make_sdesc(smem_u32(smem + Smem::q), 16, 1024), dk = make_sdesc(smem_u32(smem + Smem::k), 16, 1024);
        const uint64_t dv = make_sdesc(smem_u32(smem + Smem::v), kTileBytes, 1024);      // 192 columns: the parts one after the other
        auto scores = [&](int st) {
            six([&](int pa, int pb, uint32_t add) {
                mma_ss_4<2, 2>(tmem + kColS, sdesc_advance(dq, pa * kTileBytes), sdesc_advance(dk, st * kParts + pb * kTileBytes), idesc_s, add);
            });
            tc_commit_p(&bars->s_full);
            tc_commit_p(&bars->k_free[st]);
        };
        bool ok = mbar_wait_warp(&bars->k_full[0], 0, abort_flag, 5);
        tc_fence_after();
        if (ok) scores(0);
        int n = 0;
        for (int k0 = next_tile(0); ok && k0 < n_keys; ++n) {
            k0 = next_tile(k0 + kKeys);
            if (k0 < n_keys) {
                const int st = (n + 1) & 1;
                if (!(ok = mbar_wait_warp(&bars->k_full[st], ((n + 1) >> 1) & 1, abort_flag, 5) && mbar_wait_warp(&bars->s_free, n & 1, abort_flag, 6))) break;
                tc_fence_after();
                scores(st);
            }
            if (!(ok = mbar_wait_warp(&bars->v_full, n & 1, abort_flag, 7) && mbar_wait_warp(&bars->p_full, n & 1, abort_flag, 8))) break;
            tc_fence_after();
#pragma unroll
            for (int p = 0; p < 3; ++p) {
                // part p of P with the first 3 - p parts of V, into the last 3 - p column groups
                const uint32_t idesc = make_idesc(128, 64 * (3 - p), false, true), d = tmem + kColO + 64 * p, w = tmem + kColP + 64 * p;
                mma_ts_4<8, 128>(d, w, dv, idesc, p > 0);
                mma_ts_4<8, 128>(d, w + 32, sdesc_advance(dv, 4 * 2048), idesc, 1);
            }
            tc_commit_p(&bars->o_full);
            tc_commit_p(&bars->v_free);
        }
        __syncthreads();
    }
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);      // a wait gave up: products in flight end before TMEM is given back
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
    return !a.is_bf16 && s.D <= kDim && scale_supported(s.scale) && enough_work(s) && (long long)s.B * s.Hq * ((s.Sq + kOwnRows - 1) / kOwnRows) <= 0x7fffffffLL;
}

cudaError_t f32_tc_forward(const SimtArgs& a, cudaStream_t st)
{
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(f32_fwd_kernel, Smem::bytes, configured);
    if (e != cudaSuccess) return e;
    const int n_qt = (a.s.Sq + kOwnRows - 1) / kOwnRows;
    return launch_kernel(f32_fwd_kernel, (unsigned)(n_qt * a.s.B * a.s.Hq), kThreads, Smem::bytes, st, 1, a, n_qt);
}

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
