// Exact-fp32 backward on the tensor cores (attn_f32_sm100.cuh says how), head_dim up to 64: one launch whose CTAs have one of two
// roles, as in attn_simt_bwd.cu.  A CTA owns 128 rows and visits tiles of 64 rows of the other side:
//   dK/dV   owns K and V rows of one (batch, KV head); visits Q and dO for every query head of the group.  dV += P^T dO, dK += dS^T Q.
//   dQ      owns Q and dO rows of one (batch, head); visits K and V.  dQ += dS K.
// One owner per element and no atomics: reproducible.
//
//   warps 0-7   sums: thread = one owned row and half of the 64 columns of a tile (then 32 features of the results).
//   warps 8-13  stage: fp32 rows -> parts in shared memory; delta = rowsum(dO o O) on the way.
//   warp 14     issues the products.
//
// TMEM: own0 x in0 (scores) [0, 64), own1 x in1 (dP) [64, 128), parts of P [128, 224), parts of dS [224, 320), products with in1
// [320, 384) and with in0 [384, 448).
#include "attn_f32_sm100.cuh"

namespace sntl {
using namespace f32tc;
using namespace ptx;
namespace {

constexpr int kLoop = kFetchRows, kOwnTile = kOwnRows * kRowBytes, kInTile = kLoop * kRowBytes;
constexpr uint32_t kColS = 0, kColDp = 64, kColP = 128, kColDs = 224, kColOut1 = 320, kColOut0 = 384;

struct Bars {
    uint64_t in_full[2], in_free[2], scores_full, scores_free, weights_full, out_full, sums_full;
    uint32_t tmem_base, abort_flag, odd;
};
struct Smem {
    static constexpr int own0 = 0, own1 = 3 * kOwnTile, in0 = 6 * kOwnTile, stage_bytes = 6 * kInTile, in1 = in0 + 3 * kInTile;
    static constexpr int part = in0 + 2 * stage_bytes, terms = part + 2 * kLoop * 9 * 4, bars = terms + 2 * kLoop * 8;
    static constexpr int bytes = bars + (int)sizeof(Bars) + 1024;
};
static_assert(Smem::bytes <= 227 * 1024, "");

struct Tile {
    int g, r0;      // query head of the group (dK/dV), first row
};

template <bool kDkv>
__device__ __forceinline__ void role(const SimtArgs& a, int tile, uint8_t* smem, Bars* bars, int warp, uint32_t mark)
{
    const AttnShape& s = a.s;
    const int lane = threadIdx.x & 31, group = s.Hq / s.Hkv;
    const uint32_t tmem = bars->tmem_base;
    volatile uint32_t* abort_flag = &bars->abort_flag;
    const int heads = kDkv ? s.Hkv : s.Hq, slabs = s.B * heads, slab = tile % slabs, b = slab / heads, head = slab - b * heads;
    const int hk = kDkv ? head : head / group, h0 = kDkv ? head * group : head;
    const int own_rows = kDkv ? s.Skv : s.Sq, n_tiles = (own_rows + kOwnRows - 1) / kOwnRows;
    // the longest tiles first: the first keys, the last queries
    const int row0 = (kDkv ? tile / slabs : n_tiles - 1 - tile / slabs) * kOwnRows;
    const int shift = s.causal ? s.Skv - s.Sq : 0;             // query row r sits at position r + shift

    // the tiles to visit, in the same order for every warp
    const int q_first = s.causal ? max(0, row0 - shift) / kLoop * kLoop : 0;
    const int n_keys = s.causal ? min(min(row0 + kOwnRows, s.Sq) + shift, s.Skv) : s.Skv;
    auto settle = [&](Tile& t) {                               // t, or the first tile after it that is visible; whether there is one
        if constexpr (kDkv) {
            // past the window of the last key (and no key is global): no later query sees these keys
            const bool beyond = s.window > 0 && row0 >= s.global_tokens && t.r0 + shift > row0 + kOwnRows - 1 + s.window - 1;
            if (t.r0 >= s.Sq || beyond) t = Tile{t.g + 1, q_first};
            return t.g < group && q_first < s.Sq;
        } else {
            // tiles between the global tokens and the window of the first row are visible to no row
            while (s.window > 0 && t.r0 < n_keys && t.r0 >= s.global_tokens && t.r0 + kLoop - 1 < row0 + shift - s.window + 1) t.r0 += kLoop;
            return t.r0 < n_keys;
        }
    };
    auto first = [&](Tile& t) { t = Tile{0, kDkv ? q_first : 0}; return settle(t); };
    auto next = [&](Tile& t) { t.r0 += kLoop; return settle(t); };

    float* part = reinterpret_cast<float*>(smem + Smem::part);
    // (-LSE, -delta) of the queries of a tile, or of the owned rows; kHidden in the place of -LSE where there is no such query or it
    // sees nothing
    float2* terms = reinterpret_cast<float2*>(smem + Smem::terms);
    const long long kv_off = b * a.vkv.sb + hk * a.vkv.sh;
    auto q_off = [&](int h) { return b * a.vq.sb + h * a.vq.sh; };

    if (warp < 8) {
        setmaxnreg_inc<kSumRegs>();
        const int half = warp >> 2, r = (warp & 3) * 32 + lane, row = row0 + r;
        const uint32_t lanes = tmem + ((uint32_t)(warp & 3) << 21);
        float2 out0[16], out1[16];                             // dK and dV, or dQ; dK and dQ without the factor `scale`
        uint32_t largest_p = 0;                                // (as bits: also NaN and what should not be negative)
        float largest_ds = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) out0[i] = out1[i] = make_float2(0.f, 0.f);
        auto add_product = [&](float2 (&out)[16], uint32_t column) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t x[16];
                tmem_ld16(lanes + column + half * 32 + c * 16, x);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    out[c * 8 + i] = fadd2(out[c * 8 + i], make_float2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])));
            }
        };
        auto add_products = [&]() {
            add_product(out0, kColOut0);
            if (kDkv) add_product(out1, kColOut1);
        };
        const float2 scale = make_float2(s.scale, s.scale);
        float2 own = make_float2(0.f, 0.f);
        int n = 0;
        bool ok = true;
        Tile t;
        for (bool more = first(t); more; more = next(t), ++n) {
            // (its rows' terms are in shared memory)
            if (!(ok = mbar_wait_warp(&bars->in_full[n & 1], (n >> 1) & 1, abort_flag, 1) && mbar_wait_warp(&bars->scores_full, n & 1, abort_flag, 2))) break;
            tc_fence_after();
            float2 p[16], ds[16];
            tmem_ld32(lanes + kColS + half * 32, reinterpret_cast<uint32_t*>(p));
            tmem_ld32(lanes + kColDp + half * 32, reinterpret_cast<uint32_t*>(ds));
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(&bars->scores_free);
            const int c0 = t.r0 + half * 32;
            const float4* col = reinterpret_cast<const float4*>(terms + (n & 1) * kLoop + half * 32);
            if (!kDkv && n == 0) own = terms[r];
            bool cut;                                          // some pair of the tile may be hidden
            if (kDkv) cut = (s.causal && t.r0 + shift < row0 + kOwnRows - 1) || s.window > 0 || row0 + kOwnRows > s.Skv;
            else cut = (s.causal && t.r0 + kLoop > row0 + shift + 1) || t.r0 + kLoop > s.Skv || s.window > 0;
            if (cut) {
                const uint32_t seen = kDkv ? queries_seeing(s, row, c0 + shift) : keys_seen(s, row + shift, s.causal ? min(row + shift + 1, s.Skv) : s.Skv, c0);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    if (!(seen & (1u << (2 * i)))) p[i].x = kHidden;
                    if (!(seen & (2u << (2 * i)))) p[i].y = kHidden;
                }
            }
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const float4 term = kDkv ? col[i] : make_float4(own.x, own.y, own.x, own.y);
                p[i] = exp_pair(ffma2(p[i], scale, make_float2(term.x, term.z)));
                ds[i] = fmul2(p[i], fadd2(ds[i], make_float2(term.y, term.w)));
                largest_p = max(largest_p, max(__float_as_uint(p[i].x), __float_as_uint(p[i].y)));
                largest_ds = fmax3(largest_ds, fabsf(ds[i].x), fabsf(ds[i].y));
            }
            if (n > 0) {
                if (!(ok = mbar_wait_warp(&bars->out_full, (n - 1) & 1, abort_flag, 3))) break;
                tc_fence_after();
                add_products();
            }
            if (kDkv) put_parts<16, 32>(lanes + kColP + half * 16, p);
            put_parts<16, 32>(lanes + kColDs + half * 16, ds);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&bars->weights_full);
        }
        if (ok && n > 0 && mbar_wait_warp(&bars->out_full, (n - 1) & 1, abort_flag, 3)) {
            tc_fence_after();
            add_products();
        }
        if (largest_p >= __float_as_uint(kLargestWeight) || !(largest_ds < kLargestWeight)) bars->odd = 1;
        __syncthreads();
        const bool odd = bars->odd != 0;
        if (threadIdx.x == 0) a.odd_marks[mark] = odd;
        if (!odd) {
            if (kDkv) {
                const Rows m{nullptr, a.vkv.ss, a.vkv.sd, own_rows, s.D, a.vec_kv};
                store_row((float*)a.dk + kv_off, m, row, half * 32, out0, s.scale);
                store_row((float*)a.dv + kv_off, m, row, half * 32, out1, 1.f);
            } else {
                const Rows m{nullptr, a.vq.ss, a.vq.sd, own_rows, s.D, a.vec_q};
                store_row((float*)a.dq + q_off(h0), m, row, half * 32, out0, s.scale);
            }
        }
    } else if (warp < kIssueWarp) {
        setmaxnreg_dec<kOtherRegs>();
        const int t = threadIdx.x - kSumThreads;
        auto q_rows = [&](const void* p, int h) { return Rows{(const float*)p + q_off(h), a.vq.ss, a.vq.sd, s.Sq, s.D, a.vec_q}; };
        auto kv_rows = [&](const void* p) { return Rows{(const float*)p + kv_off, a.vkv.ss, a.vkv.sd, s.Skv, s.D, a.vec_kv}; };
        Check check;
        bool odd_terms = false;
        // the terms of kLoop queries from q0 on, of head h, whose partial sums are in `sums`, for the n-th time
        auto put_terms = [&](int n, float2* dst, const float* sums, int q0, int h) {
            mbar_arrive(&bars->sums_full);
            if (!mbar_wait_warp(&bars->sums_full, n & 1, abort_flag, 8)) return false;
            if (t < kLoop) {
                float delta = 0.f;
#pragma unroll
                for (int c = 0; c < 8; ++c) delta += sums[t * 9 + c];
                const int q = q0 + t;
                const float lse = q < s.Sq ? a.lse[b * a.vlse.sb + h * a.vlse.sh + (long long)q * a.vlse.ss] : -INFINITY;
                dst[t] = make_float2(lse > -INFINITY && lse < -kHidden ? -lse : kHidden, -delta);
                odd_terms = odd_terms || !(fabsf(delta) < kLargestWeight);
            }
            return true;
        };
        const Rows m_own0 = kDkv ? kv_rows(a.k) : q_rows(a.q, h0), m_own1 = kDkv ? kv_rows(a.v) : q_rows(a.dout, h0);
        const bool tokens = m_own0.sd != 1;
        // Pairs of half tiles: n = -2, -1 the owned rows, then the tiles to visit.  (One loop for all of them: unrolled for each, the
        // code that stages a block's first rows took longer to fetch than the rows, 23 k cycles before its first product.)
        Tile tl;
        bool more = first(tl);
        const bool any = more;
        auto rows0 = [&](int n) { return n < 0 ? m_own0 : kDkv ? q_rows(a.q, h0 + tl.g) : kv_rows(a.k); };
        auto rows1 = [&](int n) { return n < 0 ? m_own1 : kDkv ? q_rows(a.dout, h0 + tl.g) : kv_rows(a.v); };
        auto row_of = [&](int n) { return n < 0 ? row0 + (n + 2) * kFetchRows : tl.r0; };
        Fetch x, y;
        if (any) x.load(rows0(-2), row_of(-2), t);
        for (int n = -2; any; ++n) {
            const int st = n & 1, h = kDkv ? h0 + tl.g : h0, at = row_of(n);
            y.load(rows1(n), at, t);
            if (n > 1 && !mbar_wait_warp(&bars->in_free[st], ((n >> 1) - 1) & 1, abort_flag, 4)) break;
            const int pitch = n < 0 ? kOwnTile : kInTile, half_tile = st * kFetchRows * kRowBytes;
            uint8_t* dst0 = smem + (n < 0 ? Smem::own0 + half_tile : Smem::in0 + st * Smem::stage_bytes);
            uint8_t* dst1 = smem + (n < 0 ? Smem::own1 + half_tile : Smem::in1 + st * Smem::stage_bytes);
            x.put(dst0, pitch, tokens, t, check);
            if (n >= 0) more = next(tl);
            if (kDkv == (n >= 0)) {
                // y holds dO rows; a third set of registers for O would not fit
                float* sums = part + st * kLoop * 9;
                x.load(q_rows(a.o, h), at, t);
                y.put(dst1, pitch, tokens, t, check);
                y.dots(tokens, t, x, sums);
                if (more) x.load(rows0(n + 1), row_of(n + 1), t);
                if (!put_terms(kDkv ? n : n + 2, terms + st * kLoop, sums, at, h)) break;
            } else {
                if (more) x.load(rows0(n + 1), row_of(n + 1), t);
                y.put(dst1, pitch, tokens, t, check);
            }
            if (n >= 0) {
                fence_proxy_async_smem();
                mbar_arrive(&bars->in_full[st]);
            }
            if (!more) break;
        }
        if (check.odd() || odd_terms) bars->odd = 1;
        __syncthreads();
    } else if (warp > kIssueWarp) {
        setmaxnreg_dec<kOtherRegs>();
        __syncthreads();
    } else {
        setmaxnreg_dec<kOtherRegs>();
        constexpr uint32_t idesc_s = make_idesc(kOwnRows, kLoop, false, false), idesc_out = make_idesc(kOwnRows, kDim, false, true);
        const uint64_t own0 = make_sdesc(smem_u32(smem + Smem::own0), 16, 1024), own1 = make_sdesc(smem_u32(smem + Smem::own1), 16, 1024);
        const uint64_t in0 = make_sdesc(smem_u32(smem + Smem::in0), 16, 1024), in1 = make_sdesc(smem_u32(smem + Smem::in1), 16, 1024);
        auto scores = [&](int st) {
            six<kDkv>([&](int pa, int pb, uint32_t add) {      // the scores of the forward, bit by bit
                mma_ss_4<2, 2>(tmem + kColS, sdesc_advance(own0, pa * kOwnTile), sdesc_advance(in0, st * Smem::stage_bytes + pb * kInTile), idesc_s, add);
            });
            six([&](int pa, int pb, uint32_t add) {
                mma_ss_4<2, 2>(tmem + kColDp, sdesc_advance(own1, pa * kOwnTile), sdesc_advance(in1, st * Smem::stage_bytes + pb * kInTile), idesc_s, add);
            });
            tc_commit_p(&bars->scores_full);
        };
        Tile tl;
        int n = 0;
        bool more = first(tl), ok = true;
        if (more && (ok = mbar_wait_warp(&bars->in_full[0], 0, abort_flag, 5))) {
            tc_fence_after();
            scores(0);
        }
        for (; ok && more; ++n) {
            const int st = n & 1;
            more = next(tl);
            if (more) {
                if (!(ok = mbar_wait_warp(&bars->in_full[st ^ 1], ((n + 1) >> 1) & 1, abort_flag, 5) && mbar_wait_warp(&bars->scores_free, n & 1, abort_flag, 6))) break;
                tc_fence_after();
                scores(st ^ 1);
            }
            if (!(ok = mbar_wait_warp(&bars->weights_full, n & 1, abort_flag, 7))) break;
            tc_fence_after();
            if (kDkv) {
                six([&](int pa, int pb, uint32_t add) {
                    mma_ts_4<8, 128>(tmem + kColOut1, tmem + kColP + 32 * pa, sdesc_advance(in1, st * Smem::stage_bytes + pb * kInTile), idesc_out, add);
                });
            }
            six([&](int pa, int pb, uint32_t add) {
                mma_ts_4<8, 128>(tmem + kColOut0, tmem + kColDs + 32 * pa, sdesc_advance(in0, st * Smem::stage_bytes + pb * kInTile), idesc_out, add);
            });
            tc_commit_p(&bars->out_full);
            tc_commit_p(&bars->in_free[st]);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kThreads, 1) f32_bwd_kernel(const SimtArgs a, int n_dkv)
{
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + (1024 - (smem_u32(raw) & 1023)) % 1024;
    Bars* bars = reinterpret_cast<Bars*>(smem + Smem::bars);
    const int warp = warp_uniform(threadIdx.x >> 5);
    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->in_full[i], kStageThreads);
            mbar_init(&bars->in_free[i], 1);
        }
        mbar_init(&bars->scores_full, 1);
        mbar_init(&bars->scores_free, kSumThreads);
        mbar_init(&bars->weights_full, kSumThreads);
        mbar_init(&bars->out_full, 1);
        mbar_init(&bars->sums_full, kStageThreads);
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
    wait_for_stream();
    if ((int)blockIdx.x < n_dkv) {
        role<true>(a, blockIdx.x, smem, bars, warp, blockIdx.x);
    } else {
        const int slabs = a.s.B * a.s.Hq, tile = blockIdx.x - n_dkv, n_qt = (a.s.Sq + kOwnRows - 1) / kOwnRows;
        role<false>(a, tile, smem, bars, warp, n_dkv + (n_qt - 1 - tile / slabs) * slabs + tile % slabs);
    }
    if (*(volatile uint32_t*)&bars->abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);      // a wait gave up: products in flight end before TMEM is given back
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kIssueWarp) {
        tc_fence_after();
        tmem_dealloc(bars->tmem_base, 512);
    }
}

long long blocks(int S, int slabs) { return (long long)((S + kOwnRows - 1) / kOwnRows) * slabs; }

}  // namespace

bool f32_tc_backward_supported(const SimtArgs& a, size_t marks_bytes)
{
    const AttnShape& s = a.s;
    const long long n = blocks(s.Skv, s.B * s.Hkv) + blocks(s.Sq, s.B * s.Hq);
    return !a.is_bf16 && s.D <= kDim && scale_supported(s.scale) && enough_work(s) && n <= 0x7fffffffLL && (size_t)n * sizeof(uint32_t) <= marks_bytes;
}

cudaError_t f32_tc_backward(const SimtArgs& a, cudaStream_t st)
{
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(f32_bwd_kernel, Smem::bytes, configured);
    if (e != cudaSuccess) return e;
    const long long n_dkv = blocks(a.s.Skv, a.s.B * a.s.Hkv), n_dq = blocks(a.s.Sq, a.s.B * a.s.Hq);
    return launch_kernel(f32_bwd_kernel, (unsigned)(n_dkv + n_dq), kThreads, Smem::bytes, st, 1, a, (int)n_dkv);
}

cudaError_t read_and_clear_f32_bwd_status(uint32_t* word)
{
    uint32_t w = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&w, g_device_status, sizeof(w));
    if (e != cudaSuccess) return e;
    if (w != 0 && (e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(zero))) != cudaSuccess) return e;
    *word = w;
    return cudaSuccess;
}

}  // namespace sntl
