// Exact-fp32 backward on the tensor cores (attn_f32_sm100.cuh says how), head_dim up to 64: one launch whose CTAs have one of two
// roles, as in attn_simt_bwd.cu.  A CTA owns 128 rows and visits tiles of 64 rows of the other side:
//   dK/dV   owns K and V rows of one (batch, KV head); visits Q and dO for every query head of the group.  dV += P^T dO, dK += dS^T Q.
//   dQ      owns Q and dO rows of one (batch, head); visits K and V.  dQ += dS K.
// One owner per element and no atomics: reproducible.
//
//   warps 0-7   sums: thread = one owned row and half of the 64 columns of a tile (then 32 features of the results).
//   warps 8-13  stage: fp32 rows -> parts in shared memory; delta = rowsum(dO o O) on the way.
//   warp 14     issues the products.
// A CTA takes over blocks (BlockQueue).  B8 H12 S512 D64: 133 us; 166 with a block per CTA and one barrier for both staged operands; 403
// with the FMA kernels.  What bounds it is the loop over two tiles from the release of a staged operand to the products that read the
// next one in its place (staging 4000 cycles, scores 2900, sums 3500, products 1440).
// Per tile: scores own0 x in0 and own1 x in1 (dP), each six products of 64 terms, 1440 cycles; dV and dK likewise; dQ has room for
// three accumulators, dS parts against the parts of K beside each other, 888 cycles (attn_f32_fwd_sm100.cu).
//
// TMEM: scores [0, 64), dP [64, 128), parts of P [128, 224), parts of dS [224, 320), dV [320, 384) and dK [384, 448), or dQ [320, 512).
#include "attn_f32_sm100.cuh"

namespace sntl {
using namespace f32tc;
using namespace ptx;
namespace {

constexpr int kLoop = kFetchRows, kOwnTile = kOwnRows * kRowBytes, kInTile = kLoop * kRowBytes;
constexpr uint32_t kColS = 0, kColDp = 64, kColP = 128, kColDs = 224, kColDv = 320, kColDk = 384, kColDq = 320;
constexpr int kSumRegs = 152;

struct Bars {
    Queue queue;
    uint64_t own_free, in0_full[2], in0_free[2], in1_full[2], in1_free[2], scores_full, scores_free, weights_full, out_full, dots_full, block_done;
    uint32_t tmem_base, abort_flag;
    OddBlocks odd;
};
struct Smem {
    static constexpr int own0 = 0, own1 = 3 * kOwnTile, in0 = 6 * kOwnTile, stage_bytes = 6 * kInTile, in1 = in0 + 3 * kInTile;
    static constexpr int part = in0 + 2 * stage_bytes, terms = part + 2 * kLoop * 9 * 4, own_terms = terms + 2 * kLoop * 8;
    static constexpr int bars = own_terms + 2 * kOwnRows * 8, bytes = bars + (int)sizeof(Bars) + 1024;
};
static_assert(Smem::bytes <= 227 * 1024, "");

struct Tile {
    int g, r0;      // query head of the group (dK/dV), first row
};

struct Block {
    bool dkv;
    int b, hk, h0, row0, shift, q_first, n_keys;      // h0: the head, or the first head of the group
    uint32_t mark;

    __device__ __forceinline__ Block(const AttnShape& s, int block, int n_dkv)
    {
        dkv = block < n_dkv;
        const int group = s.Hq / s.Hkv, heads = dkv ? s.Hkv : s.Hq, slabs = s.B * heads;
        const int n = dkv ? block : block - n_dkv, slab = n % slabs;
        b = slab / heads;
        const int head = slab - b * heads;
        hk = dkv ? head : head / group;
        h0 = dkv ? head * group : head;
        // the longest tiles first: the first keys, the last queries
        const int tile = dkv ? n / slabs : (s.Sq + kOwnRows - 1) / kOwnRows - 1 - n / slabs;
        row0 = tile * kOwnRows;
        mark = (dkv ? 0 : n_dkv) + tile * slabs + slab;
        shift = s.causal ? s.Skv - s.Sq : 0;           // query row r sits at position r + shift
        q_first = s.causal ? max(0, row0 - shift) / kLoop * kLoop : 0;
        n_keys = s.causal ? min(min(row0 + kOwnRows, s.Sq) + shift, s.Skv) : s.Skv;
    }
    // t, or the first tile to visit after it; whether there is one
    __device__ __forceinline__ bool settle(const AttnShape& s, Tile& t) const
    {
        if (dkv) {
            // past the window of the last key (and no key is global): no later query sees these keys
            const bool beyond = s.window > 0 && row0 >= s.global_tokens && t.r0 + shift > row0 + kOwnRows - 1 + s.window - 1;
            if (t.r0 >= s.Sq || beyond) t = Tile{t.g + 1, q_first};
            return t.g < s.Hq / s.Hkv && q_first < s.Sq;
        }
        // tiles between the global tokens and the window of the first row are visible to no row
        while (s.window > 0 && t.r0 < n_keys && t.r0 >= s.global_tokens && t.r0 + kLoop - 1 < row0 + shift - s.window + 1) t.r0 += kLoop;
        return t.r0 < n_keys;
    }
    __device__ __forceinline__ bool first(const AttnShape& s, Tile& t) const
    {
        t = Tile{0, dkv ? q_first : 0};
        return settle(s, t);
    }
    __device__ __forceinline__ bool next(const AttnShape& s, Tile& t) const
    {
        t.r0 += kLoop;
        return settle(s, t);
    }
};

template <bool kVec> __global__ void __launch_bounds__(kThreads, 1) f32_bwd_kernel(const SimtArgs a, int n_dkv)
{
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + (1024 - (smem_u32(raw) & 1023)) % 1024;
    Bars* bars = reinterpret_cast<Bars*>(smem + Smem::bars);
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        bars->queue.init();
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->in0_full[i], kStageThreads);
            mbar_init(&bars->in0_free[i], 1);
            mbar_init(&bars->in1_full[i], kStageThreads);
            mbar_init(&bars->in1_free[i], 1);
        }
        mbar_init(&bars->own_free, 1);
        mbar_init(&bars->scores_full, 2);      // the products, and what the issuing warp has seen of the staging warps
        mbar_init(&bars->scores_free, kSumThreads);
        mbar_init(&bars->weights_full, kSumThreads);
        mbar_init(&bars->out_full, 1);
        mbar_init(&bars->dots_full, kStageThreads);
        mbar_init(&bars->block_done, kSumThreads);
        for (int i = 0; i < 4; ++i) bars->odd.number[i] = 0;
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

    // Counters of tiles run on over the blocks: c for this block's tile.
    const AttnShape& s = a.s;
    // (-LSE, -delta) of the queries of a tile, or of the owned rows; kHidden in the place of -LSE where there is no such query or it
    // sees nothing
    float2* terms = reinterpret_cast<float2*>(smem + Smem::terms);
    float2* own_terms = reinterpret_cast<float2*>(smem + Smem::own_terms);

    if (warp < 8) {
        setmaxnreg_inc<kSumRegs>();
        const int half = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(warp & 3) << 21);
        const float2 scale = make_float2(s.scale, s.scale);
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(s, block, n_dkv);
            const int row = w.row0 + r;
            float2 out0[16], out1[16];                             // dK and dV, or dQ, times kUp; dK and dQ without the factor `scale`
            uint32_t largest_p = 0;                                // (as bits: also NaN and what should not be negative)
            float largest_ds = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) out0[i] = out1[i] = make_float2(0.f, 0.f);
            auto add_product = [&](float2 (&out)[16], uint32_t column) {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    uint32_t y[8];
                    tmem_ld8(lanes + column + half * 32 + x * 8, y);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        out[x * 4 + i] = fadd2(out[x * 4 + i], make_float2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])));
                }
            };
            auto add_products = [&]() {
                if (w.dkv) {
                    add_product(out1, kColDv);
                    add_product(out0, kColDk);
                } else {
                    // (the small groups first; out1 is not used otherwise)
#pragma unroll 1
                    for (int p = 2; p >= 0; --p) add_product(out0, kColDq + 64 * p);
                }
            };
            bool ok = true, started = false;
            Tile t;
            for (bool more = w.first(s, t); more; more = w.next(s, t), ++c, started = true) {
                if (!(ok = mbar_wait_warp(&bars->scores_full, c & 1, abort_flag, 2))) break;
                tc_fence_after();
                float2 p[16], ds[16];
                tmem_ld32(lanes + kColS + half * 32, reinterpret_cast<uint32_t*>(p));
                tmem_ld32(lanes + kColDp + half * 32, reinterpret_cast<uint32_t*>(ds));
                tmem_ld_wait();
                // (before the scores are given back: a block of one tile more, and the terms of the block after it may come)
                const float2 own = own_terms[(u & 1) * kOwnRows + r];
                tc_fence_before();
                mbar_arrive(&bars->scores_free);
                const int c0 = t.r0 + half * 32;
                bool cut;                                          // some pair of the tile may be hidden
                if (w.dkv) cut = (s.causal && t.r0 + w.shift < w.row0 + kOwnRows - 1) || s.window > 0 || w.row0 + kOwnRows > s.Skv;
                else cut = (s.causal && t.r0 + kLoop > w.row0 + w.shift + 1) || t.r0 + kLoop > s.Skv || s.window > 0;
                if (cut) {
                    const uint32_t seen = w.dkv ? queries_seeing(s, row, c0 + w.shift)
                                                : keys_seen(s, row + w.shift, s.causal ? min(row + w.shift + 1, s.Skv) : s.Skv, c0);
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        if (!(seen & (1u << (2 * i)))) p[i].x = kHidden;
                        if (!(seen & (2u << (2 * i)))) p[i].y = kHidden;
                    }
                }
                auto weights = [&](int i, float2 lse, float2 delta) {
                    p[i] = exp_pair<true>(ffma2(p[i], scale, lse));
                    ds[i] = fmul2(p[i], fadd2(ds[i], delta));
                    largest_p = max(largest_p, max(__float_as_uint(p[i].x), __float_as_uint(p[i].y)));
                    largest_ds = fmax3(largest_ds, fabsf(ds[i].x), fabsf(ds[i].y));
                };
                if (w.dkv) {
                    const float4* col = reinterpret_cast<const float4*>(terms + (c & 1) * kLoop + half * 32);
#pragma unroll
                    for (int i = 0; i < 16; ++i) weights(i, make_float2(col[i].x, col[i].z), make_float2(col[i].y, col[i].w));
                } else {
#pragma unroll
                    for (int i = 0; i < 16; ++i) weights(i, make_float2(own.x, own.x), make_float2(own.y, own.y));
                }
                if (started) {
                    if (!(ok = mbar_wait_warp(&bars->out_full, (c - 1) & 1, abort_flag, 3))) break;
                    tc_fence_after();
                    add_products();
                }
                if (w.dkv) put_parts<16, 32>(lanes + kColP + half * 16, p);
                put_parts<16, 32>(lanes + kColDs + half * 16, ds);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&bars->weights_full);
            }
            if (!ok || !mbar_wait_warp(&bars->out_full, (c - 1) & 1, abort_flag, 3)) break;
            tc_fence_after();
            add_products();
            tc_fence_before();
            if (largest_p >= __float_as_uint(kLargestWeight) || !(largest_ds < kLargestWeight)) bars->odd.set(u);
            mbar_arrive(&bars->block_done);
            if (!mbar_wait_warp(&bars->block_done, u & 1, abort_flag, 10)) break;
            // A block with odd values is left to the FMA kernels, which find the mark.
            const bool odd = bars->odd.get(u);
            if (threadIdx.x == 0) a.odd_marks[w.mark] = odd;
            if (!odd) {
                const long long off = w.dkv ? w.b * a.vkv.sb + w.hk * a.vkv.sh : w.b * a.vq.sb + w.h0 * a.vq.sh;
                const int S = w.dkv ? s.Skv : s.Sq;
                const bool vec = w.dkv ? a.vec_kv : a.vec_q;
                store_row((float*)(w.dkv ? a.dk : a.dq) + off, a.vq.ss, a.vq.sd, S, s.D, vec, row, half * 32, out0, s.scale * kDown);
                if (w.dkv) store_row((float*)a.dv + off, a.vq.ss, a.vq.sd, S, s.D, vec, row, half * 32, out1, kDown);
            }
        }
    } else if (warp < kIssueWarp) {
        setmaxnreg_dec<other_regs(kSumRegs)>();
        const int t = threadIdx.x - kSumThreads;
        float* part = reinterpret_cast<float*>(smem + Smem::part);
        const Share<kVec> share(t, (int)a.vq.ss, (int)a.vq.sd, s.D);
        int c = 0, n_dots = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(s, block, n_dkv);
            auto q_rows = [&](const void* p, int h, int row) {
                return Source{(const float*)p + w.b * a.vq.sb + h * a.vq.sh + row * a.vq.ss, s.Sq - row};
            };
            auto kv_rows = [&](const void* p, int row) {
                return Source{(const float*)p + w.b * a.vkv.sb + w.hk * a.vkv.sh + row * a.vq.ss, s.Skv - row};
            };
            Check check;
            // Pairs of half tiles: n = -2, -1 the owned rows, then the tiles to visit; in1 first, which is free first.  (One loop for all
            // of them: unrolled for each, the code that stages a block's first rows took longer to fetch than the rows.)
            Tile tl;
            bool more = w.first(s, tl), ok = true;         // (every block has a tile to visit)
            auto head = [&]() { return w.dkv ? w.h0 + tl.g : w.h0; };
            auto row_of = [&](int n) { return n < 0 ? w.row0 + (n + 2) * kFetchRows : tl.r0; };
            // rows of Q or dO are one side's, those of K or V the other's
            auto rows = [&](int n, const void* q_like, const void* kv_like) {
                return w.dkv == (n >= 0) ? q_rows(q_like, head(), row_of(n)) : kv_rows(kv_like, row_of(n));
            };
            Fetch<kVec> x, y;
            y.load(rows(-2, a.dout, a.v), share);
            for (int n = -2;; ++n) {
                const int st = n < 0 ? n & 1 : c & 1, h = head(), at = row_of(n);
                const bool with_terms = w.dkv == (n >= 0);     // y holds dO rows
                const Source m0 = rows(n, a.q, a.k);
                x.load(with_terms ? q_rows(a.o, h, at) : m0, share);
                if (n < 0) ok = n > -2 || u == 0 || mbar_wait_warp(&bars->own_free, (u - 1) & 1, abort_flag, 11);
                else ok = c < 2 || mbar_wait_warp(&bars->in1_free[st], ((c >> 1) - 1) & 1, abort_flag, 4);
                if (!ok) break;
                const int pitch = n < 0 ? kOwnTile : kInTile, half_tile = st * kFetchRows * kRowBytes;
                y.put(smem + (n < 0 ? Smem::own1 + half_tile : Smem::in1 + st * Smem::stage_bytes), pitch, share, check);
                if (with_terms) {
                    float* sums = part + (n_dots & 1) * kLoop * 9;
                    y.dots(share, x, sums);
                    x.load(m0, share);
                    mbar_arrive(&bars->dots_full);
                    if (!(ok = mbar_wait_warp(&bars->dots_full, n_dots++ & 1, abort_flag, 8))) break;
                    if (t < kLoop) {
                        float delta = 0.f;
#pragma unroll
                        for (int i = 0; i < 8; ++i) delta += sums[t * 9 + i];
                        const int q = at + t;
                        const float lse = q < s.Sq ? a.lse[w.b * a.vlse.sb + h * a.vlse.sh + (long long)q * a.vlse.ss] : -INFINITY;
                        float2* dst = n < 0 ? own_terms + (u & 1) * kOwnRows + st * kLoop : terms + st * kLoop;
                        dst[t] = make_float2(lse > -INFINITY && lse < -kHidden ? -lse : kHidden, -delta);
                        if (!(fabsf(delta) < kLargestDelta)) bars->odd.set(u);
                    }
                }
                if (n >= 0) {
                    fence_proxy_async_smem();
                    mbar_arrive(&bars->in1_full[st]);
                    more = w.next(s, tl);
                }
                if (more) y.load(rows(n + 1, a.dout, a.v), share);
                else if (t == 0) ok = bars->queue.ask(u + 1, abort_flag);
                if (!(ok = __all_sync(0xffffffffu, ok))) break;
                if (n >= 0 && c >= 2 && !(ok = mbar_wait_warp(&bars->in0_free[st], ((c >> 1) - 1) & 1, abort_flag, 4))) break;
                x.put(smem + (n < 0 ? Smem::own0 + half_tile : Smem::in0 + st * Smem::stage_bytes), pitch, share, check);
                if (n >= 0) {
                    if (!more && check.odd()) bars->odd.set(u);
                    fence_proxy_async_smem();
                    mbar_arrive(&bars->in0_full[st]);
                    ++c;
                }
                if (!more) break;
            }
            if (!ok) break;
        }
    } else if (warp > kIssueWarp) {
        setmaxnreg_dec<other_regs(kSumRegs)>();
    } else {
        setmaxnreg_dec<other_regs(kSumRegs)>();
        constexpr uint32_t idesc_s = make_idesc(kOwnRows, kLoop, false, false), idesc_out = make_idesc(kOwnRows, kDim, false, true);
        const uint64_t own0 = make_sdesc(smem_u32(smem + Smem::own0), kInTile, 1024), own1 = make_sdesc(smem_u32(smem + Smem::own1), kInTile, 1024);
        // (the distance between the parts counts where they are taken as 192 columns)
        const uint64_t in0 = make_sdesc(smem_u32(smem + Smem::in0), kInTile, 1024), in1 = make_sdesc(smem_u32(smem + Smem::in1), kInTile, 1024);
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(s, block, n_dkv);
            // the scores of tile number n, `last` of its block
            auto scores = [&](int n, bool last) {
                const int st = n & 1;
                const uint64_t b0 = sdesc_advance(in0, st * Smem::stage_bytes), b1 = sdesc_advance(in1, st * Smem::stage_bytes);
                if (!mbar_wait_warp(&bars->in1_full[st], (n >> 1) & 1, abort_flag, 5)) return false;
                if (n > 0 && !mbar_wait_warp(&bars->scores_free, (n - 1) & 1, abort_flag, 6)) return false;
                tc_fence_after();
                six([&](int pa, int pb, uint32_t add) {
                    mma_ss_4<2, 2>(tmem + kColDp, sdesc_advance(own1, pa * kOwnTile), sdesc_advance(b1, pb * kInTile), idesc_s, add);
                });
                if (!w.dkv) tc_commit_p(&bars->in1_free[st]);
                if (!mbar_wait_warp(&bars->in0_full[st], (n >> 1) & 1, abort_flag, 5)) return false;
                tc_fence_after();
                // the scores of the forward, bit by bit
                if (w.dkv)
                    six<true>([&](int pa, int pb, uint32_t add) {
                        mma_ss_4<2, 2>(tmem + kColS, sdesc_advance(own0, pa * kOwnTile), sdesc_advance(b0, pb * kInTile), idesc_s, add);
                    });
                else
                    six([&](int pa, int pb, uint32_t add) {
                        mma_ss_4<2, 2>(tmem + kColS, sdesc_advance(own0, pa * kOwnTile), sdesc_advance(b0, pb * kInTile), idesc_s, add);
                    });
                tc_commit_p(&bars->scores_full);
                if (lane == 0) mbar_arrive(&bars->scores_full);
                __syncwarp();
                if (last) tc_commit_p(&bars->own_free);
                return true;
            };
            auto products = [&](int n) {
                const int st = n & 1;
                const uint64_t b0 = sdesc_advance(in0, st * Smem::stage_bytes), b1 = sdesc_advance(in1, st * Smem::stage_bytes);
                if (!mbar_wait_warp(&bars->weights_full, n & 1, abort_flag, 7)) return false;
                tc_fence_after();
                if (w.dkv) {
                    six([&](int pa, int pb, uint32_t add) { mma_ts_4<8, 128>(tmem + kColDv, tmem + kColP + 32 * pa, sdesc_advance(b1, pb * kInTile), idesc_out, add); });
                    tc_commit_p(&bars->in1_free[st]);
                    six([&](int pa, int pb, uint32_t add) { mma_ts_4<8, 128>(tmem + kColDk, tmem + kColDs + 32 * pa, sdesc_advance(b0, pb * kInTile), idesc_out, add); });
                } else {
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        mma_ts_4<8, 128>(tmem + kColDq + 64 * p, tmem + kColDs + 32 * p, b0, make_idesc(kOwnRows, kDim * (3 - p), false, true), p > 0);
                }
                tc_commit_p(&bars->out_full);
                tc_commit_p(&bars->in0_free[st]);
                return true;
            };
            Tile t;
            bool more = w.first(s, t);
            auto is_last = [&]() { Tile x = t; return !w.next(s, x); };
            bool ok = scores(c, is_last());
            for (; ok && more; ++c) {
                more = w.next(s, t);
                // The next scores come first, so that the sums over them run beside this tile's products; but products that could be
                // issued do not wait for rows that are still being staged.
                bool scores_first = more;
                for (int i = 0; scores_first && i < 100000 && !mbar_test(&bars->in0_full[(c + 1) & 1], ((c + 1) >> 1) & 1); ++i)
                    if (mbar_test(&bars->weights_full, c & 1)) scores_first = false;
                scores_first = __all_sync(0xffffffffu, scores_first);
                if (scores_first && !(ok = scores(c + 1, is_last()))) break;
                if (!(ok = products(c))) break;
                if (more && !scores_first && !(ok = scores(c + 1, is_last()))) break;
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

long long blocks(int S, int slabs) { return (long long)((S + kOwnRows - 1) / kOwnRows) * slabs; }

}  // namespace

bool f32_tc_backward_supported(const SimtArgs& a, size_t marks_bytes)
{
    const AttnShape& s = a.s;
    const long long n = blocks(s.Skv, s.B * s.Hkv) + blocks(s.Sq, s.B * s.Hq);
    if (a.is_bf16 || s.D > kDim || !strides_supported(a) || !scale_supported(s.scale) || n > 0x7fffffffLL || (size_t)n * sizeof(uint32_t) > marks_bytes)
        return false;
    // With either flag the bits must not depend on what else is in the call, so the rows alone decide (FMA -> here at the edge: B4 H8 S128 D64
    // 24 -> 20 us, B1 H8 S256 D32 24 -> 26).
    if (s.deterministic || s.whole_tiles) return s.Sq >= 64 && (long long)s.Sq * s.D >= 8192;
    return enough_work(s, kBackwardTiles) && f32_tc_backward_pays(s);
}

template <bool kVec> static cudaError_t launch(const SimtArgs& a, cudaStream_t st)
{
    static std::atomic<unsigned long long> configured{0};
    cudaError_t e = ensure_dynamic_smem(f32_bwd_kernel<kVec>, Smem::bytes, configured);
    if (e != cudaSuccess) return e;
    const long long n_dkv = blocks(a.s.Skv, a.s.B * a.s.Hkv), n_dq = blocks(a.s.Sq, a.s.B * a.s.Hq);
    return launch_kernel(f32_bwd_kernel<kVec>, (unsigned)(n_dkv + n_dq), kThreads, Smem::bytes, st, 1, a, (int)n_dkv);
}

cudaError_t f32_tc_backward(const SimtArgs& a, cudaStream_t st) { return a.vec_q && a.vec_kv ? launch<true>(a, st) : launch<false>(a, st); }

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
