// dQ with one owner per element: the backward's third product for SNTL_FLAG_DETERMINISTIC.  A block owns 128 query rows of one
// (batch, head) and visits the key tiles that they see: S = Q K^T, dP = dO V^T, dS = P o (dP - delta), dQ += dS K.  The sum stays in
// TMEM, in the order of the keys, so the bits depend on nothing but the block's own rows and keys, and no scratch is needed; the kernel
// for dK and dV (attn_bwd_sm100.cu) then leaves dQ out.  Seven products instead of five, against reductions of 64-bit words that
// outlasted the five: 128 KB per step at the 25.5 bytes per clock that an SM gets through to L2.
//
// Backward, us, against the 64-bit reductions: B3 Hq16 Hkv4 S1237 D128 132 -> 97; B8 Hq28 Hkv4 S1024 D128 412 -> 240; B1 Hq28 Hkv4 S8192
// D128 1910 -> 1320.  Head_dim 64 stays with the reductions (bwd_dq_has_kernel).
//
//   warps 0-15  sums: thread = one query row and a quarter of a tile's 128 keys
//   warp 16     loads (TMA), warp 17 issues the products
// TMEM: S [0, 128), dP [128, 256), dS (bf16, two buffers of 64 columns) [256, 384), dQ [384, 384 + D).
#include "block_queue.cuh"
#include "row_terms.cuh"

namespace sntl {
using namespace ptx;
namespace {

constexpr int kT = 128, kSumThreads = 512, kLoadWarp = 16, kIssueWarp = 17, kThreads = 576, kChunkBytes = kT * 128;
constexpr uint32_t kColS = 0, kColDp = 128, kColDs = 256, kColDq = 384;

struct Bars {
    BlockQueue<18> queue;
    uint64_t q_full[2], q_free[2], k_full[4], k_free[4], v_full[4], v_free[4], scores_full, scores_free, ds_full[2], dq_done[2];
    uint32_t tmem_base, abort_flag;
};
template <int D> struct Smem {
    // A K tile is read last by its tile's dQ product, so the loop from its release over the next load, scores and sums to the next
    // release spans as many tiles as there are stages: two are too few.
    static constexpr int kKStages = D == 64 ? 4 : 3, kVStages = D == 64 ? 4 : 2, kQStages = D == 64 ? 2 : 1;
    static constexpr int kTile = kT * D * 2, q = 0, dout = kQStages * kTile, k = 2 * kQStages * kTile, v = k + kKStages * kTile, bars = v + kVStages * kTile;
    static constexpr int bytes = bars + (int)sizeof(Bars) + 1024;
};
static_assert(Smem<128>::bytes <= 227 * 1024, "");

struct Params {
    AttnShape s;
    const void *lse, *delta;          // terms of the padded query rows (store_row_terms)
    __nv_bfloat16* dq;
    float* dq_mat;                    // or an fp32 feature-major matrix (MatrixOut)
    long long mat_stride;
    int n_qt;
};

struct Block {
    int b, h, bh, bh_kv, qt, n_keys;

    __device__ __forceinline__ Block(const Params& p, int block)
    {
        const AttnShape& s = p.s;
        bh = block % (s.B * s.Hq);
        b = bh / s.Hq;
        h = bh - b * s.Hq;
        bh_kv = b * s.Hkv + h / (s.Hq / s.Hkv);
        qt = p.n_qt - 1 - block / (s.B * s.Hq);             // longest query tiles first
        n_keys = s.causal ? min((qt + 1) * kT, s.Skv) : s.Skv;
    }
    // k0, or the first key tile after it that some row sees (those between the global tokens and the window of the first row: none)
    __device__ __forceinline__ int tile(const AttnShape& s, int k0) const
    {
        while (s.window > 0 && k0 < n_keys && k0 >= s.global_tokens && k0 + kT - 1 < qt * kT - s.window + 1) k0 += kT;
        return k0;
    }
};

template <int D, bool kMat>
__global__ void __launch_bounds__(kThreads, 1)
    attn_dq_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                      const __grid_constant__ CUtensorMap tmap_do, const Params p)
{
    using L = Smem<D>;
    constexpr int kChunks = D / 64;
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + (1024 - (smem_u32(raw) & 1023)) % 1024;
    Bars* bars = reinterpret_cast<Bars*>(smem + L::bars);
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        bars->queue.init();
        for (int i = 0; i < 4; ++i) {
            mbar_init(&bars->k_full[i], 1);
            mbar_init(&bars->k_free[i], 1);
            mbar_init(&bars->v_full[i], 1);
            mbar_init(&bars->v_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->q_full[i], 1);
            mbar_init(&bars->q_free[i], 1);
            mbar_init(&bars->ds_full[i], kSumThreads);
            mbar_init(&bars->dq_done[i], 1);
        }
        mbar_init(&bars->scores_full, 1);
        mbar_init(&bars->scores_free, kSumThreads);
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
    const AttnShape& s = p.s;
    if (warp < kLoadWarp) {
        const int quarter = warp >> 2, r = (warp & 3) * 32 + lane;
        const uint32_t lanes = tmem + ((uint32_t)(warp & 3) << 21);
        const float2 scale2 = make_float2(s.scale * 1.4426950408889634f, s.scale * 1.4426950408889634f);
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            const int row = w.qt * kT + r, n_row = s.causal ? min(row + 1, s.Skv) : s.Skv;
            const size_t padded = (size_t)w.bh * p.n_qt * kT + row;
            float lse, delta;      // -LSE (log2) and -delta; at head_dim 64 the record of -LSE / scale is the sum of three bf16
            if constexpr (bwd_folds_row_terms(D)) {
                auto sum = [&](const void* records) {
                    const uint2 x = __ldg(reinterpret_cast<const uint2*>(static_cast<const uint4*>(records) + padded));
                    return __uint_as_float(x.x << 16) + (__uint_as_float(x.x & 0xffff0000u) + __uint_as_float(x.y << 16));
                };
                lse = sum(p.lse) * scale2.x;
                delta = sum(p.delta);
            } else {
                lse = __ldg(static_cast<const float*>(p.lse) + padded);
                delta = __ldg(static_cast<const float*>(p.delta) + padded);
            }
            bool ok = true;
            for (int k0 = w.tile(s, 0); k0 < w.n_keys; k0 = w.tile(s, k0 + kT), ++c) {
                if (!(ok = mbar_wait_warp(&bars->scores_full, c & 1, abort_flag, 0x61))) break;
                tc_fence_after();
                uint32_t x[32], y[32];
                tmem_ld32(lanes + kColS + quarter * 32, x);
                tmem_ld32(lanes + kColDp + quarter * 32, y);
                tmem_ld_wait();
                tc_fence_before();
                mbar_arrive(&bars->scores_free);
                // every pair of the tile is visible, or a mask
                const bool cut = k0 + kT > (s.causal ? w.qt * kT + 1 : s.Skv) || s.window > 0;
                uint32_t ds[16];
                auto weights = [&](auto&& seen) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) {
                        const float2 e = ffma2(make_float2(__uint_as_float(x[2 * i]), __uint_as_float(x[2 * i + 1])), scale2, make_float2(lse, lse));
                        float2 w2 = make_float2(seen(2 * i) ? ex2(e.x) : 0.f, seen(2 * i + 1) ? ex2(e.y) : 0.f);
                        if constexpr (D == 64) {      // as the P that dV and dK are made of, whose dS is rounded three times there
                            const uint32_t rounded = pack_bf16(w2.x, w2.y);
                            w2 = make_float2(__uint_as_float(rounded << 16), __uint_as_float(rounded & 0xffff0000u));
                        }
                        const float2 d = fmul2(w2, fadd2(make_float2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])), make_float2(delta, delta)));
                        ds[i] = pack_bf16(d.x, d.y);
                    }
                };
                if (!cut) {
                    weights([](int) { return true; });
                } else {
                    const uint32_t mask = keys_seen(s, row, n_row, k0 + quarter * 32);
                    weights([&](int i) { return (mask >> i & 1u) != 0; });
                }
                // (the buffer is free once the product before last has read it)
                if (c >= 2 && !(ok = mbar_wait_warp(&bars->dq_done[c & 1], ((c >> 1) - 1) & 1, abort_flag, 0x62))) break;
                tc_fence_after();
                tmem_st16(lanes + kColDs + (c & 1) * 64 + quarter * 16, ds);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&bars->ds_full[c & 1]);
            }
            if (!ok || !mbar_wait_warp(&bars->dq_done[(c - 1) & 1], ((c - 1) >> 1) & 1, abort_flag, 0x63)) break;
            tc_fence_after();
#pragma unroll
            for (int i = 0; i < D / 64; ++i) {
                const int d0 = quarter * (D / 4) + i * 16;
                uint32_t x[16];
                tmem_ld8(lanes + kColDq + d0, x);
                tmem_ld8(lanes + kColDq + d0 + 8, x + 8);
                tmem_ld_wait();
                if (row >= s.Sq) continue;
                if constexpr (kMat) {
                    float* dst = p.dq_mat + ((long long)w.h * D + d0) * p.mat_stride + (long long)w.b * s.Sq + row;
#pragma unroll
                    for (int j = 0; j < 16; ++j) dst[j * p.mat_stride] = __uint_as_float(x[j]) * s.scale;
                } else {
                    uint4* dst = reinterpret_cast<uint4*>(p.dq + ((size_t)w.bh * s.Sq + row) * D + d0);
#pragma unroll
                    for (int j = 0; j < 2; ++j) {
                        uint32_t v[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e)
                            v[e] = pack_bf16(__uint_as_float(x[8 * j + 2 * e]) * s.scale, __uint_as_float(x[8 * j + 2 * e + 1]) * s.scale);
                        dst[j] = make_uint4(v[0], v[1], v[2], v[3]);
                    }
                }
            }
            tc_fence_before();
        }
    } else if (warp == kLoadWarp) {
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            bool ok = true;
            if (lane == 0) {
                auto load = [&](int dst, const CUtensorMap* map, uint64_t* bar, int row, int slab) {
                    for (int i = 0; i < kChunks; ++i) tma_load_3d(smem + dst + i * kChunkBytes, map, bar, i * 64, row, slab);
                };
                // Q and dO once the last scores of the block before (head_dim 64: of the one before that) have been computed
                const int sq = u % L::kQStages;
                ok = u < L::kQStages || mbar_wait(&bars->q_free[sq], (u / L::kQStages - 1) & 1, abort_flag, 0x64);
                if (ok) {
                    mbar_arrive_expect_tx(&bars->q_full[sq], 2 * L::kTile);
                    load(L::q + sq * L::kTile, &tmap_q, &bars->q_full[sq], w.qt * kT, w.bh);
                    load(L::dout + sq * L::kTile, &tmap_do, &bars->q_full[sq], w.qt * kT, w.bh);
                }
                for (int k0 = w.tile(s, 0); ok && k0 < w.n_keys; ++c) {
                    const int sk = c % L::kKStages, sv = c % L::kVStages, next = w.tile(s, k0 + kT);
                    if (c >= L::kKStages && !(ok = mbar_wait(&bars->k_free[sk], (c / L::kKStages - 1) & 1, abort_flag, 0x65))) break;
                    mbar_arrive_expect_tx(&bars->k_full[sk], L::kTile);
                    load(L::k + sk * L::kTile, &tmap_k, &bars->k_full[sk], k0, w.bh_kv);
                    if (c >= L::kVStages && !(ok = mbar_wait(&bars->v_free[sv], (c / L::kVStages - 1) & 1, abort_flag, 0x66))) break;
                    mbar_arrive_expect_tx(&bars->v_full[sv], L::kTile);
                    load(L::v + sv * L::kTile, &tmap_v, &bars->v_full[sv], k0, w.bh_kv);
                    k0 = next;
                }
                if (ok) ok = bars->queue.ask(u + 1, abort_flag);
            }
            c = warp_uniform(c);
            if (!__all_sync(0xffffffffu, ok)) break;
        }
    } else if (warp == kIssueWarp) {
        constexpr uint32_t idesc_s = make_idesc(kT, kT, false, false), idesc_dq = make_idesc(kT, D, false, true);
        const uint64_t q = make_sdesc(smem_u32(smem + L::q), 16, 1024), dout = make_sdesc(smem_u32(smem + L::dout), 16, 1024);
        const uint64_t k = make_sdesc(smem_u32(smem + L::k), 16, 1024), v = make_sdesc(smem_u32(smem + L::v), 16, 1024);
        const uint64_t k_mn = make_sdesc(smem_u32(smem + L::k), kChunkBytes, 1024);
        auto wait = [&](uint64_t* bar, int parity, uint32_t site) { return mbar_wait_warp(bar, parity & 1, abort_flag, site); };
        auto product = [&](uint32_t d, uint64_t a, uint64_t b) {
#pragma unroll
            for (int i = 0; i < kChunks; ++i) mma_ss_4<2, 2>(d, sdesc_advance(a, i * kChunkBytes), sdesc_advance(b, i * kChunkBytes), idesc_s, i > 0);
        };
        // scores of tile number n, `last` of its block
        auto scores = [&](int n, int sq, bool last) {
            const int sk = n % L::kKStages, sv = n % L::kVStages;
            if (!wait(&bars->k_full[sk], n / L::kKStages, 0x67) || !wait(&bars->v_full[sv], n / L::kVStages, 0x68)) return false;
            if (n > 0 && !wait(&bars->scores_free, n - 1, 0x69)) return false;
            tc_fence_after();
            product(tmem + kColS, sdesc_advance(q, sq * L::kTile), sdesc_advance(k, sk * L::kTile));
            product(tmem + kColDp, sdesc_advance(dout, sq * L::kTile), sdesc_advance(v, sv * L::kTile));
            tc_commit_p(&bars->scores_full);
            tc_commit_p(&bars->v_free[sv]);
            if (last) tc_commit_p(&bars->q_free[sq]);
            return true;
        };
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            const int sq = u % L::kQStages;
            int k0 = w.tile(s, 0);
            bool ok = wait(&bars->q_full[sq], u / L::kQStages, 0x6a) && scores(c, sq, w.tile(s, k0 + kT) >= w.n_keys), accumulate = false;
            for (; ok && k0 < w.n_keys; ++c) {
                const int st = c & 1, sk = c % L::kKStages;
                k0 = w.tile(s, k0 + kT);
                if (k0 < w.n_keys && !(ok = scores(c + 1, sq, w.tile(s, k0 + kT) >= w.n_keys))) break;
                if (!(ok = wait(&bars->ds_full[st], c >> 1, 0x6b))) break;
                tc_fence_after();
                const uint32_t ds = tmem + kColDs + st * 64;
                const uint64_t b = sdesc_advance(k_mn, sk * L::kTile);
                mma_ts_4<8, 128>(tmem + kColDq, ds, b, idesc_dq, accumulate);
                mma_ts_4<8, 128>(tmem + kColDq, ds + 32, sdesc_advance(b, 4 * 2048), idesc_dq, 1);
                tc_commit_p(&bars->dq_done[st]);
                tc_commit_p(&bars->k_free[sk]);
                accumulate = true;
            }
            if (!ok) break;
        }
    }
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);      // a wait gave up: copies and products in flight end before the block does
    }
    tc_fence_before();
    __syncthreads();
    if (warp == kIssueWarp) {
        tc_fence_after();
        tmem_dealloc(tmem, 512);
    }
}

template <int D, bool kMat> cudaError_t launch(const TcArgs& a, const RowTerms& terms, cudaStream_t st)
{
    const AttnShape& s = a.s;
    CUtensorMap tq, tk, tv, tdo;
    cudaError_t e;
    if ((e = encode_tmap_bf16_3d(&tq, a.q, D, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tdo, a.dout, D, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tk, a.k, D, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tv, a.v, D, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    static std::atomic<unsigned long long> configured{0};
    if ((e = ensure_dynamic_smem(attn_dq_tc_kernel<D, kMat>, Smem<D>::bytes, configured)) != cudaSuccess) return e;
    const int n_qt = (s.Sq + kT - 1) / kT;
    const long long blocks = (long long)n_qt * s.B * s.Hq;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    Params p{s, terms.lse, terms.delta, a.dq, a.mat.dq, a.mat.stride, n_qt};
    if (!s.causal) p.s.window = 0;
    return launch_kernel(attn_dq_tc_kernel<D, kMat>, (unsigned)blocks, kThreads, Smem<D>::bytes, st, 1, tq, tk, tv, tdo, p);
}

}  // namespace

cudaError_t tc_backward_dq(const TcArgs& a, cudaStream_t st)
{
    const AttnShape& s = a.s;
    const RowTerms terms = row_terms_of(a.delta, (long long)s.B * s.Hq * ((s.Sq + kT - 1) / kT) * kT, s.D, s.scale);
    return a.mat.dq ? launch<128, true>(a, terms, st) : launch<128, false>(a, terms, st);
}

cudaError_t read_and_clear_dq_status(uint32_t* word)
{
    uint32_t w = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&w, g_device_status, sizeof(w));
    if (e != cudaSuccess) return e;
    if (w != 0 && (e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(zero))) != cudaSuccess) return e;
    *word = w;
    return cudaSuccess;
}

}  // namespace sntl
