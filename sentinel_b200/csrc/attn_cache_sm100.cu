// New tokens against a KV cache (decode, continued prefill) for sm_100a: tcgen05 MMA, accumulators in TMEM, TMA-staged K and V.
//
// The rows of one unit are 128 or 256 of the (query head of the group, new token) pairs of one (batch, KV head), so K and V are
// read once per group; K/V tiles of 128 keys.  Decode is bound by HBM (K and V of the whole cache once), long continuations by
// the hand-offs between products and softmax (about 4350 cycles per tile pair for 2560 cycles of products).
//
//   * Persistent, one CTA per SM.  The key tiles of all units form one list that is cut into equal pieces, one per CTA; a piece
//     may end one unit and begin the next.  Where a unit's own tiles divide evenly over the SMs the pieces are aligned to units
//     instead (cache_plan).  Cutting at units only left 40 of 148 SMs idle in the second wave of a 64-sequence decode
//     (209 us, 0.79 of the copy rate; 175 us, 0.94 now) and 36 of 148 all the time in a 512-token continuation of a 7B-class
//     layer (46.5 us).
//   * More than 128 rows per KV head (kPair): a unit is 256 rows, stream t owns 128 of them, and every K/V tile serves both: with a
//     tile per stream a 512-token continuation is bound by the rate at which the SMs pull K and V from L2.
//   * Up to 128 rows (kSingle, kSmall): a unit is one 128-row block, and tiles alternate between two streams, each with its own S
//     and O columns, softmax warpgroup and running max / sum.  Either way one stream's softmax overlaps the other's products.  K
//     and V tiles travel through rings that run on from unit to unit; Q has two slots (one of 256 rows for kPair), so the next
//     unit's rows are there before they are needed.
//   * Few rows (decode: kSmall, at most 32 rows per unit): the Q slots shrink to 32 rows and the rings grow to three stages
//     (192 KB of K and V in flight per SM at head_dim 128); only one warp per stream has rows.  Stream t reads its Q operand
//     (t + 1) * 32 rows early, which puts the rows on TMEM lanes 32 * (t + 1): the two softmax warps and the issuing warp then sit
//     on three different schedulers.  The other lanes hold products of whatever lies before and after the Q slot and are never read.
//   * Every (unit, piece) -- and stream, unless kPair -- leaves a partial (O, LSE); cache_merge_kernel combines them.
//
// Layout: bf16 token-major, D in {64, 128}.  TMEM (512 columns): S0 [0,128) S1 [128,256) O0 [256,256+D) O1 [384,384+D); P is
// written over S.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "softmax_tile.cuh"

#include <algorithm>

namespace sntl {

using namespace ptx;

namespace {

constexpr int kM = 128, kN = 128;
constexpr int kThreads = 384;        // two softmax warpgroups, one warpgroup with the issuing warp and the TMA warp
constexpr uint32_t kTmemCols = 512;
constexpr float kRescaleThreshold = 8.0f;   // log2 units
constexpr int kSmallRows = 32;

enum CacheMode : int { kSmall = 0, kSingle = 1, kPair = 2 };   // at most 32, at most 128, more rows per KV head
__host__ __device__ constexpr int unit_rows(int mode) { return mode == kPair ? 2 * kM : kM; }

enum CacheSite : uint32_t {
    kSiteQ = 0x41, kSiteQEmpty, kSiteKFull, kSiteVFull, kSiteKEmpty, kSiteVEmpty, kSiteSReady, kSitePReady, kSiteOReady, kSiteFinal
};

struct CacheParams {
    __nv_bfloat16* o_part;   // [part][unit row][D]; unit rows: [B * Hkv][rows]
    float* lse_part;         // [part][unit row]
    int slabs, rows;         // B * Hkv; rows per slab
    int Skv, new_tokens, window, global_tokens;
    int n_list;              // key tiles each unit visits
    int stride;              // tiles a unit takes in the list (n_list, or rounded up to whole pieces)
    int per_cta;             // tiles of a piece
    long long total;         // stride * units
    float scale_log2;
};

template <int D, int kMode> struct CacheSmem {
    static constexpr int kTileBytes = 128 * D * 2;
    static constexpr int kStages = kMode == kSmall ? 3 : 2;
    static constexpr int kQRows = kMode == kSmall ? kSmallRows : 128;
    static constexpr int kQBytes = kQRows * D * 2, kQChunk = kQRows * 128;
    static constexpr int k = 0, v = kStages * kTileBytes, q = 2 * kStages * kTileBytes;
    // (small: products read 128 rows from a Q slot of 32: up to 96 rows past the last slot's second chunk)
    static constexpr int bars = q + 2 * kQBytes + (kMode == kSmall ? 96 * 128 : 0);   // two slots, or one of two blocks
};

struct CacheBarriers {
    uint64_t q_full[2], q_empty[2];
    uint64_t k_full[3], k_empty[3], v_full[3], v_empty[3];
    uint64_t s_ready[2], p_half[2], p_ready[2], o_ready[2];   // p_half: the first 64 columns of P are written (kPair)
    uint64_t final_bar;
    uint32_t tmem_base;
    uint32_t abort_flag;
};

// One CTA's walk over its piece: unit after unit, tiles [tile, tile + n) of each.  (Everything that needs a division is worked
// out once per unit: in the issuing warp's loop the divisions cost a tenth of a tile's time.)
template <int kMode>
struct Walk {
    int unit, tile, n, slab, row0;   // row0: first row of the unit in its slab
    bool both;                       // kPair: the second stream has rows
    long long pos, end;
    const CacheParams& p;
    __device__ Walk(const CacheParams& params) : p(params)
    {
        pos = (long long)blockIdx.x * p.per_cta;
        end = min(pos + p.per_cta, p.total);
        n = 0;
    }
    // the next unit of the piece; false at its end
    __device__ bool next()
    {
        while (pos < end) {
            unit = (int)(pos / p.stride);
            tile = (int)(pos - (long long)unit * p.stride);
            const int take = (int)min((long long)(p.stride - tile), end - pos);
            pos += take;
            n = min(take, p.n_list - tile);
            if (n > 0) {
                slab = unit % p.slabs;
                row0 = unit / p.slabs * unit_rows(kMode);
                both = kMode != kPair || row0 + kM < p.rows;
                return true;
            }
        }
        return false;
    }
};

template <int D, int kMode>
__global__ void __launch_bounds__(kThreads, 1)
attn_cache_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                     const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CacheParams p)
{
    using L = CacheSmem<D, kMode>;
    constexpr int kStages = L::kStages, kChunkBytes = 128 * 128, kChunks = D / 64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *sK = smem + L::k, *sV = smem + L::v, *sQ = smem + L::q;
    CacheBarriers* bars = (CacheBarriers*)(smem + L::bars);
    volatile uint32_t* abort_flag = &bars->abort_flag;
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (warp-uniform for the compiler)

    // Key tiles a unit visits, in ascending order: those holding global tokens, then from the window of the oldest new token
    // to the end of the cache.
    const int first_pos = p.Skv - p.new_tokens;
    const int g_tiles = p.window > 0 ? (p.global_tokens + kN - 1) / kN : 0;
    const int w_first = p.window > 0 ? max(g_tiles, max(0, first_pos - p.window + 1) / kN) : 0;
    auto key_tile = [&](int j) { return j < g_tiles ? j : w_first + (j - g_tiles); };

    if (warp == 9 && lane == 0) {
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->q_full[i], 1);
            mbar_init(&bars->q_empty[i], 1);
            mbar_init(&bars->s_ready[i], 1);
            mbar_init(&bars->p_ready[i], kMode == kSmall ? 32 : 128);
            mbar_init(&bars->p_half[i], 128);
            mbar_init(&bars->o_ready[i], 1);
        }
        for (int i = 0; i < 3; ++i) {
            mbar_init(&bars->k_full[i], 1);
            mbar_init(&bars->k_empty[i], 1);
            mbar_init(&bars->v_full[i], 1);
            mbar_init(&bars->v_empty[i], 1);
        }
        mbar_init(&bars->final_bar, 1);
        bars->abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 8) {
        tmem_alloc(&bars->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    wait_for_stream();      // nothing before this reads or writes global memory
    auto tmem_S = [&](int t) { return tmem + (uint32_t)t * 128u; };
    auto tmem_O = [&](int t) { return tmem + 256u + (uint32_t)t * 128u; };

    if (warp >= 10) {
        setmaxnreg_dec<72>();   // idle warps of the last warpgroup
    } else if (warp == 9) {
        setmaxnreg_dec<72>();
        // =========================== TMA producer ===========================
        if (lane == 0) {
            bool ok = true;
            int st = 0, seg = 0;              // ring stage; units so far
            uint32_t lap = 0;                 // laps of the ring
            for (Walk<kMode> w(p); ok && w.next(); ++seg) {
                const int slot = kMode == kPair ? 0 : seg & 1, use = kMode == kPair ? seg : seg >> 1;   // how often the slot was filled
                if (use > 0 && !mbar_wait(&bars->q_empty[slot], (uint32_t)(use - 1) & 1u, abort_flag, kSiteQEmpty)) break;
                const int blocks = kMode == kPair && w.both ? 2 : 1;
                mbar_arrive_expect_tx(&bars->q_full[slot], (uint32_t)(blocks * L::kQBytes));
                for (int i = 0; i < blocks; ++i)
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(sQ + (slot + i) * L::kQBytes + c * L::kQChunk, &tmap_q, &bars->q_full[slot], c * 64, w.row0 + i * kM, w.slab);
                for (int j = 0; j < w.n; ++j) {
                    const int key0 = key_tile(w.tile + j) * kN;
                    if (lap > 0 && !(ok = mbar_wait(&bars->k_empty[st], (lap - 1) & 1u, abort_flag, kSiteKEmpty))) break;
                    mbar_arrive_expect_tx(&bars->k_full[st], (uint32_t)L::kTileBytes);
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(sK + st * L::kTileBytes + c * kChunkBytes, &tmap_k, &bars->k_full[st], c * 64, key0, w.slab);
                    if (lap > 0 && !(ok = mbar_wait(&bars->v_empty[st], (lap - 1) & 1u, abort_flag, kSiteVEmpty))) break;
                    mbar_arrive_expect_tx(&bars->v_full[st], (uint32_t)L::kTileBytes);
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(sV + st * L::kTileBytes + c * kChunkBytes, &tmap_v, &bars->v_full[st], c * 64, key0, w.slab);
                    if (++st == kStages) { st = 0; ++lap; }
                }
            }
        }
    } else if (warp == 8) {
        setmaxnreg_dec<72>();
        // =========================== MMA issuer ===========================
        // All 32 lanes walk the loops, one elected lane issues the products four k-steps at a time: descriptors then live in
        // uniform registers.  With a single-lane loop 16 products took 2200 cycles to issue, and a tile of a 512-token continuation 5600.
        {
            constexpr uint32_t idesc_s = make_idesc(kM, kN, false, false);
            constexpr uint32_t idesc_pv = make_idesc(kM, D, false, true);
            const uint64_t dq0 = make_sdesc(smem_u32(sQ), 16, 1024), dk0 = make_sdesc(smem_u32(sK), 16, 1024);
            const uint64_t dv0 = make_sdesc(smem_u32(sV), kChunkBytes, 1024);
            auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t site) {
                return mbar_wait_warp(bar, parity, abort_flag, site);
            };
            auto issue_s = [&](int t, int st, int slot) {
                const uint64_t a = dq0 + (uint64_t)((slot * L::kQBytes - (kMode == kSmall ? (t + 1) * kSmallRows * 128 : 0)) >> 4);
                const uint64_t b = sdesc_advance(dk0, (uint32_t)(st * L::kTileBytes));
#pragma unroll
                for (int c = 0; c < kChunks; ++c)
                    mma_ss_4<2, 2>(tmem_S(t), sdesc_advance(a, (uint32_t)(c * L::kQChunk)), sdesc_advance(b, (uint32_t)(c * kChunkBytes)), idesc_s, c > 0);
                tc_commit_p(&bars->s_ready[t]);
            };
            // kPair: the first half of the contraction goes out as soon as the first 64 columns of P are there (the caller has
            // waited for them), the rest behind p_ready.  Returns false when a wait gave up.
            auto issue_pv = [&](int t, int st, bool accumulate, uint32_t parity) {
                const uint64_t b = sdesc_advance(dv0, (uint32_t)(st * L::kTileBytes));
                mma_ts_4<8, 128>(tmem_O(t), tmem_S(t), b, idesc_pv, accumulate);
                if (kMode == kPair) {
                    if (!wait(&bars->p_ready[t], parity, kSitePReady)) return false;
                    tc_fence_after();
                }
                mma_ts_4<8, 128>(tmem_O(t), tmem_S(t) + 32u, sdesc_advance(b, 4 * 2048), idesc_pv, 1);
                tc_commit_p(&bars->o_ready[t]);
                return true;
            };
            // S runs ahead of P V: one load, or two when the streams take turns.  Each side walks the piece by itself.
            struct Cursor {
                Walk<kMode> w;
                int j = 0, n = 0, seg = 0, st = 0;
                uint32_t lap = 0;
                bool more;
                __device__ Cursor(const CacheParams& p) : w(p) { more = w.next(); }
                __device__ bool first() const { return j == 0; }
                __device__ bool last() const { return j + 1 == w.n; }
                __device__ void advance()
                {
                    ++n;
                    if (++st == kStages) { st = 0; ++lap; }
                    if (++j == w.n) { j = 0; ++seg; more = w.next(); }
                }
            };
            Cursor s(p), v(p);
            bool ok = true;
            auto s_operands = [&]() {     // K, and with a new unit Q, of the next S product are there
                const int slot = kMode == kPair ? 0 : s.seg & 1;
                const uint32_t use = (uint32_t)(kMode == kPair ? s.seg : s.seg >> 1);
                if (s.first() && !wait(&bars->q_full[slot], use & 1u, kSiteQ)) return false;
                if (!wait(&bars->k_full[s.st], s.lap & 1u, kSiteKFull)) return false;
                tc_fence_after();
                return true;
            };
            auto s_done = [&]() {         // S products are issued in load order: behind the unit's last one its Q is free
                tc_commit_p(&bars->k_empty[s.st]);
                if (s.last()) tc_commit_p(&bars->q_empty[kMode == kPair ? 0 : s.seg & 1]);
                s.advance();
            };
            if constexpr (kMode == kPair) {
                uint32_t done[2] = {0u, 0u};      // P V products per stream
                if (s.more && (ok = s_operands())) {
                    issue_s(0, s.st, 0);
                    if (s.w.both) issue_s(1, s.st, 1);
                    s_done();
                }
                while (ok && v.more) {
                    if (!(ok = wait(&bars->v_full[v.st], v.lap & 1u, kSiteVFull))) break;
                    bool operands = false;
#pragma unroll
                    for (int t = 0; t < 2; ++t) {
                        if (t == 0 || v.w.both) {
                            if (!(ok = wait(&bars->p_half[t], done[t] & 1u, kSitePReady))) break;
                            tc_fence_after();
                            if (!(ok = issue_pv(t, v.st, v.j > 0, done[t] & 1u))) break;
                            ++done[t];
                        }
                        if (s.more && (t == 0 || s.w.both)) {
                            if (!operands && !(ok = operands = s_operands())) break;
                            issue_s(t, s.st, t);
                        }
                    }
                    if (!ok) break;
                    tc_commit_p(&bars->v_empty[v.st]);
                    v.advance();
                    if (s.more) s_done();
                }
            } else {
                for (int i = 0; i < 2 && ok && s.more; ++i)
                    if ((ok = s_operands())) {
                        issue_s(s.n & 1, s.st, s.seg & 1);
                        s_done();
                    }
                while (ok && v.more) {
                    const int t = v.n & 1;
                    if (!(ok = wait(&bars->v_full[v.st], v.lap & 1u, kSiteVFull))) break;
                    if (!(ok = wait(&bars->p_ready[t], (uint32_t)(v.n >> 1) & 1u, kSitePReady))) break;
                    tc_fence_after();
                    // a stream's first tile of a unit overwrites its O: the unit's loads are dealt to the streams in turn
                    issue_pv(t, v.st, v.j >= 2, 0);
                    tc_commit_p(&bars->v_empty[v.st]);
                    v.advance();
                    // into the S columns this product has just read P from: one thread's products run in order
                    if (s.more && (ok = s_operands())) {
                        issue_s(s.n & 1, s.st, s.seg & 1);
                        s_done();
                    }
                }
            }
            tc_commit_p(&bars->final_bar);
            wait(&bars->final_bar, 0, kSiteFinal);
        }
    } else {
        // =========================== softmax + epilogue warpgroups ===========================
        setmaxnreg_inc<216>();
        const int t = warp >> 2;
        if (kMode != kSmall || (warp & 3) == t + 1) {
            const int row = kMode == kSmall ? lane : (warp & 3) * 32 + lane + (kMode == kPair ? t * kM : 0);     // row of the unit
            const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
            bool ok = true;
            int n0 = 0;                    // loads of the piece before the current unit
            uint32_t mine = 0;             // tiles of this stream so far
            for (Walk<kMode> w(p); ok && w.next(); n0 += w.n) {
                const int grow = w.row0 + row;                          // row of the slab
                const int qpos = first_pos + grow % p.new_tokens;
                const bool live = grow < p.rows;
                float m_ref = -INFINITY, l = 0.0f;
                int count = 0;
                if (t == 1 && !w.both) continue;
                for (int j = kMode == kPair || (n0 & 1) == t ? 0 : 1; j < w.n; j += kMode == kPair ? 1 : 2, ++count, ++mine) {
                    if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->s_ready[t], mine & 1u, abort_flag, kSiteSReady)))) break;
                    tc_fence_after();
                    uint32_t s[128];
#pragma unroll
                    for (int c = 0; c < 4; ++c) tmem_ld32(tmem_S(t) + lane_off + (uint32_t)(c * 32), s + c * 32);
                    tmem_ld_wait();
                    const int key0 = key_tile(w.tile + j) * kN;
                    const int limit = min(p.Skv, qpos + 1) - key0;      // keys of the tile this row sees
                    if (limit < kN) {
#pragma unroll
                        for (int c = 0; c < kN; ++c)
                            if (c >= limit) s[c] = 0xff800000u;         // -inf
                    }
                    if (p.window > 0) {
                        const int lo = qpos - p.window + 1 - key0, glim = p.global_tokens - key0;
                        if (lo > 0 && glim < min(lo, kN)) {
#pragma unroll
                            for (int c = 0; c < kN; ++c)
                                if (c < lo && c >= glim) s[c] = 0xff800000u;
                        }
                    }
                    const float m_new = fmaxf(m_ref, row_max(s) * p.scale_log2);
                    const bool need = (m_new - m_ref) > kRescaleThreshold && live;   // false when both are -inf (NaN compare)
                    if (count == 0) {
                        m_ref = m_new;
                    } else if (__any_sync(0xffffffffu, need)) {
                        if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_ready[t], (mine - 1u) & 1u, abort_flag, kSiteOReady)))) break;
                        tc_fence_after();
                        const float factor = need ? ex2(m_ref - m_new) : 1.0f;
                        if (need) m_ref = m_new;
                        l *= factor;
#pragma unroll
                        for (int c = 0; c < D / 32; ++c) {
                            uint32_t o[32];
                            tmem_ld32(tmem_O(t) + lane_off + (uint32_t)(c * 32), o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                            tmem_st32(tmem_O(t) + lane_off + (uint32_t)(c * 32), o);
                        }
                        tmem_st_wait();
                    }
                    const float neg_m = (m_ref == -INFINITY) ? 0.0f : -m_ref;
                    uint32_t pk[32];
                    float2 sum[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                    exp_half<0>(s, p.scale_log2, neg_m, pk, sum);
                    tmem_st32(tmem_S(t) + lane_off, pk);
                    if (kMode == kPair) {
                        tmem_st_wait();
                        tc_fence_before();
                        mbar_arrive(&bars->p_half[t]);
                    }
                    exp_half<1>(s, p.scale_log2, neg_m, pk, sum);
                    tmem_st32(tmem_S(t) + lane_off + 32u, pk);
                    l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
                    tmem_st_wait();
                    tc_fence_before();
                    mbar_arrive(&bars->p_ready[t]);
                }
                if (!ok) break;
                // this stream's partial result of the unit.  The next unit's first product overwrites O only behind the P that
                // these same threads store after this.
                const long long first = (long long)w.unit * p.stride;
                const int piece = (int)(blockIdx.x - first / p.per_cta), part = kMode == kPair ? piece : 2 * piece + t;
                const size_t out_row = ((size_t)part * p.slabs + w.slab) * p.rows + grow;
                if (count == 0) {
                    if (live) p.lse_part[out_row] = -INFINITY;          // no tile: weighs nothing in the merge
                    continue;
                }
                if (!(ok = __all_sync(0xffffffffu, mbar_wait(&bars->o_ready[t], (mine - 1u) & 1u, abort_flag, kSiteOReady)))) break;
                tc_fence_after();
                const float inv = l > 0.0f ? 1.0f / l : 0.0f;
#pragma unroll
                for (int c = 0; c < D / 32; ++c) {
                    uint32_t o[32];
                    tmem_ld32(tmem_O(t) + lane_off + (uint32_t)(c * 32), o);
                    tmem_ld_wait();
                    if (live) {
                        uint4* dst = reinterpret_cast<uint4*>(p.o_part + out_row * D + c * 32);
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            dst[i] = make_uint4(pack_bf16(__uint_as_float(o[8 * i + 0]) * inv, __uint_as_float(o[8 * i + 1]) * inv),
                                                pack_bf16(__uint_as_float(o[8 * i + 2]) * inv, __uint_as_float(o[8 * i + 3]) * inv),
                                                pack_bf16(__uint_as_float(o[8 * i + 4]) * inv, __uint_as_float(o[8 * i + 5]) * inv),
                                                pack_bf16(__uint_as_float(o[8 * i + 6]) * inv, __uint_as_float(o[8 * i + 7]) * inv));
                    }
                }
                tc_fence_before();
                if (live) p.lse_part[out_row] = l > 0.0f ? (m_ref + log2f(l)) * 0.6931471805599453f : -INFINITY;
            }
        }
    }

    // ---- teardown ----
    if (*abort_flag) {
        // a wait gave up: let TMA copies that may still be in flight land before the CTA's memory is released
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 8) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

// Combines the partial results of a row: LSE = log sum_s exp(lse_s), O = sum_s exp(lse_s - LSE) * O_s; a part without a visible
// key carries LSE = -inf and weighs nothing.  D/8 lanes hold one row, 16 bytes each, with the loads of four parts in flight.
// kWide: the lane groups of a block share ONE row and take its parts in turn (decode of a few long sequences: dozens of parts
// for a few dozen rows), else a row each.  O is stored 16 bytes at a time where it starts on such a boundary.
template <int D, bool kWide>
__global__ void __launch_bounds__(256) cache_merge_kernel(const CacheParams p, int rows_per_unit, int parts_per_piece, bool o_aligned,
                                                          __nv_bfloat16* __restrict__ o, float* __restrict__ lse)
{
    constexpr int kLanes = D / 8, kGroups = 256 / kLanes;
    __shared__ float s_acc[kWide ? kGroups : 1][kWide ? D : 1], s_m[kWide ? kGroups : 1], s_l[kWide ? kGroups : 1];
    wait_for_stream();
    const int group = threadIdx.x / kLanes, l8 = threadIdx.x % kLanes * 8;
    const long long rows = (long long)p.slabs * p.rows, r = kWide ? blockIdx.x : (long long)blockIdx.x * kGroups + group;
    if (r >= rows) return;                                    // (kWide: never)
    const int slab = (int)(r / p.rows), grow = (int)(r - (long long)slab * p.rows);
    const long long first = ((long long)(grow / rows_per_unit) * p.slabs + slab) * p.stride;
    const int n_parts = parts_per_piece * (int)((first + p.stride - 1) / p.per_cta - first / p.per_cta + 1);
    float m = -INFINITY, sum = 0.0f, acc[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
    constexpr int kStep = kWide ? kGroups : 1, kAhead = 4;
    for (int part0 = kWide ? group : 0; part0 < n_parts; part0 += kAhead * kStep) {
        float x[kAhead];
        uint4 v[kAhead];
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const int part = part0 + k * kStep;
            x[k] = part < n_parts ? p.lse_part[(size_t)part * rows + r] : -INFINITY;
            v[k] = part < n_parts ? *reinterpret_cast<const uint4*>(p.o_part + ((size_t)part * rows + r) * D + l8) : make_uint4(0, 0, 0, 0);
        }
        float m_new = m;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) m_new = fmaxf(m_new, x[k]);
        const float ref = m_new > -INFINITY ? m_new : 0.0f, corr = __expf(m - ref);
        m = m_new;
        sum *= corr;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] *= corr;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            if (!(x[k] > -INFINITY)) continue;                // (its O was never written)
            const float w = __expf(x[k] - ref);
            sum += w;
            const uint32_t u[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[2 * i] = fmaf(w, __uint_as_float(u[i] << 16), acc[2 * i]);
                acc[2 * i + 1] = fmaf(w, __uint_as_float(u[i] & 0xffff0000u), acc[2 * i + 1]);
            }
        }
    }
    if constexpr (kWide) {
#pragma unroll
        for (int i = 0; i < 8; ++i) s_acc[group][l8 + i] = acc[i];
        if (l8 == 0) {
            s_m[group] = m;
            s_l[group] = sum;
        }
        __syncthreads();
        if (group != 0) return;
        m = -INFINITY;
#pragma unroll
        for (int g = 0; g < kGroups; ++g) m = fmaxf(m, s_m[g]);
        const float ref = m > -INFINITY ? m : 0.0f;
        sum = 0.0f;
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.0f;
#pragma unroll 4
        for (int g = 0; g < kGroups; ++g) {
            const float w = __expf(s_m[g] - ref);
            sum = fmaf(w, s_l[g], sum);
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i] = fmaf(w, s_acc[g][l8 + i], acc[i]);
        }
    }
    const float inv = sum > 0.0f ? 1.0f / sum : 0.0f;
    __nv_bfloat16* dst = o + (size_t)r * D + l8;
    if (o_aligned) {
        *reinterpret_cast<uint4*>(dst) = make_uint4(pack_bf16(acc[0] * inv, acc[1] * inv), pack_bf16(acc[2] * inv, acc[3] * inv),
                                                    pack_bf16(acc[4] * inv, acc[5] * inv), pack_bf16(acc[6] * inv, acc[7] * inv));
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) dst[i] = __float2bfloat16_rn(acc[i] * inv);
    }
    if (l8 == 0) lse[r] = sum > 0.0f ? m + __logf(sum) : -INFINITY;
}

struct CachePlan {
    int mode, n_list, stride, per_cta, max_parts;
    long long total;
};

// How the key tiles are dealt to CTAs, one CTA per SM.  Aligned to units when that wastes little: pieces of at least one tile
// per stream, every unit cut into the same number of them, all of them running at once.  Otherwise one list of all units'
// tiles in equal pieces; a piece that crosses from one unit to the next costs about one tile more (its Q load, first products
// and partial result).
CachePlan cache_plan(const AttnShape& s)
{
    const int n_tiles = (s.Skv + kN - 1) / kN, sms = sm_count();
    CachePlan plan;
    const long long rows = (long long)(s.Hq / s.Hkv) * s.Sq;
    plan.mode = rows <= kSmallRows ? kSmall : rows <= kM ? kSingle : kPair;
    const int streams = plan.mode == kPair ? 1 : 2;   // tiles in work at a time = partial results per piece
    plan.n_list = n_tiles;
    if (s.window > 0) {
        const int g_tiles = (s.global_tokens + kN - 1) / kN;
        const int w_first = std::max(g_tiles, std::max(0, s.Skv - s.Sq - s.window + 1) / kN);
        plan.n_list = std::min(g_tiles, n_tiles) + std::max(0, n_tiles - w_first);
    }
    const long long units = (long long)s.B * s.Hkv * ((rows + unit_rows(plan.mode) - 1) / unit_rows(plan.mode));
    const int pieces = (int)std::max(1LL, std::min<long long>((plan.n_list + streams - 1) / streams, sms / std::max(1LL, units)));
    const int per = (plan.n_list + pieces - 1) / pieces, splits = (plan.n_list + per - 1) / per;
    const long long waves = (units * splits + sms - 1) / sms, even = std::max<long long>(streams, (units * plan.n_list + sms - 1) / sms);
    if (waves == 1 && per <= even + 1) {
        plan.per_cta = per;
        plan.stride = per * splits;
        plan.max_parts = streams * splits;
    } else {
        plan.per_cta = (int)std::min<long long>(even, INT32_MAX);
        plan.stride = plan.n_list;
        plan.max_parts = streams * ((plan.n_list + plan.per_cta - 1) / plan.per_cta + 1);
    }
    plan.total = units * plan.stride;
    return plan;
}

size_t lse_bytes(const CachePlan& plan, long long rows) { return ((size_t)plan.max_parts * rows * sizeof(float) + 255) / 256 * 256; }

template <int D, int kMode>
cudaError_t launch_cache(const TcArgs& a, const CachePlan& plan, int capacity, void* workspace, cudaStream_t st)
{
    using L = CacheSmem<D, kMode>;
    const AttnShape& s = a.s;
    const int slabs = s.B * s.Hkv, rows_per_slab = s.Hq / s.Hkv * s.Sq;
    const long long rows = (long long)slabs * rows_per_slab;
    CUtensorMap tq, tk, tv;
    cudaError_t e;
    // Q [B][Hq][new][D] read as [B*Hkv][group*new][D]: the query heads of a group are consecutive heads
    if ((e = encode_tmap_bf16_3d(&tq, a.q, D, rows_per_slab, slabs, L::kQRows)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tk, a.k, D, s.Skv, slabs, 128, capacity)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tv, a.v, D, s.Skv, slabs, 128, capacity)) != cudaSuccess) return e;
    if (!aligned(16, workspace)) return cudaErrorMisalignedAddress;   // the partial results are accessed 16 bytes at a time
    CacheParams p{};
    p.lse_part = reinterpret_cast<float*>(workspace);
    p.o_part = reinterpret_cast<__nv_bfloat16*>(reinterpret_cast<uint8_t*>(workspace) + lse_bytes(plan, rows));
    const bool o_aligned = aligned(16, a.o_out), direct = plan.max_parts == 1 && o_aligned;   // one part per unit: it is the result
    if (direct) {
        p.o_part = a.o_out;
        p.lse_part = a.lse_out;
    }
    p.slabs = slabs; p.rows = rows_per_slab;
    p.Skv = s.Skv; p.new_tokens = s.Sq; p.window = s.window; p.global_tokens = s.global_tokens;
    p.n_list = plan.n_list; p.stride = plan.stride; p.per_cta = plan.per_cta; p.total = plan.total;
    p.scale_log2 = s.scale * 1.4426950408889634f;
    constexpr size_t smem = L::bars + sizeof(CacheBarriers) + 1024;
    static std::atomic<unsigned long long> configured{0};   // one bit per device
    if ((e = ensure_dynamic_smem(attn_cache_tc_kernel<D, kMode>, smem, configured)) != cudaSuccess) return e;
    const unsigned ctas = (unsigned)((plan.total + plan.per_cta - 1) / plan.per_cta);
    if ((e = launch_kernel(attn_cache_tc_kernel<D, kMode>, ctas, kThreads, smem, st, 1, tq, tk, tv, p)) != cudaSuccess) return e;
    if (direct) return cudaSuccess;
    const int per_piece = kMode == kPair ? 1 : 2;
    // more than eight parts a row: their loads want to be in flight at once
    if (plan.max_parts > 8 && rows <= 4096)
        return launch_kernel(cache_merge_kernel<D, true>, (unsigned)rows, 256, 0, st, 1, p, unit_rows(kMode), per_piece, o_aligned, a.o_out, a.lse_out);
    constexpr int kRowsPerBlock = 256 / (D / 8);
    return launch_kernel(cache_merge_kernel<D, false>, (unsigned)((rows + kRowsPerBlock - 1) / kRowsPerBlock), 256, 0, st, 1, p,
                         unit_rows(kMode), per_piece, o_aligned, a.o_out, a.lse_out);
}

}  // namespace

size_t tc_cache_workspace_bytes(const AttnShape& s)
{
    const CachePlan plan = cache_plan(s);
    const long long rows = (long long)s.B * s.Hq * s.Sq;
    return lse_bytes(plan, rows) + (size_t)plan.max_parts * rows * s.D * 2;
}

bool tc_cache_supported(const AttnShape& s)
{
    return (s.D == 64 || s.D == 128) && s.causal && s.Sq <= s.Skv;
}

cudaError_t tc_cache_forward(const TcArgs& a, int capacity, void* workspace, cudaStream_t st)
{
    const CachePlan plan = cache_plan(a.s);
    if (a.s.D == 64)
        return plan.mode == kSmall    ? launch_cache<64, kSmall>(a, plan, capacity, workspace, st)
               : plan.mode == kSingle ? launch_cache<64, kSingle>(a, plan, capacity, workspace, st)
                                      : launch_cache<64, kPair>(a, plan, capacity, workspace, st);
    return plan.mode == kSmall    ? launch_cache<128, kSmall>(a, plan, capacity, workspace, st)
           : plan.mode == kSingle ? launch_cache<128, kSingle>(a, plan, capacity, workspace, st)
                                  : launch_cache<128, kPair>(a, plan, capacity, workspace, st);
}

cudaError_t read_and_clear_cache_status(uint32_t* word)
{
    unsigned int w = 0, zero = 0;
    cudaError_t e = cudaMemcpyFromSymbol(&w, ptx::g_device_status, sizeof(w));
    if (e != cudaSuccess) return e;
    if (w != 0 && (e = cudaMemcpyToSymbol(ptx::g_device_status, &zero, sizeof(zero))) != cudaSuccess) return e;
    *word = w;
    return cudaSuccess;
}

}  // namespace sntl
