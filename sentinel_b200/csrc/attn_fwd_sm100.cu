// Causal attention forward for sm_100a: tcgen05 MMA with accumulators in TMEM, TMA-staged operands,
// warp-specialised producer / MMA / softmax roles.
//
// Replaces the reference's CudaFlashAttentionForwardWmma64Entry
// (sentinel/NeuralNet/Cuda/CudaFlashAttention.cu:1105-1266): same math -- S = scale*Q K^T, causal mask,
// online softmax, O = P V, LSE = m + ln(l) -- re-designed for Blackwell:
//
//   * head_dim 128 (attn_fwd_tc_kernel): one CTA owns 256 (small grids: 128) consecutive query rows of one (batch, head) as two
//     128-row tiles, whose key tiles are taken in halves of 64 keys; each tile has its own softmax warpgroup (one thread per query
//     row: tcgen05.ld's 32x32b shape hands thread i row i, so the row max / row sum need no shuffles) while a single MMA-issuing
//     warp (one elected lane) feeds the tensor core for both, so one tile's softmax overlaps the other tile's MMAs;
//   * head_dim 64 (attn_fwd_streams_kernel): four softmax warpgroups, each with 64 of the 128 keys of every key tile and sums and
//     an O of its own, two per query tile, and two query tiles that run independently of each other;
//   * S (fp32) and O (fp32, D columns) live in TMEM; P is written back over S as packed bf16 and consumed by the PV MMA
//     straight from TMEM (A operand in TMEM), V is consumed from shared memory as an MN-major operand, so nothing is
//     transposed and P never touches shared memory;
//   * Q/K/V tiles arrive by per-CTA TMA (128-byte swizzle, no multicast) into two-stage K and V rings
//     guarded by mbarriers; stages are released by tcgen05.commit;
//   * the softmax works in the exp2 domain with scale*log2(e) folded into one FMA, and rescales O lazily:
//     only when a row's running max grew by more than 2^8 since the last rescale;
//   * grouped-query heads index their shared K/V head directly (no repeated K/V as at
//     sentinel/NeuralNet/Cuda/CudaCausalSelfAttention.cu:27-34); CTAs are ordered heaviest-first and the query
//     heads of one group are adjacent in launch order so they share K/V tiles in L2.
//
// Layout: bf16 token-major [B][H][S][D], D in {64,128}; LSE [B][Hq][Sq] fp32 (natural log).
// TMEM map (512 columns): head_dim 128 two S of 64 columns for each tile, O0 [256,384) O1 [384,512); head_dim 64 four S of
// 64, then four O of 64.
#include "common.cuh"
#include "sm100_ptx.cuh"
#include "softmax_tile.cuh"

#include <algorithm>
#include <mutex>

namespace sntl {

using namespace ptx;

namespace {

constexpr int kM = 128;          // query rows per tile
constexpr int kN = 128;          // keys per tile
constexpr int kHalf = 64;        // keys of a tile per S product: one S buffer, or one stream
constexpr int kFwdThreads = 384; // 2 softmax warpgroups + 1 warpgroup holding the MMA warp and the TMA warp
constexpr uint32_t kTmemCols = 512;
constexpr int kOutBytes = 8 * 4096;        // staging of O
constexpr float kRescaleThreshold = 8.0f;  // log2 units

enum WaitSite : uint32_t {
    kSiteQ = 1, kSiteK0, kSitePairFull, kSitePairEmpty, kSiteSReady, kSitePReady, kSiteOReady, kSiteFinal, kSiteQEmpty = 10, kSiteNext
};

struct FwdParams {
    __nv_bfloat16* o;
    float* lse;
    int B, Hq, Hkv, Sq, Skv;
    int causal;
    int window, global_tokens;   // sliding window and always-visible first keys (0, 0: plain causal)
    int n_qblk, tiles_per_cta;   // query blocks of that many 128-row tiles per (b, h)
    int several_waves;           // CTAs ask for further blocks
    int second_blocks;           // head_dim 64: blocks of the call where two per SM are enough and every half has its own, else 0
    float scale_log2; // scale * log2(e)
    // non-null: O and LSE leave as fp32 feature-major matrices (see MatrixOut)
    float *o_mat, *lse_mat;
    long long mat_stride;
};

// What one block of the grid computes.  A CTA computes its own block and then takes over blocks that have not started yet (as the
// backward does): K, Q and the first S of one come in under the last softmax passes and the epilogue of the one before.
// us: a 512-key window over B2 Hq28 Hkv4 S8192 D128 123 -> 108; B8 Hq28 Hkv4 S1024 D128 88.5 -> 72.0, B8 Hq16 S512 20.8 -> 18.9, B2 Hq16 Hkv4 S3000
// 73.5 -> 69.9.  (A grid whose time is one long block's alone only pays for it: B1 Hq4 S8192 D128, 256 blocks of one tile, 71.5 -> 77.)
struct FwdWork {
    int bh, bh_kv, q0;         // q0: first of the one or two 128-row tiles
    int g_tiles, w_first;      // key tiles in ascending order: the g_tiles tiles holding global tokens, then from w_first up to the
                               // diagonal (without a window simply 0 .. diagonal)
    int n0, n1;                // key tiles that tile 0 / tile 1 visits; n0 < 0: no more blocks

    template <bool kWin> __device__ __forceinline__ void decode(const FwdParams& p, int block)
    {
        // heaviest query blocks first; the heads of one KV group are adjacent
        const int bh_count = p.B * p.Hq, rank = block / bh_count;
        bh = block - rank * bh_count;
        const int b = bh / p.Hq, h = bh - b * p.Hq;
        bh_kv = b * p.Hkv + h / (p.Hq / p.Hkv);
        q0 = (p.causal ? p.n_qblk - 1 - rank : rank) * p.tiles_per_cta * kM;
        const bool windowed = kWin && p.window > 0;
        g_tiles = windowed ? (p.global_tokens + kN - 1) / kN : 0;
        w_first = windowed ? max(g_tiles, max(0, q0 - p.window + 1) / kN) : 0;
        const int n_all = (p.Skv + kN - 1) / kN;
        auto visits = [&](int t) {
            const int row0 = q0 + t * kM;
            if (row0 >= p.Sq || t >= p.tiles_per_cta) return 0;
            if (!p.causal) return n_all;
            const int diag = min(n_all - 1, row0 / kN);
            return min(g_tiles, diag + 1) + max(0, diag - w_first + 1);
        };
        n0 = visits(0);
        n1 = visits(1);
    }
    __device__ __forceinline__ int n_max() const { return max(n0, n1); }      // K/V tiles the producer brings in
    __device__ __forceinline__ int key_tile(int j) const { return j < g_tiles ? j : w_first + (j - g_tiles); }
};

struct FwdBarriers {
    uint4 response;            // of the block scheduler
    uint64_t response_full, work_full[2], work_empty[2];
    FwdWork work[2];           // blocks in turn
    uint64_t q_full, q_empty, k0_full;
    // Loads come in pairs {K_{j+1}, V_j} (K_0 alone first) and are released in the same pairs, {K_0} counting as pair -1: one
    // wait and one commit per key tile for the issuing warp instead of two each.  Barrier j & 1.
    uint64_t pair_full[2], pair_empty[2];
    // [tile][S buffer].  s_ready: S is there, and the product of the P that was in the buffer before has been added to O; buffer 0
    // once more behind the last P that was in it.
    uint64_t s_ready[2][2], p_ready[2][2];
    uint64_t o_ready[2];     // the tile's last P V product has been added
    uint64_t final_bar;
    uint32_t tmem_base;
    uint32_t abort_flag;
};

// kMode: kPlain = causal / full attention of a whole sequence; kWindow adds the sliding window (separate so that the
// plain kernel carries none of its bookkeeping).
enum FwdMode : int { kPlain = 0, kWindow = 1 };

// kMat: O and LSE leave as fp32 feature-major matrices
// kMany: CTAs take over blocks (FwdWork); without it each computes its own and the bookkeeping folds away
//
// Bound by the chain of one tile between two of its softmax passes, beside 2048 cycles of exponentials and 2560 of products per step of two
// tiles.  A key tile is taken as two halves of 64 keys, each with an S buffer of its own and its P written over it: while a
// half is exponentiated, the other's P V and the S of the half after it run, which took the P V and S products (about 1150 cycles per
// step) out of that chain.  S products of 64 keys are bound by their operands in shared memory (48 cycles per k-step instead of 32).
// With 128 keys per S product, us, before -> with halves, neither taking over blocks: B1 Hq4 S8192 88.0 -> 71.2 (256 blocks of one tile), B8
// Hq16 S512 21.7 -> 20.2, B3 Hq16 Hkv4 S1237 28.7 -> 27.3, B8 Hq28 Hkv4 S1024 92.6 -> 88.0, B2 Hq28 Hkv4 S8192 within its spread (at the power
// limit: 1600 MHz).  64 columns in registers instead of 128 also leave room for taking over blocks: the 168 registers that 384 threads
// can have at compile time then spill 12 bytes (60 of loads, none of them without kMany and kWindow).
// A row's reference maximum is that of 64 keys first and is renewed per 64 keys.  Taken from a whole first key tile, bits are those of
// 128 keys per S product, and O of rows with scores of standard deviation 3 and more is 2 % nearer to its value; scores of 0.25 see no
// difference, and the forward takes 3 to 10 % longer (B3 Hq16 Hkv4 S1237 26.1 -> 26.9, one tile 5.8 -> 6.2).
template <int kMode, bool kMat, bool kMany>
__global__ void __launch_bounds__(kFwdThreads, 1)
attn_fwd_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v, const FwdParams p)
{
    constexpr int D = 128;
    constexpr int kTileBytes = 128 * D * 2;          // one 128-row tile of Q, K or V
    constexpr int kChunkBytes = 128 * 128;           // one 64-element-wide TMA box (128 rows x 128 B)
    constexpr int kChunks = D / 64;
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = smem;                               // [2][kTileBytes]
    uint8_t* sK = sQ + 2 * kTileBytes;                // [2][kTileBytes]
    uint8_t* sV = sK + 2 * kTileBytes;                // [2][kTileBytes]
    uint8_t* sOut = sV + 2 * kTileBytes;              // 4 KB per softmax warp
    FwdBarriers* bars = (FwdBarriers*)(sOut + (kMat ? 0 : kOutBytes));
    volatile uint32_t* abort_flag = &bars->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (warp-uniform for the compiler)

    constexpr bool kWin = kMode != kPlain;

    // ---- setup ----
    FwdWork own;        // (kMany: the producer's)
    if (!kMany || (warp == 9 && lane == 0)) own.decode<kWin>(p, (int)blockIdx.x);
    if (warp == 9 && lane == 0) {
        if (kMany) bars->work[0] = own;
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
        mbar_init(&bars->q_full, 1);
        mbar_init(&bars->q_empty, 1);
        mbar_init(&bars->k0_full, 1);
        mbar_init(&bars->response_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->work_full[i], 1);
            mbar_init(&bars->work_empty[i], 9);    // the issuing warp and the softmax warps
            mbar_init(&bars->pair_full[i], 1);
            mbar_init(&bars->pair_empty[i], 1);
            for (int b = 0; b < 2; ++b) {
                mbar_init(&bars->s_ready[i][b], 1);
                mbar_init(&bars->p_ready[i][b], 128);
            }
            mbar_init(&bars->o_ready[i], 1);
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
    // (computed, not looked up: a two-element array indexed by the warp's tile would live in local memory)
    auto tmem_S = [&](int t, int b) { return tmem + (uint32_t)(t * kN + b * kHalf); };
    auto tmem_O = [&](int t) { return tmem + 256u + (uint32_t)(t * D); };

    // Every role walks the same blocks, which the producer decodes into shared memory: number u is work[u & 1].  Counters of key
    // tiles run on over the blocks (all of them: c0; those of tile t: its steps), so stages and barrier phases continue where they
    // are.  next(u): done with block u; whether another follows.
    auto next = [&](int u) {
        if (!kMany) return false;
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->work_empty[u & 1]);
        return mbar_wait_prompt_warp(&bars->work_full[(u + 1) & 1], (uint32_t)((u >> 1) & 1), abort_flag, kSiteNext) && warp_uniform(bars->work[(u + 1) & 1].n0) >= 0;
    };

    auto work = [&](int u) -> const FwdWork& { return kMany ? bars->work[u & 1] : own; };
    auto uniform = [&](int x) { return kMany ? warp_uniform(x) : x; };

    // 384 threads start with 168 registers each; each role re-allocates inside its own branch
    if (warp >= 10) {
        setmaxnreg_dec<104>();   // idle warps of the last warpgroup
    } else if (warp == 9) {
        setmaxnreg_dec<104>();
        // =========================== TMA producer ===========================
        if (lane == 0) {
            int c0 = 0;
            bool ok = true;
            FwdWork& w = own;
            for (int u = 0, block = 0; block >= 0; ++u) {
                const int n_max = w.n_max();
                auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int j) {
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(dst + ((c0 + j) & 1) * kTileBytes + c * kChunkBytes, map, bar, c * 64, w.key_tile(j) * kN, w.bh_kv);
                };
                // Q and K_0 once the last S product of the block before has run: Q is free then, and K_0's stage and barrier were free
                // before (the barrier must not be armed again while the K_0 before is on its way or unseen: rows of a single
                // key tile get here that early)
                if (u > 0 && !mbar_wait_prompt(&bars->q_empty, (uint32_t)((u - 1) & 1), abort_flag, kSiteQEmpty)) break;
                mbar_arrive_expect_tx(&bars->k0_full, (uint32_t)kTileBytes);
                load(sK, &tmap_k, &bars->k0_full, 0);
                mbar_arrive_expect_tx(&bars->q_full, (uint32_t)((w.n1 > 0 ? 2 : 1) * kTileBytes));
                for (int t = 0; t < (w.n1 > 0 ? 2 : 1); ++t)
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(sQ + t * kTileBytes + c * kChunkBytes, &tmap_q, &bars->q_full, c * 64, w.q0 + t * kM, w.bh);
                for (int j = 0; j < n_max; ++j) {
                    // K_{c+1} and V_c go where K_{c-1} and V_{c-2} were: pair c - 2, the (c >> 1)-th release of this barrier for odd c
                    // (pair -1 was the first), the one before for even c
                    const int c = c0 + j;
                    if (c >= 1 && !(ok = mbar_wait_prompt(&bars->pair_empty[c & 1], (uint32_t)((c >> 1) - (c & 1 ? 0 : 1)) & 1u, abort_flag, kSitePairEmpty))) break;
                    const bool k_too = j + 1 < n_max;
                    mbar_arrive_expect_tx(&bars->pair_full[c & 1], (uint32_t)(k_too ? 2 * kTileBytes : kTileBytes));
                    if (k_too) load(sK, &tmap_k, &bars->pair_full[c & 1], j + 1);
                    load(sV, &tmap_v, &bars->pair_full[c & 1], j);
                }
                if (!ok) break;
                c0 += n_max;
                // The next block is asked for about two steps before this one ends: in time, and not so early that it would go to
                // this CTA although others are free sooner.
                block = -1;
                if constexpr (kMany) {
                    mbar_arrive_expect_tx(&bars->response_full, 16);
                    clc_try_cancel(&bars->response, &bars->response_full);
                    if (!mbar_wait_prompt(&bars->response_full, (uint32_t)(u & 1), abort_flag, kSiteNext)) break;
                    block = clc_first_block(&bars->response);
                    fence_proxy_async_smem();
                    w.n0 = -1;
                    if (block >= 0) w.decode<kWin>(p, block);
                    if (u >= 1 && !mbar_wait_prompt(&bars->work_empty[(u + 1) & 1], (uint32_t)(((u - 1) >> 1) & 1), abort_flag, kSiteNext)) break;
                    bars->work[(u + 1) & 1] = w;
                    mbar_arrive(&bars->work_full[(u + 1) & 1]);
                }
            }
        }
    } else if (warp == 8) {
        setmaxnreg_dec<104>();
        // =========================== MMA issuer ===========================
        // All 32 lanes walk the loops (warp-uniform control flow keeps descriptors and addresses in uniform registers) and
        // one elected lane issues each tcgen05 instruction.
        {
            auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t site) {
                return mbar_wait_prompt_warp(bar, parity, abort_flag, site);
            };
            const bool tl8 = lane == 0;
            (void)tl8;
            SNTL_TRACE_DECL(tn);
            constexpr uint32_t idesc_s = make_idesc(kM, kHalf, false, false);
            constexpr uint32_t idesc_pv = make_idesc(kM, D, false, true);
            constexpr uint32_t kHalfBytes = kHalf * 128;    // of a K or V tile's 64-column chunk
            // one descriptor per tile, advanced per k-step by a 64-bit add
            const uint64_t dq = make_sdesc(smem_u32(sQ), 16, 1024), dk = make_sdesc(smem_u32(sK), 16, 1024);
            const uint64_t dv = make_sdesc(smem_u32(sV), kChunkBytes, 1024);
            auto issue_s = [&](int t, int b, int st) {
                const uint64_t q = sdesc_advance(dq, (uint32_t)(t * kTileBytes)), k = sdesc_advance(dk, (uint32_t)st * kTileBytes + (uint32_t)b * kHalfBytes);
#pragma unroll
                for (int c = 0; c < kChunks; ++c)
                    mma_ss_4<2, 2>(tmem_S(t, b), sdesc_advance(q, (uint32_t)(c * kChunkBytes)), sdesc_advance(k, (uint32_t)(c * kChunkBytes)), idesc_s, c > 0);
            };
            int c0 = 0, s0 = 0, s1 = 0;        // key tiles of the blocks before: all, those of tile 0, of tile 1
            bool ok = true, more = true;
            for (int u = 0; more; more = next(u++)) {
                const int n0 = uniform(work(u).n0), n1 = uniform(work(u).n1), n_max = max(n0, n1);
                if (!(ok = wait(&bars->k0_full, (uint32_t)(u & 1), kSiteK0) && wait(&bars->q_full, (uint32_t)(u & 1), kSiteQ))) break;
                tc_fence_after();
                // (S of the last step of the block before has been read, and P over it consumed: this warp waited for p_ready and issued
                // the product; O is overwritten behind p_ready of the new block, which its warps give after their epilogue)
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int t = 0; t < 2; ++t)
                        if (t == 0 || n1 > 0) {      // (a block has rows in its first tile)
                            issue_s(t, b, c0 & 1);
                            tc_commit_p(&bars->s_ready[t][b]);
                        }
                tc_commit_p(&bars->pair_empty[(c0 - 1) & 1]);        // K_0 and the last V of the block before
                if (kMany && n_max == 1) tc_commit_p(&bars->q_empty);
                for (int j = 0; ok && j < n_max; ++j) {
                    const int c = c0 + j;
                    if (!(ok = wait(&bars->pair_full[c & 1], (uint32_t)((c >> 1) & 1), kSitePairFull))) break;
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int t = 0; t < 2; ++t) {
                            const int n = t ? n1 : n0;
                            if (!ok || j >= n) continue;
                            if (!(ok = wait(&bars->p_ready[t][b], (uint32_t)(((t ? s1 : s0) + j) & 1), kSitePReady))) continue;
                            SNTL_TRACE_EV(tl8, 0, tn, 10 + 2 * b + t);
                            tc_fence_after();
                            mma_ts_4<8, 128>(tmem_O(t), tmem_S(t, b), sdesc_advance(dv, (uint32_t)(c & 1) * kTileBytes + (uint32_t)b * kHalfBytes), idesc_pv, j > 0 || b > 0);
                            SNTL_TRACE_EV(tl8, 0, tn, 20 + 2 * b + t);
                            if (j + 1 < n) issue_s(t, b, (c + 1) & 1);
                            tc_commit_p(b == 1 && j + 1 == n ? &bars->o_ready[t] : &bars->s_ready[t][b]);
                            SNTL_TRACE_EV(tl8, 0, tn, 30 + 2 * b + t);
                        }
                    if (!ok) break;
                    if (j + 1 < n_max) tc_commit_p(&bars->pair_empty[c & 1]);
                    if (kMany && j + 2 == n_max) tc_commit_p(&bars->q_empty);
                }
                if (!ok) break;
                c0 += n_max;
                s0 += n0;
                s1 += n1;
            }
            // every MMA issued above must have retired before shared memory / TMEM are given up
            tc_commit_p(&bars->final_bar);
            wait(&bars->final_bar, 0, kSiteFinal);
        }
    } else {
        // =========================== softmax + epilogue warpgroups ===========================
        setmaxnreg_inc<200>();
        const int t = warp >> 2;                       // tile 0 or 1
        const int row = (warp & 3) * 32 + lane;        // row inside the tile == TMEM lane
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        SNTL_TRACE_DECL(tn);
        const bool tw = (warp & 3) == 0 && lane == 0;
        (void)tw;
        bool ok = true, more = true;
        uint32_t phase[2] = {0, 0}, blocks = 0;        // of the tile's s_ready barriers, blocks with rows
        for (int u = 0; ok && more; more = next(u++)) {
        const FwdWork& w = work(u);
        const int n_mine = uniform(t ? w.n1 : w.n0), q0 = uniform(w.q0);
        const int g_tiles = kWin ? uniform(w.g_tiles) : 0, w_first = kWin ? uniform(w.w_first) : 0;
        const int grow = q0 + t * kM + row;            // query row inside the (batch, head) slab
        auto key_tile = [&](int j) { return j < g_tiles ? j : w_first + (j - g_tiles); };
        float m_ref = -INFINITY, l = 0.0f;
        // Barrier tests queue behind the exponentials in the same unit and take 200-400 cycles here; where a result is likely to be
        // there already it is asked for ahead of its use, with other work in between.
        bool s_seen = false;
        const int row_lo = q0 + t * kM + (warp & 3) * 32;      // first row of the warp
        for (int h = 0; h < 2 * n_mine; ++h) {
            const int b = h & 1;
            const uint32_t tmS = tmem_S(t, b) + lane_off;
            if (!(ok = s_seen || mbar_wait_prompt_warp(&bars->s_ready[t][b], b ? phase[1] : phase[0], abort_flag, kSiteSReady))) break;
            SNTL_TRACE_EV(tw, 1 + t, tn, 1);
            tc_fence_after();
            uint32_t s[kHalf];
#pragma unroll
            for (int c = 0; c < 2; ++c) tmem_ld32(tmS + (uint32_t)(c * 32), s + c * 32);
            tmem_ld_wait();
            SNTL_TRACE_EV(tw, 1 + t, tn, 2);
            // number of visible keys of this row among these
            const int key0 = key_tile(h >> 1) * kN + b * kHalf;
            const int limit = (p.causal ? min(p.Skv, grow + 1) : p.Skv) - key0;
            // Once a row has a reference maximum, keys that the mask does not cut are exponentiated against it at once, with their
            // own maximum taken on the way: only if some row of the warp then needs a rescale (its maximum grew by more than 2^8,
            // which the lazy rule below leaves rare) is that done again.  The maximum and the decision were a quarter of a tile's time
            // in front of the exponentials.  (Under a window many tiles are cut, and with both forms of the pass in use it is slower: a
            // 512-key window over B2 Hq28 Hkv4 S2048 47.0 us, 44.4 without; 200 keys over B4 Hq16 S1024 27.5 and 26.1.)
            const int limit_lo = (p.causal ? min(p.Skv, row_lo + 1) : p.Skv) - key0;
            const int lo_hi = kWin ? row_lo + 31 - p.window + 1 - key0 : 0, glim = kWin ? p.global_tokens - key0 : 0;
            const bool cut = limit_lo < kHalf || (kWin && lo_hi > 0 && glim < min(lo_hi, kHalf));   // (some row of the warp is)
            uint32_t pk[32];
            float2 sum[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
            auto shift = [&]() { return m_ref == -INFINITY ? 0.0f : -m_ref; };   // (no finite score so far: -inf + inf would be NaN)
            // O and the sum of a row whose maximum has outgrown its reference
            auto rescale = [&](float m_new) {
                // the product of the P before has been added
                if (!(ok = mbar_wait_prompt_warp(&bars->s_ready[t][b ^ 1], b ? phase[0] ^ 1u : phase[1], abort_flag, kSiteOReady))) return;
                tc_fence_after();
                const bool need = (m_new - m_ref) > kRescaleThreshold;
                const float factor = need ? ex2(m_ref - m_new) : 1.0f;
                if (need) m_ref = m_new;
                l *= factor;
#pragma unroll 1
                for (int c = 0; c < D / 32; ++c) {
                    uint32_t o[32];
                    tmem_ld32(tmem_O(t) + lane_off + (uint32_t)(c * 32), o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                    tmem_st32(tmem_O(t) + lane_off + (uint32_t)(c * 32), o);
                }
                tmem_st_wait();
            };
            // whether some row of the warp has outgrown its reference (false when both are -inf: NaN compare)
            auto outgrown = [&](float m_new) { return __any_sync(0xffffffffu, (m_new - m_ref) > kRescaleThreshold); };
            bool plain = kMode == kPlain && h > 0 && !cut;
            if (plain) {
                RowMax mx;
                exp_row<true>(s, p.scale_log2, shift(), pk, sum, mx);
                SNTL_TRACE_EV(tw, 1 + t, tn, 3);
                if (outgrown(fmaxf(m_ref, mx.value() * p.scale_log2))) {
                    plain = false;
                    sum[0] = sum[1] = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int c = 0; c < 2; ++c) tmem_ld32(tmS + (uint32_t)(c * 32), s + c * 32);    // (kept, it would take 64 registers more)
                    tmem_ld_wait();
                }
            }
            if (!plain) {
                if (cut) {
                    if (limit < kHalf) {
#pragma unroll
                        for (int c = 0; c < kHalf; ++c)
                            if (c >= limit) s[c] = 0xff800000u;  // -inf
                    }
                    const int lo = kWin ? grow - p.window + 1 - key0 : 0;
                    if (kWin && lo > 0 && glim < min(lo, kHalf)) {      // keys below the window that are no global tokens
#pragma unroll
                        for (int c = 0; c < kHalf; ++c)
                            if (c < lo && c >= glim) s[c] = 0xff800000u;
                    }
                }
                const float m_new = fmaxf(m_ref, row_max(s) * p.scale_log2);
                if (h == 0) m_ref = m_new;
                else if (outgrown(m_new)) rescale(m_new);
                if (!ok) break;
                SNTL_TRACE_EV(tw, 1 + t, tn, 4);
                RowMax unused;
                exp_row<false>(s, p.scale_log2, shift(), pk, sum, unused);
            }
            if (b) phase[0] ^= 1u, phase[1] ^= 1u;
            s_seen = h + 1 < 2 * n_mine && __all_sync(0xffffffffu, mbar_test(&bars->s_ready[t][b ^ 1], b ? phase[0] : phase[1]));
            tmem_st32(tmS, pk);      // over S
            l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
            SNTL_TRACE_EV(tw, 1 + t, tn, 5);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&bars->p_ready[t][b]);
            SNTL_TRACE_EV(tw, 1 + t, tn, 6);
        }
        if (ok && n_mine > 0) {
            ok = mbar_wait_prompt_warp(&bars->o_ready[t], blocks, abort_flag, kSiteOReady);
            blocks ^= 1u;
            phase[0] ^= 1u;
        }
        if (ok && n_mine > 0) {
            tc_fence_after();
            const float inv = l > 0.0f ? 1.0f / l : 0.0f;
            const bool store = grow < p.Sq;
            // Coalesced store of O.  A thread holds one whole row (2*D bytes); written straight from there a warp's store
            // instruction would touch 32 rows, 16 bytes each.  So the warp's 32 rows go through 4 KB of shared memory of its own, 64
            // columns at a time, and come back out with each store instruction covering 128 bytes of four rows.  Only the rows of
            // this warp are exchanged, so a warp-level sync is all it takes; 16-byte units are XOR-swizzled by the row so
            // that both the row-wise writes and the row-wise reads spread over the banks.
            const int bh = w.bh;
            if constexpr (kMat) {
                // feature-major matrices: the 32 rows of a warp are 128 contiguous bytes of every feature's row
                const int b = bh / p.Hq, h = bh - b * p.Hq;
                float* dst = p.o_mat + (long long)h * D * p.mat_stride + (long long)b * p.Sq + grow;
#pragma unroll
                for (int c = 0; c < D / 32; ++c) {
                    uint32_t o[32];
                    tmem_ld32(tmem_O(t) + lane_off + (uint32_t)(c * 32), o);
                    tmem_ld_wait();
                    if (store) {
#pragma unroll
                        for (int i = 0; i < 32; ++i) dst[(c * 32 + i) * p.mat_stride] = __uint_as_float(o[i]) * inv;
                    }
                }
                if (store)
                    p.lse_mat[(long long)h * p.mat_stride + (long long)b * p.Sq + grow] = l > 0.0f ? (m_ref + log2f(l)) * 0.6931471805599453f : -INFINITY;
            } else {
            uint8_t* stage = sOut + warp * 4096;
            const int sub = lane >> 3, unit0 = lane & 7, warp_row0 = grow - lane;      // (first row of this warp inside the slab)
            __nv_bfloat16* dst = p.o + (size_t)bh * p.Sq * D;
#pragma unroll
            for (int half = 0; half < D / 64; ++half) {
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    uint32_t o[32];
                    tmem_ld32(tmem_O(t) + lane_off + (uint32_t)(half * 64 + c * 32), o);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint4 v;
                        v.x = pack_bf16(__uint_as_float(o[8 * i + 0]) * inv, __uint_as_float(o[8 * i + 1]) * inv);
                        v.y = pack_bf16(__uint_as_float(o[8 * i + 2]) * inv, __uint_as_float(o[8 * i + 3]) * inv);
                        v.z = pack_bf16(__uint_as_float(o[8 * i + 4]) * inv, __uint_as_float(o[8 * i + 5]) * inv);
                        v.w = pack_bf16(__uint_as_float(o[8 * i + 6]) * inv, __uint_as_float(o[8 * i + 7]) * inv);
                        *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + i) ^ (lane & 7)) << 4)) = v;
                    }
                }
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const int r = i * 4 + sub;
                    const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 128 + ((unit0 ^ (r & 7)) << 4));
                    if (warp_row0 + r < p.Sq) *reinterpret_cast<uint4*>(dst + (size_t)(warp_row0 + r) * D + half * 64 + unit0 * 8) = v;
                }
                __syncwarp();
            }
            if (store)
                p.lse[(size_t)bh * p.Sq + grow] = l > 0.0f ? (m_ref + log2f(l)) * 0.6931471805599453f : -INFINITY;
            }
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

// ---- head_dim 64 ----
// Bound by the exponentials: 2048 cycles of the special-function unit for two tiles of 128 x 128, beside 1280 of products.  With two
// softmax warps per scheduler, one per query tile, a step of two tiles took 3490 cycles: both warps wait for products, load, store
// and hand over about as long as they compute.  Here four warps per scheduler work on four independent chains (S 64 columns and O 64
// columns each fill the TMEM; the 96 registers that 640 threads can have at compile time hold 64 columns, under a window with 16 bytes
// spilled), and a step takes 2460 to 2520 cycles in long rows, 2700 to 2870 in rows of 16 key tiles.
// The two query tiles of a CTA are halves that share nothing but the TMEM allocation and the queue of blocks: the end of a block
// (4700 to 5800 cycles from its last S to the first S of the next) then passes under the other half's steps, no tile waits for
// the longer row of another, and blocks of one tile balance better.
// us, two warps per scheduler and the longer form of waits -> now: B4 Hq32 Hkv8 S4096 407 -> 343; B8 Hq12 S1024 34.6 -> 28.3; B2 Hq32 S1024 25.2 ->
// 19.5; B16 Hq8 S130 8.3 -> 7.6; a 300-key window over B4 Hq12 S2048 39.2 -> 35.7; one block of one tile 5.3 -> 5.5 (its two streams meet once
// more).  Of the first three 7 to 9 % are the waits' alone.  Also measured, when the streams took 351, 28.5 and 19.4: both tiles fed by one
// MMA warp, 351, 28.2 and 27.9; two softmax warpgroups with two S buffers of 64 columns each, 436, 32.0 and 25.2.  The key loop is
// sensitive to what the compiler does with code outside it: forms of the set-up that differ in nothing else came out up to 4 % apart.
constexpr int kStreamThreads = 640;   // four softmax warpgroups, and one holding the MMA and the TMA warps

// One half of a CTA: blocks of one query tile, two softmax warpgroups ("streams": stream b has keys [64 b, 64 b + 64) of every key
// tile), an MMA warp and a TMA warp.
struct StreamHalf {
    uint4 response;                   // of the block scheduler
    uint64_t response_full, work_full[2], work_empty[2];
    struct alignas(16) { int n, q0, bh, unused, g_tiles, w_first; } work[2];    // blocks in turn (see FwdWork); n: key tiles, -1: no more blocks
    uint64_t q_full, q_empty, k0_full, pair_full[2], pair_empty[2];    // as in FwdBarriers
    uint64_t s_ready[2];              // S_j of the stream is there, and P_{j-1} V has been added to O
    uint64_t o_ready[2];              // the last P V of a block has been.  (A phase of s_ready instead could be over before it is seen: the
                                      // next block's first S does not wait for the softmax warps.)
    uint64_t p_ready[2];
    uint64_t o_read;                  // every softmax warp has read O and ml of a block
    uint64_t final_bar;
    float2 ml[2][kM];                 // reference maximum and sum of a row, for its other stream
};
struct StreamShared {
    StreamHalf half[2];
    uint32_t tmem_base;
    uint32_t abort_flag;
    uint32_t asking, none_left;       // a lock, and what it guards: no request may follow one that has failed
};

template <int kMode, bool kMat>
__global__ void __launch_bounds__(kStreamThreads, 1)
attn_fwd_streams_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                        const __grid_constant__ CUtensorMap tmap_v, const FwdParams p)
{
    enum : uint32_t {       // (the status word tells the two kernels apart)
        kSiteQ = 33, kSiteK0, kSitePairFull, kSitePairEmpty, kSiteSReady, kSitePReady, kSiteOReady, kSiteFinal, kSiteQEmpty, kSiteNext, kSiteORead
    };
    constexpr int D = 64, kTileBytes = 128 * D * 2;
    constexpr uint32_t kHalfBytes = kHalf * 128;    // of a K or V tile
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = (uint8_t*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t* sOut = smem + 10 * kTileBytes;           // 2 KB per softmax warp
    StreamShared* shared = (StreamShared*)(sOut + (kMat ? 0 : kOutBytes));
    volatile uint32_t* abort_flag = &shared->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (warp-uniform for the compiler)
    constexpr bool kWin = kMode != kPlain;
    const int inst = warp < 16 ? warp >> 3 : (warp >> 1) & 1;    // warps 0-7 and 8-15: softmax; 16, 18: MMA; 17, 19: TMA
    StreamHalf* bars = &shared->half[inst];
    uint8_t* sQ = smem + inst * 5 * kTileBytes;       // [kTileBytes]
    uint8_t* sK = sQ + kTileBytes;                    // [2][kTileBytes]
    uint8_t* sV = sK + 2 * kTileBytes;                // [2][kTileBytes]

    // first block of this half, or -1: the second half either asks for one or has the light one that goes with the first half's heavy one
    const int first = inst == 0 ? (int)blockIdx.x
                      : p.second_blocks && 2 * (int)gridDim.x - 1 - (int)blockIdx.x < p.second_blocks ? 2 * (int)gridDim.x - 1 - (int)blockIdx.x
                                                                                                      : -1;

    // ---- setup ----
    FwdWork w{};        // (the producers')
    if (warp >= 16 && (warp & 1) && lane == 0) {
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
        mbar_init(&bars->q_full, 1);
        mbar_init(&bars->q_empty, 1);
        mbar_init(&bars->k0_full, 1);
        mbar_init(&bars->response_full, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->work_full[i], 1);
            mbar_init(&bars->work_empty[i], 9);    // the issuing warp and the softmax warps
            mbar_init(&bars->pair_full[i], 1);
            mbar_init(&bars->pair_empty[i], 1);
            mbar_init(&bars->s_ready[i], 1);
            mbar_init(&bars->o_ready[i], 1);
            mbar_init(&bars->p_ready[i], 128);
        }
        mbar_init(&bars->o_read, 8);
        mbar_init(&bars->final_bar, 1);
        shared->abort_flag = shared->asking = shared->none_left = 0;
        fence_mbar_init();
    }
    if (warp == 16) {
        tmem_alloc(&shared->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = shared->tmem_base;
    wait_for_stream();      // nothing before this reads or writes global memory
    auto tmem_S = [&](int b) { return tmem + (uint32_t)(inst * 2 * kHalf + b * kHalf); };
    auto tmem_O = [&](int b) { return tmem + 256u + (uint32_t)(inst * 2 * D + b * D); };

    // Every role walks the same blocks, which the producer decodes into shared memory: number u is work[u & 1].  Counters of key
    // tiles run on over the blocks, so stages and barrier phases continue where they are.
    constexpr int kGaveUp = -2;
    int2 win = make_int2(0, 0);   // its g_tiles, w_first
    // A warp's copy of block u (work: n, q0, bh); false when there is none, or when the wait for it gave up (n = kGaveUp).  Every
    // access to shared memory waits some 250 cycles behind the other warps' exponentials, so there are few of them, and the softmax
    // warps take the next block before their epilogue.
    auto get = [&](int u, int4& work) {
        work.x = kGaveUp;
        if (!mbar_wait_prompt_warp(&bars->work_full[u & 1], (uint32_t)((u >> 1) & 1), abort_flag, kSiteNext)) return false;
        work = *reinterpret_cast<const int4*>(&bars->work[u & 1]);
        if (kWin) win = *reinterpret_cast<const int2*>(&bars->work[u & 1].g_tiles);
        work.x = warp_uniform(work.x);
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->work_empty[u & 1]);
        return work.x >= 0;
    };

    // 640 threads start with 96 registers each
    if (warp >= 16 && (warp & 1)) {
        setmaxnreg_dec<64>();
        // =========================== TMA producer ===========================
        if (lane == 0) {
            // A block of the grid that has not started, or -1.  Both producers of the CTA ask, one at a time: none may ask once the
            // answer was that there are no more.
            uint32_t asked = 0;
            auto ask = [&]() {
                if (!p.several_waves) return -1;
                uint32_t spins = 0;
                while (atomicCAS(&shared->asking, 0u, 1u) != 0u) {
                    __nanosleep(40);
                    if (*abort_flag || ++spins > (1u << 24)) return -1;
                }
                int block = -1;
                if (!*(volatile uint32_t*)&shared->none_left) {
                    mbar_arrive_expect_tx(&bars->response_full, 16);
                    clc_try_cancel(&bars->response, &bars->response_full);
                    if (mbar_wait_prompt(&bars->response_full, asked++ & 1u, abort_flag, kSiteNext)) block = clc_first_block(&bars->response);
                    fence_proxy_async_smem();
                    if (block < 0) *(volatile uint32_t*)&shared->none_left = 1u;
                }
                __threadfence_block();
                atomicExch(&shared->asking, 0u);
                return block;
            };
            int c0 = 0, block = first >= 0 ? first : ask();
            for (int u = 0;; ++u) {
                if (block < 0) w.n0 = -1;
                else w.decode<kWin>(p, block);
                const int n = w.n0;
                if (u >= 2 && !mbar_wait_prompt(&bars->work_empty[u & 1], (uint32_t)(((u >> 1) - 1) & 1), abort_flag, kSiteNext)) break;
                bars->work[u & 1] = {n, w.q0, w.bh, 0, w.g_tiles, w.w_first};
                mbar_arrive(&bars->work_full[u & 1]);
                if (block < 0) break;
                auto load = [&](uint8_t* dst, const CUtensorMap* map, uint64_t* bar, int j) {
                    tma_load_3d(dst + ((c0 + j) & 1) * kTileBytes, map, bar, 0, w.key_tile(j) * kN, w.bh_kv);
                };
                // Q and K_0 once the last S product of the block before has run: Q is free then, and K_0's stage and barrier were free
                // before (the barrier must not be armed again while the K_0 before is on its way or unseen: rows of a single
                // key tile get here that early)
                if (u > 0 && !mbar_wait_prompt(&bars->q_empty, (uint32_t)((u - 1) & 1), abort_flag, kSiteQEmpty)) break;
                mbar_arrive_expect_tx(&bars->k0_full, (uint32_t)kTileBytes);
                load(sK, &tmap_k, &bars->k0_full, 0);
                mbar_arrive_expect_tx(&bars->q_full, (uint32_t)kTileBytes);
                tma_load_3d(sQ, &tmap_q, &bars->q_full, 0, w.q0, w.bh);
                bool ok = true;
                for (int j = 0; j < n; ++j) {
                    // (as in attn_fwd_tc_kernel)
                    const int c = c0 + j;
                    if (c >= 1 && !(ok = mbar_wait_prompt(&bars->pair_empty[c & 1], (uint32_t)((c >> 1) - (c & 1 ? 0 : 1)) & 1u, abort_flag, kSitePairEmpty))) break;
                    const bool k_too = j + 1 < n;
                    mbar_arrive_expect_tx(&bars->pair_full[c & 1], (uint32_t)(k_too ? 2 * kTileBytes : kTileBytes));
                    if (k_too) load(sK, &tmap_k, &bars->pair_full[c & 1], j + 1);
                    load(sV, &tmap_v, &bars->pair_full[c & 1], j);
                }
                if (!ok) break;
                c0 += n;
                // (about two steps before this block ends: in time, and not so early that blocks would go to this CTA although others
                // are free sooner)
                block = ask();
            }
        }
    } else if (warp >= 16) {
        setmaxnreg_dec<64>();
        // =========================== MMA issuer ===========================
        auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t site) { return mbar_wait_prompt_warp(bar, parity, abort_flag, site); };
        constexpr uint32_t idesc_s = make_idesc(kM, kHalf, false, false);
        constexpr uint32_t idesc_pv = make_idesc(kM, D, false, true);
        const uint64_t dq = make_sdesc(smem_u32(sQ), 16, 1024), dk = make_sdesc(smem_u32(sK), 16, 1024), dv = make_sdesc(smem_u32(sV), 16384, 1024);
        auto issue_s = [&](int b, int st) {
            mma_ss_4<2, 2>(tmem_S(b), dq, sdesc_advance(dk, (uint32_t)(st * kTileBytes) + (uint32_t)b * kHalfBytes), idesc_s, 0);
            tc_commit_p(&bars->s_ready[b]);
        };
        int c0 = 0;                        // key tiles of the blocks before
        bool ok = true;
        int4 work;
        for (int u = 0; ok && get(u, work); ++u) {
            const int n = work.x;
            if (!(ok = wait(&bars->k0_full, (uint32_t)(u & 1), kSiteK0) && wait(&bars->q_full, (uint32_t)(u & 1), kSiteQ))) break;
            tc_fence_after();
            // (S of the block before has been read and P over it consumed: this warp waited for p_ready and issued the product; O is
            // overwritten behind o_read)
#pragma unroll
            for (int b = 0; b < 2; ++b) issue_s(b, c0 & 1);
            tc_commit_p(&bars->pair_empty[(c0 - 1) & 1]);        // K_0 and the last V of the block before
            if (n == 1) tc_commit_p(&bars->q_empty);
            for (int j = 0; ok && j < n; ++j) {
                const int c = c0 + j;
                if (!(ok = wait(&bars->pair_full[c & 1], (uint32_t)((c >> 1) & 1), kSitePairFull))) break;
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    if (!ok || !(ok = wait(&bars->p_ready[b], (uint32_t)(c & 1), kSitePReady))) continue;
                    if (b == 0 && j == 0 && u > 0 && !(ok = wait(&bars->o_read, (uint32_t)((u - 1) & 1), kSiteORead))) continue;
                    tc_fence_after();
                    mma_ts_4<8, 128>(tmem_O(b), tmem_S(b), sdesc_advance(dv, (uint32_t)((c & 1) * kTileBytes) + (uint32_t)b * kHalfBytes), idesc_pv, j > 0);
                    if (j + 1 < n) issue_s(b, (c + 1) & 1);
                    else tc_commit_p(&bars->o_ready[b]);
                }
                if (!ok) break;
                if (j + 1 < n) tc_commit_p(&bars->pair_empty[c & 1]);
                if (j + 2 == n) tc_commit_p(&bars->q_empty);
            }
            c0 += n;
        }
        // every MMA issued above must have retired before shared memory / TMEM are given up
        tc_commit_p(&bars->final_bar);
        wait(&bars->final_bar, 0, kSiteFinal);
    } else {
        // =========================== softmax + epilogue warpgroups ===========================
        setmaxnreg_inc<104>();
        const int half = (warp >> 2) & 1;
        const int row = (warp & 3) * 32 + lane;        // row inside the tile == TMEM lane
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tmS = tmem_S(half) + lane_off, tmO = tmem_O(half) + lane_off;
        SNTL_TRACE_DECL(tn);
        const bool tw = (warp & 3) == 0 && lane == 0;
        (void)tw;
        bool ok = true;
        uint32_t phase = 0;                            // of s_ready
        int4 work;
        bool more = get(0, work);
        // The eight warps of a half meet in a named barrier, which has no limit: here and at the end of each block.  A warp whose wait
        // gave up goes there all the same and says so, and then all leave.
        more = named_barrier_all(1 + inst, 256, work.x != kGaveUp) && more;
        for (int u = 0; more; ++u) {
            const int n_mine = work.x, q0 = work.y, bh = work.z;
            const int g_tiles = kWin ? win.x : 0, w_first = kWin ? win.y : 0;
            const int grow = q0 + row;                 // query row inside the (batch, head) slab
            const int row_lo = q0 + (warp & 3) * 32;   // first row of the warp
            float m_ref = -INFINITY, l = 0.0f;
            for (int j = 0; j < n_mine; ++j) {
                if (!(ok = mbar_wait_prompt_warp(&bars->s_ready[half], phase, abort_flag, kSiteSReady))) break;
                SNTL_TRACE_EV(tw, warp >> 2, tn, 1);
                phase ^= 1u;
                tc_fence_after();
                uint32_t s[kHalf];
#pragma unroll
                for (int c = 0; c < 2; ++c) tmem_ld32(tmS + (uint32_t)(c * 32), s + c * 32);
                tmem_ld_wait();
                SNTL_TRACE_EV(tw, warp >> 2, tn, 2);
                // number of visible keys of this row among these
                const int key0 = (j < g_tiles ? j : w_first + (j - g_tiles)) * kN + half * kHalf;
                const int limit_lo = (p.causal ? min(p.Skv, row_lo + 1) : p.Skv) - key0;
                const int lo_hi = kWin ? row_lo + 31 - p.window + 1 - key0 : 0, glim = kWin ? p.global_tokens - key0 : 0;
                const bool cut = limit_lo < kHalf || (kWin && lo_hi > 0 && glim < min(lo_hi, kHalf));   // (some row of the warp is)
                uint32_t pk[32];
                float2 sum[2] = {make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)};
                auto shift = [&]() { return m_ref == -INFINITY ? 0.0f : -m_ref; };   // (no finite score so far: -inf + inf would be NaN)
                // whether some row of the warp has outgrown its reference (false when both are -inf: NaN compare)
                auto outgrown = [&](float m_new) { return __any_sync(0xffffffffu, (m_new - m_ref) > kRescaleThreshold); };
                // Keys that the mask does not cut are exponentiated against the row's reference at once, with their maximum taken on the
                // way (see attn_fwd_tc_kernel)
                bool done = j > 0 && !cut;
                if (done) {
                    RowMax mx;
                    exp_row<true>(s, p.scale_log2, shift(), pk, sum, mx);
                    if (outgrown(fmaxf(m_ref, mx.value() * p.scale_log2))) {
                        done = false;
                        sum[0] = sum[1] = make_float2(0.0f, 0.0f);
#pragma unroll
                        for (int c = 0; c < 2; ++c) tmem_ld32(tmS + (uint32_t)(c * 32), s + c * 32);
                        tmem_ld_wait();
                    }
                }
                if (!done) {
                    if (cut) {
                        const int limit = (p.causal ? min(p.Skv, grow + 1) : p.Skv) - key0;
                        if (limit < kHalf) {       // (under a window often only the other mask cuts)
#pragma unroll
                            for (int c = 0; c < kHalf; ++c)
                                if (c >= limit) s[c] = 0xff800000u;  // -inf
                        }
                        const int lo = kWin ? grow - p.window + 1 - key0 : 0;
                        if (kWin && lo > 0 && glim < min(lo, kHalf)) {      // keys below the window that are no global tokens
#pragma unroll
                            for (int c = 0; c < kHalf; ++c)
                                if (c < lo && c >= glim) s[c] = 0xff800000u;
                        }
                    }
                    const float m_new = fmaxf(m_ref, row_max(s) * p.scale_log2);
                    if (j == 0) {
                        m_ref = m_new;
                    } else if (outgrown(m_new)) {
                        // O and the sum of a row whose maximum has outgrown its reference (S_j was issued behind the product of P_{j-1})
                        const bool need = (m_new - m_ref) > kRescaleThreshold;
                        const float factor = need ? ex2(m_ref - m_new) : 1.0f;
                        if (need) m_ref = m_new;
                        l *= factor;
#pragma unroll 1
                        for (int c = 0; c < D / 8; ++c) {
                            uint32_t o[8];
                            tmem_ld8(tmO + (uint32_t)(c * 8), o);
                            tmem_ld_wait();
#pragma unroll
                            for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * factor);
                            tmem_st8(tmO + (uint32_t)(c * 8), o);
                        }
                        tmem_st_wait();
                    }
                    RowMax unused;
                    exp_row<false>(s, p.scale_log2, shift(), pk, sum, unused);
                }
                SNTL_TRACE_EV(tw, warp >> 2, tn, 3);
                tmem_st32(tmS, pk);      // over S
                l += (sum[0].x + sum[0].y) + (sum[1].x + sum[1].y);
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&bars->p_ready[half]);
                SNTL_TRACE_EV(tw, warp >> 2, tn, 4);
            }
            if (!ok || (more = get(u + 1, work), work.x == kGaveUp) || !mbar_wait_prompt_warp(&bars->o_ready[half], (uint32_t)(u & 1), abort_flag, kSiteOReady)) {
                named_barrier_all(1 + inst, 256, false);
                break;
            }
            // The two streams of a row are added here; each stores one half of the features.
            SNTL_TRACE_EV(tw, warp >> 2, tn, 5);
            bars->ml[half][row] = make_float2(m_ref, l);
            tc_fence_before();
            if (!named_barrier_all(1 + inst, 256, true)) break;
            tc_fence_after();
            const float2 ml = bars->ml[half ^ 1][row];
            uint32_t o[2][32];
            tmem_ld32(tmO + (uint32_t)(half * 32), o[0]);
            tmem_ld32(tmem_O(half ^ 1) + lane_off + (uint32_t)(half * 32), o[1]);
            const float m = fmaxf(m_ref, ml.x);
            float f0 = m_ref == -INFINITY ? 0.0f : ex2(m_ref - m), f1 = ml.x == -INFINITY ? 0.0f : ex2(ml.x - m);
            // (the same order of the two in both, for the same bits)
            const float total = half == 0 ? fmaf(l, f0, ml.y * f1) : fmaf(ml.y, f1, l * f0);
            const float inv = total > 0.0f ? 1.0f / total : 0.0f;
            f0 *= inv;
            f1 *= inv;
            tmem_ld_wait();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&bars->o_read);      // (and ml: it is written behind products that wait for this)
#pragma unroll
            for (int i = 0; i < 32; ++i) o[0][i] = __float_as_uint(fmaf(__uint_as_float(o[0][i]), f0, __uint_as_float(o[1][i]) * f1));
            const bool store = grow < p.Sq;
            if constexpr (kMat) {
                // feature-major matrices: the 32 rows of a warp are 128 contiguous bytes of every feature's row
                const int b = bh / p.Hq, h = bh - b * p.Hq;
                float* dst = p.o_mat + (long long)(h * D + half * 32) * p.mat_stride + (long long)b * p.Sq + grow;
                if (store) {
#pragma unroll
                    for (int i = 0; i < 32; ++i) dst[i * p.mat_stride] = __uint_as_float(o[0][i]);
                    if (half == 0)
                        p.lse_mat[(long long)h * p.mat_stride + (long long)b * p.Sq + grow] = total > 0.0f ? (m + log2f(total)) * 0.6931471805599453f : -INFINITY;
                }
            } else {
                // Through 2 KB of shared memory of the warp's own, so that a store instruction covers 64 bytes of each of eight rows; 16-byte
                // units are XOR-swizzled by the row so that both sides spread over the banks.
                uint8_t* stage = sOut + warp * 2048;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint4 v;
                    v.x = pack_bf16(__uint_as_float(o[0][8 * i + 0]), __uint_as_float(o[0][8 * i + 1]));
                    v.y = pack_bf16(__uint_as_float(o[0][8 * i + 2]), __uint_as_float(o[0][8 * i + 3]));
                    v.z = pack_bf16(__uint_as_float(o[0][8 * i + 4]), __uint_as_float(o[0][8 * i + 5]));
                    v.w = pack_bf16(__uint_as_float(o[0][8 * i + 6]), __uint_as_float(o[0][8 * i + 7]));
                    *reinterpret_cast<uint4*>(stage + lane * 64 + ((i ^ ((lane >> 1) & 3)) << 4)) = v;
                }
                __syncwarp();
                __nv_bfloat16* dst = p.o + (size_t)bh * p.Sq * D;
                const int sub = lane >> 2, unit = lane & 3, warp_row0 = grow - lane;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = i * 8 + sub;
                    const uint4 v = *reinterpret_cast<const uint4*>(stage + r * 64 + ((unit ^ ((r >> 1) & 3)) << 4));
                    if (warp_row0 + r < p.Sq) *reinterpret_cast<uint4*>(dst + (size_t)(warp_row0 + r) * D + half * 32 + unit * 8) = v;
                }
                __syncwarp();
                if (store && half == 0) p.lse[(size_t)bh * p.Sq + grow] = total > 0.0f ? (m + log2f(total)) * 0.6931471805599453f : -INFINITY;
            }
            SNTL_TRACE_EV(tw, warp >> 2, tn, 6);
        }
    }

    // ---- teardown ----
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);      // (see attn_fwd_tc_kernel)
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 16) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                  const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* sym = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = (EncodeTiledFn)sym;
    });
    return fn;
}

// head_dim 128.  Two query tiles per CTA overlap one tile's softmax with the other's products; on a grid that leaves SMs idle or ends
// with one long CTA, one tile per CTA finishes sooner.  The estimate counts steps of two tiles.  A step of one tile is 2/3 of one
// (1.1 us of 1.65 over rows of 2 to 8 steps).  With at most one block per SM the longest decides.  With up to two, the lightest blocks
// come second on the SMs that are free first (two sums bound that), and a second block costs 2.2 steps more than its own where a CTA has
// one tile and 1.2 where it has two: its loads, its first products and the end of the block before pass with little else to do (192 blocks
// of one tile and one or two steps 11.4 us, 148 or fewer of two steps 7.5).  With more, the SMs' average load and a tail.
// Measured with either form on 200 grids (8 to 256 heads, 100 to 8192 queries, windows, no mask): the choice is the better one, or within
// the 2 to 4 % by which two runs of such calls differ.  An estimate without the second block's cost took one tile for B4 Hq16 S333 (12.3 us, 9.5 with two) and B4 Hq12 S640
// (15.2 and 13.0), and two for B6 Hq16 S333 (15.7 and 14.7).
int fwd_tiles_per_cta(const AttnShape& s)
{
    const int n = (s.Sq + kM - 1) / kM, n_keys = (s.Skv + kN - 1) / kN, heads = s.B * s.Hq, sms = sm_count();
    if (n == 1) return 1;
    if ((long long)((n + 1) / 2) * heads > 2 * sms) return 2;
    const int reach = s.causal && s.window > 0 ? (s.window + kN - 1) / kN + 1 + (s.global_tokens + kN - 1) / kN : n_keys;
    auto time = [&](int tiles, double second) {
        const int per_head = (n + tiles - 1) / tiles, blocks = per_head * heads;
        // of the blocks of each head, in the order in which they start
        auto cost = [&](int rank) {
            const int first = (s.causal ? per_head - 1 - rank : rank) * tiles, last = std::min(n, first + tiles) - 1;
            return std::min(s.causal ? last + 1 : n_keys, reach) * (last > first ? 1.0 : 2.0 / 3.0);
        };
        auto block = [&](int i) { return cost(i / heads); };
        const double longest = std::max(cost(0), cost(std::min(1, per_head - 1)));     // (the first may be a lone tile)
        if (blocks <= sms) return longest;
        if (blocks <= 2 * sms)
            return std::max(longest, std::max(block(sms - 1) + block(sms), block(2 * sms - blocks) + block(blocks - 1)) + second);
        double sum = 0.0;
        for (int i = 0; i < per_head; ++i) sum += cost(i);
        return std::max(longest, (sum * heads + second * blocks) / sms - second + 0.2 * longest);
    };
    return time(1, 2.2) < 0.95 * time(2, 1.2) ? 1 : 2;
}

template <int D, int kMode, bool kMat>
cudaError_t launch_fwd(const TcArgs& a, cudaStream_t st)
{
    const AttnShape& s = a.s;
    CUtensorMap tq, tk, tv;
    cudaError_t e;
    if ((e = encode_tmap_bf16_3d(&tq, a.q, D, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tk, a.k, D, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tv, a.v, D, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    FwdParams p{};
    p.o = a.o_out;
    p.lse = a.lse_out;
    p.o_mat = a.mat.o; p.lse_mat = a.mat.lse; p.mat_stride = a.mat.stride;
    p.B = s.B; p.Hq = s.Hq; p.Hkv = s.Hkv; p.Sq = s.Sq; p.Skv = s.Skv;
    p.causal = s.causal;
    p.window = s.causal ? s.window : 0;
    p.global_tokens = s.global_tokens;
    p.tiles_per_cta = D == 64 ? 1 : fwd_tiles_per_cta(s);
    p.n_qblk = (s.Sq + p.tiles_per_cta * kM - 1) / (p.tiles_per_cta * kM);
    p.scale_log2 = s.scale * 1.4426950408889634f;
    const long long ctas = (long long)p.n_qblk * s.B * s.Hq;
    if (ctas > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    // At head_dim 64 a CTA has two blocks at a time.  With up to two per SM, which half takes which is settled at the launch: asked for, a
    // second block starts about 1 us later, beside whichever block is there, and a CTA that asks early may take one that an idle SM was
    // about to start.  us: B1 Hq32 S1024 (256 blocks) 15.6 -> 13.4, B1 Hq16 S2048 24.5 -> 20.7, B4 Hq16 S333 (192) 9.3 -> 8.3.
    const long long sms = sm_count();
    p.several_waves = ctas > (D == 64 ? 2 * sms : sms);
    p.second_blocks = D == 64 && ctas > sms && !p.several_waves ? (int)ctas : 0;
    const size_t smem = (D == 64 ? 10 : 6) * (size_t)(128 * D * 2) + (kMat ? 0 : kOutBytes) + (D == 64 ? sizeof(StreamShared) : sizeof(FwdBarriers)) + 1024;
    auto launch = [&](auto kernel, std::atomic<unsigned long long>& configured) {
        const cudaError_t err = ensure_dynamic_smem(kernel, smem, configured);
        return err != cudaSuccess ? err : launch_kernel(kernel, (unsigned)(p.second_blocks ? sms : ctas), D == 64 ? kStreamThreads : kFwdThreads, smem, st, 1, tq, tk, tv, p);
    };
    static std::atomic<unsigned long long> configured_one{0}, configured_many{0};   // per instantiation, one bit per device
    if constexpr (D == 64) {
        return launch(attn_fwd_streams_kernel<kMode, kMat>, configured_one);
    } else {
        if (p.several_waves) return launch(attn_fwd_tc_kernel<kMode, kMat, true>, configured_many);
        return launch(attn_fwd_tc_kernel<kMode, kMat, false>, configured_one);
    }
}

}  // namespace

// A training loop calls with the same tensors step after step (the reference's trainer even replays a captured graph
// with identical pointers, CudaLanguageModel.cu:2176-2209), and on small problems the seven driver calls that encode
// the tensor maps of one forward + backward are a visible part of the launch path.  So the last few encodings are
// kept, keyed by everything that goes into one; a tensor map holds no data, only the address and the geometry, so a
// hit is exact whatever has happened to the memory since.
namespace {
struct TmapKey {
    const void* base; int D, rows, slabs, box_rows, slab_rows;
    bool operator==(const TmapKey& o) const
    {
        return base == o.base && D == o.D && rows == o.rows && slabs == o.slabs && box_rows == o.box_rows && slab_rows == o.slab_rows;
    }
};
constexpr int kTmapCacheSize = 32;
struct TmapCache {
    std::mutex guard;
    TmapKey keys[kTmapCacheSize];
    CUtensorMap maps[kTmapCacheSize];
    int used = 0, next = 0;
};
TmapCache& tmap_cache()
{
    static TmapCache* c = new TmapCache;
    return *c;
}
}  // namespace

cudaError_t encode_tmap_bf16_3d(CUtensorMap* out, const void* base, int D, int rows, int slabs, int box_rows, int slab_rows)
{
    if (slab_rows <= 0) slab_rows = rows;   // rows of storage per slab (a KV cache holds more rows than are in use)
    const TmapKey key{base, D, rows, slabs, box_rows, slab_rows};
    TmapCache& cache = tmap_cache();
    {
        std::lock_guard<std::mutex> lock(cache.guard);
        for (int i = 0; i < cache.used; ++i)
            if (cache.keys[i] == key) { *out = cache.maps[i]; return cudaSuccess; }
    }
    const cudaError_t e = encode_tmap_bf16_3d_uncached(out, base, D, rows, slabs, box_rows, slab_rows);
    if (e == cudaSuccess) {
        std::lock_guard<std::mutex> lock(cache.guard);
        const int slot = cache.next;
        cache.keys[slot] = key;
        cache.maps[slot] = *out;
        cache.next = (slot + 1) % kTmapCacheSize;
        if (cache.used < kTmapCacheSize) ++cache.used;
    }
    return e;
}

cudaError_t encode_tmap_bf16_3d_uncached(CUtensorMap* out, const void* base, int D, int rows, int slabs, int box_rows, int slab_rows)
{
    EncodeTiledFn fn = encode_fn();
    if (!fn) return cudaErrorNotSupported;
    if (((uintptr_t)base & 15u) != 0) return cudaErrorMisalignedAddress;
    cuuint64_t dims[3] = {(cuuint64_t)D, (cuuint64_t)rows, (cuuint64_t)slabs};
    cuuint64_t strides[2] = {(cuuint64_t)D * 2, (cuuint64_t)slab_rows * D * 2};
    cuuint32_t box[3] = {64u, (cuuint32_t)box_rows, 1u};
    cuuint32_t estr[3] = {1u, 1u, 1u};
    CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(base), dims, strides, box, estr,
                    CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                    CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

bool tc_fwd_supported(const AttnShape& s)
{
    return (s.D == 64 || s.D == 128) && (!s.causal || s.Sq == s.Skv);
}

namespace {
template <int D>
cudaError_t dispatch_fwd(const TcArgs& a, cudaStream_t st)
{
    const bool win = a.s.causal && a.s.window > 0;
    if (a.mat.o) return win ? launch_fwd<D, kWindow, true>(a, st) : launch_fwd<D, kPlain, true>(a, st);
    return win ? launch_fwd<D, kWindow, false>(a, st) : launch_fwd<D, kPlain, false>(a, st);
}
}  // namespace

cudaError_t tc_forward(const TcArgs& a, cudaStream_t st)
{
    if (!aligned(16, a.q, a.k, a.v, a.o_out)) return cudaErrorMisalignedAddress;   // (matrix results go out element by element: o_out is null)
    return a.s.D == 64 ? dispatch_fwd<64>(a, st) : dispatch_fwd<128>(a, st);
}

#ifdef SNTL_TRACE
// trace build only: choose the CTA that records and read back what the last launch recorded
extern "C" int sntl_debug_trace_fwd(unsigned long long* out, int n_words, int set_cta)
{
    if (out && cudaMemcpyFromSymbol(out, ptx::g_trace, sizeof(unsigned long long) * n_words) != cudaSuccess) return 1;
    static unsigned long long zeros[ptx::kTraceRoles * ptx::kTraceDepth];
    if (cudaMemcpyToSymbol(ptx::g_trace, zeros, sizeof(zeros)) != cudaSuccess) return 2;
    unsigned int c = (unsigned int)set_cta;
    return cudaMemcpyToSymbol(ptx::g_trace_cta, &c, sizeof(c)) == cudaSuccess ? 0 : 3;
}
#endif

// Self-test of the bounded waits, one form per block, on a barrier that by construction never receives its arrival and with a limit
// of `limit_ns` instead of the kernels' one second: the wait of one thread (mbar_wait_for), its short form in one thread and in a
// warp, and eight warps of which every other one gives up before they meet in a named barrier.  The waits run out, record
// kSiteSelfTest in the status word as a stuck production wait records its own site, and the kernel returns normally (no trap, the
// context stays usable).  A form that says that the phase completed, does not set the CTA's flag, gives up before half its limit without
// being told to, or lets part of the warps go on records kSiteSelfTestFailed and its number instead.
constexpr uint32_t kSiteSelfTest = 0x7e, kSiteSelfTestFailed = 0x7d;
constexpr unsigned kSelfTestForms = 4;
__global__ void __launch_bounds__(256) wait_selftest_kernel(unsigned long long limit_ns)
{
    __shared__ uint64_t never, done;
    __shared__ uint32_t abort_word;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned form = blockIdx.x;
    if (threadIdx.x == 0) {
        ptx::mbar_init(&never, 1);
        ptx::mbar_init(&done, 1);
        abort_word = 0;
        ptx::fence_mbar_init();
    }
    __syncthreads();
    if (threadIdx.x == 0) ptx::mbar_arrive(&done);
    const unsigned long long t0 = ptx::global_timer_ns();
    const bool told = t0 < *(volatile unsigned long long*)&ptx::g_abort_until_ns;      // (by a give-up before this launch)
    bool fine = true;
    if (form == 0 && threadIdx.x == 0) fine = !ptx::mbar_wait_for(&never, 0, &abort_word, kSiteSelfTest, limit_ns);
    if (form == 1 && threadIdx.x == 0) fine = !ptx::mbar_wait_prompt(&never, 0, &abort_word, kSiteSelfTest, limit_ns);
    if (form == 2 && warp == 0) fine = !ptx::mbar_wait_prompt_warp(&never, 0, &abort_word, kSiteSelfTest, limit_ns);
    if (form == 3) {
        const bool came = ptx::mbar_wait_prompt_warp(warp & 1 ? &done : &never, 0, &abort_word, kSiteSelfTest, limit_ns);
        const bool some = ptx::named_barrier_all(1, 256, came), all = ptx::named_barrier_all(2, 256, true);     // (every warp meets in both)
        fine = came == (bool)(warp & 1) && !some && all;
    }
    const bool early = !told && (ptx::global_timer_ns() - t0) * 2 < limit_ns;
    __syncthreads();
    if (lane == 0 && (!fine || (warp == 0 && (early || *(volatile uint32_t*)&abort_word != 1u))))
        atomicExch(&ptx::g_device_status, (kSiteSelfTestFailed << 24) | form);
}

cudaError_t launch_wait_selftest(unsigned long long limit_ns, cudaStream_t st)
{
    wait_selftest_kernel<<<kSelfTestForms, 256, 0, st>>>(limit_ns);
    count_launch();
    return cudaGetLastError();
}

cudaError_t read_and_clear_fwd_status(cudaStream_t st, uint32_t* word)
{
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    unsigned int w = 0, zero = 0;
    if ((e = cudaMemcpyFromSymbol(&w, ptx::g_device_status, sizeof(w))) != cudaSuccess) return e;
    if (w != 0 && (e = cudaMemcpyToSymbol(ptx::g_device_status, &zero, sizeof(zero))) != cudaSuccess) return e;
    uint32_t cache = 0;
    if ((e = read_and_clear_cache_status(&cache)) != cudaSuccess) return e;
    uint32_t f32 = 0;
    if ((e = read_and_clear_f32_fwd_status(&f32)) != cudaSuccess) return e;
    *word = w ? w : cache ? cache : f32;
    return cudaSuccess;
}

}  // namespace sntl
