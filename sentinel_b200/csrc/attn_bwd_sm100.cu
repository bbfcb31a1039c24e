// Causal attention backward for sm_100a: dQ, dK, dV with P recomputed from the saved log-sum-exp.
//
// Replaces the reference's CudaFlashAttentionDeltaEntry + CudaFlashAttentionBackwardQueryWmma64Entry
// (sentinel/NeuralNet/Cuda/CudaFlashAttention.cu:576-596, :1269-1456).  The reference walks query tiles and
// pushes dK/dV out with global atomics after scalar FMA loops; here all five products run on tcgen05 tensor
// cores and the loop is key-tile-outer:
//
//   * one block is one 128-key tile of one (batch, KV head), or a piece of one (BwdCut): it walks the 128-query tiles that can
//     see it, for every query head of the group, so dK and dV accumulate in TMEM for the whole block and are
//     written exactly once: deterministic, no atomics, grouped-query sums done in place (the reference
//     materialises repeated K/V and reduces afterwards, CudaCausalSelfAttention.cu:27-44);
//   * everything is computed transposed (rows = keys) so that both P^T and dS^T are consumed by the next MMA
//     straight from TMEM as the A operand:
//         S^T  = K  Q^T  - 1 (LSE/scale)^T    (K, Q  K-major from shared memory)      -> TMEM
//         dP^T = V  dO^T - 1 delta^T          (V, dO K-major from shared memory)      -> TMEM
//           (the rank-one terms ride along as one extra 16-wide contraction step: a constant block of ones on the key
//            side, a 16-byte record per query on the other -- the fp32 value split exactly in three bf16 -- so no
//            per-column operand reaches the compute warps)
//         P^T  = exp2(scale*log2e * that), causal mask on the diagonal tile, bf16 back over S^T
//         dV  += P^T  dO         (A = P^T in TMEM,  B = dO tile MN-major)
//         dS^T = P^T o that, a packed bf16 product, into a shared-memory tile [key][query]
//         dQ_i = dS   K          (A = that tile read MN-major, B = K tile MN-major)
//         dK  += dS^T Q          (A = the same tile read K-major, B = Q tile MN-major)
//     the softmax scale is folded into the final dK store and the dQ conversion pass;
//   * dQ_i lands in TMEM (over the dP^T columns, which are dead by then) and a drain warpgroup adds it into an
//     fp32 accumulator in global memory with coalesced 16-byte vector reductions; the accumulator uses a
//     per-tile [d/4][row][4] order so that the 32 rows of a warp hit consecutive addresses;
//   * warp roles: 2 compute warpgroups (each owns 64 of the 128 query columns, one thread per key row),
//     1 drain warpgroup, 2 MMA-issuing warps, 1 TMA-producer warp; registers are re-allocated per role
//     (setmaxnreg).  Q (with its LSE records) has two stages and dO (with its delta records) one at D=128
//     (shared-memory capacity); three and two at D=64.
//
// A pre-pass computes the per-query terms (row_terms.cuh: from delta = rowsum(dO o O) and LSE; padded rows get a term that makes
// P = 0) and zeroes the dQ accumulator; a post-pass converts the accumulator to bf16 dQ (times scale).
//
// Long key tiles are cut into pieces (BwdCut): one CTA per (key tile, KV head, piece), each leaving its dK/dV as an fp32
// partial in scratch, and a small kernel adds the partials in piece order (deterministic) and writes the result.
//
// Under SNTL_FLAG_DETERMINISTIC (kDet) the dQ contributions of the key tiles are summed as 64-bit integers, which no order can change:
// at head_dim 64 the drain warpgroup pushes them as such; at 128 this kernel leaves dQ out and attn_dq_sm100.cu sums them (kOwnDq).
// TMEM map (512 columns): S^T/P^T [0,128)  dP^T/dQ [128,256)  then dV [256,384) dK [384,512) at head_dim 128, and
// dV [256,320) dK [320,384) plus a second S^T/P^T buffer [384,512) at head_dim 64.
#include "common.cuh"
#include "row_terms.cuh"
#include "sm100_ptx.cuh"

#include <string.h>

#include <algorithm>

namespace sntl {

using namespace ptx;

namespace {

constexpr int kMaxPieces = 16;          // of one key tile
constexpr int kT = 128;                 // tile edge: keys per CTA, queries per step
constexpr int kBwdThreads = 512;        // 2 compute WGs + drain WG + 1 WG holding the MMA warp and the producer warp
constexpr uint32_t kTmemCols = 512;

enum BwdSite : uint32_t {
    kSiteKV = 0x21, kSiteQFull, kSiteQEmpty, kSiteDoFull, kSiteDoEmpty, kSiteS, kSiteP, kSiteDP, kSiteDS, kSiteDQ,
    kSiteDrained, kSiteFinal, kSiteNext
};

struct BwdParams {
    __nv_bfloat16 *dk, *dv;
    // head_dim 64 (see bwd_folds_row_terms):
    const uint4* qaug;     // [B][Hq][Sq_pad] one 16-byte record per query: bf16 (hi, mid, lo, 0 x 5) of -LSE / scale
    const uint4* doaug;    // the same for -delta = -rowsum(dO o O)
    // head_dim 128:
    const float* lse2;     // [B][Hq][Sq_pad]  -LSE * log2(e), -inf on padded rows
    const float* delta;    // [B][Hq][Sq_pad]  -rowsum(dO o O)
    float* dq_accum;       // [B*Hq][n_qt][D/4][128][4]
    int B, Hq, Hkv, Sq, Skv, Sq_pad;
    int causal;
    int window, global_tokens;   // sliding window and always-visible first keys (0, 0: plain causal)
    int n_qt, n_kt;
    int split_tiles;       // the first split_tiles key tiles are cut into pieces (see BwdCut) of about split_steps steps,
    int split_steps, split_pieces, whole_first;   // at most split_pieces of a tile
    int piece_end[kMaxPieces];                    // blocks of all pieces up to this one (piece 0 of every cut tile, then piece 1, ...)
    int several_waves;     // more blocks than SMs
    float* dkv_part;       // [split tile][slab][piece][dV, dK][128][D] fp32
    float *dk_acc, *dv_acc;   // non-null: dK*scale / dV are ADDED into these fp32 [B*Hkv][Skv][D] tensors (no bf16 store)
    // non-null: dK / dV leave as fp32 feature-major matrices (see MatrixOut)
    float *dk_mat, *dv_mat;
    long long mat_stride;
    float scale, scale_log2;
};

// Query tiles per head that key tile kt visits (the kernel's own rule)
__host__ __device__ inline int bwd_tiles_per_head(int kt, int n_qt, int causal, int window, int global_tokens)
{
    const int qt_first = causal ? kt : 0;
    const int k0 = kt * kT;
    const int qt_last = (window > 0 && k0 >= global_tokens) ? min(n_qt - 1, (k0 + kT - 1 + window - 1) / kT) : n_qt - 1;
    return max(0, qt_last - qt_first + 1);
}

// A key tile's CTA visits `steps` (head of the group, query tile) pairs in order; a cut tile deals them to pieces of equal
// length, one CTA each.
__host__ __device__ inline int bwd_piece_count(int steps, int split_steps) { return (steps + split_steps - 1) / split_steps; }

// Which key tiles to cut, and how fine.  The CTA of key tile 0 visits every query tile of every head of its group; on a small
// grid (few sequences x KV heads, one layer's strong-scaling share, short batches) or where a window leaves only the tiles with
// global tokens long, that one CTA outlasts the average SM's whole load.  Cutting balances the grid and costs each piece its
// set-up and an fp32 partial of dK and dV: about one and a half steps for a CTA, four for a piece.  The estimate below weighs the
// two for a few piece lengths (a CTA's cost counts once per block, although blocks that follow one another in a CTA hide part of
// it).  B3 Hq16 Hkv4 S1237 D128 with reproducible dQ: 120 CTAs of up to 40 steps on 148 SMs took
// 158 us, 108 us cut.
struct BwdCut {
    int tiles = 0, steps = 1, pieces = 0;
    bool whole_first = false;      // some whole tile is longer than the pieces
};
inline size_t align256(size_t x) { return (x + 255) / 256 * 256; }
size_t bwd_base_bytes(const AttnShape& s)      // without the partials
{
    const size_t sq_pad = ((size_t)s.Sq + kT - 1) / kT * kT, rows = (size_t)s.B * s.Hq * sq_pad;
    return align256(kBwdRowAuxBytes * rows) + align256((s.deterministic ? 8 : 4) * rows * (size_t)s.D);
}
size_t bwd_part_bytes(const AttnShape& s, const BwdCut& c) { return (size_t)c.tiles * c.pieces * s.B * s.Hkv * 2 * kT * (size_t)s.D * 4; }

BwdCut bwd_cut_uncached(const AttnShape& s)
{
    const int group = s.Hq / s.Hkv, slabs = s.B * s.Hkv, sms = sm_count(), window = s.causal ? s.window : 0;
    const int n_qt = (s.Sq + kT - 1) / kT, n_kt = (s.Skv + kT - 1) / kT;
    auto steps = [&](int kt) { return bwd_tiles_per_head(kt, n_qt, s.causal, window, s.global_tokens) * group; };
    constexpr double kCta = 1.5, kPiece = 4.0;       // overhead in steps
    const int longest = steps(0);
    double total = 0.0;
    for (int kt = 0; kt < n_kt; ++kt) total += steps(kt);
    BwdCut cut;
    if (s.whole_tiles) return cut;
    if (s.deterministic) {
        // Measured with reductions of 64-bit words at either head size: steps take longer then (twice the bytes of dQ) and a piece costs
        // about four of them, so only a grid that is clearly out of balance is cut.  (At 128, where dQ has a kernel of its own now, the rule
        // stays because the cut decides the last bits of dK and dV; what it cuts still gains: 126 -> 110 for B3 Hq16 Hkv4 S1237, 256 -> 227 for
        // B6 Hq14 Hkv2 S1500, 145 -> 113 for B2 Hq28 Hkv4 S1024, 867 -> 301 for the windowed call.)  (By the SMs' average load over the longest tile; backward uncut -> cut, us): 0.08 1938 -> 526 (B1 Hq28 Hkv4 S8000
        // D128, 100-key window, 4 global tokens), 0.45 194 -> 144 (B3 Hq16 Hkv4 S1237 D128), 0.53 206 -> 165 (B6 Hq14 Hkv2 S1500 D64), 0.57
        // 271 -> 261; but 0.65 134 -> 134, 0.85 101 -> 114, 0.97 421 -> 482 (B8 Hq28 Hkv4 S1024 D128), 1.84 644 -> 714.  How a tile is cut
        // depends on the tile alone: a part of a batch that is cut gives the same bits as the whole.  Two to five pieces.
        if (longest < 24 || total * slabs / sms > 0.6 * longest) return cut;
        cut.steps = (longest + 1) / std::max(2, std::min(4, longest / 32));
        cut.pieces = bwd_piece_count(longest, cut.steps);
        while (cut.tiles < n_kt && steps(cut.tiles) * 4 > cut.steps * 5) ++cut.tiles;
        cut.whole_first = cut.tiles < n_kt && steps(cut.tiles) > cut.steps;
        return cut;
    }
    if (total * slabs / sms > 3.0 * longest) return cut;       // balanced by its many CTAs
    // Time of a cut in steps: the longest CTA, or the SMs' average load and a tail (short: the longest CTAs go first), or the
    // whole waves that the CTAs of about the longest kind need.
    auto estimate = [&](BwdCut& c) {
        double work = 0.0, last = 0.0, long_sum = 0.0, long_n = 0.0;
        c.tiles = 0;
        auto visit = [&](auto&& f) {
            bool cutting = c.steps > 0;
            for (int kt = 0; kt < n_kt; ++kt) {
                const int n = steps(kt);
                cutting = cutting && n * 4 > c.steps * 5;
                const int pieces = cutting ? bwd_piece_count(n, c.steps) : 1;
                f(cutting, (n + pieces - 1) / pieces + (cutting ? kPiece : kCta), pieces);
            }
        };
        double piece_longest = 0.0;
        visit([&](bool cutting, double len, int pieces) {
            work += len * pieces;
            last = std::max(last, len);
            c.tiles += cutting;
            if (cutting) piece_longest = std::max(piece_longest, len);
        });
        visit([&](bool, double len, int pieces) {
            if (len >= 0.75 * last) { long_sum += len * pieces; long_n += pieces; }
        });
        c.whole_first = c.tiles < n_kt && steps(c.tiles) + kCta > piece_longest;
        const double waves = (double)(((long long)long_n * slabs + sms - 1) / sms);
        return std::max({last, work * slabs / sms + 0.25 * last, waves * long_sum / long_n});
    };
    BwdCut none;
    none.steps = 0;
    BwdCut tried[17];
    double time[17], best = 0.9 * estimate(none);              // cut for a clear gain only
    int n = 0;
    for (int k = 2; k <= 16; ++k) {
        BwdCut c;
        c.steps = (longest + k - 1) / k;
        if (c.steps < 3) break;
        c.pieces = bwd_piece_count(longest, c.steps);
        time[n] = estimate(c);
        best = std::min(best, time[n]);
        tried[n++] = c;
    }
    for (int i = 0; i < n; ++i)                                // the coarsest of those that are about as good
        if (time[i] <= 1.03 * best) return tried[i];
    return cut;
}

// (asked for several times per call)
BwdCut bwd_cut(const AttnShape& s)
{
    struct Key { int B, Hq, Hkv, Sq, Skv, D, causal, window, global_tokens, deterministic, whole_tiles, sms; };
    static thread_local Key last{};
    static thread_local BwdCut cut;
    const Key key{s.B, s.Hq, s.Hkv, s.Sq, s.Skv, s.D, s.causal, s.window, s.global_tokens, s.deterministic, s.whole_tiles, sm_count()};
    if (memcmp(&key, &last, sizeof key) != 0) {
        cut = bwd_cut_uncached(s);
        last = key;
    }
    return cut;
}

// What one block of the grid computes.  A CTA computes its own block and then takes over blocks that have not started yet, one at
// a time (clc_try_cancel), so that the loads and first products of one run under the epilogue of the one before, and barriers
// and TMEM are set up once.  A block's fixed cost of about 2 us was a third of a short one: B8 Hq12 S1024 D64, 768 blocks of 1 to 8
// steps, took 83 us for the whole backward and takes 73; B2 Hq32 S1024 D64 54 -> 49; a 300-key window over B2 Hq16 Hkv4 S4096
// D128 159 -> 149.  Grids that fit the SMs at once have nothing to take over and do not ask.
struct BwdWork {
    int kt, slab, piece;       // key tile, b * Hkv + hk, piece of a cut tile
    int n_iter;                // steps
    int qt_first, per_head;    // query tiles of a head: from qt_first, per_head of them
    int g_first, r_first;      // head and query tile of the first step
    int split;

    template <bool kWin, bool kSplit> __device__ __forceinline__ void decode(const BwdParams& p, int block)
    {
        // whole tiles as one block per (tile, slab), cut ones as one per (piece, tile, slab); the kind with the longest blocks
        // first, and key tile 0, which sees every query tile, before the others
        const int slabs = p.B * p.Hkv, group = p.Hq / p.Hkv;
        const int n_whole = (p.n_kt - p.split_tiles) * slabs, n_pieces = kSplit ? p.piece_end[p.split_pieces - 1] : 0;
        split = kSplit && (p.whole_first ? block >= n_whole : block < n_pieces);
        int idx = block - (!kSplit ? 0 : p.whole_first ? (split ? n_whole : 0) : (split ? 0 : n_pieces));
        piece = 0;
        if (split) {
            while (idx >= p.piece_end[piece]) ++piece;
            if (piece > 0) idx -= p.piece_end[piece - 1];
        }
        kt = idx / slabs;
        slab = idx - kt * slabs;
        if (!split) kt += p.split_tiles;
        qt_first = p.causal ? kt : 0;
        // with a sliding window the last query that sees this tile is (last key + window - 1), unless the tile holds
        // global tokens, which every later query sees
        const int qt_last = (kWin && kt * kT >= p.global_tokens) ? min(p.n_qt - 1, (kt * kT + kT - 1 + p.window - 1) / kT) : p.n_qt - 1;
        per_head = qt_last - qt_first + 1;
        n_iter = per_head > 0 ? per_head * group : 0;
        int i0 = 0;
        if (split) {
            const int pieces = bwd_piece_count(n_iter, p.split_steps), len = (n_iter + pieces - 1) / pieces;
            i0 = piece * len;
            n_iter = min(len, n_iter - i0);
        }
        g_first = per_head > 0 ? i0 / per_head : 0;
        r_first = i0 - g_first * per_head;
    }
};

struct BwdBarriers {
    uint4 response;           // of the block scheduler
    uint64_t response_full, work_full[2], work_empty[2];
    BwdWork work[2];          // blocks in turn
    uint64_t k_full, v_full;
    uint64_t q_full[3], q_empty[3], do_full[2], do_empty[2];
    uint64_t s_ready[2], p_ready[2], dp_ready, ds_ready, dq_ready, dq_drained, final_bar;
    uint32_t tmem_base;
    uint32_t abort_flag;
};

// Shared-memory descriptor of an unswizzled K-major operand of ONE contraction step (16 bf16 = two 8-element column
// blocks): a column block is rows of 16 bytes, eight rows forming one 128-byte core matrix (SBO = 128 to the next eight
// rows); LBO is the distance from the first column block to the second.
__device__ __forceinline__ uint64_t make_sdesc_plain(uint32_t smem_addr, uint32_t lbo_bytes)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);
    d |= (uint64_t)((lbo_bytes >> 4) & 0x3fffu) << 16;
    d |= (uint64_t)(128u >> 4) << 32;
    d |= (uint64_t)1 << 46;  // descriptor version (Blackwell); swizzle field 0 = none
    return d;
}

// One dQ tile (this thread's row in registers) -> staging buffers -> asynchronous bulk add-reductions into the accumulator
// tile, kStageCols columns per piece.  Called by all 128 threads of the drain warpgroup (named barrier 1); `elected` is the
// one thread that owns the bulk groups.  kStagingBytes of staging in all; `piece` counts pieces over the CTA's lifetime, so
// that the rotation carries on from tile to tile (a buffer is rewritten only after the kStages - 1 groups issued since
// its last use are all that may still be reading).  A warp whose wait for the tile gave up takes part in the first barrier only,
// with named_barrier_all(1, 128, false): then nothing is pushed and the result is false in all of them.
template <int D, bool kDet, int kStageCols, int kStagingBytes>
__device__ __forceinline__ bool push_dq_tile(const uint32_t (&r)[D], float* tile, uint8_t* sStage, int row, bool elected, uint32_t& piece)
{
    constexpr int kStageBytes = kStageCols * kT * 4;
    constexpr int kStages = kStagingBytes / kStageBytes;
    static_assert(kStages >= 2 && kStages * kStageBytes == kStagingBytes, "staging must hold whole pieces");
    auto stage_free = [&](int c) {
        if (elected) bulk_wait_read<kStages - 1>();
        if (c == 0) return named_barrier_all(1, 128, true);
        named_barrier_sync(1, 128);
        return true;
    };
    if constexpr (!kDet) {
#pragma unroll
        for (int c = 0; c < D / kStageCols; ++c) {
            uint8_t* stage = sStage + (piece++ % kStages) * kStageBytes;
            if (!stage_free(c)) return false;
#pragma unroll
            for (int v = 0; v < kStageCols / 4; ++v)
                *reinterpret_cast<uint4*>(stage + ((size_t)v * kT + row) * 16) =
                    make_uint4(r[c * kStageCols + 4 * v], r[c * kStageCols + 4 * v + 1], r[c * kStageCols + 4 * v + 2], r[c * kStageCols + 4 * v + 3]);
            fence_proxy_async_smem();
            named_barrier_sync(1, 128);
            if (elected) {
                bulk_reduce_add_f32(tile + (size_t)c * kStageCols * kT, stage, (uint32_t)kStageBytes);
                bulk_commit();
            }
        }
    } else {
        // Order-independent form: each fp32 value times 2^32 is an integer that fits 64 bits exactly (24-bit
        // mantissa, |value| < 2^31), and integer addition is associative, so the accumulated sum is the same
        // whatever order the key tiles arrive in.  Same staging buffers, half as many columns per piece; the
        // accumulator tile is [d/2][row][2] 64-bit words, so a piece is still one contiguous block.
        constexpr int kDetCols = kStageCols / 2;
        unsigned long long* tile64 = reinterpret_cast<unsigned long long*>(tile);
#pragma unroll
        for (int c = 0; c < D / kDetCols; ++c) {
            uint8_t* stage = sStage + (piece++ % kStages) * kStageBytes;
            if (!stage_free(c)) return false;
#pragma unroll
            for (int v = 0; v < kDetCols / 2; ++v) {
                const long long a = __float2ll_rn(__uint_as_float(r[c * kDetCols + 2 * v]) * 4294967296.0f);
                const long long b2 = __float2ll_rn(__uint_as_float(r[c * kDetCols + 2 * v + 1]) * 4294967296.0f);
                *reinterpret_cast<ulonglong2*>(stage + ((size_t)v * kT + row) * 16) =
                    make_ulonglong2((unsigned long long)a, (unsigned long long)b2);
            }
            fence_proxy_async_smem();
            named_barrier_sync(1, 128);
            if (elected) {
                bulk_reduce_add_u64(tile64 + (size_t)c * kDetCols * kT, stage, (uint32_t)kStageBytes);
                bulk_commit();
            }
        }
    }
    return true;
}

// Epilogue of a compute warpgroup: its accumulator (dV for warpgroup 0, dK for warpgroup 1; `src` = TMEM address of this
// thread's row) leaves as an fp32 partial (cut tiles), is added into the caller's fp32 accumulators, or is stored as bf16
// through `stage` (4 KB of shared memory of this warp's own).
template <int D, bool kMat>
__device__ __forceinline__ void write_dkv(const BwdParams& p, bool ok, bool split, int n_iter, int wg, int warp, int lane, int row,
                                          uint32_t src, int kt, int slab, int slabs, int piece, int k0, uint8_t* stage)
{
    if (split) {
        // this CTA's share of dV (warpgroup 0) / dK (warpgroup 1) as an fp32 partial; zeros if it saw no query
        float* dst = p.dkv_part + ((((size_t)kt * slabs + slab) * p.split_pieces + piece) * 2 + wg) * (size_t)(kT * D) + (size_t)row * D;
        if (ok) tc_fence_after();
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            if (ok) {
                tmem_ld32(src + (uint32_t)(c * 32), r);
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int v = 0; v < 32; ++v) r[v] = 0u;
            }
#pragma unroll
            for (int v = 0; v < 8; ++v)
                *reinterpret_cast<uint4*>(dst + c * 32 + v * 4) = make_uint4(r[4 * v], r[4 * v + 1], r[4 * v + 2], r[4 * v + 3]);
        }
    } else if (!kMat && ok && p.dk_acc != nullptr) {
        // accumulate form: this CTA is the only writer of its 128 key rows in this launch
        tc_fence_after();
        const int key = k0 + row;
        const bool store = key < p.Skv;
        const float mul = wg == 0 ? 1.0f : p.scale;
        float* dst = (wg == 0 ? p.dv_acc : p.dk_acc) + ((size_t)slab * p.Skv + (size_t)(store ? key : 0)) * D;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            tmem_ld32(src + (uint32_t)(c * 32), r);
            tmem_ld_wait();
            if (store) {
#pragma unroll
                for (int v = 0; v < 8; ++v) {
                    float4 a = *reinterpret_cast<const float4*>(dst + c * 32 + v * 4);
                    a.x = fmaf(__uint_as_float(r[4 * v + 0]), mul, a.x);
                    a.y = fmaf(__uint_as_float(r[4 * v + 1]), mul, a.y);
                    a.z = fmaf(__uint_as_float(r[4 * v + 2]), mul, a.z);
                    a.w = fmaf(__uint_as_float(r[4 * v + 3]), mul, a.w);
                    *reinterpret_cast<float4*>(dst + c * 32 + v * 4) = a;
                }
            }
        }
    } else if (kMat && ok) {
        // feature-major matrices: the 32 keys of a warp are 128 contiguous bytes of every feature's row
        tc_fence_after();
        const int key = k0 + row;
        const float mul = wg == 0 ? 1.0f : p.scale;
        const int b = slab / p.Hkv, hk = slab - b * p.Hkv;
        float* dst = (wg == 0 ? p.dv_mat : p.dk_mat) + (long long)hk * D * p.mat_stride + (long long)b * p.Skv + key;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) {
            uint32_t r[32];
            tmem_ld32(src + (uint32_t)(c * 32), r);
            tmem_ld_wait();
            if (key < p.Skv) {
#pragma unroll
                for (int v = 0; v < 32; ++v) dst[(c * 32 + v) * p.mat_stride] = __uint_as_float(r[v]) * mul;
            }
        }
    } else if (ok) {
        tc_fence_after();
        const int key = k0 + row;
        const float mul = wg == 0 ? 1.0f : p.scale;
        // Coalesced bf16 store: a thread holds one whole key row, so the warp's 32 rows go through shared memory, 64 columns at a
        // time, and leave with each store instruction covering 128 bytes of four rows; 16-byte units are XOR-swizzled by the row
        // against bank conflicts.  The staging rows are the warp's own rows of the dS tile: every product that read them has
        // retired, and only this warp writes them again.  (K and V are not: the next block's may be on their way.)
        __nv_bfloat16* out = (wg == 0 ? p.dv : p.dk) + (size_t)slab * p.Skv * D;
        const int sub = lane >> 3, unit0 = lane & 7, key_warp0 = key - lane;
#pragma unroll
        for (int half = 0; half < D / 64; ++half) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t r[32];
                tmem_ld32(src + (uint32_t)(half * 64 + c * 32), r);
                tmem_ld_wait();
#pragma unroll
                for (int v = 0; v < 4; ++v) {
                    uint4 w;
                    w.x = pack_bf16(__uint_as_float(r[8 * v + 0]) * mul, __uint_as_float(r[8 * v + 1]) * mul);
                    w.y = pack_bf16(__uint_as_float(r[8 * v + 2]) * mul, __uint_as_float(r[8 * v + 3]) * mul);
                    w.z = pack_bf16(__uint_as_float(r[8 * v + 4]) * mul, __uint_as_float(r[8 * v + 5]) * mul);
                    w.w = pack_bf16(__uint_as_float(r[8 * v + 6]) * mul, __uint_as_float(r[8 * v + 7]) * mul);
                    *reinterpret_cast<uint4*>(stage + lane * 128 + (((c * 4 + v) ^ (lane & 7)) << 4)) = w;
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const int rr = i * 4 + sub;
                const uint4 w = *reinterpret_cast<const uint4*>(stage + rr * 128 + ((unit0 ^ (rr & 7)) << 4));
                if (key_warp0 + rr < p.Skv) *reinterpret_cast<uint4*>(out + (size_t)(key_warp0 + rr) * D + half * 64 + unit0 * 8) = w;
            }
            __syncwarp();
        }
    } else if (n_iter == 0 && p.dk_acc == nullptr) {
        // a key tile no query can see (cannot happen for causal with Sq == Skv; kept for safety): zero grads
        const int key = k0 + row;
        if (key < p.Skv && kMat) {
            const int b = slab / p.Hkv, hk = slab - b * p.Hkv;
            float* dst = (wg == 0 ? p.dv_mat : p.dk_mat) + (long long)hk * D * p.mat_stride + (long long)b * p.Skv + key;
            for (int d = 0; d < D; ++d) dst[d * p.mat_stride] = 0.0f;
        } else if (key < p.Skv) {
            __nv_bfloat16* dst = (wg == 0 ? p.dv : p.dk) + ((size_t)slab * p.Skv + key) * D;
            for (int d = 0; d < D; d += 8) *reinterpret_cast<uint4*>(dst + d) = make_uint4(0, 0, 0, 0);
        }
    }
}

// kSplit: the grid may hold pieces of cut key tiles (a separate instantiation, so that the plain kernel carries none
// of that bookkeeping)
// kDet: dQ contributions leave as 64-bit fixed point (see the drain warpgroup), or dQ is left to attn_dq_sm100.cu (kOwnDq): no dQ
// product then, nothing to drain
// kMat: dK and dV leave as feature-major fp32 matrices (an instantiation of its own: with that store in the common kernel it is
// 3 % slower at head_dim 128; the accumulate form, in contrast, is better left in: without it the kernel is 3 % slower too)
template <int D, bool kWin, bool kSplit, bool kDet, bool kMat>
__global__ void __launch_bounds__(kBwdThreads, 1)
attn_bwd_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k,
                   const __grid_constant__ CUtensorMap tmap_v, const __grid_constant__ CUtensorMap tmap_do, const BwdParams p)
{
    constexpr int kTileBytes = kT * D * 2;
    constexpr int kChunkBytes = kT * 128;          // 128 rows x 128 B
    constexpr int kChunks = D / 64;
    constexpr int kDoStages = (D == 128) ? 1 : 2;  // shared-memory capacity: 227 KB
    // head_dim 64 leaves 128 TMEM columns and 60 KB of shared memory unused: S^T gets a second buffer there, so that
    // S^T_{i+2} is computed while the compute warps are still busy with step i+1 and they never wait for the dV_i, S^T_{i+1}
    // pair behind their own P^T_i; Q then needs a third stage (Q_{i+2} is loaded while dK_i still reads Q_i)
    constexpr int kSBufs = (D == 128) ? 1 : 2;
    constexpr int kQStages = (D == 128) ? 2 : 3;
    // ... and the dS tile a second buffer, which lets dK_i be issued after the next dP^T instead of before it: the chain
    // dS_i -> dQ_i -> drain -> dP^T_{i+1} -> dS_{i+1} then no longer carries the issue time of dK_i (with one buffer dK_i must
    // have read the tile before dP^T_{i+1} lets the compute warps overwrite it)
    constexpr int kDsBufs = (D == 128) ? 1 : 2;
    // columns of a dQ tile per bulk reduction (kStageCols columns x 128 rows fp32 = one piece): 8 KB pieces at head_dim 128,
    // where the tile loads of Q and dO queue behind the reductions on the SM's path to L2 and shorter pieces let them through
    // sooner (-3 % kernel time); 16 KB pieces at head_dim 64 (there the finer split costs 1 %, and 4 KB pieces cost 10-20 %
    // at either size)
    constexpr int kStageCols = (D == 128) ? 16 : 32;
    constexpr int kStagingBytes = 32 * 1024;       // dQ staging in all
    // The extra contraction step (head_dim 64).  S^T and dP^T each get one more 16-wide k-step whose operands are not tile data: on the
    // key side a constant block (1, 1, 1, 0, ...), on the query side a 16-byte record per query, (hi, mid, lo, 0, ...) with
    // hi + mid + lo = -LSE/scale (for S^T) or -delta (for dP^T): the fp32 value split exactly in three bf16.  The tensor core then delivers
    // S^T - LSE/scale and dP^T - delta, and the compute warps need no per-column operand from shared memory at all:
    // P^T = exp2(scale*log2e * that) and dS^T = P^T o that.  One column block (8 bf16) per operand is real; the second
    // block of the constant operand is zeros, so the second block of the record operand may alias the first (LBO 0).
    constexpr bool kAug = bwd_folds_row_terms(D);
    constexpr bool kOwnDq = kDet && bwd_dq_has_kernel(D);
    constexpr int kAugBytes = kT * 16;             // 128 records
    constexpr int kDsBytes = kT * kT * 2;          // dS^T tile: [128 keys][128 queries] bf16 as two 64-query chunks
    // The layout uses every byte of the 227 KB a CTA may have (D = 128), so there is no room for an alignment
    // pad: the kernel has no static shared memory, which puts the dynamic window at the 1024-byte aligned start
    // of the CTA's shared memory; that is verified below instead of assumed.
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;
    uint8_t* sK = smem;
    uint8_t* sV = sK + kTileBytes;
    uint8_t* sQ = sV + kTileBytes;                 // [kQStages]
    uint8_t* sDo = sQ + kQStages * kTileBytes;     // [kDoStages]
    uint8_t* sDs = sDo + kDoStages * kTileBytes;   // [kDsBufs]
    uint8_t* sStage = sDs + kDsBufs * kDsBytes;    // kStagingBytes
    // per-query terms: with the extra contraction step its operands, else -LSE*log2e and -delta as plain fp32 columns
    uint8_t* sTail = sStage + kStagingBytes;
    uint8_t* sOnes = sTail;                        // [2][kAugBytes]: the constant block, then zeros
    uint8_t* sQaug = sOnes + 2 * kAugBytes;        // [kQStages][kAugBytes]
    uint8_t* sDoaug = sQaug + kQStages * kAugBytes;   // [kDoStages][kAugBytes]
    float* sLse = (float*)sTail;                   // [kQStages][128]
    float* sDelta = sLse + kQStages * kT;          // [kQStages][128]
    constexpr int kTailBytes = kAug ? (2 + kQStages + kDoStages) * kAugBytes : 2 * kQStages * kT * 4;
    BwdBarriers* bars = (BwdBarriers*)(sTail + kTailBytes);
    volatile uint32_t* abort_flag = &bars->abort_flag;

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;   // (warp-uniform for the compiler)
    if ((smem_u32(smem_raw) & 1023u) != 0u) {      // uniform over the CTA: nothing has been set up yet
        if (threadIdx.x == 0) atomicCAS(&g_device_status, 0u, (0x3fu << 24) | (blockIdx.x & 0xffffffu));
        wait_for_stream();
        return;
    }

    const int group = p.Hq / p.Hkv;
    BwdWork w;          // (the producer's)
    if (warp == 13 && lane == 0) {
        w.decode<kWin, kSplit>(p, (int)blockIdx.x);
        bars->work[0] = w;
        prefetch_tensormap(&tmap_q);
        prefetch_tensormap(&tmap_k);
        prefetch_tensormap(&tmap_v);
        prefetch_tensormap(&tmap_do);
        mbar_init(&bars->response_full, 1);
        mbar_init(&bars->k_full, 1);
        mbar_init(&bars->v_full, 1);
        for (int i = 0; i < 3; ++i) {
            mbar_init(&bars->q_full[i], 1);
            mbar_init(&bars->q_empty[i], 2);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->work_full[i], 1);
            mbar_init(&bars->work_empty[i], 14);    // every warp but the idle one and the producer
            mbar_init(&bars->do_full[i], 1);
            mbar_init(&bars->do_empty[i], 2);
            mbar_init(&bars->s_ready[i], 1);
            mbar_init(&bars->p_ready[i], 256);
        }
        mbar_init(&bars->dp_ready, 1);
        mbar_init(&bars->ds_ready, 256);
        mbar_init(&bars->dq_ready, 1);
        mbar_init(&bars->dq_drained, 128);
        mbar_init(&bars->final_bar, 2);
        bars->abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 12) {
        tmem_alloc(&bars->tmem_base, kTmemCols);
        tmem_relinquish();
    }
    if (kAug && threadIdx.x < kT) {
        reinterpret_cast<uint4*>(sOnes)[threadIdx.x] = make_uint4(0x3f803f80u, 0x00003f80u, 0u, 0u);   // bf16 (1, 1, 1, 0, 0, 0, 0, 0)
        reinterpret_cast<uint4*>(sOnes + kAugBytes)[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
        fence_proxy_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = bars->tmem_base;
    wait_for_stream();      // nothing before this reads or writes global memory
    // S^T / P^T [0,128)   dP^T / dQ [128,256)   head_dim 128: dV [256,384) dK [384,512)   64: dV [256,320) dK [320,384) 2nd S^T [384,512)
    const uint32_t tm_S = tmem, tm_dP = tmem + 128u, tm_dV = tmem + 256u, tm_dK = tmem + (D == 128 ? 384u : 320u);
    constexpr uint32_t kSBufStride = 384u;         // columns from the first S^T buffer to the second

    // 512 threads start with 128 registers each; the issuing/producer warpgroup needs few, the others get the rest
    // (each role re-allocates registers inside its own branch so that the compiler sees which register count applies where)

    // Every role walks the same blocks, which the producer decodes into shared memory: number u is work[u & 1].  Step counters run
    // on over the blocks (n0: steps before this block, blocks: how many before it had steps), so stages and barrier phases continue
    // where they are.  next(u): done with block u; whether another follows (agree: whether the wait for it came through, for all warps that
    // have to leave together).
    auto next = [&](int u, auto agree) {
        __syncwarp();
        if (lane == 0) mbar_arrive(&bars->work_empty[u & 1]);
        return agree(mbar_wait_prompt_warp(&bars->work_full[(u + 1) & 1], (uint32_t)((u >> 1) & 1), abort_flag, kSiteNext)) && bars->work[(u + 1) & 1].n_iter >= 0;
    };
    auto alone = [](bool came) { return came; };

    if (warp == 15) {
        setmaxnreg_dec<56>();
        // idle warps of the last warpgroup
    } else if (warp == 13) {
        setmaxnreg_dec<56>();
        // =========================== TMA producer ===========================
        if (lane == 0) {
            int n0 = 0, blocks = 0;
            bool ok = true;
            for (int u = 0, block = 0; block >= 0; ++u) {
                // K and V: once every product of the block before has read them
                if (w.n_iter > 0) {
                    ok = blocks == 0 || mbar_wait_prompt(&bars->final_bar, (uint32_t)((blocks - 1) & 1), abort_flag, kSiteFinal);
                    if (!ok) break;
                    mbar_arrive_expect_tx(&bars->k_full, (uint32_t)kTileBytes);
                    for (int c = 0; c < kChunks; ++c) tma_load_3d(sK + c * kChunkBytes, &tmap_k, &bars->k_full, c * 64, w.kt * kT, w.slab);
                    ++blocks;
                }
                const int bh0 = w.slab * group;      // b * Hq + hk * group
                int g = w.g_first, r = w.r_first;
                for (int i = 0; i < w.n_iter; ++i) {
                    const int qt = w.qt_first + r, bh = bh0 + g, n = n0 + i;
                    if (++r == w.per_head) { r = 0; ++g; }
                    const int sq = n % kQStages;
                    if (n >= kQStages && !(ok = mbar_wait_prompt(&bars->q_empty[sq], (uint32_t)(((n / kQStages) - 1) & 1), abort_flag, kSiteQEmpty))) break;
                    mbar_arrive_expect_tx(&bars->q_full[sq], (uint32_t)(kTileBytes + (kAug ? kAugBytes : 2 * kT * 4)));
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(sQ + sq * kTileBytes + c * kChunkBytes, &tmap_q, &bars->q_full[sq], c * 64, qt * kT, bh);
                    if constexpr (kAug) {
                        bulk_load_1d(sQaug + sq * kAugBytes, p.qaug + (size_t)bh * p.Sq_pad + (size_t)qt * kT, kAugBytes, &bars->q_full[sq]);
                    } else {
                        bulk_load_1d(sLse + sq * kT, p.lse2 + (size_t)bh * p.Sq_pad + (size_t)qt * kT, kT * 4, &bars->q_full[sq]);
                        bulk_load_1d(sDelta + sq * kT, p.delta + (size_t)bh * p.Sq_pad + (size_t)qt * kT, kT * 4, &bars->q_full[sq]);
                    }
                    if (i == 0) {
                        mbar_arrive_expect_tx(&bars->v_full, (uint32_t)kTileBytes);
                        for (int c = 0; c < kChunks; ++c) tma_load_3d(sV + c * kChunkBytes, &tmap_v, &bars->v_full, c * 64, w.kt * kT, w.slab);
                    }
                    const int sd = n % kDoStages;
                    if (n >= kDoStages &&
                        !(ok = mbar_wait_prompt(&bars->do_empty[sd], (uint32_t)(((n / kDoStages) - 1) & 1), abort_flag, kSiteDoEmpty)))
                        break;
                    mbar_arrive_expect_tx(&bars->do_full[sd], (uint32_t)(kTileBytes + (kAug ? kAugBytes : 0)));
                    if constexpr (kAug)
                        bulk_load_1d(sDoaug + sd * kAugBytes, p.doaug + (size_t)bh * p.Sq_pad + (size_t)qt * kT, kAugBytes, &bars->do_full[sd]);
                    for (int c = 0; c < kChunks; ++c)
                        tma_load_3d(sDo + sd * kTileBytes + c * kChunkBytes, &tmap_do, &bars->do_full[sd], c * 64, qt * kT, bh);
                }
                if (!ok) break;
                n0 += w.n_iter;
                // The next block is asked for one or two steps before this one ends, in time to have the answer: asked for at its
                // start, it would go to this CTA even if others are free sooner (B3 Hq16 Hkv4 S1237 D128, reproducible: 183 us instead of
                // 134; blocks left to the hardware's own order: 138).
                block = -1;
                if (p.several_waves) {
                    mbar_arrive_expect_tx(&bars->response_full, 16);
                    clc_try_cancel(&bars->response, &bars->response_full);
                    if (!mbar_wait_prompt(&bars->response_full, (uint32_t)(u & 1), abort_flag, kSiteNext)) break;
                    block = clc_first_block(&bars->response);
                    fence_proxy_async_smem();
                }
                w.n_iter = -1;
                if (block >= 0) w.decode<kWin, kSplit>(p, block);
                if (u >= 1 && !mbar_wait_prompt(&bars->work_empty[(u + 1) & 1], (uint32_t)(((u - 1) >> 1) & 1), abort_flag, kSiteNext)) break;
                bars->work[(u + 1) & 1] = w;
                mbar_arrive(&bars->work_full[(u + 1) & 1]);
            }
        }
    } else if (warp == 12 || warp == 14) {
        setmaxnreg_dec<56>();
        // =========================== MMA issuers ===========================
        // Two issuing threads on two different schedulers, because a lone issuing warp shares its scheduler with
        // ALU-dense compute warps and gets too few issue slots to keep the tensor pipe fed:
        //   warp 12 ("P side"):   dV_i += P^T dO_i ,  S^T_{i+1} = K Q_{i+1}^T
        //   warp 14 ("dS side"):  dK_i += dS^T Q_i ,  dQ_i = dS K ,  dP^T_{i+1} = V dO_{i+1}^T
        // Every TMEM region with a write-after-read hazard is touched by one of the two only (S^T/P^T by warp 12,
        // dP^T/dS^T/dQ by warp 14), so the in-order execution of one thread's MMAs still covers those hazards.  The Q
        // and dO stages are read by both and are released when both have committed (barrier count 2).  Each commits its
        // share of a dO stage right after its own product that reads it: with one dO stage (head_dim 128) the next dO tile
        // can only be loaded once both have, and dP^T_{i+1} waits for that load.
        // (Two, not more: MMAs issued by different warps interleave in the tensor pipe k-step by k-step, each on another
        // accumulator, and a third issuing warp for dK measured 7-20 % slower than this split at either head size.)
        if (warp == 12) {
            // P side: all 32 lanes walk the loop (warp-uniform control flow lets descriptors and addresses live in uniform
            // registers) and one elected lane issues the products four k-steps at a time (mma_ss_4).
            SNTL_TRACE_DECL(tn);
            const bool tl = lane == 0;
            (void)tl;
            constexpr uint32_t idesc_st = make_idesc(kT, kT, false, false);
            constexpr uint32_t idesc_kv = make_idesc(kT, D, false, true);
            auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t site) { return mbar_wait_prompt_warp(bar, parity, abort_flag, site); };
            const uint64_t d_ones = make_sdesc_plain(smem_u32(sOnes), kAugBytes), d_qaug0 = make_sdesc_plain(smem_u32(sQaug), 0);
            // the D/16 steps over the head dimension, then the extra step that subtracts LSE/scale (see kAugBytes)
            auto issue_kmajor = [&](uint32_t d_tmem, uint64_t a, uint64_t b, uint64_t aug) {
#pragma unroll
                for (int c = 0; c < kChunks; ++c)
                    mma_ss_4<2, 2>(d_tmem, sdesc_advance(a, (uint32_t)(c * kChunkBytes)), sdesc_advance(b, (uint32_t)(c * kChunkBytes)), idesc_st, c > 0);
                if constexpr (kAug) mma_ss_1(d_tmem, d_ones, aug, idesc_st);
            };
            auto issue_from_tmem = [&](uint32_t d_tmem, uint32_t a_tmem, uint64_t b, bool accumulate) {
                mma_ts_4<8, 128>(d_tmem, a_tmem, b, idesc_kv, accumulate);
                mma_ts_4<8, 128>(d_tmem, a_tmem + 64u, sdesc_advance(b, 4 * 2048), idesc_kv, 1);
            };
            const uint64_t dK_k = make_sdesc(smem_u32(sK), 16, 1024);
            const uint64_t dQ_k0 = make_sdesc(smem_u32(sQ), 16, 1024), dDo_mn0 = make_sdesc(smem_u32(sDo), kChunkBytes, 1024);
            int n0 = 0, blocks = 0;
            bool ok = true;
            bool more = true;
            for (int u = 0; more; more = next(u++, alone)) {
                const int end = n0 + bars->work[u & 1].n_iter;
                if (end == n0) continue;
                if (!(ok = wait(&bars->k_full, (uint32_t)(blocks & 1), kSiteKV))) break;
                // S^T of the first kSBufs steps; after that S^T_{n+kSBufs} follows dV_n into the buffer that P^T_n leaves
                for (int n = n0; n < n0 + kSBufs && n < end; ++n) {
                    const int sq = n % kQStages, sb = n % kSBufs;
                    if (!(ok = wait(&bars->q_full[sq], (uint32_t)((n / kQStages) & 1), kSiteQFull))) break;
                    tc_fence_after();
                    issue_kmajor(tm_S + (uint32_t)sb * kSBufStride, dK_k, sdesc_advance(dQ_k0, sq * kTileBytes), sdesc_advance(d_qaug0, sq * kAugBytes));
                    tc_commit_p(&bars->s_ready[sb]);
                }
                for (int n = n0; ok && n < end; ++n) {
                    const int sq = n % kQStages, sd = n % kDoStages, sb = n % kSBufs;
                    const uint32_t tm_Si = tm_S + (uint32_t)sb * kSBufStride;
                    // one barrier per S^T buffer: with two buffers the threads of one warpgroup can be through step n + 1 while a
                    // warp of the other has not stored its P^T_n yet, and a single barrier would count their second arrival for it
                    if (!(ok = wait(&bars->p_ready[sb], (uint32_t)((n / kSBufs) & 1), kSiteP))) break;
                    if (!(ok = wait(&bars->do_full[sd], (uint32_t)((n / kDoStages) & 1), kSiteDoFull))) break;
                    SNTL_TRACE_EV(tl, 0, tn, 1);
                    tc_fence_after();
                    // (the first dV of a block overwrites the accumulator: the compute warps arrive at p_ready behind their epilogue)
                    issue_from_tmem(tm_dV, tm_Si, sdesc_advance(dDo_mn0, sd * kTileBytes), n > n0);
                    tc_commit_p(&bars->do_empty[sd]);
                    tc_commit_p(&bars->q_empty[sq]);
                    SNTL_TRACE_EV(tl, 0, tn, 2);
                    if (n + kSBufs < end) {
                        const int nq = (n + kSBufs) % kQStages;
                        if (!(ok = wait(&bars->q_full[nq], (uint32_t)(((n + kSBufs) / kQStages) & 1), kSiteQFull))) break;
                        tc_fence_after();
                        issue_kmajor(tm_Si, dK_k, sdesc_advance(dQ_k0, nq * kTileBytes), sdesc_advance(d_qaug0, nq * kAugBytes));
                        tc_commit_p(&bars->s_ready[sb]);
                        SNTL_TRACE_EV(tl, 0, tn, 9);
                    }
                }
                if (!ok) break;
                tc_commit_p(&bars->final_bar);
                n0 = end;
                ++blocks;
            }
            if (!ok) tc_commit_p(&bars->final_bar);
            else if (blocks > 0) wait(&bars->final_bar, (uint32_t)((blocks - 1) & 1), kSiteFinal);
        } else {
            // dS side, in the same form
            const bool tl14 = lane == 0;
            (void)tl14;
            auto wait = [&](uint64_t* bar, uint32_t parity, uint32_t site) { return mbar_wait_prompt_warp(bar, parity, abort_flag, site); };
            SNTL_TRACE_DECL(tn);
            constexpr uint32_t idesc_st = make_idesc(kT, kT, false, false);   // S^T, dP^T
            constexpr uint32_t idesc_kv = make_idesc(kT, D, false, true);     // dV, dK: A in TMEM, B MN-major
            constexpr uint32_t idesc_dq = make_idesc(kT, D, true, true);      // dQ: both operands MN-major
            const uint64_t d_ones = make_sdesc_plain(smem_u32(sOnes), kAugBytes), d_doaug0 = make_sdesc_plain(smem_u32(sDoaug), 0);
            // C[128 x 128] = A[128 x D] * B[128 x D]^T, both K-major tiles: the D/16 steps over the head dimension, then the extra
            // step that subtracts delta (see kAugBytes)
            auto issue_kmajor = [&](uint32_t d_tmem, uint64_t a, uint64_t b, uint64_t aug) {
#pragma unroll
                for (int c = 0; c < kChunks; ++c)
                    mma_ss_4<2, 2>(d_tmem, sdesc_advance(a, (uint32_t)(c * kChunkBytes)), sdesc_advance(b, (uint32_t)(c * kChunkBytes)), idesc_st, c > 0);
                if constexpr (kAug) mma_ss_1(d_tmem, d_ones, aug, idesc_st);
            };
            const uint64_t dV_k = make_sdesc(smem_u32(sV), 16, 1024), dDo_k0 = make_sdesc(smem_u32(sDo), 16, 1024);
            const uint64_t dK_mn = make_sdesc(smem_u32(sK), kChunkBytes, 1024), dDs_mn = make_sdesc(smem_u32(sDs), kChunkBytes, 1024);
            const uint64_t dDs_k = make_sdesc(smem_u32(sDs), 16, 1024);
            const uint64_t dQ_mn0 = make_sdesc(smem_u32(sQ), kChunkBytes, 1024);
            int n0 = 0, blocks = 0;
            bool ok = true;
            bool more = true;
            for (int u = 0; more; more = next(u++, alone)) {
                const int end = n0 + bars->work[u & 1].n_iter;
                if (end == n0) continue;
                // dP^T of step n, into the columns that dQ of the step before has left
                auto issue_dp = [&](int n) {
                    const int nd = n % kDoStages;
                    // (kOwnDq: dP^T of the step before has been read, this warp has seen ds_ready)
                    if (!kOwnDq && n > 0 && !wait(&bars->dq_drained, (uint32_t)((n - 1) & 1), kSiteDrained)) return false;
                    SNTL_TRACE_EV(tl14, 4, tn, 5);
                    if (!wait(&bars->do_full[nd], (uint32_t)((n / kDoStages) & 1), kSiteDoFull)) return false;
                    tc_fence_after();
                    issue_kmajor(tm_dP, dV_k, sdesc_advance(dDo_k0, nd * kTileBytes), sdesc_advance(d_doaug0, nd * kAugBytes));
                    tc_commit_p(&bars->dp_ready);
                    // this warp's share of releasing dO_n, committed at once: with a single dO stage the load of the
                    // next tile starts as soon as this product and dV_n have read the stage
                    tc_commit_p(&bars->do_empty[nd]);
                    SNTL_TRACE_EV(tl14, 4, tn, 6);
                    return true;
                };
                if (!(ok = wait(&bars->k_full, (uint32_t)(blocks & 1), kSiteKV) && wait(&bars->v_full, (uint32_t)(blocks & 1), kSiteKV) && issue_dp(n0))) break;
                for (int n = n0; n < end; ++n) {
                    const int sq = n % kQStages;
                    if (!(ok = wait(&bars->ds_ready, (uint32_t)(n & 1), kSiteDS))) break;
                    SNTL_TRACE_EV(tl14, 4, tn, 3);
                    tc_fence_after();
                    // dQ first: it gates the drain and with it the next dP^T
                    const uint32_t ds_off = (uint32_t)((n % kDsBufs) * kDsBytes);
                    const uint64_t ds_mn = sdesc_advance(dDs_mn, ds_off);
                    if constexpr (!kOwnDq) {
                        mma_ss_4<128, 128>(tm_dP, ds_mn, dK_mn, idesc_dq, 0);
                        mma_ss_4<128, 128>(tm_dP, sdesc_advance(ds_mn, 4 * 2048), sdesc_advance(dK_mn, 4 * 2048), idesc_dq, 1);
                        tc_commit_p(&bars->dq_ready);
                    }
                    SNTL_TRACE_EV(tl14, 4, tn, 4);
                    // dK += dS^T Q with dS^T read from its shared-memory tile as a K-major A operand (rows = keys, the 64
                    // contiguous elements run along the queries).  Q_n is ready: ds_ready implies its load was seen.  With
                    // one dS buffer it goes before the next dP^T: by the time the compute warps see that dP^T and rewrite the
                    // tile, this product has read it (one thread's MMAs run in order).  With two it goes after, and the
                    // buffer it reads is rewritten only behind dP^T_{n+2}, which this thread issues later still.
                    auto issue_dk = [&]() {
                        const uint64_t a = sdesc_advance(dDs_k, ds_off), bq = sdesc_advance(dQ_mn0, sq * kTileBytes);
                        mma_ss_4<2, 128>(tm_dK, a, bq, idesc_kv, n > n0);
                        mma_ss_4<2, 128>(tm_dK, sdesc_advance(a, kChunkBytes), sdesc_advance(bq, 4 * 2048), idesc_kv, 1);
                        tc_commit_p(&bars->q_empty[sq]);    // this warp's share: dK_n
                    };
                    if constexpr (kDsBufs == 1) issue_dk();
                    if (n + 1 < end && !(ok = issue_dp(n + 1))) break;
                    if constexpr (kDsBufs == 2) issue_dk();
                }
                if (!ok) break;
                // every MMA of this thread has retired once its commit lands; the epilogue waits for both issuers
                tc_commit_p(&bars->final_bar);
                n0 = end;
                ++blocks;
            }
            if (!ok) tc_commit_p(&bars->final_bar);
            else if (blocks > 0) wait(&bars->final_bar, (uint32_t)((blocks - 1) & 1), kSiteFinal);
        }
    } else if (warp >= 8) {
        setmaxnreg_inc<152>();
        // =========================== dQ drain warpgroup ===========================
        const int row = (warp & 3) * 32 + lane;                 // query row inside the tile == TMEM lane
        SNTL_TRACE_DECL(tn);
        const bool tw = warp == 8 && lane == 0;
        (void)tw;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const bool elected = warp == 8 && lane == 0;
        bool ok = true;
        uint32_t piece = 0;
        int n = 0;
        bool more = true;
        for (int u = 0; ok && more; ++u) {
        const BwdWork w = bars->work[u & 1];
        const int bh0 = w.slab * group;      // b * Hq + hk * group
        int g = w.g_first, tile_r = w.r_first;
        for (const int end = n + (kOwnDq ? 0 : w.n_iter); n < end; ++n) {
            const int qt = w.qt_first + tile_r, bh = bh0 + g;
            if (++tile_r == w.per_head) { tile_r = 0; ++g; }
            // fp32 accumulator: kT*D words per tile; fixed-point accumulator: kT*D 64-bit words per tile
            float* tile = p.dq_accum + ((size_t)bh * p.n_qt + qt) * (size_t)(kT * D) * (kDet ? 2 : 1);
            ok = mbar_wait_prompt_warp(&bars->dq_ready, (uint32_t)(n & 1), abort_flag, kSiteDQ);
            SNTL_TRACE_EV(tw, 3, tn, 1);
            if (!ok) {
                named_barrier_all(1, 128, false);
                break;
            }
            tc_fence_after();
            // The whole dQ tile goes to registers first so that the TMEM columns are handed back to the MMA warp at
            // once; pushing 64 KB (D = 128) through the reduction path (~30 bytes/clock per SM) is the slow part and
            // overlaps the next step.  The data leave through the TMA engine, not the load/store unit: reductions
            // issued as instructions queue up in the unit that also carries the compute warps' shared-memory and
            // TMEM traffic and stall them.  kStageCols columns at a time: registers -> staging buffer -> one asynchronous
            // bulk add-reduction (contiguous in the accumulator thanks to its [d/4][row][4] order).  The staging buffers
            // (32 KB in all) rotate; the elected thread makes sure a buffer's previous reduction has finished reading it
            // before it is overwritten.
            uint32_t r[D];
#pragma unroll
            for (int c = 0; c < D / 32; ++c) tmem_ld32(tm_dP + lane_off + (uint32_t)(c * 32), r + c * 32);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(&bars->dq_drained);
            SNTL_TRACE_EV(tw, 3, tn, 2);
            ok = push_dq_tile<D, kDet, kStageCols, kStagingBytes>(r, tile, sStage, row, elected, piece);
            SNTL_TRACE_EV(tw, 3, tn, 3);
            if (!ok) break;
        }
        if (!ok) break;
        more = next(u, [&](bool came) { return ok = named_barrier_all(1, 128, came); });      // (the four warps leave together)
        }
        if (elected) bulk_wait_all();   // the reductions read shared memory and must land before the CTA retires
    } else {
        setmaxnreg_inc<152>();
        // =========================== compute warpgroups ===========================
        const int wg = warp >> 2;                                // owns query columns [64*wg, 64*wg+64)
        const int row = (warp & 3) * 32 + lane;                  // key row inside the tile == TMEM lane
        SNTL_TRACE_DECL(tn);
        const bool tw = (warp & 3) == 0 && lane == 0;
        (void)tw;
        const uint32_t lane_off = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t col0 = (uint32_t)(wg * 64);
        uint8_t* ds_row0 = sDs + wg * kChunkBytes + row * 128;   // this thread's 128-byte row of its 64-query chunk
        bool ok = true;
        int n = 0, blocks = 0;
        bool more = true;
        for (int u = 0; ok && more; more = next(u++, alone)) {
        const BwdWork& w = bars->work[u & 1];
        const int qt_first = w.qt_first, per_head = w.per_head, n_iter = w.n_iter;
        const int kt = w.kt, k0 = kt * kT;
        int tile_r = w.r_first;
        for (const int end = n + n_iter; n < end; ++n) {
            const int qt = qt_first + tile_r;
            if (++tile_r == per_head) tile_r = 0;
            const uint32_t ph = (uint32_t)(n & 1);
            // ---- P^T ----
            const uint32_t tm_Si = tm_S + (uint32_t)(n % kSBufs) * kSBufStride;
            // (the Q stage's barrier also covers the LSE and delta columns this warp reads when they come as plain columns)
            ok = (kAug || mbar_wait_prompt_warp(&bars->q_full[n % kQStages], (uint32_t)((n / kQStages) & 1), abort_flag, kSiteQFull)) &&
                 mbar_wait_prompt_warp(&bars->s_ready[n % kSBufs], (uint32_t)((n / kSBufs) & 1), abort_flag, kSiteS);
            SNTL_TRACE_EV(tw, 1 + wg, tn, 1);
            if (!ok) break;
            tc_fence_after();
            uint32_t s[64];
            tmem_ld32(tm_Si + lane_off + col0, s);
            tmem_ld32(tm_Si + lane_off + col0 + 32u, s + 32);
            tmem_ld_wait();
            SNTL_TRACE_EV(tw, 1 + wg, tn, 2);
            // tiles the mask cuts through: the diagonal one and, with a window, those reaching past (first key + window - 1)
            const bool diag = (p.causal && qt == kt) || (kWin && qt * kT + kT - 1 > k0 + p.window - 1);
            uint32_t pk[32];
            const float2 sc2 = make_float2(p.scale_log2, p.scale_log2);
            const float4* lse4 = reinterpret_cast<const float4*>(sLse + (n % kQStages) * kT + col0);
            // exponents of four columns: with the extra contraction step the product already holds S^T - LSE/scale and one
            // packed multiply per pair gives them; else x = s*scale*log2(e) - LSE*log2(e) is one packed FMA per pair
            auto exponents = [&](int c, float2& x01, float2& x23) {
                const float2 s01 = make_float2(__uint_as_float(s[4 * c + 0]), __uint_as_float(s[4 * c + 1]));
                const float2 s23 = make_float2(__uint_as_float(s[4 * c + 2]), __uint_as_float(s[4 * c + 3]));
                if constexpr (kAug) {
                    x01 = fmul2(s01, sc2);
                    x23 = fmul2(s23, sc2);
                } else {
                    const float4 l = lse4[c];
                    x01 = ffma2(s01, sc2, make_float2(l.x, l.y));
                    x23 = ffma2(s23, sc2, make_float2(l.z, l.w));
                }
            };
            // branch-free main body (the mask test lives in its own copy of the loop, taken only on the diagonal tile,
            // so that the common copy is one basic block the compiler can software-pipeline)
            if (!diag) {
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    float2 x01, x23;
                    exponents(c, x01, x23);
                    pk[2 * c] = pack_bf16(ex2(x01.x), ex2(x01.y));
                    pk[2 * c + 1] = pack_bf16(ex2(x23.x), ex2(x23.y));
                }
            } else {
                // this thread's key sees the queries from itself (causal) up to key + window - 1 (global keys: all)
                const int key = k0 + row;
                const int first_q = p.causal ? key - qt * kT : -1;
                const int last_q = (kWin && key >= p.global_tokens) ? key + p.window - 1 - qt * kT : kT;
#pragma unroll
                for (int c = 0; c < 16; ++c) {
                    float2 x01, x23;
                    exponents(c, x01, x23);
                    const int q = (int)col0 + 4 * c;   // visible: first_q <= query (column) <= last_q
                    const float p0 = (q + 0 < first_q || q + 0 > last_q) ? 0.0f : ex2(x01.x);
                    const float p1 = (q + 1 < first_q || q + 1 > last_q) ? 0.0f : ex2(x01.y);
                    const float p2 = (q + 2 < first_q || q + 2 > last_q) ? 0.0f : ex2(x23.x);
                    const float p3 = (q + 3 < first_q || q + 3 > last_q) ? 0.0f : ex2(x23.y);
                    pk[2 * c] = pack_bf16(p0, p1);
                    pk[2 * c + 1] = pack_bf16(p2, p3);
                }
            }
            SNTL_TRACE_EV(tw, 1 + wg, tn, 3);
            tmem_st32(tm_Si + lane_off + col0, pk);
            tmem_st_wait();
            tc_fence_before();
            mbar_arrive(&bars->p_ready[n % kSBufs]);
            SNTL_TRACE_EV(tw, 1 + wg, tn, 4);
            // ---- dS^T ----
            ok = mbar_wait_prompt_warp(&bars->dp_ready, ph, abort_flag, kSiteDP);
            SNTL_TRACE_EV(tw, 1 + wg, tn, 5);
            if (!ok) break;
            tc_fence_after();
            tmem_ld32(tm_dP + lane_off + col0, s);
            tmem_ld32(tm_dP + lane_off + col0 + 32u, s + 32);
            tmem_ld_wait();
            SNTL_TRACE_EV(tw, 1 + wg, tn, 6);
            const float4* dl4 = reinterpret_cast<const float4*>(sDelta + (n % kQStages) * kT + col0);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                if constexpr (kAug) {
                    // the product already holds dP^T - delta, and dS^T = P^T o that is a packed bf16 product: the second
                    // factor is rounded to bf16 first, the product once more (dS^T is a bf16 MMA operand either way)
                    pk[2 * c] = mul_bf16x2(pk[2 * c], pack_bf16(__uint_as_float(s[4 * c + 0]), __uint_as_float(s[4 * c + 1])));
                    pk[2 * c + 1] = mul_bf16x2(pk[2 * c + 1], pack_bf16(__uint_as_float(s[4 * c + 2]), __uint_as_float(s[4 * c + 3])));
                } else {
                    const float4 dl = dl4[c];   // holds -delta
                    const float2 pa = make_float2(__uint_as_float(pk[2 * c] << 16), __uint_as_float(pk[2 * c] & 0xffff0000u));
                    const float2 pb = make_float2(__uint_as_float(pk[2 * c + 1] << 16), __uint_as_float(pk[2 * c + 1] & 0xffff0000u));
                    const float2 da = fmul2(pa, fadd2(make_float2(__uint_as_float(s[4 * c + 0]), __uint_as_float(s[4 * c + 1])), make_float2(dl.x, dl.y)));
                    const float2 db = fmul2(pb, fadd2(make_float2(__uint_as_float(s[4 * c + 2]), __uint_as_float(s[4 * c + 3])), make_float2(dl.z, dl.w)));
                    pk[2 * c] = pack_bf16(da.x, da.y);
                    pk[2 * c + 1] = pack_bf16(db.x, db.y);
                }
            }
            // into shared memory, rows of 128 bytes with the 128-byte swizzle the MMA expects (both the dQ and the dK
            // product read this tile)
            uint8_t* ds_row = ds_row0 + (n % kDsBufs) * kDsBytes;
#pragma unroll
            for (int j = 0; j < 8; ++j) {
                uint4 w = make_uint4(pk[4 * j], pk[4 * j + 1], pk[4 * j + 2], pk[4 * j + 3]);
                *reinterpret_cast<uint4*>(ds_row + ((j ^ (row & 7)) << 4)) = w;
            }
            fence_proxy_async_smem();
            SNTL_TRACE_EV(tw, 1 + wg, tn, 7);
            tc_fence_before();   // orders this thread's TMEM loads of dP^T before the MMA that overwrites those columns
            mbar_arrive(&bars->ds_ready);
            SNTL_TRACE_EV(tw, 1 + wg, tn, 8);
        }
        // ---- epilogue: dV (warpgroup 0) and dK (warpgroup 1) ----
        const bool done = ok && n_iter > 0 && mbar_wait_prompt_warp(&bars->final_bar, (uint32_t)(blocks & 1), abort_flag, kSiteFinal);
        if (n_iter > 0) {
            ok = done;
            ++blocks;
        }
        write_dkv<D, kMat>(p, done, w.split != 0, n_iter, wg, warp, lane, row, (wg == 0 ? tm_dV : tm_dK) + lane_off, kt, w.slab, p.B * p.Hkv, w.piece, k0,
                               sDs + warp * 32 * 128);
        }
    }

    // ---- teardown ----
    if (*abort_flag) {
        for (int i = 0; i < 64; ++i) __nanosleep(2000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 12) {
        tc_fence_after();
        tmem_dealloc(tmem, kTmemCols);
    }
}

template <int D> constexpr int kPreRows = D == 64 ? 128 : 64;   // query rows per block of bwd_pre_kernel

// Per padded query row: the terms the main kernel wants (store_row_terms) from delta = rowsum(dO o O) and LSE, and the dQ
// accumulator zeroed.  Bound by HBM: D/8 lanes per row with 16 bytes of O and of dO each and four rows per lane group in flight,
// 8 warps x 8 (16 at head_dim 64) rows per block, whose part of the accumulator is contiguous.  kWide: O and dO start on 16-byte
// boundaries; else on 8-byte ones (nothing else in the backward reads O, so it needs no more).
template <int D, bool kWide>
__global__ void __launch_bounds__(256) bwd_pre_kernel(const __nv_bfloat16* __restrict__ o, const __nv_bfloat16* __restrict__ dout,
                                                      const float* __restrict__ lse, const RowTerms terms, float* __restrict__ dq_accum, int Sq,
                                                      int Sq_pad, int acc_words_per_row)
{
    wait_for_stream();
    constexpr int kLanes = D / 8, kGroups = 32 / kLanes, kPer = 4, kRows = 8 * kGroups * kPer;   // rows per block
    static_assert(kRows == kPreRows<D>, "grid");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, l = lane % kLanes;
    const long long r0 = (long long)blockIdx.x * kRows;
    auto load = [](const __nv_bfloat16* p) {
        if constexpr (kWide) return __ldg(reinterpret_cast<const uint4*>(p));
        const uint2 a = __ldg(reinterpret_cast<const uint2*>(p)), b = __ldg(reinterpret_cast<const uint2*>(p) + 1);
        return make_uint4(a.x, a.y, b.x, b.y);
    };
    uint4 x[kPer], y[kPer];
    int s[kPer];
    long long bh[kPer];
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const long long r = r0 + (i * 8 + warp) * kGroups + lane / kLanes;
        bh[i] = r / Sq_pad;
        s[i] = (int)(r - bh[i] * Sq_pad);
        const bool live = s[i] < Sq;
        const size_t off = ((size_t)bh[i] * Sq + s[i]) * D + l * 8;
        x[i] = live ? load(o + off) : make_uint4(0, 0, 0, 0);
        y[i] = live ? load(dout + off) : make_uint4(0, 0, 0, 0);
    }
    const int words = kRows * acc_words_per_row;       // (rows_padded is a multiple of 128: every block has all its rows)
    float4* z = reinterpret_cast<float4*>(dq_accum + r0 * acc_words_per_row);
    for (int i = threadIdx.x; i < words / 4; i += 256) z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        const uint32_t xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, ys[4] = {y[i].x, y[i].y, y[i].z, y[i].w};
        float acc = 0.0f;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            acc = fmaf(__uint_as_float(xs[k] << 16), __uint_as_float(ys[k] << 16), acc);
            acc = fmaf(__uint_as_float(xs[k] & 0xffff0000u), __uint_as_float(ys[k] & 0xffff0000u), acc);
        }
#pragma unroll
        for (int m = kLanes / 2; m > 0; m >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, m);
        const long long r = r0 + (i * 8 + warp) * kGroups + lane / kLanes;
        if (l == 0) store_row_terms<D>(terms, r, s[i] < Sq, s[i] < Sq ? lse[(size_t)bh[i] * Sq + s[i]] : 0.0f, acc);
    }
}

// dQ (bf16, [B][Hq][Sq][D]) = scale * accumulator, undoing the per-tile [d/4][row][4] order; one block per tile.  A thread
// takes 16 features of a row at a time: four loads that are contiguous over the rows of a warp, one whole 32-byte sector out,
// and all its loads (16 at head_dim 128) in flight before the first store.
template <int D>
__global__ void __launch_bounds__(256, 2) bwd_post_kernel(const float* __restrict__ dq_accum, __nv_bfloat16* __restrict__ dq, int Sq,
                                                       int n_qt, float scale)
{
    wait_for_stream();
    const size_t t = blockIdx.x, bh = t / n_qt;
    const int qt = (int)(t - bh * n_qt), row = threadIdx.x & 127, half = threadIdx.x >> 7, s = qt * kT + row;
    if (s >= Sq) return;
    const float4* src = reinterpret_cast<const float4*>(dq_accum + t * (size_t)(kT * D)) + row;
    constexpr int kPer = D / 32;
    float4 x[kPer][4];
#pragma unroll
    for (int g = 0; g < kPer; ++g)
#pragma unroll
        for (int i = 0; i < 4; ++i) x[g][i] = src[(size_t)((2 * g + half) * 4 + i) * kT];
    __nv_bfloat16* dst = dq + (bh * Sq + s) * D;
#pragma unroll
    for (int g = 0; g < kPer; ++g) {
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            w[2 * i] = pack_bf16(x[g][i].x * scale, x[g][i].y * scale);
            w[2 * i + 1] = pack_bf16(x[g][i].z * scale, x[g][i].w * scale);
        }
        uint4* out = reinterpret_cast<uint4*>(dst + (2 * g + half) * 16);
        out[0] = make_uint4(w[0], w[1], w[2], w[3]);
        out[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}

// The same for the 64-bit fixed-point accumulator (tiles of [d/2][row][2] words in units of 2^-32): the one rounding
// of the exact integer sum happens here.
template <int D>
__global__ void __launch_bounds__(256) bwd_post_det_kernel(const unsigned long long* __restrict__ dq_accum, __nv_bfloat16* __restrict__ dq,
                                                           int Sq, int n_qt, float scale)
{
    wait_for_stream();
    const size_t t = blockIdx.x, bh = t / n_qt;
    const int qt = (int)(t - bh * n_qt), row = threadIdx.x & 127, half = threadIdx.x >> 7, s = qt * kT + row;
    if (s >= Sq) return;
    const longlong2* src = reinterpret_cast<const longlong2*>(dq_accum + t * (size_t)(kT * D)) + row;
    __nv_bfloat16* dst = dq + (bh * Sq + s) * D;
#pragma unroll 2
    for (int g = half; g < D / 16; g += 2) {
        longlong2 x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = src[(size_t)(g * 8 + i) * kT];
        uint32_t w[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            w[i] = pack_bf16((float)((double)x[i].x * (1.0 / 4294967296.0)) * scale, (float)((double)x[i].y * (1.0 / 4294967296.0)) * scale);
        uint4* out = reinterpret_cast<uint4*>(dst + g * 16);
        out[0] = make_uint4(w[0], w[1], w[2], w[3]);
        out[1] = make_uint4(w[4], w[5], w[6], w[7]);
    }
}


// How many partials each cut key tile has.
struct BwdPieces {
    int n_qt, causal, window, global_tokens, group, steps, stride;
    __device__ int of(int kt) const { return bwd_piece_count(bwd_tiles_per_head(kt, n_qt, causal, window, global_tokens) * group, steps); }
};

// dV / dK of the key tiles that were cut: the partials of a tile are added in piece order and written as
// bf16 (dK times the softmax scale).  One thread per 8 consecutive features of one key row.
template <int D>
__global__ void __launch_bounds__(256) bwd_dkv_reduce_kernel(const float* __restrict__ part, __nv_bfloat16* __restrict__ dk,
                                                             __nv_bfloat16* __restrict__ dv, const BwdPieces pieces, int slabs, int Skv,
                                                             float scale, long long n_units)
{
    wait_for_stream();
    const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n_units) return;
    constexpr int kPerRow = D / 8;
    const int d8 = (int)(u % kPerRow) * 8;
    long long r = u / kPerRow;
    const int row = (int)(r % kT); r /= kT;
    const int which = (int)(r & 1); r >>= 1;              // 0: dV, 1: dK
    const int slab = (int)(r % slabs);
    const int kt = (int)(r / slabs);
    const int key = kt * kT + row;
    if (key >= Skv) return;
    const float* src = part + (((size_t)kt * slabs + slab) * pieces.stride * 2 + which) * (size_t)(kT * D) + (size_t)row * D + d8;
    const int n = pieces.of(kt);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int g = 0; g < n; ++g) {
        const float4 a = *reinterpret_cast<const float4*>(src + (size_t)g * 2 * kT * D);
        const float4 c = *reinterpret_cast<const float4*>(src + (size_t)g * 2 * kT * D + 4);
        acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
        acc[4] += c.x; acc[5] += c.y; acc[6] += c.z; acc[7] += c.w;
    }
    const float mul = which ? scale : 1.0f;
    uint4 w;
    w.x = pack_bf16(acc[0] * mul, acc[1] * mul);
    w.y = pack_bf16(acc[2] * mul, acc[3] * mul);
    w.z = pack_bf16(acc[4] * mul, acc[5] * mul);
    w.w = pack_bf16(acc[6] * mul, acc[7] * mul);
    *reinterpret_cast<uint4*>((which ? dk : dv) + ((size_t)slab * Skv + key) * D + d8) = w;
}

// The same sums into fp32 feature-major matrices: consecutive threads take consecutive keys.
template <int D>
__global__ void __launch_bounds__(256) bwd_dkv_reduce_matrix_kernel(const float* __restrict__ part, float* __restrict__ dk, float* __restrict__ dv,
                                                                    long long stride, const BwdPieces pieces, int Hkv, int slabs, int Skv, float scale,
                                                                    long long n_units)
{
    wait_for_stream();
    const long long u = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (u >= n_units) return;
    constexpr int kPerRow = D / 8;
    const int row = (int)(u % kT);
    long long r = u / kT;
    const int d8 = (int)(r % kPerRow) * 8; r /= kPerRow;
    const int which = (int)(r & 1); r >>= 1;              // 0: dV, 1: dK
    const int slab = (int)(r % slabs), kt = (int)(r / slabs), key = kt * kT + row;
    if (key >= Skv) return;
    const float* src = part + (((size_t)kt * slabs + slab) * pieces.stride * 2 + which) * (size_t)(kT * D) + (size_t)row * D + d8;
    const int n = pieces.of(kt);
    float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int g = 0; g < n; ++g)
#pragma unroll
        for (int i = 0; i < 8; i += 4) {
            const float4 x = *reinterpret_cast<const float4*>(src + (size_t)g * 2 * kT * D + i);
            acc[i] += x.x; acc[i + 1] += x.y; acc[i + 2] += x.z; acc[i + 3] += x.w;
        }
    const int b = slab / Hkv, hk = slab - b * Hkv;
    float* dst = (which ? dk : dv) + (long long)(hk * D + d8) * stride + (long long)b * Skv + key;
#pragma unroll
    for (int i = 0; i < 8; ++i) dst[i * stride] = acc[i] * (which ? scale : 1.0f);
}

// dQ as an fp32 feature-major matrix = scale * accumulator: four features of one query per thread, consecutive threads on
// consecutive queries, in either form of the accumulator (fp32 [d/4][row][4] or 2^-32 fixed point [d/2][row][2]).
template <int D, bool kDet>
__global__ void __launch_bounds__(256) bwd_post_matrix_kernel(const float* __restrict__ dq_accum, float* __restrict__ dq, long long stride, int Hq,
                                                              int Sq, int n_qt, float scale)
{
    wait_for_stream();
    const size_t t = blockIdx.x;                          // tile: (b, h, query tile)
    const int bh = (int)(t / n_qt), qt = (int)(t - (size_t)bh * n_qt), b = bh / Hq, h = bh - b * Hq;
    const int row = threadIdx.x & 127, s = qt * kT + row;
    if (s >= Sq) return;
    const float* src = dq_accum + t * (size_t)(kT * D) * (kDet ? 2 : 1);
    float* dst = dq + (long long)h * D * stride + (long long)b * Sq + s;
#pragma unroll 4
    for (int c = threadIdx.x >> 7; c < D / 4; c += 2) {
        float x[4];
        if constexpr (!kDet) {
            const float4 v = *reinterpret_cast<const float4*>(src + ((size_t)c * kT + row) * 4);
            x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
        } else {
            const longlong2* w = reinterpret_cast<const longlong2*>(src);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const longlong2 v = w[(size_t)(2 * c + i) * kT + row];
                x[2 * i] = (float)((double)v.x * (1.0 / 4294967296.0));
                x[2 * i + 1] = (float)((double)v.y * (1.0 / 4294967296.0));
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) dst[(4 * c + i) * stride] = x[i] * scale;
    }
}

template <int D, bool kWin, bool kSplit, bool kDet, bool kMat>
cudaError_t launch_bwd(const TcArgs& a, cudaStream_t st)
{
    const AttnShape& s = a.s;
    const int n_qt = (s.Sq + kT - 1) / kT, n_kt = (s.Skv + kT - 1) / kT;
    const int Sq_pad = n_qt * kT;
    const long long rows_padded = (long long)s.B * s.Hq * Sq_pad;
    // workspace: [delta records | LSE records] then the accumulator (see tc_backward_workspace_bytes)
    constexpr bool kAug = bwd_folds_row_terms(D), kOwnDq = kDet && bwd_dq_has_kernel(D);
    const RowTerms terms = row_terms_of(a.delta, rows_padded, D, s.scale);
    cudaError_t e;
    const int phases = a.phases ? a.phases : (kBwdPre | kBwdMain | kBwdPost);
    if (phases & kBwdPre) {
        const long long blocks = rows_padded / kPreRows<D>;
        if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
        auto kernel = aligned(16, a.o, a.dout) ? bwd_pre_kernel<D, true> : bwd_pre_kernel<D, false>;
        if ((e = launch_kernel(kernel, (unsigned)blocks, 256, 0, st, 1, a.o, a.dout, a.lse, terms, a.dq_accum, s.Sq, Sq_pad, kOwnDq ? 0 : kDet ? 2 * D : D)) !=
            cudaSuccess)
            return e;
    }
    // dQ before dK and dV, which may lie where K and V lie; and where dQ lies on an input itself, it waits in the unused accumulator
    [[maybe_unused]] const size_t q_bytes = 2 * (size_t)s.B * s.Hq * s.Sq * D, kv_bytes = 2 * (size_t)s.B * s.Hkv * s.Skv * D;
    [[maybe_unused]] bool apart = true;
    if constexpr (kOwnDq) {
        auto clear_of = [&](const void* x, size_t bytes) { return (uintptr_t)x + bytes <= (uintptr_t)a.dq || (uintptr_t)a.dq + q_bytes <= (uintptr_t)x; };
        apart = kMat || (clear_of(a.q, q_bytes) && clear_of(a.dout, q_bytes) && clear_of(a.k, kv_bytes) && clear_of(a.v, kv_bytes));
        TcArgs b = a;
        if (!apart) b.dq = reinterpret_cast<__nv_bfloat16*>(a.dq_accum);
        if ((e = tc_backward_dq(b, st)) != cudaSuccess) return e;
    }
    if (phases & kBwdMain) {
    CUtensorMap tq, tk, tv, tdo;
    if ((e = encode_tmap_bf16_3d(&tq, a.q, D, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tdo, a.dout, D, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tk, a.k, D, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tv, a.v, D, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    BwdParams p{};
    p.dk = a.dk; p.dv = a.dv;
    p.qaug = (const uint4*)terms.lse; p.doaug = (const uint4*)terms.delta; p.lse2 = (const float*)terms.lse;
    p.delta = (const float*)terms.delta; p.dq_accum = a.dq_accum;
    p.B = s.B; p.Hq = s.Hq; p.Hkv = s.Hkv; p.Sq = s.Sq; p.Skv = s.Skv; p.Sq_pad = Sq_pad;
    p.causal = s.causal;
    p.window = s.causal ? s.window : 0;
    p.global_tokens = s.global_tokens;
    p.n_qt = n_qt; p.n_kt = n_kt;
    const BwdCut cut = kSplit ? bwd_cut(s) : BwdCut{};
    p.split_tiles = cut.tiles; p.split_steps = cut.steps; p.split_pieces = cut.pieces; p.whole_first = cut.whole_first;
    p.dkv_part = reinterpret_cast<float*>(reinterpret_cast<char*>(a.dq_accum) + align256((kDet ? 8 : 4) * (size_t)rows_padded * D));
    p.dk_acc = a.dk_acc; p.dv_acc = a.dv_acc;
    p.dk_mat = a.mat.dk; p.dv_mat = a.mat.dv; p.mat_stride = a.mat.stride;
    p.scale = s.scale;
    p.scale_log2 = s.scale * 1.4426950408889634f;
    const int slabs = s.B * s.Hkv;
    long long ctas = (long long)(n_kt - p.split_tiles) * slabs, n_pieces = 0;
    if (cut.pieces > kMaxPieces) return cudaErrorInvalidValue;
    for (int piece = 0; piece < cut.pieces; ++piece) {      // (a later tile has no more steps than an earlier one)
        for (int kt = 0; kt < cut.tiles; ++kt) {
            const int steps = bwd_tiles_per_head(kt, n_qt, s.causal, p.window, s.global_tokens) * (s.Hq / s.Hkv);
            const int pieces = bwd_piece_count(steps, cut.steps), len = (steps + pieces - 1) / pieces;
            if (piece * len < steps) n_pieces += slabs;
        }
        p.piece_end[piece] = (int)n_pieces;
    }
    ctas += n_pieces;
    p.several_waves = ctas > sm_count();
    if (ctas > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    static std::atomic<unsigned long long> configured{0};   // per instantiation, one bit per device
    {
        constexpr int kDoStages = (D == 128) ? 1 : 2;
        // K, V, Q stages, dO stages; the dS tile (two at head_dim 64); dQ staging; the per-query terms (see sTail in the kernel)
        constexpr int kQStages = (D == 128) ? 2 : 3;
        const size_t smem = (size_t)(128 * D * 2) * (2 + kQStages + kDoStages) + (D == 128 ? 1 : 2) * 128 * 128 * 2 + 32 * 1024 +
                            (kAug ? (size_t)(2 + kQStages + kDoStages) * 128 * 16 : (size_t)2 * kQStages * 128 * 4) + sizeof(BwdBarriers);
        if ((e = ensure_dynamic_smem(attn_bwd_tc_kernel<D, kWin, kSplit, kDet, kMat>, smem, configured)) != cudaSuccess) return e;
        if ((e = launch_kernel(attn_bwd_tc_kernel<D, kWin, kSplit, kDet, kMat>, (unsigned)ctas, kBwdThreads, smem, st, 1, tq, tk, tv, tdo, p)) !=
            cudaSuccess)
            return e;
    }
    if (p.split_tiles > 0) {
        const long long n_units = (long long)p.split_tiles * slabs * 2 * kT * (D / 8);
        const unsigned blocks = (unsigned)((n_units + 255) / 256);
        const BwdPieces pieces{n_qt, p.causal, p.window, p.global_tokens, s.Hq / s.Hkv, cut.steps, cut.pieces};
        if constexpr (kMat)
            e = launch_kernel(bwd_dkv_reduce_matrix_kernel<D>, blocks, 256, 0, st, 1, p.dkv_part, a.mat.dk, a.mat.dv, a.mat.stride, pieces,
                              s.Hkv, slabs, s.Skv, s.scale, n_units);
        else
            e = launch_kernel(bwd_dkv_reduce_kernel<D>, blocks, 256, 0, st, 1, p.dkv_part, a.dk, a.dv, pieces, slabs, s.Skv, s.scale, n_units);
        if (e != cudaSuccess) return e;
    }
    }   // kBwdMain
    if (!(phases & kBwdPost)) return cudaSuccess;
    const unsigned tiles = (unsigned)((long long)s.B * s.Hq * n_qt);
    if constexpr (kOwnDq)
        return apart ? cudaSuccess : cudaMemcpyAsync(a.dq, a.dq_accum, q_bytes, cudaMemcpyDeviceToDevice, st);
    else if constexpr (kMat)
        return launch_kernel(bwd_post_matrix_kernel<D, kDet>, tiles, 256, 0, st, 1, a.dq_accum, a.mat.dq, a.mat.stride, s.Hq, s.Sq, n_qt, s.scale);
    else if constexpr (kDet)
        return launch_kernel(bwd_post_det_kernel<D>, tiles, 256, 0, st, 1, reinterpret_cast<const unsigned long long*>(a.dq_accum), a.dq, s.Sq,
                             n_qt, s.scale);
    else
        return launch_kernel(bwd_post_kernel<D>, tiles, 256, 0, st, 1, a.dq_accum, a.dq, s.Sq, n_qt, s.scale);
}

}  // namespace

bool tc_bwd_supported(const AttnShape& s)
{
    return (s.D == 64 || s.D == 128) && (!s.causal || s.Sq == s.Skv);
}

// [delta records: B*Hq*Sq_pad x 16 bytes][LSE records: same], 256-byte aligned, then the fp32 dQ accumulator B*Hq*Sq_pad*D, then the fp32
// dK/dV partials of the key tiles that are cut into pieces (none for most shapes)
size_t tc_backward_workspace_bytes(const AttnShape& s) { return bwd_base_bytes(s) + align256(bwd_part_bytes(s, bwd_cut(s))); }

namespace {
template <int D, bool kMat>
cudaError_t dispatch_bwd(const TcArgs& a, cudaStream_t st)
{
    const bool win = a.s.causal && a.s.window > 0;
    const bool cut = bwd_cut(a.s).tiles > 0;
    if (a.s.deterministic) {
        if (cut) return win ? launch_bwd<D, true, true, true, kMat>(a, st) : launch_bwd<D, false, true, true, kMat>(a, st);
        return win ? launch_bwd<D, true, false, true, kMat>(a, st) : launch_bwd<D, false, false, true, kMat>(a, st);
    }
    if (cut) return win ? launch_bwd<D, true, true, false, kMat>(a, st) : launch_bwd<D, false, true, false, kMat>(a, st);
    return win ? launch_bwd<D, true, false, false, kMat>(a, st) : launch_bwd<D, false, false, false, kMat>(a, st);
}
template <int D>
cudaError_t dispatch_bwd_out(const TcArgs& a, cudaStream_t st)
{
    // the accumulate form (backward in pieces) has no window, no fixed-point dQ and no cut key tiles: their fp32 partials
    // would need a second adding pass
    if (a.dk_acc) return launch_bwd<D, false, false, false, false>(a, st);
    return a.mat.dk ? dispatch_bwd<D, true>(a, st) : dispatch_bwd<D, false>(a, st);
}
}  // namespace

cudaError_t tc_backward(const TcArgs& a, cudaStream_t st)
{
    // Every address is looked at before the first launch: operands go through tensor maps, the rest is accessed 16 bytes at a time
    // (O and, by the pre-pass alone, dO 8).  Matrix results are stored element by element; unused pointers are null.
    const int phases = a.phases ? a.phases : (kBwdPre | kBwdMain | kBwdPost);
    bool ok = aligned(16, a.delta, a.dq_accum);
    if (phases & kBwdPre) ok = ok && aligned(8, a.o, a.dout);
    if (phases & kBwdMain) ok = ok && aligned(16, a.q, a.k, a.v, a.dout, a.dk, a.dv, a.dk_acc, a.dv_acc);
    if (phases & kBwdPost) ok = ok && aligned(16, a.dq);
    if (!ok) return cudaErrorMisalignedAddress;
    return a.s.D == 64 ? dispatch_bwd_out<64>(a, st) : dispatch_bwd_out<128>(a, st);
}

#ifdef SNTL_TRACE
// trace build only: choose the CTA that records and read back what the last launch recorded
extern "C" int sntl_debug_trace_bwd(unsigned long long* out, int n_words, int set_cta)
{
    if (out && cudaMemcpyFromSymbol(out, ptx::g_trace, sizeof(unsigned long long) * n_words) != cudaSuccess) return 1;
    static unsigned long long zeros[ptx::kTraceRoles * ptx::kTraceDepth];
    if (cudaMemcpyToSymbol(ptx::g_trace, zeros, sizeof(zeros)) != cudaSuccess) return 2;
    unsigned int c = (unsigned int)set_cta;
    return cudaMemcpyToSymbol(ptx::g_trace_cta, &c, sizeof(c)) == cudaSuccess ? 0 : 3;
}
#endif

cudaError_t read_and_clear_bwd_status(cudaStream_t st, uint32_t* word)
{
    cudaError_t e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) return e;
    unsigned int w = 0, zero = 0;
    if ((e = cudaMemcpyFromSymbol(&w, ptx::g_device_status, sizeof(w))) != cudaSuccess) return e;
    if (w != 0 && (e = cudaMemcpyToSymbol(ptx::g_device_status, &zero, sizeof(zero))) != cudaSuccess) return e;
    uint32_t f32 = 0, dq = 0;
    if ((e = read_and_clear_f32_bwd_status(&f32)) != cudaSuccess || (e = read_and_clear_dq_status(&dq)) != cudaSuccess) return e;
    *word = w ? w : f32 ? f32 : dq;
    return cudaSuccess;
}

}  // namespace sntl
