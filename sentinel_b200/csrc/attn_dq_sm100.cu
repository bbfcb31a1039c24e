// dQ with one owner per element: the backward's third product for SNTL_FLAG_DETERMINISTIC at head_dim 128.  A block owns 128 query rows
// of one (batch, head) and visits the key tiles that they see: S = Q K^T, dP = dO V^T, dS = P o (dP - delta), dQ += dS K; the kernel for dK
// and dV (attn_bwd_sm100.cu) then leaves dQ out.  P, dS and the contribution of a key tile are rounded as that kernel rounds them, and the
// contributions are summed as it sums them under the flag at head_dim 64: exactly, as 64-bit integers (2^-32 units), rounded once at the
// end.  dQ so has the bits that reductions of 64-bit words give, and no scratch is needed.  Seven products instead of five, against
// reductions that outlasted the five: 128 KB per step at the 25.5 bytes per clock that an SM gets through to L2.
//
// Backward, us, against the 64-bit reductions: B3 Hq16 Hkv4 S1237 D128 133 -> 110; B8 Hq28 Hkv4 S1024 417 -> 255 (336 and 294 for gradients
// 10^3 and 10^5 times as large, WideSums); B1 Hq28 Hkv4 S8192 2140 -> 1575; B1 Hq28 Hkv4 S256 66 -> 42; one head of 2048 tokens 73 -> 64, of
// 16384 (a chain of 128 tiles on most SMs) 298 -> 320.  (The exact sums cost 6 to 13 % of this: with fp32 sums in TMEM, which cut off towards
// zero, B3 S1237 took 98, B8 S1024 240.)  A tile takes about 2750 cycles for 1536 of products, 1024 of exponentials and 1024 of fp32
// additions: dP goes where dS was, so from dS of a tile over its dQ product and the next dP to the next dS is one loop.  A block costs
// about 7500 more (loads of Q and dO, the first scores, the last sums).
//
//   warps 0-15   weights: thread = one query row and a quarter of a tile's 128 keys
//   warps 16-23  sums: thread = one query row and half of the features, 64 integers in registers (128 of its 160)
//   warp 24      loads (TMA), warp 25 issues the products
// TMEM: S [0, 128); dP [128, 256), over it the bf16 dS of each quarter of the keys; two contributions to dQ [256, 384), [384, 512).  The
// scores of a tile are computed under the second half of the work on the tile before.
#include "block_queue.cuh"
#include "row_terms.cuh"

namespace sntl {
using namespace ptx;
namespace {

constexpr int kD = 128, kT = 128, kWeightThreads = 512, kSumThreads = 256, kSumWarp = 16, kLoadWarp = 24, kIssueWarp = 25, kThreads = 896, kChunks = kD / 64, kChunkBytes = kT * 128;
constexpr uint32_t kColS = 0, kColDp = 128, kColDq = 256;
// (72 registers a thread at launch)
constexpr int kWeightRegs = 40, kSumRegs = 160, kOtherRegs = 24;
static_assert(kWeightThreads * kWeightRegs + kSumThreads * kSumRegs + 128 * kOtherRegs <= kThreads * 72, "");

struct Bars {
    BlockQueue<26> queue;
    uint64_t q_full, q_free, k_full[3], k_free[3], v_full[2], v_free[2], s_full, s_free, dp_full, ds_full, dq_full[2], dq_free[2];
    uint32_t tmem_base, abort_flag;
};
struct Smem {
    // A K tile is read last by its tile's dQ product, so the loop from its release over the next load, scores and sums to the next
    // release spans as many tiles as there are stages: two are too few.
    static constexpr int kKStages = 3, kVStages = 2;
    static constexpr int kTile = kT * kD * 2, q = 0, dout = kTile, k = 2 * kTile, v = k + kKStages * kTile, bars = v + kVStages * kTile;
    static constexpr int bytes = bars + (int)sizeof(Bars) + 1024;
};
static_assert(Smem::bytes <= 227 * 1024, "");
using L = Smem;

template <int N> struct Int { static constexpr int value = N; };

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

// A thread's sums of 64 elements in units of 2^-32; every contribution is rounded to such a unit to nearest even, as __float2ll_rn(2^32 x)
// does.  That conversion has the rate of the exponentials and would share their pipe, and 64-bit additions take as long again, so the usual
// case is done in 32 bits: x + 1.5 2^14 has its last bit at 2^-9, what that leaves of x plus 1.5 2^-9 at 2^-32, and the bits of the two
// are integers in these units but for constants, which are subtracted at the end.  Once |x| reaches 2^13 (the exponent of the first sum
// would be another) or is not finite, the warp goes on with conversions and 64-bit sums for the rest of the block (WideSums).
constexpr uint32_t kHighBits = 0x46c00000u, kLowBits = 0x3b400000u;     // 1.5 2^14, 1.5 2^-9
constexpr float kUnit = 2.3283064365386963e-10f;                        // 2^-32
struct Sums {
    uint32_t high[64], low[64];
    int n = 0;         // contributions in them

    __device__ __forceinline__ Sums()
    {
#pragma unroll
        for (int i = 0; i < 64; ++i) high[i] = low[i] = 0;
    }
    static __device__ __forceinline__ void split(float2 y, float2& t, float2& u)
    {
        const float2 h = make_float2(__uint_as_float(kHighBits), __uint_as_float(kHighBits)), l = make_float2(__uint_as_float(kLowBits), __uint_as_float(kLowBits));
        t = fadd2(y, h);
        u = fadd2(ffma2(fadd2(t, make_float2(-h.x, -h.y)), make_float2(-1.f, -1.f), y), l);
    }
    // contributions to the elements from i0 on, and the sum of their squares; kTakeOut: taken out again
    template <int i0, bool kTakeOut> __device__ __forceinline__ void add(const uint32_t (&x)[16], float2& squares)
    {
#pragma unroll
        for (int i = 0; i < 16; i += 2) {
            const float2 y = make_float2(__uint_as_float(x[i]), __uint_as_float(x[i + 1]));
            float2 t, u;
            split(y, t, u);
            if constexpr (kTakeOut) {
                high[i0 + i] -= __float_as_uint(t.x);
                high[i0 + i + 1] -= __float_as_uint(t.y);
                low[i0 + i] -= __float_as_uint(u.x);
                low[i0 + i + 1] -= __float_as_uint(u.y);
            } else {
                high[i0 + i] += __float_as_uint(t.x);
                high[i0 + i + 1] += __float_as_uint(t.y);
                low[i0 + i] += __float_as_uint(u.x);
                low[i0 + i + 1] += __float_as_uint(u.y);
                squares = ffma2(y, y, squares);
            }
        }
    }
    // |high| grows by up to 2^22 per tile, |low| too: every 256 tiles `low` is carried over.  False: `high` may not have room for as many more.
    __device__ __forceinline__ bool carry_over()
    {
        const uint32_t h0 = n * kHighBits, l0 = n * kLowBits;
        uint32_t large = 0;
#pragma unroll
        for (int i = 0; i < 64; ++i) {
            const uint32_t l = low[i] - l0;
            high[i] = high[i] - h0 + (uint32_t)((int)l >> 23);
            low[i] = l & 0x7fffffu;
            large |= high[i] + (1u << 29);
        }
        n = 0;
        return __all_sync(0xffffffffu, large >> 30 == 0);
    }
    // Scale times the sums, as fp32 in the place of `high`: the integers rounded to fp32, to nearest even, by one FMA of two that fp32 holds,
    // high + carry and the low 23 bits (signed).  (Conversions, with the rate of the exponentials again, took 3300 cycles of a block, 7200
    // beside them.)  False, and nothing done: some |high| is 2^21 or more (with the carry it has to be below 2^22).
    __device__ __forceinline__ bool finish(float scale)
    {
        const uint32_t h0 = n * kHighBits, l0 = n * kLowBits - (1u << 22);
        uint32_t large = 0;
#pragma unroll
        for (int i = 0; i < 64; ++i) large |= high[i] - (h0 - (1u << 21));
        if (__any_sync(0xffffffffu, large >> 22 != 0)) return false;
        constexpr uint32_t kTwo23 = 0x4b000000u;      // 2^23 in fp32, whose last bit is 1
        const float2 h1 = make_float2(-12582912.f, -12582912.f), unit = make_float2(kUnit, kUnit);
#pragma unroll
        for (int i = 0; i < 64; i += 2) {
            float2 h, l;
            auto parts = [&](int j, float& hf, float& lf) {
                const uint32_t low_up = low[j] - l0;       // low + 2^22
                hf = __uint_as_float(high[j] - (h0 - kTwo23 - (1u << 22)) + (uint32_t)((int)low_up >> 23));
                lf = __uint_as_float((low_up & 0x7fffffu) | kTwo23);
            };
            parts(i, h.x, l.x);
            parts(i + 1, h.y, l.y);
            const float2 sum = ffma2(fadd2(h, h1), make_float2(8388608.f, 8388608.f), fadd2(l, h1));
            const float2 y = fmul2(fmul2(sum, unit), make_float2(scale, scale));
            high[i] = __float_as_uint(y.x);
            high[i + 1] = __float_as_uint(y.y);
        }
        return true;
    }
};
struct WideSums {
    long long sum[64];

    __device__ __forceinline__ explicit WideSums(const Sums& s)
    {
        const uint32_t h0 = s.n * kHighBits, l0 = s.n * kLowBits;
#pragma unroll
        for (int i = 0; i < 64; ++i) sum[i] = (long long)(int)(s.high[i] - h0) * (1 << 23) + (int)(s.low[i] - l0);
    }
    template <int i0> __device__ __forceinline__ void add(const uint32_t (&x)[16])
    {
#pragma unroll
        for (int i = 0; i < 16; ++i) sum[i0 + i] += __float2ll_rn(__uint_as_float(x[i]) * 4294967296.0f);
    }
    __device__ __forceinline__ float result(int i, float scale) const { return (float)(double)sum[i] * kUnit * scale; }
};

template <bool kMat>
__global__ void __launch_bounds__(kThreads, 1)
    attn_dq_tc_kernel(const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
                      const __grid_constant__ CUtensorMap tmap_do, const Params p)
{
    extern __shared__ uint8_t raw[];
    uint8_t* smem = raw + (1024 - (smem_u32(raw) & 1023)) % 1024;
    Bars* bars = reinterpret_cast<Bars*>(smem + L::bars);
    const int warp = warp_uniform(threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        bars->queue.init();
        mbar_init(&bars->q_full, 1);
        mbar_init(&bars->q_free, 1);
        for (int i = 0; i < L::kKStages; ++i) {
            mbar_init(&bars->k_full[i], 1);
            mbar_init(&bars->k_free[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bars->v_full[i], 1);
            mbar_init(&bars->v_free[i], 1);
            mbar_init(&bars->dq_full[i], 1);
            mbar_init(&bars->dq_free[i], kSumThreads);
        }
        mbar_init(&bars->dp_full, 1);
        mbar_init(&bars->ds_full, kWeightThreads);
        mbar_init(&bars->s_full, 1);
        mbar_init(&bars->s_free, kWeightThreads);
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
    const int part = warp >> 2, half = part & 1, r = (warp & 3) * 32 + lane;
    const uint32_t lanes = tmem + ((uint32_t)(warp & 3) << 21);
    if (warp < kSumWarp) {
        setmaxnreg_dec<kWeightRegs>();
        const float2 scale2 = make_float2(s.scale * 1.4426950408889634f, s.scale * 1.4426950408889634f);
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            const int row = w.qt * kT + r, n_row = s.causal ? min(row + 1, s.Skv) : s.Skv;
            const size_t padded = (size_t)w.bh * p.n_qt * kT + row;
            const float lse = __ldg(static_cast<const float*>(p.lse) + padded);        // -LSE (log2)
            const float delta = __ldg(static_cast<const float*>(p.delta) + padded);    // -delta
            bool ok = true;
            for (int k0 = w.tile(s, 0); k0 < w.n_keys; k0 = w.tile(s, k0 + kT), ++c) {
                const uint32_t scores = lanes + kColS + part * 32, dp = lanes + kColDp + part * 32;
                if (!(ok = mbar_wait_warp(&bars->s_full, c & 1, abort_flag, 0x61))) break;
                tc_fence_after();
                uint32_t ds[16];       // P, then dS, as pairs of bf16
                uint32_t x[2][8];
                tmem_ld8(scores, x[0]);
                auto weights = [&](auto&& seen) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        tmem_ld_wait();
                        if (j < 3) {
                            tmem_ld8(scores + (j + 1) * 8, x[(j + 1) & 1]);
                        } else {
                            tc_fence_before();
                            mbar_arrive(&bars->s_free);
                        }
                        const uint32_t* y = x[j & 1];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const float2 e = ffma2(make_float2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])), scale2, make_float2(lse, lse));
                            ds[4 * j + i] = pack_bf16(seen(8 * j + 2 * i) ? ex2(e.x) : 0.f, seen(8 * j + 2 * i + 1) ? ex2(e.y) : 0.f);
                        }
                    }
                };
                // every pair of the tile is visible, or a mask
                if (!(k0 + kT > (s.causal ? w.qt * kT + 1 : s.Skv) || s.window > 0)) {
                    weights([](int) { return true; });
                } else {
                    const uint32_t mask = keys_seen(s, row, n_row, k0 + part * 32);
                    weights([&](int i) { return (mask >> i & 1u) != 0; });
                }
                if (!(ok = mbar_wait_warp(&bars->dp_full, c & 1, abort_flag, 0x62))) break;
                tc_fence_after();
                tmem_ld8(dp, x[0]);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    tmem_ld_wait();
                    if (j < 3) tmem_ld8(dp + (j + 1) * 8, x[(j + 1) & 1]);
                    const uint32_t* y = x[j & 1];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        uint32_t& z = ds[4 * j + i];
                        const float2 d = fmul2(make_float2(__uint_as_float(z << 16), __uint_as_float(z & 0xffff0000u)),
                                               fadd2(make_float2(__uint_as_float(y[2 * i]), __uint_as_float(y[2 * i + 1])), make_float2(delta, delta)));
                        z = pack_bf16(d.x, d.y);
                    }
                    if (j & 1) tmem_st8(dp + (j - 1) * 4, ds + (j - 1) * 4);
                }
                tmem_st_wait();
                tc_fence_before();
                mbar_arrive(&bars->ds_full);
            }
            if (!ok) break;
        }
    } else if (warp < kLoadWarp) {
        setmaxnreg_inc<kSumRegs>();
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            const int row = w.qt * kT + r;
            bool ok = true;
            int k0 = w.tile(s, 0);
            auto next_tile = [&]() {
                tc_fence_before();
                mbar_arrive(&bars->dq_free[c & 1]);
                k0 = w.tile(s, k0 + kT);
                ++c;
            };
            // f(first column, sixteen values) for a thread's 64 columns of the contribution
            auto all = [&](auto&& f) {
                const uint32_t dq = lanes + kColDq + (c & 1) * 128 + half * 64;
                auto sixteen = [&](auto j_) {
                    constexpr int j = decltype(j_)::value;
                    uint32_t x[16];
                    tmem_ld8(dq + j * 16, x);
                    tmem_ld8(dq + j * 16 + 8, x + 8);
                    tmem_ld_wait();
                    f(Int<j * 16>{}, x);
                };
                sixteen(Int<0>{}); sixteen(Int<1>{}); sixteen(Int<2>{}); sixteen(Int<3>{});
            };
            auto store = [&](auto&& result) {
                if (row < s.Sq && kMat) {
                    float* dst = p.dq_mat + ((long long)w.h * kD + half * 64) * p.mat_stride + (long long)w.b * s.Sq + row;
#pragma unroll
                    for (int i = 0; i < 64; ++i, dst += p.mat_stride) *dst = result(i);
                } else if (row < s.Sq) {
                    uint4* dst = reinterpret_cast<uint4*>(p.dq + ((size_t)w.bh * s.Sq + row) * kD + half * 64);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        auto two = [&](int i) { return pack_bf16(result(8 * j + i), result(8 * j + i + 1)); };
                        dst[j] = make_uint4(two(0), two(2), two(4), two(6));
                    }
                }
            };
            Sums sums;
            bool wide = false, have = false;      // (the same in all lanes; have: the tile that is waited for already)
            while (k0 < w.n_keys) {
                if (!(ok = mbar_wait_warp(&bars->dq_full[c & 1], (c >> 1) & 1, abort_flag, 0x63))) break;
                tc_fence_after();
                float2 squares = make_float2(0.f, 0.f);
                all([&](auto i0, const uint32_t (&x)[16]) { sums.template add<decltype(i0)::value, false>(x, squares); });
                // below 2^26 all |x| are below 2^13
                if (__any_sync(0xffffffffu, !(squares.x + squares.y < 67108864.0f))) {
                    all([&](auto i0, const uint32_t (&x)[16]) { sums.template add<decltype(i0)::value, true>(x, squares); });
                    wide = have = true;
                    break;
                }
                next_tile();
                if (++sums.n == 256 && !sums.carry_over()) {
                    wide = true;
                    break;
                }
            }
            if (!ok) break;
            if (!wide && sums.finish(s.scale)) {
                store([&](int i) { return __uint_as_float(sums.high[i]); });
            } else {
                WideSums sums64(sums);
                for (; k0 < w.n_keys; have = false) {
                    if (!have && !(ok = mbar_wait_warp(&bars->dq_full[c & 1], (c >> 1) & 1, abort_flag, 0x63))) break;
                    tc_fence_after();
                    all([&](auto i0, const uint32_t (&x)[16]) { sums64.template add<decltype(i0)::value>(x); });
                    next_tile();
                }
                if (!ok) break;
                store([&](int i) { return sums64.result(i, s.scale); });
            }
            __syncwarp();
        }
    } else if (warp == kLoadWarp) {
        setmaxnreg_dec<kOtherRegs>();
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            bool ok = true;
            if (lane == 0) {
                auto load = [&](int dst, const CUtensorMap* map, uint64_t* bar, int row, int slab) {
                    for (int i = 0; i < kChunks; ++i) tma_load_3d(smem + dst + i * kChunkBytes, map, bar, i * 64, row, slab);
                };
                // Q and dO once the last scores of the block before have been computed
                ok = u == 0 || mbar_wait(&bars->q_free, (u - 1) & 1, abort_flag, 0x64);
                if (ok) {
                    mbar_arrive_expect_tx(&bars->q_full, 2 * L::kTile);
                    load(L::q, &tmap_q, &bars->q_full, w.qt * kT, w.bh);
                    load(L::dout, &tmap_do, &bars->q_full, w.qt * kT, w.bh);
                }
                for (int k0 = w.tile(s, 0); ok && k0 < w.n_keys; k0 = w.tile(s, k0 + kT), ++c) {
                    const int sk = c % L::kKStages, sv = c % L::kVStages;
                    if (c >= L::kKStages && !(ok = mbar_wait(&bars->k_free[sk], (c / L::kKStages - 1) & 1, abort_flag, 0x65))) break;
                    mbar_arrive_expect_tx(&bars->k_full[sk], L::kTile);
                    load(L::k + sk * L::kTile, &tmap_k, &bars->k_full[sk], k0, w.bh_kv);
                    if (c >= L::kVStages && !(ok = mbar_wait(&bars->v_free[sv], (c / L::kVStages - 1) & 1, abort_flag, 0x66))) break;
                    mbar_arrive_expect_tx(&bars->v_full[sv], L::kTile);
                    load(L::v + sv * L::kTile, &tmap_v, &bars->v_full[sv], k0, w.bh_kv);
                }
                if (ok) ok = bars->queue.ask(u + 1, abort_flag);
            }
            c = warp_uniform(c);
            if (!__all_sync(0xffffffffu, ok)) break;
        }
    } else if (warp == kIssueWarp) {
        setmaxnreg_dec<kOtherRegs>();
        constexpr uint32_t idesc_s = make_idesc(kT, kT, false, false), idesc_dq = make_idesc(kT, kD, false, true);
        const uint64_t q = make_sdesc(smem_u32(smem + L::q), 16, 1024), dout = make_sdesc(smem_u32(smem + L::dout), 16, 1024);
        const uint64_t k = make_sdesc(smem_u32(smem + L::k), 16, 1024), v = make_sdesc(smem_u32(smem + L::v), 16, 1024);
        const uint64_t k_mn = make_sdesc(smem_u32(smem + L::k), kChunkBytes, 1024);
        auto wait = [&](uint64_t* bar, int parity, uint32_t site) { return mbar_wait_warp(bar, parity & 1, abort_flag, site); };
        auto product = [&](uint32_t d, uint64_t a, uint64_t b) {
#pragma unroll
            for (int i = 0; i < kChunks; ++i) mma_ss_4<2, 2>(d, sdesc_advance(a, i * kChunkBytes), sdesc_advance(b, i * kChunkBytes), idesc_s, i > 0);
        };
        // of tile number n; dP of the `last` of its block.  dP goes over the dS of the tile before, whose product has been issued.
        auto scores = [&](int n) {
            const int sk = n % L::kKStages;
            if (!wait(&bars->k_full[sk], n / L::kKStages, 0x67) || (n > 0 && !wait(&bars->s_free, n - 1, 0x68))) return false;
            tc_fence_after();
            product(tmem + kColS, q, sdesc_advance(k, sk * L::kTile));
            tc_commit_p(&bars->s_full);
            return true;
        };
        auto weight_gradients = [&](int n, bool last) {
            const int sv = n % L::kVStages;
            if (!wait(&bars->v_full[sv], n / L::kVStages, 0x69)) return false;
            tc_fence_after();
            product(tmem + kColDp, dout, sdesc_advance(v, sv * L::kTile));
            tc_commit_p(&bars->dp_full);
            tc_commit_p(&bars->v_free[sv]);
            if (last) tc_commit_p(&bars->q_free);
            return true;
        };
        int c = 0;
        for (int u = 0, block = blockIdx.x; block >= 0; block = bars->queue.get(++u, abort_flag)) {
            const Block w(p, block);
            int k0 = w.tile(s, 0), next = w.tile(s, k0 + kT);
            bool ok = wait(&bars->q_full, u, 0x6a) && scores(c) && weight_gradients(c, next >= w.n_keys);
            for (; ok && k0 < w.n_keys; ++c) {
                const int sk = c % L::kKStages, st = c & 1;
                const bool more = next < w.n_keys;
                if (more && !(ok = scores(c + 1))) break;
                if (!(ok = wait(&bars->ds_full, c, 0x6b) && (c < 2 || wait(&bars->dq_free[st], (c >> 1) - 1, 0x6c)))) break;
                tc_fence_after();
                const uint64_t b = sdesc_advance(k_mn, sk * L::kTile);
#pragma unroll
                for (int i = 0; i < 4; ++i) mma_ts_2<8, 128>(tmem + kColDq + st * 128, tmem + kColDp + 32 * i, sdesc_advance(b, i * 2 * 2048), idesc_dq, i > 0);
                tc_commit_p(&bars->dq_full[st]);
                tc_commit_p(&bars->k_free[sk]);
                k0 = next;
                next = w.tile(s, k0 + kT);
                if (more && !(ok = weight_gradients(c + 1, next >= w.n_keys))) break;
            }
            if (!ok) break;
        }
    } else {
        setmaxnreg_dec<kOtherRegs>();
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

template <bool kMat> cudaError_t launch(const TcArgs& a, const RowTerms& terms, cudaStream_t st)
{
    const AttnShape& s = a.s;
    CUtensorMap tq, tk, tv, tdo;
    cudaError_t e;
    if ((e = encode_tmap_bf16_3d(&tq, a.q, kD, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tdo, a.dout, kD, s.Sq, s.B * s.Hq, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tk, a.k, kD, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    if ((e = encode_tmap_bf16_3d(&tv, a.v, kD, s.Skv, s.B * s.Hkv, 128)) != cudaSuccess) return e;
    static std::atomic<unsigned long long> configured{0};
    if ((e = ensure_dynamic_smem(attn_dq_tc_kernel<kMat>, Smem::bytes, configured)) != cudaSuccess) return e;
    const int n_qt = (s.Sq + kT - 1) / kT;
    const long long blocks = (long long)n_qt * s.B * s.Hq;
    if (blocks > 0x7fffffffLL) return cudaErrorInvalidConfiguration;
    Params p{s, terms.lse, terms.delta, a.dq, a.mat.dq, a.mat.stride, n_qt};
    if (!s.causal) p.s.window = 0;
    return launch_kernel(attn_dq_tc_kernel<kMat>, (unsigned)blocks, kThreads, Smem::bytes, st, 1, tq, tk, tv, tdo, p);
}

}  // namespace

cudaError_t tc_backward_dq(const TcArgs& a, cudaStream_t st)
{
    const AttnShape& s = a.s;
    const RowTerms terms = row_terms_of(a.delta, (long long)s.B * s.Hq * ((s.Sq + kT - 1) / kT) * kT, s.D, s.scale);
    return a.mat.dq ? launch<true>(a, terms, st) : launch<false>(a, terms, st);
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
