// Exact fp32 calls that both the FMA kernels (attn_simt_*.cu) and the split products on the tensor cores (attn_f32_*_sm100.cu) take: which of
// them a call goes to.  The split products do a tile in a fraction of the time, but their blocks have 128 rows, a set-up, one chain of
// tiles with no split over the keys, and a second launch behind them that looks for marks; the FMA kernels choose smaller tiles and
// spread the keys over a cluster where a grid is small.  Both times are estimated from the tiles that the mask leaves, counted as the
// kernels visit them: the larger of the longest chain and of an SM's share of everything.
//
// The constants (us) are fitted to 190 calls, which the estimates meet within 15 % for nearly all and for which they choose the slower side
// by more than 3 % five times (by 14 % once, B8 Hq16 Hkv8 S191 D16 backward, 43 / 49).  FMA against split
// products, us:
//   forward   cached T64 L8192, H4 D32 53 / 197, D64 85 / 200, H12 D64 104 / 200; T256 L2048 H4 D32 29 / 56; T512 L2048 H4 D64 82 / 57
//             B1 H1 D64, S1024 22.4 / 33.2, S2048 74 / 57; D16 S2048 37 / 55; B8 H12 S512 D64 118 / 42; window 16 of B1 H12 S1024 D32 14.4 / 15.6,
//             window 256 29 / 19
//   backward  B3 H16 S224 D16 25.7 / 28.2, D32 36 / 29.5; B1 H1 S1024 D64 113 / 65; B8 H12 S512 D64 404 / 135
#include "common.cuh"

#include <algorithm>

namespace sntl {
namespace {

struct Visits {
    double longest = 0, all = 0;      // tiles of `cols` that a tile of `rows` visits: the longest chain, the sum
};
// (up to 64 tiles are looked at, evenly spread: the sum is that of a sample for more)
template <typename F> Visits count(int rows_in_all, int rows, F&& visited)
{
    const int n = (rows_in_all + rows - 1) / rows, step = std::max(1, n / 64);
    Visits v;
    int seen = 0;
    for (int i = 0; i < n; i += step, ++seen) {
        const double x = visited(i * rows);
        v.longest = std::max(v.longest, x);
        v.all += x;
    }
    v.longest = std::max(v.longest, (double)visited((n - 1) * rows));
    v.all *= (double)n / seen;
    return v;
}
int shift_of(const AttnShape& s) { return s.causal ? s.Skv - s.Sq : 0; }
// query tiles: the key tiles between the global tokens and the window of the first row are skipped
Visits query_tiles(const AttnShape& s, int rows, int cols)
{
    return count(s.Sq, rows, [&](int r0) {
        const int end = s.causal ? std::min(std::min(r0 + rows, s.Sq) + shift_of(s), s.Skv) : s.Skv, n = (end + cols - 1) / cols;
        if (s.window <= 0) return n;
        const int global = std::min((std::min(s.global_tokens, end) + cols - 1) / cols, n), first = std::max(0, r0 + shift_of(s) - s.window + 1) / cols;
        return std::min(n, global + std::max(0, n - std::max(global, first)));
    });
}
// key tiles: the queries from the first that sees a key to the last whose window reaches one
Visits key_tiles(const AttnShape& s, int rows, int cols)
{
    return count(s.Skv, rows, [&](int k0) {
        const int first = s.causal ? std::max(0, k0 - shift_of(s)) / cols : 0;
        const int end = s.window > 0 && k0 >= s.global_tokens ? (int)std::min<long long>(s.Sq, (long long)k0 + rows - 1 + s.window - shift_of(s)) : s.Sq;
        return std::max(0, (end + cols - 1) / cols - first);
    });
}

// us per visit of a tile of 16, 32 or 64 rows at head_dim up to 16, 32, 64: in a chain of its own, and of an SM's time when its CTAs share
// it (a CTA's set-up counts as half a visit there)
struct Cost {
    double chain[3][3], share[3][3];
};
constexpr Cost kForward = {{{1.9, 2.6, 4.3}, {2.4, 3.4, 5.5}, {4.8, 6.6, 10.0}}, {{0.95, 1.35, 2.4}, {1.0, 1.55, 2.6}, {2.25, 2.75, 4.5}}};
constexpr Cost kBackward = {{{3.2, 4.9, 7.6}, {4.0, 6.0, 9.0}, {7.0, 10.0, 15.0}}, {{1.1, 1.8, 3.2}, {1.7, 2.8, 5.0}, {3.4, 4.8, 8.0}}};
int index(int rows) { return rows / 32; }                         // 16, 32, 64
int dim_index(int D) { return D <= 16 ? 0 : D <= 32 ? 1 : 2; }
// blocks of a CTA that takes over blocks, one per SM: a second one is shared by few
double turns(double blocks_per_sm, double tail)
{
    return blocks_per_sm <= 1 ? blocks_per_sm : std::max(blocks_per_sm, std::min(2.0, blocks_per_sm + tail));
}

}  // namespace

bool f32_tc_forward_pays(const AttnShape& s)
{
    const double heads = (double)s.B * s.Hq, sms = sm_count();
    const SimtTiles t = simt_forward_tiles(s);
    const Visits f = query_tiles(s, t.rows, 64), m = query_tiles(s, 128, 128);
    const int i = index(t.rows), d = dim_index(s.D);
    const double ctas = (double)((s.Sq + t.rows - 1) / t.rows) * t.split, tiles = (s.Sq + 127) / 128, load = tiles * heads / sms;
    const double fma = 5 + std::max(f.longest / t.split * kForward.chain[i][d], (f.all + 0.5 * ctas) * heads / sms * kForward.share[i][d]);
    const double split_products = 4 + std::max(5 + 3 * m.longest + 3 * std::min(1.0, load), (3 * m.all / tiles + 4) * turns(load, 0.5));
    return split_products < fma;
}

bool f32_tc_backward_pays(const AttnShape& s)
{
    const int group = s.Hq / s.Hkv, rows = simt_backward_rows(s), i = index(rows), d = dim_index(s.D);
    const double heads = (double)s.B * s.Hq, sms = sm_count();
    auto both = [&](int rows_, int cols) {
        const Visits q = query_tiles(s, rows_, cols), k = key_tiles(s, rows_, cols);
        return Visits{std::max(q.longest, k.longest * group), (q.all + k.all) * heads};
    };
    auto blocks = [&](int rows_) { return (double)s.B * ((s.Sq + rows_ - 1) / rows_ * (double)s.Hq + (s.Skv + rows_ - 1) / rows_ * (double)s.Hkv); };
    const Visits f = both(rows, 64), m = both(128, 64);
    const double fma = 5 + std::max(f.longest * kBackward.chain[i][d], (f.all + 0.5 * blocks(rows)) / sms * kBackward.share[i][d]);
    const double split_products = std::max(13.3 + 3.3 * m.longest, 5 + (3.1 * m.all / blocks(128) + 5.5) * turns(blocks(128) / sms, 0.75));
    return split_products < fma;
}

}  // namespace sntl
