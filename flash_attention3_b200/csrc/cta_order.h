// Host-side choice of the CTA launch order for the causal backward.
//
// A CTA that owns key tile kt walks the query tiles that see it (n_tiles - kt of
// them per query head when seqlen_q == seqlen_k), so work per CTA falls with kt.
// The B200 block scheduler hands the
// next block index to whichever SM frees up first, which is greedy list
// scheduling; the plan below simulates exactly that for a few candidate orders
// and keeps the one with the smallest modelled makespan.  This plays the role
// of the reference's choose_causal_cta_order / modeled_causal_max_work
// (reference src/fused_bwd_kernel.cpp:1285-1358), whose model is a fixed
// round-robin over 48 compute units; the permutation itself
// (remap_k_tile) keeps the reference's serpentine form as one candidate.
#pragma once

#include <algorithm>
#include <array>
#include <functional>
#include <queue>
#include <vector>

#include "geometry.h"

namespace fa3b200 {

// Tile grid of one head: which query tiles each key tile visits.
struct TileWork {
    int n_k_tiles = 0;
    Band band{};
    bool causal = false;  // the band is bounded: work differs between key tiles
    int steps(int kt) const { return q_tiles_of_k_tile(kt, band); }
    static TileWork of(const Band& band) {
        TileWork w;
        w.n_k_tiles = tiles_of(band.seqlen_k);
        w.band = band;
        w.causal = !band_is_full(band);
        return w;
    }
    static TileWork square(int n_tiles, bool causal) {
        return of(make_band(n_tiles * kTileRows, n_tiles * kTileRows, causal, -1, -1));
    }
};

enum CtaOrderMode : int {
    kOrderHeavyFirst = 0,  // key tile index ascending: longest work first (LPT)
    kOrderLightFirst = 1,
    kOrderSerpentine = 2,
};

// dQ-accumulator bytes that the CTAs running at the same time may spread over (about half of L2;
// 16 and 32 MB measured slower on the S=8192 shapes)
constexpr long long kDqL2BudgetBytes = 64LL << 20;

struct CtaOrderPlan {
    int mode = kOrderHeavyFirst;
    int width = 1;
    // Heads are taken in groups of `head_group`; inside a group the order is tile slot major, head
    // minor: block = (group * n_tiles + tile slot) * head_group + head in group.  head_group = all
    // heads is the globally heaviest-first order; a small group keeps the CTAs that run together on
    // a few heads, so their Q/dO tiles and the dQ-accumulator lines they add into stay in L2.
    int head_group = 1;
    long long makespan = 0;  // modelled, in query-tile steps
};

inline int host_remap_k_tile(int physical, int count, int mode, int width) {
    if (mode == kOrderHeavyFirst) return physical;
    if (mode == kOrderLightFirst) return count - 1 - physical;
    const int round = physical / width;
    const int base = round * width;
    const int slot = physical - base;
    const int span = std::min(width, count - base);
    return base + ((round & 1) == 0 ? slot : span - 1 - slot);
}

// Greedy list scheduling of blocks 0..n-1 (block = physical tile * bh + head)
// on `sms` machines; cost of a block = steps of its logical key tile + a fixed
// prologue/epilogue charge.
inline long long modelled_makespan(const TileWork& work, int bh_count, int group, int sms,
                                   int mode, int width, int head_group = 0) {
    const int n_tiles = work.n_k_tiles;
    if (head_group <= 0 || head_group > bh_count) head_group = bh_count;
    std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free_at;
    for (int i = 0; i < sms; ++i) free_at.push(0);
    long long makespan = 0;
    const long long blocks = (long long)n_tiles * bh_count;
    const long long per_group = (long long)n_tiles * head_group;
    for (long long idx = 0; idx < blocks; ++idx) {
        const long long hg = idx / per_group;
        const int heads_here = int(std::min<long long>(head_group, bh_count - hg * head_group));
        const int physical = int((idx - hg * per_group) / heads_here);
        const int kt = host_remap_k_tile(physical, n_tiles, mode, width);
        const long long cost = 1 + (long long)group * work.steps(kt);
        const long long start = free_at.top();
        free_at.pop();
        free_at.push(start + cost);
        makespan = std::max(makespan, start + cost);
    }
    return makespan;
}

inline long long modelled_makespan(int n_tiles, int bh_count, int group, bool causal, int sms,
                                   int mode, int width, int head_group = 0) {
    return modelled_makespan(TileWork::square(n_tiles, causal), bh_count, group, sms, mode, width,
                             head_group);
}

// dq_bytes_per_head: bytes of fp32 dQ accumulator that the CTAs of one (batch, KV head) add into.
inline CtaOrderPlan plan_cta_order(const TileWork& work, int bh_count, int group, int sms,
                                   long long dq_bytes_per_head = 0) {
    const int n_tiles = work.n_k_tiles;
    const bool causal = work.causal;
    CtaOrderPlan best;
    best.head_group = bh_count;
    best.makespan = modelled_makespan(work, bh_count, group, sms, kOrderHeavyFirst, 1);
    const long long heavy_first = best.makespan;
    const int max_width = std::min(n_tiles, 16);
    for (int width = 2; causal && width <= max_width; ++width) {
        const long long m =
            modelled_makespan(work, bh_count, group, sms, kOrderSerpentine, width);
        if (m < best.makespan) {
            best.mode = kOrderSerpentine;
            best.width = width;
            best.makespan = m;
        }
    }
    // Cache-friendly grouping: the smallest head group (so the dQ-accumulator lines and Q/dO tiles of
    // the CTAs that run together stay in L2) whose modelled makespan is within 2 % of plain
    // heaviest-first, and whose accumulator share stays within the L2 budget.  Measured on B200:
    // +7..+14 % throughput on the S=4096..8192 shapes against the global heaviest-first order.
    if (dq_bytes_per_head > 0) {
        long long g_max = kDqL2BudgetBytes / dq_bytes_per_head;
        if (g_max < 1) g_max = 1;
        if (g_max > bh_count - 1) g_max = bh_count - 1;
        for (long long g = 1; g <= g_max; ++g) {
            const long long m = modelled_makespan(work, bh_count, group, sms, kOrderHeavyFirst, 1, int(g));
            if (m * 100 <= heavy_first * 102) {
                best.mode = kOrderHeavyFirst;
                best.width = 1;
                best.head_group = int(g);
                best.makespan = m;
                break;
            }
        }
    }
    return best;
}

inline CtaOrderPlan plan_cta_order(int n_tiles, int bh_count, int group, bool causal, int sms,
                                   long long dq_bytes_per_head = 0) {
    return plan_cta_order(TileWork::square(n_tiles, causal), bh_count, group, sms, dq_bytes_per_head);
}

// How the forward hands out its query tiles.  splits: how many CTAs (a cluster of 1, 2, 4 or 8) share the key tiles
// of a pair of neighbouring query tiles.  fold: a CTA takes the last and the first query tile, the last but one and
// the second, and so on, where a causal mask gives the later ones more keys.
// Pairs are launched heaviest first when the mask makes them unequal; a cluster needs its SMs at the same
// time, so the model hands the pairs to as many gangs of SMs as the device holds clusters of that size (gangs[0 .. 3];
// fewer than sms / splits, because a cluster does not cross a GPC) as these free up.  A CTA costs its key tiles plus
// what corresponds to 3 of them (set-up, first loads, pipeline fill, output), and a split one 2 to 3 more (partial
// outputs exchanged through distributed shared memory).  A key tile that only one of the two query tiles sees costs
// 5/6, so folded pairs do more work in sum but are nearly equal: they pay for up to about one wave of CTAs.  (Of
// 1.93 us per key tile at D=128, 1.47 at D=64, the model is within 5 % for 4 to 96 heads of 384 to 3072 rows.)  A plan
// further down the list has to be 2 % better than those in front of it.
// us per call, one CTA per pair of neighbours against the planned number: S=2048, 4 heads, D=128 causal 33.1 and 18.0;
// S=1024, 1 head 19.2 and 13.2; 300 queries x 8000 keys, 2 heads 156 and 24.  Neighbours against folded pairs, causal:
// 16 heads x 2048, D=128 37.1 and 32.3, D=64 29.8 and 24.7; 32 x 1024, D=128 21.9 and 19.1; 48 x 512 14.4 and 13.2.
struct FwdPlan {
    int splits = 1;
    bool fold = false;
};

using FwdGangs = std::array<int, 4>;  // clusters of 1, 2, 4, 8 CTAs that run at the same time; 0: the device runs none

// (packed sequences have different numbers of tiles: not folded)
inline FwdPlan plan_fwd(const Band& band, long long bh_count, const FwdGangs& gangs, bool packed) {
    const int q_tiles = tiles_of(band.seqlen_q), pairs = (q_tiles + 1) / 2;
    FwdPlan best;
    if (pairs * bh_count > 8LL * gangs[0]) return best;  // many waves: nothing stands idle for long
    const FwdPlan options[] = {{1, false}, {1, true}, {2, false}, {4, false}, {8, false}};
    long long best_cost = -1;
    for (const FwdPlan& option : options) {
        if (option.fold && (packed || band.left < kUnbounded || band.right >= kUnbounded)) continue;  // (every tile starts at the first key)
        std::priority_queue<long long, std::vector<long long>, std::greater<long long>> free_at;
        const int gang = option.splits == 8 ? 3 : option.splits / 2;
        if (option.splits > 1 && gangs[size_t(gang)] <= 0) continue;
        for (int i = 0; i < std::max(1, gangs[size_t(gang)]); ++i) free_at.push(0);
        long long makespan = 0;
        for (int slot = 0; slot < pairs; ++slot) {
            const TilePair tiles_here = tile_pair_of_slot(slot, q_tiles, true, option.fold);
            const int a = tiles_here.a, b = tiles_here.b;
            const int most_a = k_tiles_of_q_tile(a, band), most_b = b < q_tiles ? k_tiles_of_q_tile(b, band) : 0;
            int first = kUnbounded, last = -1;
            if (most_a > 0) first = first_k_tile(a, band), last = last_k_tile(a, band);
            if (most_b > 0) first = std::min(first, first_k_tile(b, band)), last = std::max(last, last_k_tile(b, band));
            const int tiles = last >= first ? last - first + 1 : 0, both = std::max(0, most_a + most_b - tiles);
            // in sixths of a key tile
            const long long cost = option.splits == 1 ? 6 * (3 + both) + 5 * (tiles - both)
                                                      : 6 * (3 + (tiles + option.splits - 1) / option.splits) + (option.splits == 2 ? 13 : option.splits == 4 ? 15 : 18);
            for (long long i = 0; i < bh_count; ++i) {
                const long long end = free_at.top() + cost;
                free_at.pop();
                free_at.push(end);
                makespan = std::max(makespan, end);
            }
        }
        if (best_cost < 0 || makespan * 102 < best_cost * 100) {
            best_cost = makespan;
            best = option;
        }
    }
    return best;
}

// A CTA that takes over tiles has warps that wait for the next one from the start of a tile to its end (who works it out; a softmax
// warpgroup whose query tile has fewer keys), and a wait gives up after 2e9 cycles.  A step takes 4000; longer tiles than this stay
// with one per CTA, where no wait spans more than a step, and where the set-up saved is nothing beside them.
constexpr long long kMostStepsTakenOver = 1 << 16;

// Whether the CTAs of the dK/dV and five-GEMM kernels take over key tiles of CTAs that have not started: where there are more tiles than
// SMs.  us per call, one CTA per tile and this:
// full, 80 heads x 512, D=128 60.3 and 55.2; 32 x 512 x B=8, D=64 101 and 91; 16 x 1024 x B=8, D=64 144 and 139; causal, 40 x 512, D=128
// 27.8 and 25.8; 16 x 1000 x B=4 91.5 and 85; 32 x 300 x B=8 84.3 and 78; D=64, 16 x 2048 x B=2 81.4 and 76; 8 x 4096 65.2 and 65.1; 176 tiles (1111
// queries x 1300 keys) 46.4 and 46.6; reproducible gradients (dK/dV kernel), causal, 32 x 300 x B=8, D=128 108 and 93.6; 16 x 2048 x B=2 156 and
// 154.  (Long shapes run under the power limit: the same within its spread.)  Packed, where blocks without rows are passed over by
// the warp that works tiles out instead of starting: 9 x 4096, 16 heads, D=128 832 and 794; 16 heads, 2048 and 20 x 128, D=64 causal 116 and
// 73; 1 head, 4096 and 40 x 30 (72 tiles in 1312 blocks), causal, D=64 55.9 and 54.8, reproducible 61.9 and 51.2, D=128 reproducible 74.8
// and 64.5, but 77.3 and 84.1 when such calls follow one another (alone they take the same).
inline bool bwd_takes_over(const Band& band, long long blocks, int group, int sms) {
    return blocks > sms && (long long)group * tiles_of(band.seqlen_q) <= kMostStepsTakenOver;
}

// Whether the CTAs of the forward take over pairs of query tiles of CTAs that have not started: from two pairs with rows per SM
// on.  us per call, one CTA per pair and this: causal, 32 x 300 x B=8, D=128 38.6 and 32.0; 32 on 8 heads x 1024 x B=8, D=128 108.4 and 98,
// D=64 88.4 and 87; full, 32 x 512 x B=8, D=64 41.6 and 35.2.  With fewer the longer code costs more than it gives: 256 pairs (16 x 2048 x
// B=2, causal) D=128 42.3 and 41.2, D=64 35.6 and 38.3; 240 (80 x 700, D=64) 22.8 and 24.5; 160 (40 x 1000, D=128) 22.4 and 23.8.  (Long shapes
// run under the power limit: the same within its spread.)
// Packed (total_rows > 0): the grid is sized for the longest sequence, and most blocks may have no rows; a sequence fills half of its
// last pair on average.  D=64, causal and full: 8 heads, one sequence of 1000 and 20 of 40 (192 pairs in 672 blocks) 16.6 and 18.1, 19.9 and
// 23.0; 4 heads, 4096 and 15 of 100 (124 in 1024) 49.2 and 53.2, 54.3 and 58.5; 16 heads, 2048 and 20 of 128 (448 in 2688) 42.2 and 41.2, 51.0
// and 58.0; 16 heads, 1024 and 50 of 30 (864 in 3264) 47.9 and 45.2, 48.7 and 47.8; 32 heads, 2048 and 20 of 128 (896 in 5376) 80.4 and 72.4,
// 92.7 and 89.2.  Full attention, where the pairs of a sequence are equally long, needs more of them.
inline bool fwd_takes_over(const Band& band, long long pairs, long long heads, int batch, long long total_rows, int sms) {
    if (tiles_of(band.seqlen_k) > kMostStepsTakenOver) return false;
    if (total_rows <= 0) return pairs >= 2LL * sms;
    const long long with_rows = std::min(pairs, heads * (total_rows + kTileRows * (long long)batch) / (2 * kTileRows));
    return 2 * with_rows >= (band_is_full(band) ? 7LL : 4LL) * sms;
}

}  // namespace fa3b200
