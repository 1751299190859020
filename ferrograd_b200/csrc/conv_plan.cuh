// How the conversion kernel's work is split over the SMs: host arithmetic on sizes and counts alone, free of CUDA, so that it can be
// compiled and checked without a device.
#pragma once
#include <atomic>
#include <stdint.h>

constexpr uint32_t kConvTileM = 128;
struct ConvShape { uint32_t M, N, K, batch; };
struct ConvPlan {
    uint32_t bn, split;      // tile width; K-shares of a tile
    double cycles;           // estimate; 0: cannot run
};

// SMs that a kernel whose CTAs stay to its end may count on: while a gradient exchange runs beside it, `reserved` are the
// exchange's (see fg_comm_init).
inline uint64_t fg_sms_beside(int sms, bool exchange, int reserved) { return (uint64_t)(exchange && reserved > 0 && reserved < sms ? sms - reserved : sms); }

// CTAs of a launch: one for each K-share, or no more than SMs that walk the units.
inline uint64_t conv_grid(uint64_t units, uint32_t split, uint64_t sms) { return split > 1 ? units * split : units < sms ? units : sms; }

// What a launch is estimated by, in SM cycles: with tiles 128 and 64 wide, a k-block of `kblock`, storing a tile beside the next one's
// k-blocks and what a ragged N adds to that, the same for the last tile of a CTA, and what a ragged N adds to a meeting of shares,
// divided among them; set-up and first loads, and the meeting itself.
struct ConvCosts {
    uint32_t kblock;
    double kb[2], store[2], ragged[2], last[2], ragged_last[2], ragged_shares[2], around, meet;
};
// The conversion kernel, fitted to whole launches: per k-block 0.55 us with 128 x 128 tiles and 0.33 us with 128 x 64 ones (0.34 - 0.37
// with a long k), storing a tile 2.6 and 1.5 us (the last wide one 1.2, by twice the warps), 3.5 us of set-up and first loads, 2 - 3 us
// for the shares' sums to meet; where a ragged N is stored word by word 0.5 to 2 us more, and 3.6 us divided among the shares.  (With a wide
// tile's store at 2.1 us, products of a few k-blocks and several units per CTA took wide tiles: 15064 x 400 x 1 17.3 us, 15.7 with narrow ones,
// 4390 x 632 x 2 11.1 and 9.8, dA of 1920 x 96 x 1384 10.6 and 9.0.)
constexpr ConvCosts kConvCosts = {32, {1050.0, 630.0}, {5000.0, 2800.0}, {1500.0, 2000.0}, {2000.0, 2800.0}, {1000.0, 3900.0}, {6800.0, 3500.0}, 6500.0, 5500.0};

// Estimated SM cycles of one launch for one or two products (the one with the longer k first) on `sms` SMs.  clusters(bn, split):
// clusters of `split` CTAs that run at once, below one if there are none.
template <class Clusters>
ConvPlan conv_plan(const ConvShape* sh, int n, uint64_t sms, Clusters clusters, const ConvCosts& cost = kConvCosts) {
    ConvPlan best{128, 1, 0.0};
    for (uint32_t bn = 128; bn >= 64; bn -= 64) {
        uint64_t units[2] = {0, 0}, nkb[2] = {0, 0}, min_kb = ~0ull;
        for (int i = 0; i < n; ++i) {
            units[i] = (uint64_t)((sh[i].M + kConvTileM - 1) / kConvTileM) * ((sh[i].N + bn - 1) / bn) * sh[i].batch;
            nkb[i] = (sh[i].K + cost.kblock - 1) / cost.kblock;
            if (nkb[i] < min_kb) min_kb = nkb[i];
        }
        const uint64_t all = units[0] + units[1];
        const int w = bn == 128 ? 0 : 1;
        const double kb = cost.kb[w], store = cost.store[w], around = cost.around;
        const bool ragged = sh[0].N % 4 != 0 || (n > 1 && sh[1].N % 4 != 0);
        const double edge = ragged ? cost.ragged[w] : 0.0;
        // whole units: the first CTA's units are one of every sms
        const uint64_t rounds = (all + sms - 1) / sms, rounds0 = units[0] / sms + (units[0] % sms != 0);
        auto unit = [&](int i) { return (double)nkb[i] * kb > store + edge ? (double)nkb[i] * kb : store + edge; };
        double c = around + cost.last[w] + (ragged ? cost.ragged_last[w] : 0.0) + (double)rounds0 * unit(0) + (double)(rounds - rounds0) * unit(1);
        if (best.cycles == 0.0 || c < best.cycles) best = ConvPlan{bn, 1, c};
        for (uint32_t split = 2; split <= 8 && split * 2 <= min_kb && all * split <= 2 * sms; ++split) {
            const int fit = clusters(bn, split);
            if (fit < 1) continue;
            const uint64_t turns = (all + fit - 1) / fit;
            const double share = (double)((nkb[0] + split - 1) / split) * kb;
            c = (double)turns * (share + around + cost.meet + (ragged ? cost.ragged_shares[w] / split : 0.0));
            if (c < best.cycles) best = ConvPlan{bn, split, c};
        }
    }
    return best;
}

// Tile width and K-shares as given (option gemm_conv), with fewer shares where the shorter k or the clusters do not allow them.  The
// cost is the least there is: such a plan is taken.
template <class Clusters>
ConvPlan conv_plan_fixed(const ConvShape* sh, int n, uint32_t bn, uint32_t split, Clusters clusters, uint32_t kblock = kConvCosts.kblock) {
    uint32_t k = sh[0].K;
    if (n > 1 && sh[1].K < k) k = sh[1].K;
    while (split > 1 && (split * 2 > (k + kblock - 1) / kblock || clusters(bn, split) < 1)) --split;
    return ConvPlan{bn, split, 1.0};
}

// Two products walked by `pairs` workers in one launch: worker p takes tiles p, p + pairs, ... of the n0 of the first, which cost w0
// each, then a run of the n1 tiles of the second (w1 <= w0 each), longer for those with fewer of the first.  Workers below `extra`
// have one more of the first and take run[0] of the second, the others run[1]; the largest sum is `cost`, the least there is.
struct PairRuns { uint64_t pairs; uint32_t extra, run[2]; double cost; };
inline PairRuns pair_runs(uint64_t pairs, uint64_t n0, double w0, uint64_t n1, double w1) {
    const uint64_t c0 = n0 / pairs, extra = n0 % pairs;
    PairRuns best{pairs, (uint32_t)extra, {0, 0}, 0.0};
    const double more = (double)(extra ? c0 + 1 : c0) * w0, less = (double)c0 * w0;
    // the cost is a worker's own: `more` or `less` and a whole number of w1
    const uint64_t most = (n1 + pairs - 1) / pairs + (uint64_t)(w0 / w1) + 2;
    for (uint64_t i = 0; i <= most; ++i)
        for (int from = 0; from < 2; ++from) {
            const double cost = (from ? more : less) + (double)i * w1;
            if (cost < more || (best.cost > 0.0 && cost >= best.cost)) continue;
            const uint64_t s0 = (uint64_t)((cost - more) / w1 + 1e-6), s1 = (uint64_t)((cost - less) / w1 + 1e-6);
            if (extra * s0 + (pairs - extra) * s1 < n1) continue;
            best.run[0] = (uint32_t)s0; best.run[1] = (uint32_t)s1;
            best.cost = cost;
        }
    return best;
}

// Of `fit` clusters that run at once on `all` SMs, those that do on `sms` of them: the exchange's CTAs may sit anywhere.
inline int conv_clusters_beside(int fit, uint64_t sms, uint64_t all) {
    if (fit < 1 || sms >= all) return fit;
    const int n = (int)((uint64_t)fit * sms / all);
    return n < 1 ? 1 : n;
}

// A property of the device: asked until an answer has been given (query(&value) is true then, whatever the value), kept from then on.
// `known` starts at zero and holds the value plus one.  A query that fails says nothing about the device: `fallback` for this call.
template <class Query>
int fg_asked_once(std::atomic<int>& known, int fallback, Query query) {
    const int k = known.load(std::memory_order_acquire);
    if (k > 0) return k - 1;
    int n = 0;
    if (!query(&n) || n < 0) return fallback;
    known.store(n + 1, std::memory_order_release);      // the same value whoever asks
    return n;
}
