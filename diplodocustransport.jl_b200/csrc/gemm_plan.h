// Plans of the batched gain GEMM: the tile shapes and K splits that the autotuner may choose from.
// Host arithmetic only.
#pragma once

#include <algorithm>
#include <vector>

namespace dtb {

// One way to run a group's gain GEMM: the kernel (one SM per tile, or an SM pair sharing a
// 256 x 256 MMA), the column tile width and the requested number of K splits.
struct GemmPlan {
    int pair = 0;
    int bn = 256;
    int splits = 1;
    double us = 0;  // measured time of one GEMM with this plan (0: not measured)
};

// What a plan is chosen for: the group's 128-row tiles, its K tiles (N1 input-1 states in each of
// n_cb 64-wide input-2 blocks) and the columns; the SMs and the SM pairs that run at once.
struct GemmShape {
    int m_tiles, n_cb, N1, cols;
    int sms, max_pairs;
};

// The K splits a plan runs with.
struct GemmSplits {
    int n_splits, tiles_per_split;
    int per_cb;  // > 0: every split lies inside one input-2 block
};

// The splits are aligned to the 64-wide input-2 blocks when that keeps nearly every requested
// split: a split then never reloads its f2 block in mid-stream.
inline GemmSplits gemm_splits(const GemmShape& g, const GemmPlan& p) {
    const int T = g.n_cb * g.N1;
    const int S = std::max(1, std::min(p.splits, T));
    GemmSplits s;
    s.tiles_per_split = (T + S - 1) / S;
    s.n_splits = (T + s.tiles_per_split - 1) / s.tiles_per_split;
    s.per_cb = 0;
    const int k_cb = S / g.n_cb;
    if (k_cb >= 1 && k_cb <= g.N1 && (double)(k_cb * g.n_cb) >= 0.95 * S) {
        s.per_cb = k_cb;
        s.n_splits = k_cb * g.n_cb;
    }
    return s;
}

// A GEMM kernel spreads a split's hi*hi products over 512 / bn - 1 tensor-memory accumulators (one
// on SM pairs), round robin by K tile. Each is FP32 and its error grows with the number of MMAs it
// sums (measured: about 2e-5 relative after 3,328 K values in one accumulator; three species of 576
// states reached 3e-4 in their state after 5,000 steps with 20,736 K values per accumulator), so the
// bound keeps the gain term's error at a few 1e-6: 16 K tiles per accumulator on one SM, 32 on SM
// pairs (where a second fill would double the tensor-bound step's partial traffic).
constexpr int kMaxTilesPerAccSm = 16;
constexpr int kMaxTilesPerAccPair = 32;
constexpr int kMaxWaves = 4;
inline int gemm_accumulators(const GemmPlan& p) { return p.pair ? 1 : 512 / p.bn - 1; }
inline int gemm_acc_bound(const GemmPlan& p) { return p.pair ? kMaxTilesPerAccPair : kMaxTilesPerAccSm; }
// K tiles in the fullest hi*hi accumulator of a plan
inline int gemm_tiles_per_acc(const GemmShape& g, const GemmPlan& p) {
    const GemmSplits s = gemm_splits(g, p);
    const int longest = s.per_cb > 0 ? (g.N1 + s.per_cb - 1) / s.per_cb : s.tiles_per_split;
    const int n = gemm_accumulators(p);
    return (longest + n - 1) / n;
}

// K splits that fill the device once, or a whole number of times (at most kMaxWaves) when one fill
// would leave a hi*hi accumulator more K tiles than its bound.
inline int gemm_fill_splits(const GemmShape& g, int pair, int bn) {
    const int n_tiles = (g.cols + bn - 1) / bn;
    const double units = pair ? (double)(g.m_tiles / 2 * n_tiles) : (double)(g.m_tiles * n_tiles);
    const double cap = pair ? g.max_pairs : g.sms;  // CTAs (pairs) the device runs at once
    // rounded down: one CTA more than the device holds would run in a second wave on its own
    const int fill = std::max(1, (int)(cap / units));
    const int per_split = pair ? kMaxTilesPerAccPair : kMaxTilesPerAccSm * (512 / bn - 1);
    const int T = g.n_cb * g.N1;
    const int need = (T + per_split - 1) / per_split;
    const int waves = std::min(kMaxWaves, std::max(1, (need + fill - 1) / fill));
    if (waves == 1) return fill;
    // several waves: as many splits as whole waves hold (the last wave then runs nearly full)
    return std::max(fill * waves, (int)(waves * cap / units));
}

// Whether a plan can run and sums no more K tiles into an accumulator than its bound or than the
// plan that fills the device (which exceeds the bound only where kMaxWaves caps its waves).
inline bool gemm_plan_valid(const GemmShape& g, const GemmPlan& p) {
    if (p.bn != 64 && p.bn != 128 && p.bn != 256) return false;
    if (p.splits < 1) return false;
    if (p.pair && (p.bn != 256 || g.m_tiles % 2 != 0 || g.max_pairs <= 0)) return false;
    GemmPlan fill = p;
    fill.splits = gemm_fill_splits(g, p.pair, p.bn);
    return gemm_tiles_per_acc(g, p) <= std::max(gemm_acc_bound(p), gemm_tiles_per_acc(g, fill));
}

// Without timing: the widest tile the columns fill, on SM pairs when the rows pair up.
inline GemmPlan gemm_heuristic_plan(const GemmShape& g) {
    GemmPlan p;
    p.bn = g.cols >= 192 ? 256 : (g.cols > 64 ? 128 : 64);
    p.pair = (p.bn == 256 && g.m_tiles % 2 == 0 && g.max_pairs > 0) ? 1 : 0;
    p.splits = gemm_fill_splits(g, p.pair, p.bn);
    return p;
}

// The plans worth timing: per tile width and kernel the splits that fill the device; where those
// are short (at most kShortSplit K tiles), also two thirds and half of them, within the
// accumulators' bound. Fewer splits mean fewer partials to gather.
constexpr int kShortSplit = 16;
inline std::vector<GemmPlan> gemm_plan_candidates(const GemmShape& g) {
    std::vector<GemmPlan> cands;
    const int T = g.n_cb * g.N1;
    for (int bn : {64, 128, 256}) {
        if (bn > 64 && bn / 2 >= g.cols) continue;  // half the tile or more would be padding
        for (int pair : {0, 1}) {
            GemmPlan p;
            p.bn = bn;
            p.pair = pair;
            if (pair && (bn != 256 || g.m_tiles % 2 != 0 || g.max_pairs <= 0)) continue;
            const int fill = p.splits = gemm_fill_splits(g, pair, bn);
            cands.push_back(p);
            if (T > kShortSplit * fill) continue;
            for (int part : {2, 1}) {
                p.splits = fill * part / (part + 1);
                if (gemm_plan_valid(g, p)) cands.push_back(p);
            }
        }
    }
    return cands;
}

}  // namespace dtb
