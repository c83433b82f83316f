// linear_plan.hpp — which tiles a projection of many tokens is cut into (linear_tc.cu: linear_pair_kernel), and in
// which order they are listed.  Plain C++ so that the list can be walked without a GPU.
#pragma once

#ifdef __CUDACC__
#define HC_PLAN_FN __host__ __device__ __forceinline__
#define HC_PLAN_UNROLL _Pragma("unroll")
#else
#define HC_PLAN_FN inline
#define HC_PLAN_UNROLL
#endif

namespace hc {

constexpr int kLinJobs = 4;

// Tiles of two widths.  A job's columns are cut in wide tiles, and if half of one or less is left, that is a half tile (more
// is a wide tile with zeros: as two halves 4096 tokens to 904 columns were a round more, 31 us instead of 23).
// The list has n_wide of the wide tiles, then the halves of the others and the odd halves, so that a launch's last
// round of pairs can be one of half tiles.
struct LinWide {
    int job, col, tm, width;
};
template <int BN>
HC_PLAN_FN int wide_tiles(int columns) {
    return (columns + BN / 2 - 1) / BN;
}
template <int BN>
HC_PLAN_FN int odd_tiles(int columns) {
    return columns > wide_tiles<BN>(columns) * BN ? 1 : 0;
}
// Args: n_jobs, job[].out_features, tiles_m, n_wide.
template <int BN, typename Args>
HC_PLAN_FN LinWide decode_wide(const Args& args, int tile) {
    LinWide t{0, 0, 0, BN};
    int all = 0;                                             // wide tiles of all jobs
    HC_PLAN_UNROLL
    for (int j = 0; j < kLinJobs; ++j) {
        if (j < args.n_jobs) all += wide_tiles<BN>(args.job[j].out_features) * args.tiles_m;
    }
    int wide = tile, half = 0;
    if (tile >= args.n_wide) {
        t.width = BN / 2;
        wide = args.n_wide + ((tile - args.n_wide) >> 1);
        half = (tile - args.n_wide) & 1;
    }
    const bool odd = wide >= all;
    int left = odd ? tile - args.n_wide - 2 * (all - args.n_wide) : wide;
    HC_PLAN_UNROLL
    for (int j = 0; j < kLinJobs; ++j) {
        const int columns = j < args.n_jobs ? args.job[j].out_features : 0;
        const int tiles = (odd ? odd_tiles<BN>(columns) : wide_tiles<BN>(columns)) * args.tiles_m;
        if (left >= 0 && left < tiles) {
            t.job = j;
            t.col = left / args.tiles_m;
            t.tm = left - t.col * args.tiles_m;
            t.col = odd ? wide_tiles<BN>(columns) * BN : t.col * BN + half * (BN / 2);
        }
        left -= tiles;
    }
    return t;
}

// The column tile whose rounds of pairs take least, and for 256 columns the list above.
struct LinPlan {
    int width;
    long long n_wide, n_tiles;
    double steps;                                            // clocks of a K step, all rounds together
};
inline LinPlan plan_pairs(const int* out_features, int n_jobs, int tiles_m, int pairs) {
    // A K step costs an SM the larger of its MMAs (2 clocks a column) and of (128 + BN / 2) x 128 bytes out of L2, of which
    // about 60 arrive per clock and SM with all of them loading: 546 clocks for 256 columns, 478, 443, 410.  Measured on 4096,
    // 1024, 600 and 300 tokens of the three geometries: the choice is the fastest of the four or within a few percent of it.
    const int widths[4] = {256, 192, 160, 128};
    const double step[4] = {546.0, 478.0, 443.0, 410.0};
    LinPlan plan{};
    for (int i = 0; i < 4; ++i) {
        long long tiles = 0;
        for (int j = 0; j < n_jobs; ++j) tiles += (long long)tiles_m * ((out_features[j] + widths[i] - 1) / widths[i]);
        const double t = double((tiles + pairs - 1) / pairs) * step[i];
        if (i == 0 || t < plan.steps) plan = LinPlan{widths[i], 0, tiles, t};
    }
    // Or wide tiles in whole rounds and half tiles for the rest, in the last round or two: 4096 tokens to 2880 columns are two
    // rounds of 256 and one of 128 instead of three of 256 (81.2 us, now 77.8; 2048 tokens to q, k and v of 4096 and 512 columns
    // 48.7, now 46.0).  Where another choice is predicted as fast it is faster: its K steps are of one size, its ring deeper
    // (600 tokens of 2816 to 8192 columns 28.7 against 31.6).
    long long wide = 0, odd = 0;
    for (int j = 0; j < n_jobs; ++j) {
        wide += (long long)tiles_m * wide_tiles<256>(out_features[j]);
        odd += (long long)tiles_m * odd_tiles<256>(out_features[j]);
    }
    if (plan.width == 256) plan.n_wide = wide;               // (as many tiles as predicted: wide ones and the odd halves)
    for (long long rounds = 1; rounds * pairs <= wide; ++rounds) {
        const long long n = rounds * pairs, tiles = n + 2 * (wide - n) + odd, total = (tiles + pairs - 1) / pairs;
        const double t = double(rounds) * step[0] + double(total - rounds) * step[3];
        if (t < plan.steps) plan = LinPlan{256, n, tiles, t};
    }
    return plan;
}

}  // namespace hc
