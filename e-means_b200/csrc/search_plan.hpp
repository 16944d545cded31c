// How a search's work is split over the grid: host arithmetic without CUDA.
//
// tc_nsplit and simt_plan choose the column splits of the two search kernels from the
// rows and centroids; search_part_rows is what a training run reserves for them, since
// its batches may not allocate.
#pragma once
#include <algorithm>
#include <cstddef>

namespace emb {

// Rows and centroids of a tile: the tensor-core search (kernels_tc.cuh) and the two
// forms of the FP32 SIMT search (kernels_simt.cuh).
constexpr int kPlanTcM = 128, kPlanTcN = 256;
constexpr int kPlanSimtLargeM = 128, kPlanSimtLargeN = 256, kPlanSimtSmallM = 64, kPlanSimtSmallN = 64;

// Column splits of the tensor-core search: the one with the fewest waves of items
// times the tiles an item takes plus two tiles' time for its rows and the drain of
// its accumulators, a larger split only when it saves 3%. 394 row tiles on 148 SMs:
// 3 splits, 8 waves of 22 tiles, against 3 waves of 64 unsplit. Half a tile for an
// item split too much: 20,011 x 100 rows against 1031 centroids 55 -> 38 us (three
// terms) and 91 -> 38 us (single term), 19,000 x 4096 single term 81 -> 57 us; 3 or
// 5 tiles measured the same as 2 or slower.
//
// Splits with the same tiles per CTA form runs of consecutive counts, and within
// a run the waves never decrease with the count, so only the first count of each
// run can be chosen: visiting those (O(sqrt(tiles)) of them) picks the same split
// as trying every count from 1 to the number of tiles.
inline int tc_nsplit(int sm_count, size_t m, size_t k) {
    const long row_tiles = (long)((m + kPlanTcM - 1) / kPlanTcM);
    const int ntiles = (int)((k + kPlanTcN - 1) / kPlanTcN);
    const long sms = std::max(1, sm_count);
    int best = 1;
    double best_cost = 0.0;
    for (int ns = 1; ns <= ntiles;) {
        const int per_cta = (ntiles + ns - 1) / ns;
        const double waves = (double)((row_tiles * ns + sms - 1) / sms);
        const double cost = waves * ((double)per_cta + 2.0);
        if (ns == 1 || cost < 0.97 * best_cost) {
            best = ns;
            best_cost = cost;
        }
        if (per_cta == 1) break;
        ns = (ntiles + per_cta - 2) / (per_cta - 1);  // first count with fewer tiles per CTA
    }
    return best;
}

// Tile and column splits of the FP32 SIMT search: 128 x 256 tiles (one CTA per SM),
// or 64 x 64 (two) while those would leave SMs without work; the split with the
// fewest waves of CTAs times the tiles each takes plus half a tile for its start and
// merge.
struct SimtPlan {
    bool small;
    int row_tiles, nsplit;
};
inline SimtPlan simt_plan(int sms, size_t m, size_t k) {
    SimtPlan p;
    sms = std::max(1, sms);
    p.small = (m + kPlanSimtLargeM - 1) / kPlanSimtLargeM * ((k + kPlanSimtLargeN - 1) / kPlanSimtLargeN) < (size_t)sms;
    const size_t bm = p.small ? kPlanSimtSmallM : kPlanSimtLargeM, bn = p.small ? kPlanSimtSmallN : kPlanSimtLargeN;
    const long slots = p.small ? 2L * sms : sms;
    p.row_tiles = (int)((m + bm - 1) / bm);
    const int ntiles = (int)((k + bn - 1) / bn);
    p.nsplit = 1;
    double best = 0.0;
    for (int ns = 1; ns <= std::min(ntiles, 64); ns++) {
        const int per = (ntiles + ns - 1) / ns;
        const double cost = (double)(((long)p.row_tiles * ns + slots - 1) / slots) * (per + 0.5);
        if (ns == 1 || cost < 0.97 * best) {
            best = cost;
            p.nsplit = ns;
        }
    }
    return p;
}

// Most partial rows (splits x rows) that a search of any batch of up to m rows writes.
// Fewer rows can take more splits, and the splits are the same for every batch of one
// count of row tiles: the largest batch of each count is looked at, by 128 rows and,
// where the small SIMT form with its 64-row tiles is taken, half way between.
inline size_t search_part_rows(int sms, size_t m, size_t k, bool tc) {
    size_t rows = 0;
    for (size_t top = kPlanTcM;; top += kPlanTcM) {
        const size_t mm = std::min(top, m);
        if (tc) {
            rows = std::max(rows, (size_t)tc_nsplit(sms, mm, k) * mm);
        } else {
            const SimtPlan p = simt_plan(sms, mm, k);
            rows = std::max(rows, (size_t)p.nsplit * mm);
            const size_t lower = top - kPlanSimtSmallM;
            if (p.small && lower < m) rows = std::max(rows, (size_t)simt_plan(sms, lower, k).nsplit * lower);
        }
        if (mm == m) return rows;
    }
}

}  // namespace emb
