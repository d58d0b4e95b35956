/*
 * ntlp_stage64.h -- which stage capacity the FP64 deposition takes for a box,
 * and the order of a batch's tiles by it.  Host code without CUDA.
 */
#ifndef NTLP_STAGE64_H
#define NTLP_STAGE64_H

#include <cmath>
#include <vector>

namespace ntlp {

/* droplets that a tile stages (56 bytes each): three CTAs per SM with the
 * first two, one with the third; a tile above its capacity merges from
 * global memory */
constexpr int kDepCap64[3] = {640, 1280, 3840};

/* Index of the capacity for a box of n droplets (the number, not the room for
 * them) in ncells cells whose tiles take the droplets of tile_cells cells.
 * The lines are in droplets per tile, since the tile shapes differ (425 to 585
 * cells).  Deposition with 640 / 1280 / 3840 by that mean, boxes of 64^3 and 128^3:
 *   446   0.0976 / 0.1116 / 0.2015 ms   0.540 / 0.646 / 1.333 ms
 *   594   0.1635 / 0.1362 / 0.2480      0.750 / 0.795 / 1.658
 *   1089  (1040) 0.358 / 0.201 / 0.349  2.540 / 1.241 / 2.435
 *   1287  (1228) 0.373 / 0.285 / 0.396  2.601 / 2.298 / 2.645
 *   1404  0.4154 / 0.4346 / 0.4329
 *   1732  0.558 / 0.566 / 0.504         3.947 / 3.964 / 3.396
 *   3168  (3267) 1.015 / 1.024 / 0.842  7.412 / 7.228 / 5.558
 *   3960  1.224 / 1.231 / 1.356
 * So: 640 while four standard deviations of a random spread fit; 1280 although
 * the fuller half of the tiles may exceed it, up to 1300; 3840 again while four
 * standard deviations fit; above, where every tile merges from global memory,
 * the smallest, whose CTAs come and go fastest. */
inline int deposit64_cap(long long n, long long ncells, int tile_cells) {
    const double mean = (double)n / (double)ncells * tile_cells;
    const double most = mean + 4.0 * std::sqrt(mean);
    if (most <= kDepCap64[0]) return 0;
    if (mean <= 1300.0) return 1;
    return most <= kDepCap64[2] ? 2 : 0;
}

/* consecutive tiles of the tile table with one stage capacity: one launch */
struct TileRun {
    int first, count, cap;
    bool operator==(const TileRun &o) const { return first == o.first && count == o.count && cap == o.cap; }
};

/* The boxes of a batch in the order of the tile table, and its runs: the boxes
 * of the 3840 stage apart from the others (its one CTA per SM costs a sparse box
 * 2.4 times the 640 stage), which share the larger of theirs (1.15 times).  Two
 * launches at most: one per change of capacity took 1.65 ms, not 0.76, for 48
 * boxes of 32^3 that take turns between 0.28 and 1.67 droplets per cell. */
inline void deposit64_order(const std::vector<int> &cap, const std::vector<int> &tiles, std::vector<int> &order,
                            std::vector<TileRun> &runs) {
    order.clear();
    runs.clear();
    int first = 0;
    for (int big = 0; big < 2; ++big) {
        TileRun r{first, 0, big ? 2 : 0};
        for (size_t b = 0; b < cap.size(); ++b) {
            if ((cap[b] == 2) != (big == 1)) continue;
            order.push_back((int)b);
            r.count += tiles[b];
            if (cap[b] > r.cap) r.cap = cap[b];
        }
        if (r.count > 0) runs.push_back(r);
        first += r.count;
    }
}

}  // namespace ntlp

#endif
