// ss_rules.hpp -- which of two kernels runs, where neither is the faster one everywhere: rules on sizes, with the times they
// were fitted to. Plain C++, so that a CPU test can hold them against those times.
#pragma once

#include <algorithm>
#include <cmath>

namespace ssg {

// Sync-free sweep (ss_trsv.cu): mean rows of a level above which k_sweep_wide is faster than k_sweep. The one polling loop of
// k_sweep grows with the lanes of a level, the lane-by-lane waits of k_sweep_wide hardly. G: lanes a row; batch: several
// systems in one matrix, whose rows read near each other.
// Measured, us a forward and a backward sweep together, k_sweep / k_sweep_wide, by rows a level:
//   FP64 batches, 8 lanes   5-point 100^2 16,000 1,213 / 1,744, 21,000 1,568 / 1,734, 30,000 2,170 / 1,753; 7-point 24^3 20,900
//                           584 / 670, 30,000 802 / 693; 27-point 14^3 16,000 612 / 965; 1,024 curl-curl systems of 8 to 32
//                           voxels 58,000: a whole pass 1,033 / 633 ms
//   FP64, one system        random order, 7-point 10,300 102 / 106, 14,600 126 / 112, 18,100 154 / 119, 22,000 189 / 139; 5-point
//                           11,400 89 / 81; curl-curl (16 lanes) 7,300 422 / 481, 11,200 594 / 554
//   complex batches, 8      5-point 100^2 9,000 2,972 / 3,310, 12,000 3,700 / 3,416, 16,000 4,664 / 3,561; 27-point 14^3 9,000
//                           1,398 / 2,342
//   complex, one system     random order, 8 lanes, 7-point 10,300 329 / 267; 4 lanes 10,300 221 / 252, 18,100 314 / 278; 16 lanes,
//                           curl-curl 2,900 701 / 655, 4,700 1,100 / 892
//   FP32 batches, 8         5-point 100^2 4,500 305 / 492, 6,500 614 / 528; 7-point 24^3 4,500 129 / 185, 6,500 210 / 200
//   FP32 complex batches    5-point 100^2 16,000 716 / 970; 7-point 24^3 20,900 271 / 271, 30,000 371 / 252
inline double sweep_wide_rows(bool fp32, bool complex_values, int G, bool batch) {
    if (complex_values && !fp32) return (batch ? 11264.0 : 8192.0) * 8.0 / G;
    if (fp32 && !complex_values) return 5632.0;
    return batch ? 22528.0 : 11264.0;
}

// Batched FP64 ICCG (ss_batch.cu): one CTA an instance that runs all of its iterations, or the launches? Estimates of an
// iteration's time in us, fitted to 325 measured batches (1 to 2,048 instances, 400 to 16,000 rows each, of curl-curl, grid,
// banded and random systems, equal and mixed sizes); over them the engine chosen is 2 % slower than the better one on average
// (complex 1 %), where the persistent one everywhere is 48 % (15 %) and the launches everywhere 20 % (38 %).
//   persistent  the largest instance's levels (a barrier each), rows and entries; more instances than about a third of the SMs
//               share SMs and memory
//   launches    the launches, the levels of the longest instance at a cost that grows with their width up to the lane-by-lane
//               sweep's, and the entries; with the tile sweeps (a handle's own batch) a level costs about a third
// Measured, us an iteration, persistent / launches: 5-point 20^2 1 instance 56 / 144, 1,024 217 / 314; 7-point 8^3 64 instances
// 59 / 138; 50^2 64 318 / 364; curl-curl 8^3 64 344 / 388, 10^3 64 787 / 599, 14^3 64 1,880 / 860; random sparse of 5,000 rows
// 16 374 / 160; complex curl-curl 10^3 256 1,157 / 1,980, 14^3 16 2,260 / 1,200.
struct BatchShape {
    double instances, rows, nnz;   // of the whole batch
    double max_rows, max_nnz;      // of its largest instance
    double levels;                 // of the instance with most
    int sms;
    bool complex_values, tiles;    // tiles: the launches run the tile sweeps
};
inline double batch_persistent_us(const BatchShape &b) {
    const bool c = b.complex_values;
    const double lev = (c ? 1.2 : 1.3) * b.levels, row = c ? 0.080 : 0.042, ent = c ? 0.0062 : 0.0030;
    const double alone = lev + row * b.max_rows + ent * b.max_nnz;
    const double mean = lev + (row * b.rows + ent * b.nnz) / b.instances;
    const double share = b.instances / ((c ? 0.92 : 0.30) * b.sms);
    return share <= 1.0 ? alone : std::max(alone, mean * std::pow(share, c ? 0.68 : 0.34));
}
inline double batch_launches_us(const BatchShape &b) {
    const bool c = b.complex_values;
    // a quarter off: the persistent estimate is up to half too low where levels hold one row
    if (b.tiles) return 0.75 * (c ? 90.0 + 1.5 * b.levels : 75.0 + 0.75 * b.levels);
    const double width = b.rows / std::max(b.levels, 1.0);
    const double level = std::min(c ? 3.6 + 1.0e-3 * width : 2.3 + 2.26e-4 * width, c ? 23.5 : 29.0);
    return (c ? 114.0 : 90.0) + b.levels * level + (c ? 3.65e-5 : 7.2e-6) * b.nnz;
}
inline bool batch_persists(const BatchShape &b) { return batch_persistent_us(b) < batch_launches_us(b); }

}  // namespace ssg
