// ss_rules.hpp -- which of two kernels runs, where neither is the faster one everywhere: rules on sizes, with the times they
// were fitted to. Plain C++, so that a CPU test can hold them against those times.
#pragma once

namespace ssg {

// Sync-free sweep (ss_trsv.cu): mean rows of a level above which k_sweep_wide is faster than k_sweep. The one polling loop of
// k_sweep grows with the lanes of a level, the lane-by-lane waits of k_sweep_wide hardly. G: lanes a row; batch: several
// systems in one matrix, whose rows read near each other.
// Measured, us a forward and a backward sweep together, k_sweep / k_sweep_wide, by rows a level:
//   FP64 batches, 8 lanes   5-point 100^2 16,000 1,213 / 1,744, 21,000 1,568 / 1,734, 30,000 2,170 / 1,753; 7-point 24^3 20,900
//                           584 / 670, 30,000 802 / 693; 27-point 14^3 16,000 612 / 965; 1,024 curl-curl systems of 8 to 32
//                           voxels 58,000: a whole pass 1,033 / 683 ms
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

}  // namespace ssg
