// Lanes per row of the plain SpMV (kernels: cuda/spmv.cu, cuda/krylov.cu).
//
// A twelfth of the average row, so that a lane has several entries in flight and a
// warp reads few lines at a time, and more in matrices too small to fill the chip
// that way (up to about a row's entries: there the longest row counts).  Measured
// us by lanes, 1 / 2 / 4 / 8 / 16 / 32:
//   FP64 2.05 M rows of 7:    39.6 / 62 / 79 / 133 / 317 / 747
//   FP64 250 k rows of 55:    60 / 44 / 41 / 65 / 83 / 110
//   int 250 k rows of 55:     42 / 28 / 26 / 30 / 39 / 58
//   int 125 k rows of 81:     42 / 26 / 24 / 19 / 22 / 31
//   FP64 20.8 k rows of 339:  76 / 37 / 27 / 26 / 26 / 28
//   FP64 2.5 k rows of 258:   71 / 40 / 24 / 14 / 9.9 / 8.7
//
// A row far longer than the others (a dense row among sparse ones) would take the
// product's time by itself: its lanes take 0.3 us for every four entries each, one
// round after the other, while a thread costs the whole product 11 ps (the last
// columns of the first lines above).  Its lanes are doubled while that pays.
// 200 k rows of 5 and one of 200 k, by the average alone / with the longest row:
// FP64 15,589 / 674 us, int 8,918 / 380 us, FP32 (at most 8 lanes) 11,289 / 1,062 us.
#pragma once
#include <algorithm>
#include <cstdint>

namespace sagb {

inline int longest_row(const int *rptr, int n) {
    int m = 0;
    for (int i = 0; i < n; i++) m = std::max(m, rptr[i + 1] - rptr[i]);
    return m;
}

// most: largest number of lanes
inline int spmv_lanes(int n, int64_t nnz, int longest, int most = 32) {
    if (n == 0) return 1;
    const double avg = (double)nnz / n;
    int g = 1;
    while (g < most && avg > 12 * 1.414 * g) g *= 2;
    while (g < most && (int64_t)n * g < 131072 && g < 0.75 * avg) g *= 2;
    const double round = 0.3, thread = 11e-6;  // us
    while (g < most && longest / (4.0 * g) * round > 4 + 2.0 * g * n * thread) g *= 2;
    return g;
}

}  // namespace sagb
