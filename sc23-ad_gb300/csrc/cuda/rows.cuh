// A lane's part of one CSR row's sum, for kernels that give a row G lanes.
//
// Bound by memory latency and, with one lane a row, by the L1 cache (each load
// of a warp touches as many lines as rows): four entries a lane are in flight,
// the last one to three in one predicated round, and the kernels stay at 32
// registers (FP32 with eight sums a lane: 40), so that an SM holds all its threads.
// Poisson 127^3 (FP64, 2.05 M
// rows of 7 entries), one lane a row: 39.6 us = 5.4 TB/s; one entry at a time
// and four lanes a row, 131 us.  Copying the entries of 256 rows into shared
// memory first was slower: 42 us, with the next 256 rows' copy behind the sums
// 48 us.  A lane adds its entries in their order.
#pragma once
#include <type_traits>

#include "../sagb_internal.hpp"
#include "common.cuh"

namespace sagb {

template <bool EXACT>
__device__ __forceinline__ long long row_add(long long a, int v, int x) {
    return wadd(a, (long long)v * (long long)x);
}
template <bool EXACT>  // multiply and add rounded one by one
__device__ __forceinline__ double row_add(double a, double v, double x) {
    return EXACT ? __dadd_rn(a, __dmul_rn(v, x)) : a + v * x;
}
template <bool EXACT>
__device__ __forceinline__ float row_add(float a, float v, float x) {
    return EXACT ? __fadd_rn(a, __fmul_rn(v, x)) : a + v * x;
}

// entries a + lane, a + lane + G, ... below b, in S sums in turn; SINGLY: the last one to
// three one by one
template <int G, bool EXACT = false, int S = 1, bool SINGLY = false, typename V>
__device__ __forceinline__ auto row_part(int a, int b, int lane, const int *__restrict__ cind, const V *__restrict__ val,
                                         const V *__restrict__ x) {
    static_assert(S == 1 || S == 2, "one sum or two");
    std::conditional_t<std::is_same<V, int>::value, long long, V> acc[S] = {};
    int j = a + lane;
    for (; j + 3 * G < b; j += 4 * G) {
        int c[4];
        V v[4], xv[4];
#pragma unroll
        for (int q = 0; q < 4; q++) {
            c[q] = __ldg(cind + j + q * G);
            v[q] = __ldg(val + j + q * G);
        }
#pragma unroll
        for (int q = 0; q < 4; q++) xv[q] = __ldg(x + c[q]);
#pragma unroll
        for (int q = 0; q < 4; q++) acc[q % S] = row_add<EXACT>(acc[q % S], v[q], xv[q]);
    }
    if constexpr (SINGLY) {
        static_assert(S == 1, "one sum");
        for (; j < b; j += G) acc[0] = row_add<EXACT>(acc[0], __ldg(val + j), __ldg(x + __ldg(cind + j)));
    } else if (j + G < b) {
        const bool third = j + 2 * G < b;
        int c[3];
        V v[3], xv[3];
#pragma unroll
        for (int q = 0; q < 3; q++) {
            c[q] = q < 2 || third ? __ldg(cind + j + q * G) : 0;
            v[q] = q < 2 || third ? __ldg(val + j + q * G) : V(0);
        }
#pragma unroll
        for (int q = 0; q < 3; q++) xv[q] = q < 2 || third ? __ldg(x + c[q]) : V(0);
#pragma unroll
        for (int q = 0; q < 2; q++) acc[q % S] = row_add<EXACT>(acc[q % S], v[q], xv[q]);
        if (third) acc[0] = row_add<EXACT>(acc[0], v[2], xv[2]);
    } else if (j < b) {
        acc[0] = row_add<EXACT>(acc[0], __ldg(val + j), __ldg(x + __ldg(cind + j)));
    }
    if constexpr (S == 2) return acc[0] + acc[1];
    else return acc[0];
}

// The sum that G * V lanes a row give, taken by G: lane g keeps the V partial sums
// of lanes g, g + G, ..., adds them as their butterfly would, and leaves the rest of
// the butterfly to the G lanes.  FP32 rows keep their order this way.
template <int G, int V, typename T>
__device__ __forceinline__ T row_part_of(int a, int b, int lane, const int *__restrict__ cind, const T *__restrict__ val,
                                         const T *__restrict__ x) {
    T acc[V];
#pragma unroll
    for (int v = 0; v < V; v++) acc[v] = 0;
    for (int base = a + lane; base < b; base += G * V) {
        int c[V];
        T p[V], q[V];
#pragma unroll
        for (int v = 0; v < V; v++) {
            c[v] = base + v * G < b ? __ldg(cind + base + v * G) : -1;
            p[v] = base + v * G < b ? __ldg(val + base + v * G) : T(0);
        }
#pragma unroll
        for (int v = 0; v < V; v++) q[v] = c[v] >= 0 ? __ldg(x + c[v]) : T(0);
#pragma unroll
        for (int v = 0; v < V; v++)
            if (c[v] >= 0) acc[v] += p[v] * q[v];
    }
#pragma unroll
    for (int o = V / 2; o > 0; o >>= 1)
#pragma unroll
        for (int v = 0; v < o; v++) acc[v] += acc[v + o];
    return acc[0];
}

// FP64: the lane's entries in two sums, so that a row is as exact as by about as many
// lanes as it has entries (a running sum past a large diagonal was up to 1.4 times as
// far off).  HALVES: the first half and one more (the diagonal of a symmetric row is its
// last), then the rest; else alternating, for lanes with few entries.  An FP64 addition
// keeps a scheduler busy for 64 cycles, so this costs one: Poisson 127^3 with one sum 36
// us, two 37, four 54, the eight of the lanes before 58.
template <int G, bool HALVES>
__device__ __forceinline__ double row_pair(int a, int b, int lane, const int *__restrict__ cind, const double *__restrict__ val,
                                           const double *__restrict__ x) {
    if constexpr (HALVES) {
        const int mid = min(b, a + ((b - a + G - 1) / G / 2 + 1) * G);
        const double first = row_part<G>(a, mid, lane, cind, val, x);
        return first + row_part<G>(mid, b, lane, cind, val, x);
    } else {
        return row_part<G, false, 2>(a, b, lane, cind, val, x);
    }
}

// FP64, about as many lanes as entries: one or two entries a lane.  An addition keeps a
// scheduler busy for 64 cycles also where few lanes of the warp take it, so the lanes take
// their last entries one by one, whatever number of them each has.  (32 lanes, one row a
// warp: only where it has no more than two a lane.)  12,000 rows of 9 entries 5.2 -> 4.2
// us, of 0 to 14 5.1 -> 4.2, 1.5 M rows of 0 to 2 entries 12.4 -> 10.3.
template <int G>
__device__ __forceinline__ double row_few(int a, int b, int lane, const int *__restrict__ cind, const double *__restrict__ val,
                                          const double *__restrict__ x) {
    if constexpr (G == 32)
        if (b - a > 2 * G) return row_part<G>(a, b, lane, cind, val, x);
    return row_part<G, false, 1, true>(a, b, lane, cind, val, x);
}

// FP64, one lane and few entries a row, as in interpolations (rows of one next to rows of
// four): the two sums' entries pair by pair, for the same reason.  1.5 M rows of 0 to 4
// entries 26.8 -> 17.4 us, of 0 to 6 27.2 -> 22.7, but of 0 to 8 38.9 -> 43.2 and of 3
// each 14.5 -> 17.5: only below 2.6 entries a row.
__device__ __forceinline__ double row_two(int a, int b, const int *__restrict__ cind, const double *__restrict__ val,
                                          const double *__restrict__ x) {
    double first = 0, second = 0;
    for (int j = a; j < b; j += 2) {
        const bool two = j + 1 < b;
        const int c0 = __ldg(cind + j), c1 = two ? __ldg(cind + j + 1) : 0;
        const double v0 = __ldg(val + j), v1 = two ? __ldg(val + j + 1) : 0.0;
        const double x0 = __ldg(x + c0), x1 = two ? __ldg(x + c1) : 0.0;
        first += v0 * x0;
        if (two) second += v1 * x1;
    }
    return first + second;
}

// the lane's part of an FP row by DevCsr::sums
template <int G, int V, typename T>
__device__ __forceinline__ T row_sums(int a, int b, int lane, const int *__restrict__ cind, const T *__restrict__ val,
                                      const T *__restrict__ x) {
    if constexpr (std::is_same<T, double>::value) {
        if constexpr (V == 1) return row_few<G>(a, b, lane, cind, val, x);
        else if constexpr (V == SUMS_PAIRS) return row_two(a, b, cind, val, x);
        else return row_pair<G, V == SUMS_HALVES>(a, b, lane, cind, val, x);
    } else if constexpr (V == 1) return row_part<G>(a, b, lane, cind, val, x);
    else return row_part_of<G, V>(a, b, lane, cind, val, x);
}

}  // namespace sagb
