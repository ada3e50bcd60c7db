// What a sweep level by level costs on the GPU, in us: models that upload picks
// among k_sweep, k_tri_cta and k_tri (cuda/trsv.cu) with.
//
// Fitted to the 178 levels of 42 hierarchies (2D and 3D Poisson, anisotropic,
// lognormal, convection-diffusion and 27-point systems of 1,600 to 250,000 rows)
// with each of the orders natural, 40 blocks, chunks of rows and colours, in int32,
// FP64 and FP32, timed on one GB300: k_tri_cta's is 6 % off on average (FP64 8 %),
// k_tri's 16 % (18 %), k_sweep's 10 %.
#pragma once
#include "schedule.hpp"

namespace sagb {

constexpr int kTriThreads = 256;   // k_tri: threads of a CTA
constexpr int kTriBatch = 4;       // and entries that a lane reads together
constexpr int kCtaThreads = 1024;  // k_tri_cta: threads, the last warp copies
constexpr int kCtaSlots = 8;       // and levels in flight
constexpr size_t kCtaVecMax = 150 * 1024;  // and the largest vector

// shared memory of k_tri_cta beside its copy ring: vector, bookkeeping of nlev levels
inline size_t cta_fixed_smem(int n, int es, int nlev) {
    return ((size_t)n * es + 15) / 16 * 16 + (4 * (2 * (size_t)nlev + 1) + 15) / 16 * 16 + (8 + 4) * kCtaSlots;
}
inline bool cta_fits(int n, int es, int nlev, size_t smem) {
    return (size_t)n * es <= kCtaVecMax && cta_fixed_smem(n, es, nlev) + 4096 <= smem;
}

// k_tri_cta: levels, passes of its 31 warps over each level, rounds of four entries a
// lane in the longest row of each pass; rows and entries come through one CTA
double cta_us(const TriSchedule &s, int lanes, int es);
// the same from below, by the number of levels alone
inline double cta_least_us(int nlev, int es) { return 2.1 + (es == 8 ? 0.60 : 0.67) * nlev; }

// k_tri, played through warp by warp: CTAs claim chunks in order, a warp's rows of a
// pass wait for all values that they read, and each round of kTriBatch entries a lane
// costs the way to the L2 (two of them for FP64: flag and value)
double spread_us(const TriSchedule &s, int lanes, int es, int ctas);
// the same from below, by the length of the longest chain of rows
inline double spread_least_us(int chain, int es) { return 4.0 + (es == 8 ? 2.7 : 0.9) * chain; }

}  // namespace sagb
