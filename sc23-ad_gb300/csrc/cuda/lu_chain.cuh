// The dense LU solve of a coarsest level by one thread-block cluster: integers and
// FP64 (FP32 sums keep an order that the chain does not have).
#pragma once
#include <type_traits>
#include <vector>

#include "acc.cuh"

namespace sagb {

// LUflex::Solve / LU<T>::Solve (solver/lu.hpp:91-94, 30-33): ltri forward then
// dutri backward on the coarsest operator's exact LU factors (30-45% dense at
// these sizes), stored as 32 x 32 blocks of the triangles, 16 bytes of a row
// together and the 32 rows of a block side by side (block_at).  Rows beyond n
// are zero.
//
// k_lu_chain: one cluster of kLuCtas CTAs.  Both substitutions are one chain of
// n rows, which a single warp walks (lane = row of the panel): it takes a
// panel's diagonal block and the blocks of the kLuNear panels after it from shared
// memory, and in each of 32 steps broadcasts one value by a shuffle and
// subtracts its column from the panel and from the next ones.  What the chain
// costs is the step's latency (integers: shift, shuffle, multiply-add); all else
// is kept off it.  The products with the columns further back are summed by the
// other warps of the cluster, each for its own panels, as the values come in; a
// panel's sum is needed only kLuNear panels after the last value it takes.  Values
// and sums travel as st.async into the other CTA's shared memory, counted by
// one mbarrier each; a loader warp brings the chain's blocks ahead of it.
// Integer sums wrap, so their order does not matter; FP64 sums are taken in
// another order than the reference's (the sequential-order mode uses k_dense_lu).
// Every wait is bounded in time (ST_TIMEOUT); after one that ran out the waits
// of that CTA no longer wait.
// FP64: the backward chain runs on t = x / dinv, with the columns of U multiplied
// by dinv beforehand (one rounding an entry, as the product t dinv has), so that a
// step of it has one multiply-add and no product.
// A step is 75-80 cycles for integers.  An FP64 multiply-add keeps a scheduler
// busy for 64: 190 cycles, 155 without the next panel's.  One solve,
// against one CTA with 32-row panels (k_dense_lu on row-major factors): int n = 512
// 164 -> 43 us, n = 1013 338 -> 82 us, n = 1769 637 -> 142 us; FP64 n = 1013 605 ->
// 209 us, n = 1872 1,520 -> 381 us.

constexpr int kLuCtas = 8;         // k_lu_chain: CTAs of the cluster
constexpr int kLuWarps = 8;        // and warps of each
// panels whose sums are kept: a sum is taken before the values two panels on exist
constexpr int kLuParts = 4;
constexpr size_t kLuChainSmem = kSmemMax - 256;  // (the rest is static)
constexpr int kLuSlots = 3;        // panels of the chain's blocks in shared memory
constexpr int kLuHelpers = (kLuCtas - 1) * kLuWarps;
// blocks after the diagonal one that the chain takes along: they cover the way of
// a panel's values to the other CTAs and of a sum back, and cost the chain a
// multiply-add a step.  1 / 2 / 3 of them: int n = 1769 142 / 146 / 160 us, FP64
// n = 1872 521 / 653 us / -
constexpr int kLuNear = 1;

// index of element (i, c) of a block triangle: lower (column panel by column
// panel, downwards from the diagonal) or upper (upwards from the diagonal)
__host__ __device__ __forceinline__ size_t block_lower(int npan, int q, int p) {
    return (size_t)p * npan - (size_t)p * (p - 1) / 2 + (q - p);
}
__host__ __device__ __forceinline__ size_t block_upper(int q, int p) { return (size_t)p * (p + 1) / 2 + (p - q); }
template <typename V>
__host__ __device__ __forceinline__ int block_at(int i, int c) {  // within a block
    constexpr int per = 16 / (int)sizeof(V);
    return (c / per) * (32 * per) + i * per + c % per;
}

// host copy of the factors as blocks
template <typename V>
struct LuBlocks {
    int n, npan;
    std::vector<V> L, U, dinv;
    explicit LuBlocks(int n_) : n(n_), npan((n_ + 31) / 32), L(size(n_), V(0)), U(size(n_), V(0)), dinv(n_ > 0 ? n_ : 1, V(0)) {}
    static size_t size(int n) {
        const size_t p = n > 0 ? (n + 31) / 32 : 1;
        return p * (p + 1) / 2 * 1024;
    }
    size_t lower(int i, int c) const { return block_lower(npan, i >> 5, c >> 5) * 1024 + block_at<V>(i & 31, c & 31); }
    size_t upper(int i, int c) const { return block_upper(i >> 5, c >> 5) * 1024 + block_at<V>(i & 31, c & 31); }
    void scale_columns() {
        for (int c = 0; c < n; c++)
            for (int i = 0; i < c; i++) U[upper(i, c)] *= dinv[c];
    }
};

// ------------------------------------------------- the chain in one cluster
__device__ __forceinline__ void st_async_u32(unsigned addr, unsigned v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(addr), "r"(v), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void st_async_u64(unsigned addr, unsigned long long v, unsigned bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr), "l"(v), "r"(bar)
                 : "memory");
}
template <typename T>
__device__ __forceinline__ unsigned long long bits_of(T v) {
    if constexpr (std::is_same<T, double>::value) return (unsigned long long)__double_as_longlong(v);
    else return (unsigned long long)v;
}
template <typename T>
__device__ __forceinline__ T of_bits(unsigned long long v) {
    if constexpr (std::is_same<T, double>::value) return __longlong_as_double((long long)v);
    else return (T)v;
}

// acc + d * x (integers wrap)
template <int VT>
__device__ __forceinline__ acc_t<VT> acc_add(acc_t<VT> a, vt_t<VT> d, vt_t<VT> x) {
    if constexpr (VT == VT_I32) return wadd(a, (long long)d * (long long)x);
    else return a + d * x;
}

struct LuSmem {  // byte offsets
    int ready, xbar, xs, part, ring, bytes;
};
template <int VT>
__host__ __device__ __forceinline__ LuSmem lu_smem(int npan) {
    const int es = (int)sizeof(vt_t<VT>);
    LuSmem s;
    s.ready = 0;                          // CTA 0: panel k's blocks and sum are there (both directions)
    s.xbar = s.ready + 2 * npan * 8;      // panel k's values are there
    s.xs = (s.xbar + 2 * npan * 8 + 127) / 128 * 128;  // the values, panel by panel in the chain's order
    s.part = s.xs + npan * 32 * es;       // CTA 0: the sums
    s.ring = s.part + kLuParts * 32 * 8;  // CTA 0: kLuSlots panels of blocks
    s.bytes = s.ring + kLuSlots * (1 + kLuNear) * 1024 * es;
    return s;
}

template <int VT>
struct LuChain {
    int n, bitL, bitU, dbitU;
    const vt_t<VT> *L, *U;  // FP64: U's columns times their dinv
    const vt_t<VT> *dinv;
    const vt_t<VT> *in;
    vt_t<VT> *out;
    int ld;  // between the elements of in and out
};

// one solve by the cluster of the calling CTA; PDL: in is read, and out written,
// after the programmatic-launch wait
template <int VT, bool PDL>
__device__ __forceinline__ void lu_chain(const LuChain<VT> &a, unsigned *flags) {
    using V = vt_t<VT>;
    using T = acc_t<VT>;
    constexpr int NEAR = kLuNear;
    constexpr int PER = 16 / (int)sizeof(V), QB = 32 / PER;  // entries of a quad; quads of a block's row
    constexpr unsigned BB = 1024 * sizeof(V);                // bytes of a block
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int npan = (a.n + 31) / 32, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = cluster_rank();
    const LuSmem o = lu_smem<VT>(npan);
    unsigned long long *ready = (unsigned long long *)(smem_raw + o.ready);
    unsigned long long *xbar = (unsigned long long *)(smem_raw + o.xbar);
    V *xs = (V *)(smem_raw + o.xs);
    __shared__ int s_taken, s_dead;  // panels the chain is done with; a wait ran out
    const V *L = a.L, *U = a.U;
    const int n = a.n, bitL = a.bitL, bitU = a.bitU, dbitU = a.dbitU;
    if (threadIdx.x == 0) {
        s_taken = 0;
        s_dead = 0;
    }
    for (int k = threadIdx.x; k < 2 * npan; k += 32 * kLuWarps) {
        mbar_init(ready + k, 1);
        mbar_init(xbar + k, 1);
    }
    fence_mbar_init();
    __syncthreads();
    for (int k = threadIdx.x; k < 2 * npan; k += 32 * kLuWarps) mbar_expect_tx(xbar + k, 32 * sizeof(V));
    if (PDL) pdl_wait();
    cluster_sync_all();

    auto wait = [&](unsigned long long *bar) {
        if (mbar_try_wait(bar, 0) || *(volatile int *)&s_dead) return;
        const unsigned long long t0 = globaltimer_ns();
        while (!mbar_try_wait(bar, 0))
            if (*(volatile int *)&s_dead || globaltimer_ns() - t0 > kSpinLimitNs) {
                *(volatile int *)&s_dead = 1;
                atomicOr(flags, ST_TIMEOUT);
                return;
            }
    };

    if (rank == 0 && warp == 0) {
        // ------------------------------------------------------- the chain
        const V *in = a.in, *dinv = a.dinv;
        V *out = a.out;
        const long long ld = a.ld;
        const unsigned long long *part = (const unsigned long long *)(smem_raw + o.part);
        unsigned xs_at[kLuCtas], bar_at[kLuCtas];
#pragma unroll
        for (int r = 0; r < kLuCtas; r++) {
            xs_at[r] = map_rank(smem_addr(xs), r);
            bar_at[r] = map_rank(smem_addr(xbar), r);
        }
        bool ovf = false;
        for (int dir = 0; dir < 2; dir++) {
            const bool fwd = dir == 0;
            T near[NEAR];  // the products of the panels before with the next ones
#pragma unroll
            for (int j = 0; j < NEAR; j++) near[j] = T(0);
            auto row_of = [&](int k) { return (fwd ? k : npan - 1 - k) * 32 + lane; };
            auto start = [&](int k) {  // the row's input, and its inverse diagonal
                const int i = row_of(k);
                return k < npan && i < n ? (fwd ? in[i * ld] : out[i * ld]) : V(0);
            };
            auto dinv_of = [&](int k) {
                const int i = row_of(k);
                return !fwd && k < npan && i < n ? __ldg(dinv + i) : V(0);
            };
            V s0 = start(0), dv = dinv_of(0);
            for (int k = 0; k < npan; k++) {
                const int i = row_of(k);
                wait(ready + dir * npan + k);
                T sum = near[0];
                if (k > NEAR) {
                    const T far = of_bits<T>(part[k % kLuParts * 32 + lane]);
                    if constexpr (VT == VT_I32) sum = wadd(sum, far);
                    else sum += far;
                }
#pragma unroll
                for (int j = 0; j + 1 < NEAR; j++) near[j] = near[j + 1];
                near[NEAR - 1] = T(0);
                T t = acc_init<VT>(s0, fwd ? bitL : bitU);
                if constexpr (VT == VT_I32) t = wsub(t, sum);
                else t -= sum;
                const V d_here = dv;
                s0 = start(k + 1);
                dv = dinv_of(k + 1);
                const uint4 *blk = (const uint4 *)(smem_raw + o.ring + (dir * npan + k) % kLuSlots * (1 + NEAR) * BB) + lane;
                const int bit = fwd ? bitL : bitU;
                // integers: u = ~t, so that a step is one multiply-add
                if constexpr (VT == VT_I32) t = ~t;
                auto value = [&](bool &bad) {  // x of this lane's row as t stands
                    if constexpr (VT == VT_I32) {
                        if (fwd) {
                            const long long s = ~(t >> bit);
                            bad = !fits32(s);
                            return lo32(s);
                        }
                        bad = false;
                        return acc_finish<VT>(~t, d_here, bitU, dbitU, bad);
                    } else {
                        bad = false;
                        return t;
                    }
                };
                auto steps = [&](auto forward) {
                    constexpr bool F = decltype(forward)::value;
                    // FP64: the next panel's multiply-adds one group of columns late, or they
                    // come before this panel's in the pipe and hold up the chain
                    constexpr bool kLate = VT == VT_F64;
                    [[maybe_unused]] V le[PER][NEAR], lx[PER];
                    if constexpr (kLate) {
#pragma unroll
                        for (int e = 0; e < PER; e++) {
                            lx[e] = V(0);
#pragma unroll
                            for (int j = 0; j < NEAR; j++) le[e][j] = V(0);
                        }
                    }
#pragma unroll (kLate ? 1 : QB)
                    for (int g = 0; g < QB; g++) {
                        const int gq = F ? g : QB - 1 - g;
                        uint4 q[1 + NEAR];
#pragma unroll
                        for (int j = 0; j <= NEAR; j++) q[j] = blk[j * (BB / 16) + gq * 32];
#pragma unroll
                        for (int e = 0; e < PER; e++) {
                            const int ec = F ? e : PER - 1 - e, c = gq * PER + ec;
                            bool bad;
                            V xc;
                            if constexpr (VT == VT_I32 && F) xc = ~(int)__funnelshift_r((unsigned)t, (unsigned)((unsigned long long)t >> 32), bit);
                            else xc = value(bad);
                            xc = __shfl_sync(0xffffffffu, xc, c);
                            auto entry = [&](const uint4 &w) {
                                if constexpr (VT == VT_F64) return ec == 0 ? __hiloint2double((int)w.y, (int)w.x) : __hiloint2double((int)w.w, (int)w.z);
                                else {
                                    const unsigned u = ec == 0 ? w.x : ec == 1 ? w.y : ec == 2 ? w.z : w.w;
                                    return (int)u;
                                }
                            };
                            if constexpr (VT == VT_I32) t = acc_add<VT>(t, entry(q[0]), xc);
                            else if (F ? lane > c : lane < c) t -= entry(q[0]) * xc;  // (0 * inf is no 0)
#pragma unroll
                            for (int j = 0; j < NEAR; j++) {
                                if constexpr (kLate) {
                                    near[j] = acc_add<VT>(near[j], le[e][j], lx[e]);
                                    le[e][j] = entry(q[1 + j]);
                                } else {
                                    near[j] = acc_add<VT>(near[j], entry(q[1 + j]), xc);
                                }
                            }
                            if constexpr (kLate) lx[e] = xc;
                        }
                    }
                    if constexpr (kLate) {
#pragma unroll
                        for (int e = 0; e < PER; e++)
#pragma unroll
                            for (int j = 0; j < NEAR; j++) near[j] = acc_add<VT>(near[j], le[e][j], lx[e]);
                    }
                };
                if (fwd) steps(std::true_type());
                else steps(std::false_type());
                bool bad;
                V x = value(bad);
                if (i >= n) {
                    x = V(0);
                    bad = false;
                }
                ovf |= bad;
                // to every CTA of the cluster
                const unsigned at = (unsigned)((k * 32 + lane) * sizeof(V)), bt = (unsigned)((dir * npan + k) * 8);
#pragma unroll
                for (int r = 0; r < kLuCtas; r++) {
                    if constexpr (sizeof(V) == 8) st_async_u64(xs_at[r] + at, bits_of<V>(x), bar_at[r] + bt);
                    else st_async_u32(xs_at[r] + at, (unsigned)bits_of<V>(x), bar_at[r] + bt);
                }
                if (i < n) {
                    if constexpr (VT == VT_I32) out[i * ld] = x;
                    else out[i * ld] = fwd ? x : x * d_here;
                }
                __syncwarp();
                if (lane == 0) *(volatile int *)&s_taken = dir * npan + k + 1;
            }
        }
        if (ovf) atomicOr(flags, ST_OVERFLOW);
    } else if (rank == 0 && warp == 1) {
        // ------------------------------------- the loader of the chain's blocks
        if (lane == 0) {
            for (int m = 0; m < 2 * npan; m++) {
                const int k = m < npan ? m : m - npan, have = min(1 + NEAR, npan - k);
                const unsigned long long t0 = globaltimer_ns();
                while (*(volatile int *)&s_taken + kLuSlots <= m) {
                    if (*(volatile int *)&s_dead) break;
                    if (globaltimer_ns() - t0 > kSpinLimitNs) {
                        *(volatile int *)&s_dead = 1;
                        atomicOr(flags, ST_TIMEOUT);
                    }
                }
                if (*(volatile int *)&s_dead) break;
                const unsigned bytes = have * BB, sum = k > NEAR ? 32 * 8 : 0;
                mbar_expect_tx(ready + m, bytes + sum);
                // column panel k: the diagonal block and the ones after it lie side by side
                const V *src = m < npan ? L + block_lower(npan, k, k) * 1024 : U + block_upper(npan - 1 - k, npan - 1 - k) * 1024;
                bulk_g2s(smem_raw + o.ring + m % kLuSlots * (1 + NEAR) * BB, src, bytes, ready + m);
            }
        }
    } else if (rank != 0) {
        // --------------------- sums of a panel's products with the far columns
        const int h = ((int)rank - 1) * kLuWarps + warp;
        const unsigned part0 = map_rank(smem_addr(smem_raw + o.part), 0), ready0 = map_rank(smem_addr(ready), 0);
        for (int dir = 0; dir < 2; dir++) {
            // (panel NEAR + 1 is the first with far columns)
            for (int k = NEAR + 1 + h; k < npan; k += kLuHelpers) {
                T sa = T(0), sb = T(0);
                auto block = [&](int j) {  // block (panel k, column panel j), both in the chain's order
                    const V *base = dir == 0 ? L + block_lower(npan, k, j) * 1024
                                             : U + block_upper(npan - 1 - k, npan - 1 - j) * 1024;
                    return (const uint4 *)base + lane;
                };
                uint4 w[QB];
#pragma unroll
                for (int g = 0; g < QB; g++) w[g] = __ldg(block(0) + g * 32);
                for (int j = 0; j < k - NEAR; j++) {
                    wait(xbar + dir * npan + j);
                    __syncwarp();
                    const uint4 *xq = (const uint4 *)(xs + j * 32);
                    const uint4 *nb = block(min(j + 1, k - NEAR - 1));
#pragma unroll
                    for (int g = 0; g < QB; g++) {
                        const uint4 x = xq[g], v = w[g];
                        w[g] = __ldg(nb + g * 32);
                        if constexpr (VT == VT_F64) {
                            sa = acc_add<VT>(sa, __hiloint2double((int)v.y, (int)v.x), __hiloint2double((int)x.y, (int)x.x));
                            sb = acc_add<VT>(sb, __hiloint2double((int)v.w, (int)v.z), __hiloint2double((int)x.w, (int)x.z));
                        } else {
                            sa = acc_add<VT>(sa, (int)v.x, (int)x.x);
                            sb = acc_add<VT>(sb, (int)v.y, (int)x.y);
                            sa = acc_add<VT>(sa, (int)v.z, (int)x.z);
                            sb = acc_add<VT>(sb, (int)v.w, (int)x.w);
                        }
                    }
                }
                if constexpr (VT == VT_I32) sa = wadd(sa, sb);
                else sa += sb;
                st_async_u64(part0 + (unsigned)(k % kLuParts * 32 + lane) * 8, bits_of<T>(sa), ready0 + (unsigned)(dir * npan + k) * 8);
            }
        }
    }
    // no CTA leaves while a value may still be on its way into its shared memory; CTA 0
    // has waited for its blocks and sums, unless a wait ran out
    if (warp == kLuWarps - 1) {
        const unsigned long long t0 = globaltimer_ns();
        auto arrived = [&](unsigned long long *bar) {
            for (int m = lane; m < 2 * npan; m += 32)
                while (!mbar_try_wait(bar + m, 0) && globaltimer_ns() - t0 <= kSpinLimitNs) {
                }
        };
        arrived(xbar);
        if (rank == 0 && *(volatile int *)&s_dead) arrived(ready);
    }
    __syncthreads();
    cluster_sync_all();
}

}  // namespace sagb
