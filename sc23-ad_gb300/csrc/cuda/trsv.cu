// Gauss-Seidel / SOR sweeps and the coarse LU solve in the reference's
// dependency order.
//
// Integer sweeps follow ldtri::CSRflex::SpTRSV (matrix/trimat/ldtri.hpp:172-183)
// and its block-Jacobi form BJCSRflex (ldtri.hpp:511-525):
//   t = in_i << bit;  t -= sum_j a_ij * out_j;  out_i = (int)((t >> bit) * dinv_i >> dbit)
// FP sweeps follow ldtri::CSR<T> / BJCSR<T> (ldtri.hpp:49-58, 398-412).
// Rows are grouped into dependency levels (host/schedule.hpp); every row of a
// level only reads rows of earlier levels, so computing level after level gives
// the integer results of the sequential loop.
//
// Three kernels, picked at upload by what they are expected to take
// (host/sweep_plan.cpp, host/tri_cost.hpp):
//  * k_sweep: contiguous blocks of rows, one CTA each, the block's values in
//    shared memory, every level's row data copied ahead by the lanes that use
//    them; one block where the vector fits one CTA's shared memory and the
//    levels are small.  It needs every row of a block to read rows of the same
//    or of earlier blocks.
//  * k_tri_cta (few levels of many rows, the vector fits in shared memory): one
//    CTA.  The result vector lives in shared memory, seeded with `in` (a row
//    reads its own input once and then overwrites it).  Each level's row data
//    is one 16-byte aligned block that a bulk copy (cp.async.bulk + mbarrier)
//    brings into a byte ring in shared memory (all of it not taken by the
//    vector) up to kCtaSlots levels ahead, so a level costs shared memory
//    traffic and one block barrier.
//  * k_tri (few levels of many rows in larger triangles; what k_sweep's plan
//    cannot hold: large multicolour sweeps, whose rows also read later rows,
//    and triangles that reach back too far for the shared memory): one CTA per
//    SM claims chunks of level-ordered rows
//    by ticket; a row waits only for the rows it reads.  Integer and FP32
//    results are published as one 64-bit word {epoch, value}, so a dependency
//    costs one L2 load; FP64 results use an epoch flag with release/acquire.
//    Each lane reads a batch of dependencies at once and spins only on those
//    not yet published.  Chunks are claimed in level order and depend only on
//    earlier chunks, so the waits cannot deadlock.
// All waits are bounded in time (ST_TIMEOUT); ticket and epoch are advanced by
// the last CTA, so all of them replay from a CUDA graph.
#include <algorithm>
#include <cstring>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>
#include <type_traits>

#include "../host/sweep_plan.hpp"
#include "../sagb_internal.hpp"
#include "acc.cuh"
#include "common.cuh"
#include "lu_chain.cuh"

namespace sagb {

constexpr int kBatch = kTriBatch;  // dependencies read together per lane (k_tri)

__device__ __forceinline__ bool aborted(const unsigned *flags) {
    return (*(volatile const unsigned *)flags & ST_TIMEOUT) != 0;
}

// ============================================================== multi-CTA

struct TriArgs {
    int n, nchunks, bit, dbit;
    const int *perm, *prp, *pci;
    const void *pval, *dinv;
    const int *chunk_lv, *sub_bound;
    unsigned long long *pk;
    unsigned *flag;
    TriSync *sync;
};

// spin on one packed {epoch, value} word until it carries epoch ep (bounded;
// the shared status word is read only on the slow path)
__device__ __forceinline__ unsigned long long wait_packed(unsigned long long *pk, int c, unsigned ep,
                                                          unsigned *flags) {
    const unsigned long long t0 = globaltimer_ns();
    for (unsigned it = 1;; it++) {
        const unsigned long long w = ld_relaxed_u64(pk + c);
        if ((unsigned)(w >> 32) == ep) return w;
        if ((it & 255u) == 0) {
            if (globaltimer_ns() - t0 > kSpinLimitNs) {
                atomicOr(flags, ST_TIMEOUT);
                return w;
            }
            if (aborted(flags)) return w;
        }
    }
}

__device__ __forceinline__ void wait_flag(const unsigned *flag, int c, unsigned ep, unsigned *flags) {
    const unsigned long long t0 = globaltimer_ns();
    for (unsigned it = 1;; it++) {
        if (ld_relaxed_u32(flag + c) == ep) return;
        if ((it & 255u) == 0) {
            if (globaltimer_ns() - t0 > kSpinLimitNs) {
                atomicOr(flags, ST_TIMEOUT);
                return;
            }
            if (aborted(flags)) return;
        }
    }
}

__device__ __forceinline__ double ld_relaxed_f64(const double *p) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(p) : "memory");
    return v;
}

// one row, G lanes; each lane reads kBatch dependencies at a time, all
// together, and spins only on those not yet published
template <int VT, int G, bool EXACT>
__device__ __forceinline__ void tri_row(const TriArgs &a, int p, bool valid, int g, unsigned ep, const void *in_,
                                        void *out_, unsigned *flags, bool &ovf) {
    using V = vt_t<VT>;
    const V *in = (const V *)in_;
    V *out = (V *)out_;
    const V *pv = (const V *)a.pval;
    acc_t<VT> t = 0;
    int row = 0;
    if (valid) {
        row = __ldg(a.perm + p);
        if (g == 0) t = acc_init<VT>(__ldg(in + row), a.bit);
        const int jb = __ldg(a.prp + p), je = __ldg(a.prp + p + 1);
        for (int j0 = jb + g; j0 < je; j0 += G * kBatch) {
            int c[kBatch];
            V v[kBatch];
#pragma unroll
            for (int k = 0; k < kBatch; k++) {
                const int j = j0 + k * G;
                c[k] = j < je ? __ldg(a.pci + j) : -1;
                v[k] = j < je ? __ldg(pv + j) : V(0);
            }
            if constexpr (VT == VT_F64) {
                unsigned f[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) f[k] = c[k] >= 0 ? ld_relaxed_u32(a.flag + c[k]) : ep;
#pragma unroll
                for (int k = 0; k < kBatch; k++)
                    if (f[k] != ep) wait_flag(a.flag, c[k], ep, flags);
                fence_acq_rel_gpu();  // the flags were released after the values
#pragma unroll
                for (int k = 0; k < kBatch; k++)
                    if (c[k] >= 0) t = acc_sub<VT, EXACT>(t, v[k], ld_relaxed_f64((const double *)out + c[k]));
            } else {
                unsigned long long w[kBatch];
#pragma unroll
                for (int k = 0; k < kBatch; k++) w[k] = c[k] >= 0 ? ld_relaxed_u64(a.pk + c[k]) : 0ull;
#pragma unroll
                for (int k = 0; k < kBatch; k++) {
                    if (c[k] < 0) continue;
                    if ((unsigned)(w[k] >> 32) != ep) w[k] = wait_packed(a.pk, c[k], ep, flags);
                    V o;
                    if constexpr (VT == VT_I32) o = (int)(unsigned)w[k];
                    else o = __uint_as_float((unsigned)w[k]);
                    t = acc_sub<VT, EXACT>(t, v[k], o);
                }
            }
        }
    }
    t = acc_reduce<VT>(t, G);
    if (valid && g == 0) {
        const V r = acc_finish<VT>(t, __ldg((const V *)a.dinv + p), a.bit, a.dbit, ovf);
        out[row] = r;
        if constexpr (VT == VT_F64) {
            st_release_u32(a.flag + row, ep);
        } else if constexpr (VT == VT_I32) {
            st_relaxed_u64(a.pk + row, ((unsigned long long)ep << 32) | (unsigned)r);
        } else {
            st_relaxed_u64(a.pk + row, ((unsigned long long)ep << 32) | __float_as_uint(r));
        }
    }
}

template <int VT, int G, bool EXACT>
__global__ void __launch_bounds__(kTriThreads) k_tri(TriArgs a, const void *in, void *out, unsigned *flags) {
    __shared__ int s_chunk;
    __shared__ unsigned s_epoch;
    if (threadIdx.x == 0) s_epoch = ld_acquire_u32(&a.sync->epoch) + 1;
    __syncthreads();
    const unsigned ep = s_epoch;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int RPW = 32 / G;  // rows per warp per pass
    constexpr int NW = kTriThreads / 32;
    const int g = lane % G, sub = lane / G;
    bool ovf = false;
    for (;;) {
        if (threadIdx.x == 0) s_chunk = aborted(flags) ? a.nchunks : (int)atomicAdd(&a.sync->ticket, 1u);
        __syncthreads();
        const int ch = s_chunk;
        if (ch >= a.nchunks) break;
        const int s0 = __ldg(a.chunk_lv + ch), s1 = __ldg(a.chunk_lv + ch + 1);
        for (int s = s0; s < s1; s++) {
            const int p0 = __ldg(a.sub_bound + s), p1 = __ldg(a.sub_bound + s + 1);
            for (int base = p0 + warp * RPW; base < p1; base += NW * RPW) {
                const int p = base + sub;
                tri_row<VT, G, EXACT>(a, p, p < p1, g, ep, in, out, flags, ovf);
            }
            if (s + 1 < s1) __syncthreads();
        }
        __syncthreads();
    }
    if (ovf) atomicOr(flags, ST_OVERFLOW);
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned d = atomicAdd(&a.sync->done, 1u);
        if (d == gridDim.x - 1) {
            a.sync->ticket = 0;
            a.sync->done = 0;
            __threadfence();
            st_release_u32(&a.sync->epoch, ep);
        }
    }
}

// ============================================================= single CTA
//
// Level block (host layout, 16-byte aligned, size a multiple of 16):
//   int32 header[8] = {R, E, off_val, off_dinv, off_perm, off_rp, 0, 0}
//   val[E] (V), dinv[R] (V), perm[R], rp[R+1] (0-based inside the block), pci[E]

template <int VT, int G, bool EXACT>
__device__ __forceinline__ void cta_level(const unsigned char *blk, vt_t<VT> *s_out, int bit, int dbit, int warp,
                                          int sub, int g, bool &ovf) {
    using V = vt_t<VT>;
    constexpr int RPW = 32 / G;
    constexpr int NW = kCtaThreads / 32 - 1;  // the last warp issues the bulk copies
    const int *hdr = (const int *)blk;
    const int R = hdr[0];
    const V *val = (const V *)(blk + hdr[2]);
    const V *dv = (const V *)(blk + hdr[3]);
    const int *perm = (const int *)(blk + hdr[4]);
    const int *rp = (const int *)(blk + hdr[5]);
    const int *pci = rp + R + 1;
    for (int base = warp * RPW; base < R; base += NW * RPW) {
        const int r = base + sub;
        const bool valid = r < R;
        acc_t<VT> t = 0;
        int row = 0;
        if (valid) {
            row = perm[r];
            const int jb = rp[r], je = rp[r + 1];
            if (g == 0) t = acc_init<VT>(s_out[row], bit);
            // four entries of the lane at a time: their loads are issued
            // together, the products are taken in the lane's order
            int j = jb + g;
            for (; j + 3 * G < je; j += 4 * G) {
                const int c0 = pci[j], c1 = pci[j + G], c2 = pci[j + 2 * G], c3 = pci[j + 3 * G];
                const V v0 = val[j], v1 = val[j + G], v2 = val[j + 2 * G], v3 = val[j + 3 * G];
                const V o0 = s_out[c0], o1 = s_out[c1], o2 = s_out[c2], o3 = s_out[c3];
                t = acc_sub<VT, EXACT>(t, v0, o0);
                t = acc_sub<VT, EXACT>(t, v1, o1);
                t = acc_sub<VT, EXACT>(t, v2, o2);
                t = acc_sub<VT, EXACT>(t, v3, o3);
            }
            for (; j < je; j += G) t = acc_sub<VT, EXACT>(t, val[j], s_out[pci[j]]);
        }
        t = acc_reduce<VT>(t, G);
        if (valid && g == 0) s_out[row] = acc_finish<VT>(t, dv[r], bit, dbit, ovf);
    }
}

// Shared memory of the single-CTA kernel: the result vector, a byte ring for
// the level blocks, kCtaSlots mbarriers, the ring position of each level in
// flight, the block offsets and the rows of each level.  The first lane of
// the last warp (the producer; that warp computes no rows, so issuing copies
// never delays a level) places every block contiguously in the ring, in level
// order (at the write position, or at the ring's start when the end has no
// room), as soon as the ring has room and fewer than kCtaSlots levels are in
// flight; a block larger than the whole ring is read from global memory
// instead.  Level d is always placed by the time the CTA reaches it: the
// producer places it right after the barrier of level d-1 at the latest, when
// every earlier level has been consumed and the ring is empty.
//
// (A variant without the barrier per level, each row waiting on done bits of
// the rows it reads, ran about twice as slow on the coarse levels of Poisson
// 128^3: the waiting rows' shared-memory polling slowed the rows being
// computed more than the barrier costs.)
template <int VT, int G, bool EXACT>
__global__ void __launch_bounds__(kCtaThreads, 1)
k_tri_cta(const unsigned char *__restrict__ blocks, const unsigned *__restrict__ blk_off, int nlev, int n,
          int bit, int dbit, int ring_bytes, const void *in_, void *out_, unsigned *flags) {
    using V = vt_t<VT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    V *s_out = (V *)smem_raw;
    const size_t vec_bytes = ((size_t)n * sizeof(V) + 15) & ~(size_t)15;
    unsigned char *ring = smem_raw + vec_bytes;
    unsigned long long *bar = (unsigned long long *)(ring + ring_bytes);
    unsigned *s_pos = (unsigned *)(bar + kCtaSlots);  // ring offset of each level in flight
    unsigned *s_off = s_pos + kCtaSlots;              // block offsets in 16-byte units
    const unsigned *s_rows = s_off + nlev + 1;     // rows of each level
    const V *in = (const V *)in_;
    V *out = (V *)out_;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane % G, sub = lane / G;
    constexpr int kProducerWarp = kCtaThreads / 32 - 1;
    const bool compute = warp != kProducerWarp;
    const bool producer = warp == kProducerWarp && lane == 0;
    bool ovf = false;

    if (producer) {
        for (int s = 0; s < kCtaSlots; s++) mbar_init(bar + s, 1);
        fence_mbar_init();
    }
    for (int i = threadIdx.x; i < n; i += kCtaThreads) s_out[i] = in[i];
    for (int i = threadIdx.x; i <= 2 * nlev; i += kCtaThreads) s_off[i] = __ldg(blk_off + i);
    __syncthreads();
    auto bytes_of = [&](int d) { return (s_off[d + 1] - s_off[d]) * 16u; };
    auto staged = [&](int d) { return bytes_of(d) <= (unsigned)ring_bytes; };
    // the producer's ring state: levels [consumed, issued) are in flight; the
    // nst staged ones among them occupy [lo, head), wrapped once when head <= lo
    int issued = 0, nst = 0;
    unsigned lo = 0, head = 0;
    auto issue_more = [&](int consumed) {  // producer only
        while (issued < nlev && issued - consumed < kCtaSlots) {
            const int d = issued;
            if (staged(d)) {
                const unsigned b = bytes_of(d);
                unsigned pos;
                if (nst == 0) {
                    pos = 0;
                    lo = 0;
                } else if (head > lo) {  // [lo, head): room at the end, else at the start
                    if (b <= (unsigned)ring_bytes - head) pos = head;
                    else if (b <= lo) pos = 0;
                    else break;
                } else {  // [lo, ring) and [0, head): room between head and lo
                    if (b <= lo - head) pos = head;
                    else break;
                }
                head = pos + b;
                nst++;
                const int s = d % kCtaSlots;
                // the region's previous readers passed the level barrier
                // before this copy is issued (no proxy fence is needed for a
                // bulk copy into memory that generic loads only read)
                s_pos[s] = pos;  // published to the waiting threads by the arrive below
                mbar_expect_tx(bar + s, b);
                bulk_g2s(ring + pos, blocks + (size_t)s_off[d] * 16, b, bar + s);
            }
            issued++;
        }
    };
    if (producer) issue_more(0);
    unsigned phase = 0;  // bit s: parity of slot s's next completion
    int stuck = -1;      // level whose copy did not arrive in time
    for (int d = 0; d < nlev; d++) {
        const bool st = staged(d);
        const int s = d % kCtaSlots;
        const unsigned char *blk = blocks + (size_t)s_off[d] * 16;
        bool timed_out = false;
        // a warp with no row in this level neither waits for its block nor
        // reads it (it only keeps the slot parities)
        constexpr int kRowsPerWarp = 32 / G;
        const bool mine = compute && warp * kRowsPerWarp < (int)s_rows[d];
        if (st && !mine) {
            phase ^= 1u << s;
        } else if (st) {
            // bounded wait for the bulk copy of this level
            const unsigned par = (phase >> s) & 1u;
            if (!mbar_try_wait(bar + s, par)) {
                const unsigned long long t0 = globaltimer_ns();
                while (!mbar_try_wait(bar + s, par)) {
                    if (globaltimer_ns() - t0 > kSpinLimitNs) {
                        timed_out = true;
                        break;
                    }
                }
            }
            phase ^= 1u << s;
            blk = ring + s_pos[s];
        }
        if (mine && !timed_out) cta_level<VT, G, EXACT>(blk, s_out, bit, dbit, warp, sub, g, ovf);
        // one barrier per level: results visible, the level's ring space free
        if (__syncthreads_or(timed_out)) {
            stuck = d;
            break;
        }
        if (producer) {
            if (st && --nst > 0) {
                for (int e = d + 1; e < issued; e++)
                    if (staged(e)) {
                        lo = s_pos[e % kCtaSlots];
                        break;
                    }
            }
            issue_more(d + 1);
        }
    }
    if (stuck >= 0) {
        // report, then wait (bounded) for the copies this CTA still has in
        // flight before its shared memory goes away
        if (producer) {
            atomicOr(flags, ST_TIMEOUT);
            const unsigned long long t0 = globaltimer_ns();
            for (int dd = stuck; dd < issued; dd++) {
                if (!staged(dd)) continue;
                const int s = dd % kCtaSlots;
                // the stuck level's wait already flipped its parity bit
                const unsigned par = ((phase >> s) & 1u) ^ (dd == stuck ? 1u : 0u);
                while (!mbar_try_wait(bar + s, par) && globaltimer_ns() - t0 < kSpinLimitNs) {
                }
            }
        }
        __syncthreads();
        return;
    }
    for (int i = threadIdx.x; i < n; i += kCtaThreads) out[i] = s_out[i];
    if (ovf) atomicOr(flags, ST_OVERFLOW);
}

// ================================================================ blocks
//
// k_sweep runs the plan of host/sweep_plan.hpp: CTA b (blocks claimed in order,
// so the blocks it reads are running or done) keeps the values of its rows and
// of its imports in shared memory and takes its rows level by level.
//
// What bounds it is the chain of dependency levels, so a step has to be short:
// its static data (entries as shared memory offsets, inverse diagonals) are
// copied to shared memory kSweepStage - 1 records ahead (each lane its own
// part, so a record needs no barrier) and are in registers before the step's
// barrier; a step is then one gather from shared memory, the products, the sum
// over a row's lanes, the row rule, one store and the barrier of the CTA's
// compute warps.  It has next to no branches: one warp runs alone on its
// scheduler, where a branch costs about as much as a round of the sum.
// A few more warps (importers) poll the published values of earlier blocks and
// copy them into the import slots ahead of their use, so that a step waits for
// another CTA only when this one has caught up with it.
//
// A row that later blocks read is published as 64-bit words {epoch, value}
// (two of them for FP64, each with half of the value), which need no reset; the
// words of a block's rows of one level are neighbours, so that a poll of 32 of
// them takes few sectors (the pollers share the SM's load path with the sweep).
//
// Measured on one GB300 against the kernels it took the place of (one CTA with
// a barrier of 31 warps and row data in level blocks; k_tri with two passes of
// dependent loads a level): int sweeps of all nine levels of Poisson 128^3, 11.4
// -> 3.1 ms (level 0, 382 dependency levels, 1.14 -> 0.23 ms; level 5, 1,112
// levels of 22 rows of 164 entries, 1.66 -> 0.60 ms), of Poisson 181^2 1.29 ->
// 0.32 ms (0.18-0.23 us a level), FP64 convection-diffusion 41^3 5.97 -> 1.13 ms.
// What was slower: mbarrier-tracked bulk copies instead of the per-lane copies
// (a try_wait and a vote a record: 0.25 instead of 0.18 us a level), records in
// registers by plain loads (too few scoreboards to keep several records in
// flight), lanes a row chosen per step (branches), importers that poll several
// groups at once (their polls take the sweep's share of the load path), words
// by row number (a poll of 32 rows took 32 sectors: level 0 0.44 ms).
//
// Every wait for a published value is bounded in time: it raises ST_TIMEOUT
// when it runs out and the sweep goes on with the values there are.
struct SweepBlock {
    int row0, row1, imp0, imp1, grp0, grp1, steps, pad;  // rows, imports, entries of grp; barriers
};
struct SweepArgs {
    int warps, importers_log, bit, dbit;  // 2^importers_log importers (several blocks)
    const SweepBlock *blocks;  // gridDim.x of them
    const long long *stream;   // first record of (block, warp)
    const uint4 *data;
    const int *imp_place, *grp;
    unsigned long long *pk;
    TriSync *sync;
};

__device__ __forceinline__ void ld_relaxed_v2(const unsigned long long *p, unsigned long long &a,
                                              unsigned long long &b) {
    asm volatile("ld.relaxed.gpu.global.v2.u64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
}
__device__ __forceinline__ void st_relaxed_v2(unsigned long long *p, unsigned long long a, unsigned long long b) {
    asm volatile("st.relaxed.gpu.global.v2.u64 [%0], {%1, %2};" ::"l"(p), "l"(a), "l"(b) : "memory");
}
__device__ __forceinline__ int ld_acquire_cta(const int *p) {
    int v;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta(int *p, int v) {
    asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}

// a published row as read: its words, whether they are of this epoch, its value
struct Published {
    unsigned long long a, b;
};
template <int VT>
__device__ __forceinline__ Published sweep_peek(const unsigned long long *pk, int row) {
    Published w{0ull, 0ull};
    if constexpr (VT == VT_F64) ld_relaxed_v2(pk + 2 * (size_t)row, w.a, w.b);
    else w.a = ld_relaxed_u64(pk + row);
    return w;
}
template <int VT>
__device__ __forceinline__ bool sweep_ready(const Published &w, unsigned ep) {
    return (unsigned)(w.a >> 32) == ep && (VT != VT_F64 || (unsigned)(w.b >> 32) == ep);
}
template <int VT>
__device__ __forceinline__ vt_t<VT> sweep_value(const Published &w) {
    if constexpr (VT == VT_F64) return __hiloint2double((int)(unsigned)w.b, (int)(unsigned)w.a);
    else if constexpr (VT == VT_I32) return (int)(unsigned)w.a;
    else return __uint_as_float((unsigned)w.a);
}
template <int VT>
__device__ __forceinline__ void sweep_publish(unsigned long long *pk, int row, unsigned ep, vt_t<VT> v) {
    const unsigned long long hi = (unsigned long long)ep << 32;
    if constexpr (VT == VT_F64)
        st_relaxed_v2(pk + 2 * (size_t)row, hi | (unsigned)__double2loint(v), hi | (unsigned)__double2hiint(v));
    else if constexpr (VT == VT_I32)
        st_relaxed_u64(pk + row, hi | (unsigned)v);
    else
        st_relaxed_u64(pk + row, hi | __float_as_uint(v));
}

// the sum of 2^LG neighbouring lanes; 32 lanes of 64-bit integers as three
// REDUX of 22, 21 and 21 bits (their sums fit 32 bits)
template <int VT, int LG>
__device__ __forceinline__ acc_t<VT> sweep_sum(acc_t<VT> t) {
    if constexpr (VT == VT_I32 && LG == 5) {
        const unsigned long long u = (unsigned long long)t;
        const unsigned a = __reduce_add_sync(0xffffffffu, (unsigned)u & 0x3fffffu);
        const unsigned b = __reduce_add_sync(0xffffffffu, (unsigned)(u >> 22) & 0x1fffffu);
        const unsigned c = __reduce_add_sync(0xffffffffu, (unsigned)(u >> 43));
        return (long long)((unsigned long long)a + ((unsigned long long)b << 22) + ((unsigned long long)c << 43));
    } else {
#pragma unroll
        for (int o = 1 << LG >> 1; o > 0; o >>= 1) {
            if constexpr (VT == VT_I32) t = wadd(t, shfl_xor(t, o));
            else t += shfl_xor(t, o);
        }
        return t;
    }
}

// shared memory by 32-bit address (volatile: they keep their order around the
// barriers)
template <typename V>
__device__ __forceinline__ V lds_val(unsigned a) {
    V v;
    if constexpr (sizeof(V) == 8) asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
    else if constexpr (std::is_same<V, float>::value) asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a));
    else asm volatile("ld.shared.s32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
// (a store that is skipped where `no` is not zero)
template <typename V>
__device__ __forceinline__ void sts_unless(unsigned no, unsigned a, V v) {
#define SAGB_STS(TYPE, C)                                                                                     \
    asm volatile("{\n .reg .pred p;\n setp.eq.u32 p, %2, 0;\n @p st.shared." TYPE " [%0], %1;\n}\n" ::"r"(a), \
                 C(v), "r"(no)                                                                                \
                 : "memory")
    if constexpr (sizeof(V) == 8) SAGB_STS("f64", "d");
    else if constexpr (std::is_same<V, float>::value) SAGB_STS("f32", "f");
    else SAGB_STS("s32", "r");
#undef SAGB_STS
}
__device__ __forceinline__ uint4 lds_quad(unsigned a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
// 16 bytes to this lane's own part of shared memory, counted by copy groups
__device__ __forceinline__ void copy_quad(unsigned dst, const uint4 *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

constexpr int kSweepThreads = 32 * (kSweepMaxWarps + kSweepImporters);

// N: lanes that one stands for, each with a sum of its own (FP32, see fixed_order)
template <int VT, bool EXACT, int LG, int E, int N = 1>
__global__ void __launch_bounds__(kSweepThreads, 1)
k_sweep(SweepArgs a, const void *in_, void *out_, unsigned *flags) {
    using V = vt_t<VT>;
    constexpr int Q = 1 + E + (VT == VT_F64);  // quads of a record
    constexpr unsigned RB = Q * 512;           // its bytes
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int W = a.warps, IM = 1 << a.importers_log;
    int *s_misc = (int *)smem_raw;  // block, epoch
    int *s_done = s_misc + 4;       // import groups each importer has filled
    unsigned char *stage = smem_raw + 128;
    V *slots = (V *)(stage + W * kSweepStage * RB);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool many = gridDim.x > 1;
    if (threadIdx.x == 0) {
        s_misc[0] = many ? (int)atomicAdd(&a.sync->ticket, 1u) : 0;
        s_misc[1] = many ? (int)(ld_acquire_u32(&a.sync->epoch) + 1) : 0;
    }
    if (threadIdx.x < kSweepImporters) s_done[threadIdx.x] = 0;
    __syncthreads();
    const int blk = s_misc[0];
    const unsigned ep = (unsigned)s_misc[1];
    const SweepBlock B = a.blocks[blk];
    const int rows = B.row1 - B.row0, nimp = B.imp1 - B.imp0;

    if (warp >= W) {
        // ------------------------------------------------------ importers
        const int w = warp - W, groups = B.grp1 - B.grp0 - 1;
        V *sv = slots + rows;
        // the place of this lane's row in group k
        auto import_of = [&](int k, int &idx) {
            if (k >= groups) return -1;
            idx = __ldg(a.grp + B.grp0 + k) + lane;
            return idx < __ldg(a.grp + B.grp0 + k + 1) ? __ldg(a.imp_place + B.imp0 + idx) : -1;
        };
        // places two groups ahead, a first look at the values one ahead: a
        // group whose values are there already costs no round trip of its own
        int idx0 = 0, idx1 = 0, filled = 0;
        int row0 = import_of(w, idx0), row1 = import_of(w + IM, idx1);
        Published v0{0ull, 0ull};
        if (row0 >= 0) v0 = sweep_peek<VT>(a.pk, row0);
        for (int k = w; k < groups; k += IM) {
            Published v1{0ull, 0ull};
            if (row1 >= 0) v1 = sweep_peek<VT>(a.pk, row1);
            int idx2 = 0;
            const int row2 = import_of(k + 2 * IM, idx2);
            if (row0 >= 0) {
                if (!sweep_ready<VT>(v0, ep)) {
                    const unsigned long long t0 = globaltimer_ns();
                    for (unsigned it = 1;; it++) {
                        v0 = sweep_peek<VT>(a.pk, row0);
                        if (sweep_ready<VT>(v0, ep)) break;
                        if ((it & 255u) == 0) {
                            if (globaltimer_ns() - t0 > kSpinLimitNs) {
                                atomicOr(flags, ST_TIMEOUT);
                                break;
                            }
                            if (aborted(flags)) break;
                        }
                    }
                }
                sv[idx0] = sweep_value<VT>(v0);
            }
            idx0 = idx1;
            row0 = row1;
            v0 = v1;
            idx1 = idx2;
            row1 = row2;
            __threadfence_block();
            __syncwarp();
            if (lane == 0) st_release_cta(s_done + w, ++filled);
        }
        return;
    }

    // ------------------------------------------------------------ compute
    const long long r0 = a.stream[(size_t)blk * W + warp];
    const int nrec = (int)(a.stream[(size_t)blk * W + warp + 1] - r0);
    // (the streams are padded: copies past a warp's last record stay inside)
    const uint4 *src = a.data + (size_t)r0 * (Q * 32) + lane;
    const unsigned mine = smem_addr(stage) + warp * (kSweepStage * RB) + lane * 16;
    auto copy = [&](unsigned at) {
#pragma unroll
        for (int q = 0; q < Q; q++) copy_quad(mine + at + q * 512, src + q * 32);
        copy_commit();
        src += Q * 32;
    };
#pragma unroll
    for (int k = 0; k < kSweepStage - 1; k++) copy(k * RB);
    const unsigned char *ahead = (const unsigned char *)(a.data + (size_t)r0 * (Q * 32)) + lane * 128;
    if (lane < 4 * Q)
        for (int k = kSweepStage; k < kSweepAhead; k++) prefetch_l2(ahead + (size_t)k * RB);
    ahead += (size_t)kSweepAhead * RB;
    {
        const V *in = (const V *)in_ + B.row0;
#pragma unroll 8
        for (int i = threadIdx.x; i < rows; i += W * 32) slots[i] = in[i];
        if (threadIdx.x < 2) slots[rows + nimp + threadIdx.x] = V(0);
    }
    asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
    const unsigned sl = smem_addr(slots);
    int step = 0, need = 0;  // barriers passed, import groups needed
    bool ovf = false, fresh = true;
    acc_t<VT> t = 0, tn[N] = {};
    unsigned to = (kSweepStage - 1) * RB, from = RB;  // where the next copy goes and the next record is
    // one record, in registers in r; the next one is brought into n
    auto record = [&](const uint4(&r)[Q], uint4(&n)[Q], bool odd) {
        const unsigned c = r[0].x;
        for (unsigned k = c >> 18 & 127u; k > 0; k--) {
            asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
            step++;
        }
        asm volatile("{\n .reg .pred p;\n setp.ne.u32 p, %0, 0;\n @p bar.sync 1, %1;\n}\n" ::"r"(c & (1u << 17)), "r"(W * 32)
                     : "memory");
        step += (int)(c >> 17 & 1u);
        if (c >> 25) {
            // importer w has filled its groups w, w + IM, ...
            need += (int)(c >> 25);
            const int w = lane & (IM - 1), want = (need - w + IM - 1) >> a.importers_log;
            if (ld_acquire_cta(s_done + w) < want) {
                const unsigned long long t0 = globaltimer_ns();
                while (ld_acquire_cta(s_done + w) < want)
                    if (globaltimer_ns() - t0 > 2 * kSpinLimitNs) {
                        atomicOr(flags, ST_TIMEOUT);
                        break;
                    }
            }
            __syncwarp();
        }
        V x[2 * E];
#pragma unroll
        for (int h = 0; h < 2 * E; h++) {
            if constexpr (VT == VT_F64) {
                const uint4 &o = r[1 + E];
                const unsigned w = h / 2 == 0 ? o.x : h / 2 == 1 ? o.y : h / 2 == 2 ? o.z : o.w;
                x[h] = lds_val<V>(sl + (h & 1 ? w >> 16 : w & 0xffffu) * 8);
            } else {
                x[h] = lds_val<V>(sl + (h & 1 ? r[1 + h / 2].z : r[1 + h / 2].x));
            }
        }
        const unsigned row = sl + (c & 0xffffu) * (unsigned)sizeof(V);
        const V own = lds_val<V>(row);
        // the record kSweepStage - 1 ahead goes where the last one was
        copy(to);
        to = to == (kSweepStage - 1) * RB ? 0 : to + RB;
        if (odd) {  // two records are 8 Q lines, at most one a lane: of four pairs' 40 or 48, the first 32
            if (lane < 8 * Q) prefetch_l2(ahead);
            ahead += 2 * RB;
        }
        copy_wait<kSweepStage - 2>();
#pragma unroll
        for (int q = 0; q < Q; q++) n[q] = lds_quad(mine + from + q * 512);
        from = from == (kSweepStage - 1) * RB ? 0 : from + RB;
        const bool more = c & (1u << 16);  // the row goes on
        acc_t<VT> s;
        if constexpr (VT == VT_F32) {  // the lanes' sums in their order; the first starts from the input
            acc_t<VT> sn[N];
#pragma unroll
            for (int k = 0; k < N; k++) sn[k] = k > 0 ? tn[k] : !fresh ? tn[0] : (lane & ((1 << LG) - 1)) == 0 ? own : V(0);
#pragma unroll
            for (int h = 0; h < 2 * E; h++) {
                const uint4 &v = r[1 + h / 2];
                sn[h % N] = acc_sub<VT, EXACT>(sn[h % N], __uint_as_float(h & 1 ? v.w : v.y), x[h]);
            }
#pragma unroll
            for (int k = 0; k < N; k++) tn[k] = more ? sn[k] : V(0);
#pragma unroll
            for (int o = N / 2; o > 0; o >>= 1)
#pragma unroll
                for (int k = 0; k < o; k++) sn[k] += sn[k + o];
            s = sn[0];
        } else {
            s = t;
            acc_t<VT> s2 = 0;  // (two chains a record where the order is free)
            if constexpr (VT == VT_F64 && LG == 0) s = fresh ? own : t;  // one lane a row: it starts from the input
#pragma unroll
            for (int h = 0; h < 2 * E; h++) {
                const uint4 &v = r[1 + h / 2];
                acc_t<VT> &sum = h < E || EXACT ? s : s2;
                if constexpr (VT == VT_I32)  // the products, subtracted at the end
                    sum = wadd(sum, (long long)(int)(h & 1 ? v.w : v.y) * (long long)x[h]);
                else
                    sum = acc_sub<VT, EXACT>(sum, h & 1 ? __hiloint2double((int)v.w, (int)v.z) : __hiloint2double((int)v.y, (int)v.x), x[h]);
            }
            if constexpr (VT == VT_I32) s = wadd(s, s2);
            else if constexpr (!EXACT) s += s2;
            t = more ? s : acc_t<VT>(0);
        }
        fresh = !more;
        s = sweep_sum<VT, LG>(s);
        V dinv;
        if constexpr (VT == VT_F64) dinv = __hiloint2double((int)r[0].w, (int)r[0].z);
        else if constexpr (VT == VT_I32) dinv = (int)r[0].z;
        else dinv = __uint_as_float(r[0].z);
        if constexpr (VT == VT_I32) s = wsub(wshl((long long)own, a.bit), s);
        else if constexpr (LG > 0 && VT == VT_F64) s += own;
        // every lane of a row has its result and stores it
        const V v = acc_finish<VT>(s, dinv, a.bit, a.dbit, ovf);
        sts_unless<V>(c & (1u << 16), row, v);
        if ((int)r[0].y >= 0) sweep_publish<VT>(a.pk, (int)r[0].y, ep, v);
    };
    uint4 ra[Q], rb[Q];
    copy_wait<kSweepStage - 2>();
#pragma unroll
    for (int q = 0; q < Q; q++) ra[q] = lds_quad(mine + q * 512);
    for (int i = 0; i < nrec; i += 2) {
        record(ra, rb, false);
        if (i + 1 < nrec) record(rb, ra, true);
    }
    copy_wait<0>();
    for (; step < B.steps; step++) asm volatile("bar.sync 1, %0;" ::"r"(W * 32) : "memory");
    // the block's values are complete
    V *out = (V *)out_ + B.row0;
    for (int i = threadIdx.x; i < rows; i += W * 32) out[i] = slots[i];
    if (ovf) atomicOr(flags, ST_OVERFLOW);
    if (many && threadIdx.x == 0) {
        // this CTA's importers are done: its warps waited for every import
        __threadfence();
        const unsigned d = atomicAdd(&a.sync->done, 1u);
        if (d == gridDim.x - 1) {
            a.sync->ticket = 0;
            a.sync->done = 0;
            __threadfence();
            st_release_u32(&a.sync->epoch, ep);
        }
    }
}

// ================================================================ upload

void DevTri::release() {
    dfree(perm);
    dfree(prp);
    dfree(pci);
    dfree(pval);
    dfree(dinv);
    dfree(chunk_lv);
    dfree(sub_bound);
    dfree(pk);
    dfree(flag);
    if (!data) dfree(sync);  // (a sweep by blocks: behind pk; its small arrays: behind blocks)
    dfree(blocks);
    dfree(data);
    dfree(blk_off);
    perm = prp = pci = chunk_lv = sub_bound = nullptr;
    pval = dinv = nullptr;
    pk = nullptr;
    flag = nullptr;
    sync = nullptr;
    blocks = data = nullptr;
    blk_off = nullptr;
    stream = nullptr;
    imp_place = grp = nullptr;
}

template <typename T>
static void gather_vals(const TriSchedule &s, const T *vals, std::vector<T> &pv, std::vector<T> &dv) {
    pv.resize(s.src_idx.size());
    for (size_t j = 0; j < s.src_idx.size(); j++) pv[j] = vals[s.src_idx[j]];
    dv.assign(s.n, T(0));
    for (int p = 0; p < s.n; p++)
        if (s.diag_src[p] >= 0) dv[p] = vals[s.diag_src[p]];
}

static size_t up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// one block per level (see the layout above k_tri_cta)
template <typename T>
static void build_blocks(const TriSchedule &s, const std::vector<T> &pv, const std::vector<T> &dv,
                         std::vector<unsigned char> &blob, std::vector<long long> &off) {
    off.assign(s.nlev + 1, 0);
    blob.clear();
    for (int l = 0; l < s.nlev; l++) {
        const int p0 = s.lvl_ptr[l], p1 = s.lvl_ptr[l + 1];
        const int R = p1 - p0;
        const int e0 = s.prp[p0], e1 = s.prp[p1];
        const int E = e1 - e0;
        const size_t o_val = 32;
        const size_t o_dinv = up(o_val + sizeof(T) * E, 8);
        const size_t o_perm = up(o_dinv + sizeof(T) * R, 4);
        const size_t o_rp = o_perm + 4 * (size_t)R;
        const size_t o_pci = o_rp + 4 * (size_t)(R + 1);
        const size_t size = up(o_pci + 4 * (size_t)E, 16);
        const size_t base = blob.size();
        blob.resize(base + size, 0);
        unsigned char *b = blob.data() + base;
        int hdr[8] = {R, E, (int)o_val, (int)o_dinv, (int)o_perm, (int)o_rp, 0, 0};
        memcpy(b, hdr, sizeof hdr);
        memcpy(b + o_val, pv.data() + e0, sizeof(T) * E);
        memcpy(b + o_dinv, dv.data() + p0, sizeof(T) * R);
        memcpy(b + o_perm, s.perm.data() + p0, 4 * (size_t)R);
        int *rp = (int *)(b + o_rp);
        for (int r = 0; r <= R; r++) rp[r] = s.prp[p0 + r] - e0;
        memcpy(b + o_pci, s.pci.data() + e0, 4 * (size_t)E);
        off[l + 1] = (long long)blob.size();
    }
}

static int pow2_at_least(double x) {
    int g = 1;
    while (g < 32 && g < x) g <<= 1;
    return g;
}

// Lanes a row in k_tri_cta and k_tri: a quarter of its average length (off the
// diagonal), one in the sequential-order mode.
constexpr int kRowShare = 4;
static int tri_lanes(const Ctx &c, const TriSource &t, int vt) {
    if (vt != VT_I32 && c.fp_exact) return 1;
    return pow2_at_least((t.n ? ((double)t.rptr[t.n] - t.n) / t.n : 0.0) / kRowShare);
}

// Whether a row's sum has one order: in the sequential-order mode, and in FP32.  FP32
// solves converge in a number of iterations that follows the last bits of their
// V-cycles, so an FP32 row is summed by all kernels as by tri_lanes lanes, which
// depend on its triangle alone: lane g takes entries g, g + G, ... in their order,
// lane 0 starts from the input, and the lanes are added by a butterfly.  k_sweep may
// let a lane stand for up to eight of them.  (Lanes and order free, and the coarsest
// solve on the cluster: an FP32 V-cycle of a 383^2 grid with 40 blocks 714 us
// instead of 910; but solves of 27-point and variable-coefficient systems took
// another number of iterations or ended 1e-8 apart.)
static bool fixed_order(const Ctx &c, int vt) { return vt == VT_F32 || (vt == VT_F64 && c.fp_exact); }

static SweepPlan plan_tri(const Ctx &c, const TriSource &t, int vt) {
    SweepLimits lim;
    lim.sms = c.num_sms;
    lim.smem = (int)kSmemMax;
    lim.integer = vt == VT_I32;
    lim.lanes = tri_lanes(c, t, vt);
    if (fixed_order(c, vt)) lim.lanes_log = __builtin_ctz(lim.lanes);
    return build_sweep_plan(t.rptr, t.cind, t.vals, (int)vt_size(vt), t.n, lim, t.level_hint);
}

static DevTri upload_tri(const Ctx &c, const TriSource &src, int vt, const SweepPlan &p) {
    const int n = src.n;
    const void *vals = src.vals;
    DevTri d;
    d.n = n;
    d.small = (size_t)n * vt_size(vt) <= kSmallSweep;
    d.kind = TRI_LD;
    d.vt = vt;
    d.bit = src.bit;
    d.dbit = src.dbit;
    d.nlev = p.nlev;
    d.max_level_rows = p.max_level_rows;
    d.nnz_off = p.nnz_off;
    if (p.ok()) {
        d.grid = p.blocks;
        d.warps = p.warps;
        d.importers = p.importers;
        d.lg = p.lg;
        d.lines = p.lines;
        d.virt = p.virt;
        // the small arrays in one buffer (blocks, streams, imports, groups), the
        // records in another
        std::vector<SweepBlock> bl(p.blocks);
        for (int b = 0; b < p.blocks; b++)
            bl[b] = SweepBlock{p.row0[b], p.row0[b + 1], p.imp_ptr[b], p.imp_ptr[b + 1], p.grp_ptr[b], p.grp_ptr[b + 1], p.steps[b], 0};
        std::vector<unsigned char> small;
        auto put = [&](const void *v, size_t bytes) {
            const size_t at = (small.size() + 15) / 16 * 16;
            small.resize(at + bytes + 16);
            if (bytes) memcpy(small.data() + at, v, bytes);
            return at;
        };
        const size_t o_bl = put(bl.data(), bl.size() * sizeof(SweepBlock)), o_st = put(p.stream.data(), p.stream.size() * 8),
                     o_im = put(p.imp_place.data(), p.imp_place.size() * 4), o_gr = put(p.grp.data(), p.grp.size() * 4);
        unsigned char *base = dupload(small);
        d.blocks = base + o_bl;
        d.stream = (long long *)(base + o_st);
        d.imp_place = (int *)(base + o_im);
        d.grp = (int *)(base + o_gr);
        const size_t rec = (size_t)p.quads * 512, bytes = (size_t)p.stream.back() * rec, pad = (kSweepAhead + 4) * rec;
        d.data = dmalloc(bytes + pad);
        SAGB_CUDA(cudaMemset((unsigned char *)d.data + bytes, 0, pad));
        SAGB_CUDA(cudaMemcpy(d.data, p.data.get(), bytes, cudaMemcpyHostToDevice));
        d.smem = sweep_fixed_smem(p.warps, p.quads) + (size_t)p.max_slots * vt_size(vt);
        if (p.blocks > 1 && !d.small) {
            const size_t words = (size_t)n * (vt == VT_F64 ? 2 : 1), all = sizeof(unsigned long long) * words + sizeof(TriSync);
            d.pk = (unsigned long long *)dmalloc(all);
            SAGB_CUDA(cudaMemset(d.pk, 0, all));
            d.sync = (TriSync *)(d.pk + words);
        }
        return d;
    }
    const TriSchedule &s = *p.levels;
    d.group = tri_lanes(c, src, vt);
    d.one_cta = p.one_cta;
    d.nlev = s.nlev;
    d.max_level_rows = s.max_level_rows;
    d.nnz_off = (int64_t)s.pci.size();
    d.nchunks = s.nchunks();
    std::vector<unsigned char> blob;
    std::vector<long long> off;
    auto put_vals = [&](auto tag) {
        using T = decltype(tag);
        std::vector<T> pv, dv;
        gather_vals(s, (const T *)vals, pv, dv);
        if (d.one_cta) {
            build_blocks(s, pv, dv, blob, off);
        } else {
            d.pval = pv.empty() ? dmalloc(16) : (void *)dupload(pv);
            d.dinv = dupload(dv);
        }
    };
    if (vt == VT_I32) put_vals(int32_t());
    else if (vt == VT_F64) put_vals(double());
    else put_vals(float());
    if (d.one_cta) {
        d.blocks = blob.empty() ? dmalloc(16) : (void *)dupload(blob);
        // block offsets in 16-byte units (nlev + 1), then the rows of each level (nlev)
        std::vector<unsigned> off16(off.size() + s.nlev);
        for (size_t i = 0; i < off.size(); i++) off16[i] = (unsigned)(off[i] / 16);
        for (int l = 0; l < s.nlev; l++) off16[off.size() + l] = (unsigned)(s.lvl_ptr[l + 1] - s.lvl_ptr[l]);
        d.blk_off = dupload(off16);
        d.stage_bytes = (int)((kSmemMax - cta_fixed_smem(n, (int)vt_size(vt), s.nlev)) / 16 * 16);
        d.smem = cta_fixed_smem(n, (int)vt_size(vt), s.nlev) + (size_t)d.stage_bytes;
        d.grid = 1;
        return d;
    }
    d.perm = dupload(s.perm);
    d.prp = dupload(s.prp);
    d.pci = s.pci.empty() ? (int *)dmalloc(16) : dupload(s.pci);
    d.chunk_lv = dupload(s.chunk_lv);
    d.sub_bound = dupload(s.sub_bound);
    d.grid = std::max(1, std::min(d.nchunks, c.num_sms));
    if (d.small) return d;
    if (vt == VT_F64) {
        d.flag = (unsigned *)dmalloc(sizeof(unsigned) * std::max(n, 1));
        SAGB_CUDA(cudaMemset(d.flag, 0, sizeof(unsigned) * std::max(n, 1)));
    } else {
        d.pk = (unsigned long long *)dmalloc(sizeof(unsigned long long) * std::max(n, 1));
        SAGB_CUDA(cudaMemset(d.pk, 0, sizeof(unsigned long long) * std::max(n, 1)));
    }
    d.sync = (TriSync *)dmalloc(sizeof(TriSync));
    SAGB_CUDA(cudaMemset(d.sync, 0, sizeof(TriSync)));
    return d;
}

std::vector<DevTri> upload_tris(const Ctx &c, const std::vector<TriSource> &src, int vt) {
    const int n = (int)src.size();
    std::vector<SweepPlan> plans(n);
    std::vector<std::exception_ptr> failed(n);
    auto plan = [&](int k) {
        try {
            plans[k] = plan_tri(c, src[k], vt);
        } catch (...) {
            failed[k] = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(n);
    for (int k = 0; k < n; k++) {
        try {
            pool.emplace_back(plan, k);
        } catch (const std::system_error &) {  // no more threads to be had
            plan(k);
        }
    }
    for (auto &t : pool) t.join();
    for (auto &f : failed)
        if (f) std::rethrow_exception(f);
    std::vector<DevTri> out;
    for (int k = 0; k < n; k++) {
        out.push_back(upload_tri(c, src[k], vt, plans[k]));
        plans[k] = SweepPlan();
    }
    return out;
}

template <int VT, int G, bool EXACT>
static void launch_tri(Ctx &c, const DevTri &T, const void *in, void *out) {
    c.launches++;
    if (T.one_cta) {
        k_tri_cta<VT, G, EXACT><<<1, kCtaThreads, T.smem, c.stream>>>((const unsigned char *)T.blocks, T.blk_off, T.nlev, T.n, T.bit,
                                                                      T.dbit, T.stage_bytes, in, out, c.d_flags);
        return;
    }
    TriArgs a{T.n, T.nchunks, T.bit, T.dbit, T.perm, T.prp, T.pci, T.pval, T.dinv,
              T.chunk_lv, T.sub_bound, T.pk, T.flag, T.sync};
    if (T.small) {
        a.pk = c.sweep->pk;
        a.flag = c.sweep->flag;
        a.sync = &c.sweep->sync;
    }
    k_tri<VT, G, EXACT><<<T.grid, kTriThreads, 0, c.stream>>>(a, in, out, c.d_flags);
}

using SweepKernel = void (*)(SweepArgs, const void *, void *, unsigned *);
template <int VT, bool EXACT, int LG>
static SweepKernel sweep_kernel_of(int lines, int virt) {
    if constexpr (VT == VT_F32) {  // (eight entries a record)
        if constexpr (LG <= 4)
            if (virt == 1) return k_sweep<VT, EXACT, LG, 4, 2>;
        if constexpr (LG <= 3)
            if (virt == 2) return k_sweep<VT, EXACT, LG, 4, 4>;
        if constexpr (LG <= 2)
            if (virt == 3) return k_sweep<VT, EXACT, LG, 4, 8>;
    }
    return lines == 1 ? k_sweep<VT, EXACT, LG, 1> : lines == 2 ? k_sweep<VT, EXACT, LG, 2> : k_sweep<VT, EXACT, LG, 4>;
}
template <int VT, bool EXACT>
static SweepKernel sweep_kernel(int lg, int lines, int virt) {
    switch (lg) {
        case 0: return sweep_kernel_of<VT, EXACT, 0>(lines, virt);
        case 1: return sweep_kernel_of<VT, EXACT, 1>(lines, virt);
        case 2: return sweep_kernel_of<VT, EXACT, 2>(lines, virt);
        case 3: return sweep_kernel_of<VT, EXACT, 3>(lines, virt);
        case 4: return sweep_kernel_of<VT, EXACT, 4>(lines, virt);
        default: return sweep_kernel_of<VT, EXACT, 5>(lines, virt);
    }
}

template <int VT, bool EXACT>
static void tri_by_group(Ctx &c, const DevTri &T, const void *in, void *out) {
    if (T.data) {
        int ilog = 0;
        while (2 << ilog <= T.importers) ilog++;
        SweepArgs a{T.warps, ilog, T.bit, T.dbit, (const SweepBlock *)T.blocks, T.stream, (const uint4 *)T.data, T.imp_place,
                    T.grp, T.pk, T.sync};
        if (T.small) {
            a.pk = c.sweep->pk;
            a.sync = &c.sweep->sync;
        }
        sweep_kernel<VT, EXACT>(T.lg, T.lines, T.virt)<<<T.grid, 32 * (T.warps + T.importers), T.smem,
                                                 c.stream>>>(a, in, out, c.d_flags);
        c.launches++;
        return;
    }
    switch (T.group) {
        case 1: return launch_tri<VT, 1, EXACT>(c, T, in, out);
        case 2: return launch_tri<VT, 2, EXACT>(c, T, in, out);
        case 4: return launch_tri<VT, 4, EXACT>(c, T, in, out);
        case 8: return launch_tri<VT, 8, EXACT>(c, T, in, out);
        case 16: return launch_tri<VT, 16, EXACT>(c, T, in, out);
        default: return launch_tri<VT, 32, EXACT>(c, T, in, out);
    }
}

void trsv(Ctx &c, const DevTri &T, const void *in, void *out) {
    if (T.n == 0) return;
    if (T.vt == VT_I32) return tri_by_group<VT_I32, false>(c, T, in, out);
    if (T.vt == VT_F64) {
        if (c.fp_exact) return tri_by_group<VT_F64, true>(c, T, in, out);
        return tri_by_group<VT_F64, false>(c, T, in, out);
    }
    if (c.fp_exact) return tri_by_group<VT_F32, true>(c, T, in, out);
    return tri_by_group<VT_F32, false>(c, T, in, out);
}

// ================================================ sweep without allocation
//
// For callers that cannot allocate device memory while they solve (their GPU
// memory is already claimed by another allocator, or they cannot afford the
// device-wide synchronisation cudaMalloc/cudaFree imply).  A sweep by several CTAs
// needs per-row scratch (the packed {epoch, value} words and the ticket/epoch
// block); small levels have their context's (SweepScratch), larger ones take it
// here from the file-scope array below instead of the schedule's own allocation.
// The array is sized for kNoAllocRows rows (two words each for FP64: 4 MiB) and
// every GPU that loads the library holds it
// until the process exits.  All calls share it and it keeps the last call's
// contents, so before each call the words of this level's rows and the
// ticket, done and epoch counters are cleared (a previous call may have left
// words of another precision there): every call starts at epoch 1 against
// zeroed words.  Calls that overlap on the GPU race on this array.
constexpr int kNoAllocRows = 262144;
static __device__ __align__(256) unsigned long long g_noalloc_scratch[2 * kNoAllocRows + 2];

static std::mutex g_noalloc_mu;
static void *g_noalloc_addr[64];

// The array's device address, looked up once per device with that device
// current (in host code the symbol is only a host-side stand-in).
static unsigned long long *noalloc_scratch(int device) {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (device < 0 || device >= 64) throw CudaError{"device index out of range"};
    if (!g_noalloc_addr[device]) {
        int cur = -1;
        SAGB_CUDA(cudaGetDevice(&cur));
        if (cur != device) SAGB_CUDA(cudaSetDevice(device));
        void *p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if (cur != device) cudaSetDevice(cur);
        if (e != cudaSuccess || !p) throw CudaError{std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e)};
        g_noalloc_addr[device] = p;
    }
    return (unsigned long long *)g_noalloc_addr[device];
}

void trsv_noalloc(Ctx &c, const DevTri &T, const void *in, void *out) {
    if (T.n == 0 || T.small || (T.data && T.grid == 1)) return trsv(c, T, in, out);  // the context's scratch, or none
    if (T.n > kNoAllocRows)
        throw CudaError{"level has more than 262144 rows, the limit of the no-allocation sweep"};
    unsigned long long *s = noalloc_scratch(c.device);
    DevTri U = T;  // same schedule and operator, scratch from the static array
    U.pk = s;
    U.flag = (unsigned *)s;
    U.sync = (TriSync *)(s + 2 * kNoAllocRows);
    SAGB_CUDA(cudaMemsetAsync(s, 0, sizeof(unsigned long long) * (size_t)T.n * (T.vt == VT_F64 ? 2 : 1), c.stream));
    SAGB_CUDA(cudaMemsetAsync(U.sync, 0, sizeof(TriSync), c.stream));  // ticket, done, epoch
    if (U.vt == VT_I32) return tri_by_group<VT_I32, false>(c, U, in, out);
    if (U.vt == VT_F64) {
        if (c.fp_exact) return tri_by_group<VT_F64, true>(c, U, in, out);
        return tri_by_group<VT_F64, false>(c, U, in, out);
    }
    if (c.fp_exact) return tri_by_group<VT_F32, true>(c, U, in, out);
    return tri_by_group<VT_F32, false>(c, U, in, out);
}

// ======================================================== dense coarse LU
//
// LUflex::Solve / LU<T>::Solve (solver/lu.hpp:91-94, 30-33) by k_lu_chain (see
// lu_chain.cuh).  k_dense_lu, one CTA and 32-row panels, left looking, solves FP32
// (whose sums keep their order, see fixed_order; the chain took 64 us instead of 158
// at n = 1013), FP64 systems of one panel, the sequential-order mode and fixed-point
// shifts outside 0..31:
// warps reduce a panel's rows against the solved part, lanes over the columns (one
// thread a row in column order in the sequential-order mode), then a warp solves
// the diagonal block.  Its factors are stored row by row.
constexpr int kLuThreads = 1024;

template <int VT, bool EXACT>
__global__ void __launch_bounds__(kLuThreads, 1)
k_dense_lu(int n, const void *__restrict__ L_, const void *__restrict__ U_, const void *__restrict__ dinv_,
           int bitL, int bitU, int dbitU, const void *__restrict__ in_, void *__restrict__ out_, unsigned *flags) {
    using V = vt_t<VT>;
    using T = acc_t<VT>;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    T *t = (T *)smem_raw;                           // n accumulators
    V *x = (V *)(smem_raw + sizeof(T) * (size_t)n); // n solved values
    const V *L = (const V *)L_;
    const V *U = (const V *)U_;
    const V *dinv = (const V *)dinv_;
    const V *in = (const V *)in_;
    V *out = (V *)out_;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    bool ovf = false;

    // ---------------- forward: unit lower, t = in << bit
    for (int i = tid; i < n; i += kLuThreads) t[i] = acc_init<VT>(in[i], bitL);
    __syncthreads();
    for (int k0 = 0; k0 < n; k0 += 32) {
        const int kb = min(32, n - k0);
        // panel rows against columns [0, k0)
        if (k0 > 0) {
            if constexpr (EXACT && VT != VT_I32) {
                if (tid < kb) {
                    const V *row = L + (size_t)(k0 + tid) * n;
                    T acc = t[k0 + tid];
                    for (int c = 0; c < k0; c++) acc = acc_sub<VT, true>(acc, row[c], x[c]);
                    t[k0 + tid] = acc;
                }
            } else if (warp < kb) {
                const V *row = L + (size_t)(k0 + warp) * n;
                T acc = 0;
                for (int c = lane; c < k0; c += 32) acc = acc_sub<VT, false>(acc, __ldg(row + c), x[c]);
                acc = acc_reduce<VT>(acc, 32);
                if (lane == 0) {
                    if constexpr (VT == VT_I32) t[k0 + warp] = wadd(t[k0 + warp], acc);
                    else t[k0 + warp] += acc;
                }
            }
        }
        __syncthreads();
        if (warp == 0) {
            V dblk[32];
            const V *row = L + (size_t)(k0 + lane) * n + k0;
#pragma unroll
            for (int c = 0; c < 32; c++) dblk[c] = (lane < kb && c < lane) ? __ldg(row + c) : V(0);
            T tr = lane < kb ? t[k0 + lane] : T(0);
#pragma unroll
            for (int c = 0; c < 32; c++) {
                if (c < kb) {
                    V xc;
                    if constexpr (VT == VT_I32) {
                        const long long s = tr >> bitL;
                        if (lane == c) ovf |= !fits32(s);
                        xc = __shfl_sync(0xffffffffu, lo32(s), c);
                    } else {
                        xc = __shfl_sync(0xffffffffu, tr, c);
                    }
                    if (lane > c) tr = acc_sub<VT, EXACT>(tr, dblk[c], xc);
                    if (lane == c) x[k0 + c] = xc;
                }
            }
        }
        __syncthreads();
    }
    // ---------------- backward: D^-1 U, last panel first
    for (int i = tid; i < n; i += kLuThreads) t[i] = acc_init<VT>(x[i], bitU);
    __syncthreads();
    for (int k1 = n; k1 > 0; k1 -= 32) {
        const int kb = min(32, k1);
        const int k0 = k1 - kb;
        if (k1 < n) {
            if constexpr (EXACT && VT != VT_I32) {
                if (tid < kb) {
                    const V *row = U + (size_t)(k0 + tid) * n;
                    T acc = t[k0 + tid];
                    for (int c = n - 1; c >= k1; c--) acc = acc_sub<VT, true>(acc, row[c], x[c]);
                    t[k0 + tid] = acc;
                }
            } else if (warp < kb) {
                const V *row = U + (size_t)(k0 + warp) * n;
                T acc = 0;
                for (int c = k1 + lane; c < n; c += 32) acc = acc_sub<VT, false>(acc, __ldg(row + c), x[c]);
                acc = acc_reduce<VT>(acc, 32);
                if (lane == 0) {
                    if constexpr (VT == VT_I32) t[k0 + warp] = wadd(t[k0 + warp], acc);
                    else t[k0 + warp] += acc;
                }
            }
        }
        __syncthreads();
        if (warp == 0) {
            V dblk[32];
            const V *row = U + (size_t)(k0 + lane) * n + k0;
#pragma unroll
            for (int c = 0; c < 32; c++) dblk[c] = (lane < kb && c > lane && c < kb) ? __ldg(row + c) : V(0);
            T tr = lane < kb ? t[k0 + lane] : T(0);
            const V dv = lane < kb ? dinv[k0 + lane] : V(0);
#pragma unroll
            for (int c = 31; c >= 0; c--) {
                if (c < kb) {
                    V xc = V(0);
                    if (lane == c) xc = acc_finish<VT>(tr, dv, bitU, dbitU, ovf);
                    xc = __shfl_sync(0xffffffffu, xc, c);
                    if (lane < c) tr = acc_sub<VT, EXACT>(tr, dblk[c], xc);
                    if (lane == c) x[k0 + c] = xc;
                }
            }
        }
        __syncthreads();
    }
    for (int i = tid; i < n; i += kLuThreads) out[i] = x[i];
    if (ovf) atomicOr(flags, ST_OVERFLOW);
}

template <int VT>
__global__ void __launch_bounds__(32 * kLuWarps, 1) k_lu_chain(LuChain<VT> a, unsigned *flags) {
    lu_chain<VT, false>(a, flags);
}

void DevDenseLU::release() {
    dfree(L);
    dfree(U);
    dfree(Lb);
    dfree(Ub);
    dfree(dinv);
    L = U = Lb = Ub = dinv = nullptr;
}

// (FP64, one panel: there is nothing to hand to another CTA, and a step of the chain with
// the next panel's product takes 190 cycles; n = 2 / 13 / 32 by the cluster 10.8 us, by
// k_dense_lu 6.0 / 8.3 / 10.7)
static bool chain_takes(int vt, int bitL, int n) {
    return vt == VT_F64 ? n > 32 : vt == VT_I32 && bitL >= 0 && bitL < 32;
}

template <typename V>
static void upload_lu(DevDenseLU &d, const int *Lrptr, const int *Lcind, const V *Lval, const int *Urptr,
                      const int *Ucind, const V *Uval) {
    const int n = d.n;
    std::vector<V> dinv(std::max(n, 1), V(0));
    for (int i = 0; i < n; i++)  // dutri rows: D^-1 first, then the strict upper entries
        if (Urptr[i + 1] > Urptr[i]) dinv[i] = Uval[Urptr[i]];
    if (chain_takes(d.vt, d.bitL, d.n)) {
        LuBlocks<V> B(n);
        B.dinv = dinv;
        for (int i = 0; i < n; i++) {
            for (int j = Lrptr[i]; j < Lrptr[i + 1]; j++)
                if (Lcind[j] < i) B.L[B.lower(i, Lcind[j])] = Lval[j];
            for (int j = Urptr[i] + 1; j < Urptr[i + 1]; j++)
                if (Ucind[j] > i) B.U[B.upper(i, Ucind[j])] = Uval[j];
        }
        if (d.vt == VT_F64) B.scale_columns();
        d.Lb = dupload(B.L);
        d.Ub = dupload(B.U);
    }
    if (d.vt != VT_I32 || !d.Lb) {
        std::vector<V> L((size_t)std::max(n, 1) * n + 1, V(0)), U(L);
        for (int i = 0; i < n; i++) {
            for (int j = Lrptr[i]; j < Lrptr[i + 1]; j++) L[(size_t)i * n + Lcind[j]] = Lval[j];
            for (int j = Urptr[i] + 1; j < Urptr[i + 1]; j++) U[(size_t)i * n + Ucind[j]] = Uval[j];
        }
        d.L = dupload(L);
        d.U = dupload(U);
    }
    d.dinv = dupload(dinv);
}

DevDenseLU upload_dense_lu(const int *Lrptr, const int *Lcind, const void *Lval, const int *Urptr,
                           const int *Ucind, const void *Uval, int n, int vt, int bitL, int bitU, int dbitU) {
    DevDenseLU d;
    d.n = n;
    d.vt = vt;
    d.bitL = bitL;
    d.bitU = bitU;
    d.dbitU = dbitU;
    if (vt == VT_I32) upload_lu(d, Lrptr, Lcind, (const int32_t *)Lval, Urptr, Ucind, (const int32_t *)Uval);
    else if (vt == VT_F64) upload_lu(d, Lrptr, Lcind, (const double *)Lval, Urptr, Ucind, (const double *)Uval);
    else upload_lu(d, Lrptr, Lcind, (const float *)Lval, Urptr, Ucind, (const float *)Uval);
    return d;
}

template <int VT>
static void launch_chain(Ctx &c, const DevDenseLU &LU, const void *in, void *out) {
    using V = vt_t<VT>;
    LuChain<VT> a;
    a.n = LU.n;
    a.L = (const V *)LU.Lb;
    a.U = (const V *)LU.Ub;
    a.dinv = (const V *)LU.dinv;
    a.bitL = LU.bitL;
    a.bitU = LU.bitU;
    a.dbitU = LU.dbitU;
    a.in = (const V *)in;
    a.out = (V *)out;
    a.ld = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(kLuCtas);
    cfg.blockDim = dim3(32 * kLuWarps);
    cfg.dynamicSmemBytes = lu_smem<VT>((LU.n + 31) / 32).bytes;
    cfg.stream = c.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kLuCtas;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    SAGB_CUDA(cudaLaunchKernelEx(&cfg, k_lu_chain<VT>, a, c.d_flags));
}

template <int VT, bool EXACT>
static void launch_lu(Ctx &c, const DevDenseLU &LU, const void *in, void *out) {
    c.launches++;
    if constexpr (!EXACT && VT != VT_F32) {
        if (chain_takes(VT, LU.bitL, LU.n)) return launch_chain<VT>(c, LU, in, out);
    }
    const size_t smem = (sizeof(acc_t<VT>) + sizeof(vt_t<VT>)) * (size_t)LU.n;
    k_dense_lu<VT, EXACT><<<1, kLuThreads, smem, c.stream>>>(LU.n, LU.L, LU.U, LU.dinv, LU.bitL, LU.bitU,
                                                                LU.dbitU, in, out, c.d_flags);
}

template <int VT, bool EXACT>
static void cta_attrs() {
    const int mx = (int)kSmemMax;
    for (int lg = 0; lg <= 5; lg++)
        for (int lines = 1; lines <= 4; lines *= 2)
            for (int virt = 0; virt <= (VT == VT_F32 && lines == 4 ? std::min(3, 5 - lg) : 0); virt++)
                SAGB_CUDA(cudaFuncSetAttribute(sweep_kernel<VT, EXACT>(lg, lines, virt), cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_tri_cta<VT, 1, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_tri_cta<VT, 2, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_tri_cta<VT, 4, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_tri_cta<VT, 8, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_tri_cta<VT, 16, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_tri_cta<VT, 32, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    SAGB_CUDA(cudaFuncSetAttribute(k_dense_lu<VT, EXACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, mx));
    if constexpr (!EXACT && VT != VT_F32)
        SAGB_CUDA(cudaFuncSetAttribute(k_lu_chain<VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLuChainSmem));
}

void init_kernel_attributes() {
    cta_attrs<VT_I32, false>();
    cta_attrs<VT_F64, false>();
    cta_attrs<VT_F64, true>();
    cta_attrs<VT_F32, false>();
    cta_attrs<VT_F32, true>();
}

void lu_solve(Ctx &c, const DevDenseLU &LU, const void *in, void *out) {
    if (LU.n == 0) return;
    if ((size_t)LU.n * 16 > kSmemMax) throw CudaError{"coarsest level too large for the dense LU kernel"};
    if (LU.vt == VT_I32) return launch_lu<VT_I32, false>(c, LU, in, out);
    if (LU.vt == VT_F64) return c.fp_exact ? launch_lu<VT_F64, true>(c, LU, in, out)
                                           : launch_lu<VT_F64, false>(c, LU, in, out);
    return c.fp_exact ? launch_lu<VT_F32, true>(c, LU, in, out) : launch_lu<VT_F32, false>(c, LU, in, out);
}

}  // namespace sagb
