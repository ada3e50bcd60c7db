#include "sweep_plan.hpp"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <mutex>
#include <system_error>
#include <thread>

#include "csr.hpp"

namespace sagb {

namespace {

int threads_for(int n, int64_t work) {  // a thread pays from about 20,000 units of work (rows and entries)
    return (int)std::max<int64_t>(1, std::min<int64_t>({n, (int64_t)std::thread::hardware_concurrency(), work / 20000}));
}
// f(i) for i < n on T threads
template <typename F>
void on_threads(int T, int n, F &&f) {
    std::atomic<int> next(0);
    std::exception_ptr first;
    std::mutex mu;
    auto work = [&] {
        try {
            for (int i; (i = next++) < n;) f(i);
        } catch (...) {
            std::lock_guard<std::mutex> g(mu);
            if (!first) first = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(T);
    try {
        for (int t = 1; t < T; t++) pool.emplace_back(work);
    } catch (const std::system_error &) {  // no more threads to be had: fewer do it
    }
    work();
    for (auto &th : pool) th.join();
    if (first) std::rethrow_exception(first);
}

struct Triangle {
    const int *rptr, *cind;
    const unsigned char *vals;
    int es, n;
    int begin(int i) const { return rptr[i]; }
    int len(int i) const { return std::max(0, rptr[i + 1] - 1 - rptr[i]); }
    bool has_diag(int i) const { return rptr[i + 1] > rptr[i]; }
};

// What a step of one block costs, in cycles: a model that the plan's shape is
// picked with, fitted to 5,300 timed sweeps on one GB300 (Poisson, lognormal,
// convection-diffusion and 27-point levels of 2,000 to 2,000,000 rows, every warp
// count, lanes a row and record size, 1 to 152 blocks).  It is 8 % off on
// average; its pick is 4 % slower than the fastest of those.
struct Costs {
    double record, line, round, sum32;  // a record; a pair of entries a lane; a shuffle round; 32 lanes
};
constexpr Costs kCostInt = {102, 13, 25, 58};  // (32 integer lanes: three REDUX)
constexpr Costs kCostF32 = {178, 20, 35, 176};
constexpr Costs kCostF64 = {295, 71, 122, 610};
constexpr double kCostStep = 150, kCostWarp = 7.7;  // a step; each warp at its barrier
constexpr double kCostSlot = 4.8;   // shared memory: each entry of a lane, over all records of the step
constexpr double kCostImport = 84;  // a step that waits for imports
constexpr double kCostFetch = 1.5;  // an import
constexpr double kCostHop = 1490;   // a value published by one block and used by the next (0.8 us)
constexpr double kCostBytes = 21;   // bytes of records one CTA streams a cycle (40 GB/s)

struct Shape {
    int blocks = 0, warps = 1, lg = 0, lines = 1;
    double cost = 1e300;
    double queued = 0;  // records after the third of a warp and step, in the slowest block of each step
};

// A shape's time in us, to compare it with the other kernels': the launch, the
// cycles, and what the model above leaves out because it hardly differs between
// shapes: a step with many records a warp waits for their copies, of which
// kSweepStage - 1 are on their way.
double sweep_us(const Shape &s, int es, bool integer) {
    const double cycles = es == 8 ? 1.0 : integer ? 0.87 : 0.66, record = es == 8 ? 0.11 : integer ? 0.053 : 0.031;
    return 4.3 + cycles * s.cost / 1900 + record * s.queued;
}
// The estimates are 10 to 15 % off, so k_tri_cta, where the vector fits it, and k_tri
// elsewhere are left where another kernel promises 12 % less (k_tri for k_tri_cta: 20 %,
// its estimate is the roughest).  Over the levels that the estimates were fitted to, the
// kernel picked then took at most 1.13 times as long as the one left, but for one level
// of 1.27.
constexpr double kCostMargin = 0.88, kCostSpread = 1.1;

// first row of each of P blocks: rows weighted by their entries and three more
std::vector<int> cut_rows(const int *rptr, int n, int P) {
    std::vector<int> row0(P + 1, 0);
    const double total = (double)rptr[n] + 3.0 * n;
    int i = 0;
    for (int b = 1; b < P; b++) {
        int lo = i, hi = n;
        while (lo < hi) {
            const int mid = lo + (hi - lo) / 2;
            if ((double)rptr[mid] + 3.0 * mid < total * b / P) lo = mid + 1;
            else hi = mid;
        }
        row0[b] = i = lo;
    }
    row0[P] = n;
    return row0;
}

// the cheapest shape with P blocks: a level takes as long as its slowest block
// (the mean over some levels); by_level, level_ptr: the rows level by level
Shape pick_shape(const Triangle &A, const std::vector<int> &by_level, const std::vector<int> &level_ptr,
                 const std::vector<int> &row0, int reach, const SweepLimits &lim) {
    const int P = (int)row0.size() - 1, nlev = (int)level_ptr.size() - 1;
    const int stride = std::max(1, nlev / std::max(16, std::min(64, 1024 / P))), kept = (nlev + stride - 1) / stride;
    struct Step {
        int level, rows, longest, entries;
    };
    std::vector<Step> steps;
    double work_kept = 0;
    for (int k = 0; k < kept; k++) {
        int b = -1;
        for (int j = level_ptr[k * stride]; j < level_ptr[k * stride + 1]; j++) {
            const int i = by_level[j], len = A.len(i);
            if (b < 0 || i >= row0[b + 1]) {  // (a level's rows are in increasing order)
                b = (int)(std::upper_bound(row0.begin() + b + 1, row0.end(), i) - row0.begin()) - 1;
                steps.push_back(Step{k, 0, 0, 0});
            }
            Step &q = steps.back();
            q.rows++;
            q.longest = std::max(q.longest, len);
            q.entries += len;
            work_kept += len + 1;
        }
    }
    const double work = (double)A.rptr[A.n];
    // a block reads up to `reach` rows before it, over all its steps
    const double fetch = P > 1 ? kCostFetch * reach * P / ((double)steps.size() * stride) : 0;
    const Costs &c = A.es == 8 ? kCostF64 : lim.integer ? kCostInt : kCostF32;
    Shape best;
    best.blocks = P;
    std::vector<double> slowest(kept);
    // (a lane that stands for several takes eight entries a record, one or more of each)
    for (int lg = std::max(lim.lanes_log - 3, 0); lg <= (lim.lanes_log >= 0 ? lim.lanes_log : 5); lg++)
        for (int lines = lg < lim.lanes_log ? 4 : 1; lines <= 4; lines *= 2)
            for (int w = 2; w <= kSweepMaxWarps; w *= 2) {
                const int per = 32 >> lg, lane = 2 * lines << lg;
                const double rec = c.record + c.line * lines + (lg == 5 ? c.sum32 : c.round * lg);
                double records = 0;
                std::fill(slowest.begin(), slowest.end(), 0.0);
                for (const Step &q : steps) {
                    const int tasks = (q.rows + per - 1) / per;
                    const int first = std::max(1, (q.longest + lane - 1) / lane);
                    const double rest = std::max(1.0, (double)q.entries / q.rows / lane);
                    const double all = first + (tasks - 1) * rest;
                    const double cycles = kCostStep + kCostWarp * w + rec * (first + ((tasks + w - 1) / w - 1) * rest) +
                                          kCostSlot * 2 * lines * all + (P > 1 ? kCostImport : 0);
                    slowest[q.level] = std::max(slowest[q.level], std::max(cycles, fetch));
                    records += all;
                }
                double step = 0;
                for (double v : slowest) step += v / kept;
                const double bytes = records * (work / work_kept) * (1 + lines + (A.es == 8)) * 512;
                const double waves = std::max(1.0, (double)P / lim.sms);
                const double cost = std::max(nlev * step * waves, bytes / kCostBytes / std::min(P, lim.sms)) +
                                    (kCostHop + fetch) * (P - 1);
                if (cost < best.cost) {
                    best.cost = cost;
                    best.warps = w;
                    best.lg = lg;
                    best.lines = lines;
                }
            }
    const int per = 32 >> best.lg, lane = 2 * best.lines << best.lg;
    std::fill(slowest.begin(), slowest.end(), 0.0);
    for (const Step &q : steps) {
        const int tasks = (q.rows + per - 1) / per, first = std::max(1, (q.longest + lane - 1) / lane);
        const double rest = std::max(1.0, (double)q.entries / q.rows / lane);
        slowest[q.level] = std::max(slowest[q.level], first + ((tasks + best.warps - 1) / best.warps - 1) * rest);
    }
    for (double v : slowest) best.queued += std::max(0.0, v - (kSweepStage - 1)) * nlev / kept;
    return best;
}

struct Plan {  // what the blocks of one plan share
    const Triangle &A;
    const std::vector<int> &level;
    const std::vector<int> &sorted, &place;  // rows block by block, level by level; where each row is there
    const std::vector<unsigned char> &exported;
    int warps, lg, lines, quads;
    int reach;  // a row reads at most this far back
};

// one record: rows order[k] .. order[k + here) of the block, part `part` of them
// (here 0: an empty record)
struct Record {
    int k, here, part;
    uint32_t bits;  // of the control word
};

struct Block {
    int b0 = 0, b1 = 0, steps = 0;
    std::vector<int> order;         // its rows, level by level, the longest first
    std::vector<int> seen;          // import index of row b0 - reach + k, -1 for none
    std::vector<int> imports, grp;  // imported rows in the order of first use, in groups
    std::vector<std::vector<Record>> records;  // per warp

    uint32_t number(const Plan &p, int c) const {  // slot of row c
        return (uint32_t)(c >= b0 ? c - b0 : b1 - b0 + seen[c - b0 + p.reach]);
    }

    // imports and records of rows [first, last)
    void build(const Plan &p, int first, int last) {
        const Triangle &A = p.A;
        b0 = first;
        b1 = last;
        const int rows = b1 - b0;
        order.assign(p.sorted.begin() + b0, p.sorted.begin() + b1);
        seen.assign(b0 > 0 ? p.reach : 0, -1);
        auto slot = [&](int c) -> int & { return seen[c - b0 + p.reach]; };
        // a group of at most kSweepGroup imports for one level, by their places
        grp.assign(1, 0);
        std::vector<int> found, need;  // need: groups each level asks for
        for (int q = 0; q < rows;) {
            const int lv = p.level[order[q]], q0 = q;
            found.clear();
            for (; q < rows && p.level[order[q]] == lv; q++)
                for (int j = A.begin(order[q]), e = j + A.len(order[q]); j < e; j++) {
                    const int c = A.cind[j];
                    if (c >= b0 || slot(c) >= 0) continue;
                    slot(c) = 0;
                    found.push_back(c);
                }
            std::sort(found.begin(), found.end(), [&](int x, int y) { return p.place[x] < p.place[y]; });
            for (int c : found) {
                slot(c) = (int)imports.size();
                imports.push_back(c);
                if ((int)imports.size() - grp.back() > kSweepGroup) grp.push_back((int)imports.size() - 1);
            }
            if ((int)imports.size() > grp.back()) grp.push_back((int)imports.size());
            // (rows of a level read rows of earlier levels: all imports so far)
            need.push_back((int)grp.size() - 1);
            const auto longer = [&](int x, int y) { return A.len(x) > A.len(y); };
            if (!std::is_sorted(order.begin() + q0, order.begin() + q, longer))
                std::stable_sort(order.begin() + q0, order.begin() + q, longer);
        }
        records.resize(p.warps);
        std::vector<int> at(p.warps, 0), got(p.warps, 0);  // barriers passed and groups asked for by each warp
        const int per = 32 >> p.lg, lane = 2 * p.lines << p.lg;
        for (int q = 0; q < rows; steps++) {
            const int lv = p.level[order[q]], q0 = q;
            while (q < rows && p.level[order[q]] == lv) q++;
            for (int t = 0, k = q0; k < q; t++, k += per) {
                const int w = t % p.warps;
                std::vector<Record> &out = records[w];
                // what does not fit the control word's fields goes into empty records
                while (steps - at[w] > 128 || need[steps] - got[w] > 127) {
                    const int nb = std::min(127, steps - at[w]), ng = std::min(127, need[steps] - got[w]);
                    out.push_back(Record{0, 0, 0, (uint32_t)nb << 18 | (uint32_t)ng << 25});
                    at[w] += nb;
                    got[w] += ng;
                }
                const int parts = std::max(1, (A.len(order[k]) + lane - 1) / lane), nb = steps - at[w];
                for (int part = 0; part < parts; part++) {
                    uint32_t bits = (uint32_t)(part < parts - 1) << 16;
                    if (part == 0)
                        bits |= (uint32_t)(nb > 0) << 17 | (uint32_t)std::max(0, nb - 1) << 18 | (uint32_t)(need[steps] - got[w]) << 25;
                    out.push_back(Record{k, std::min(per, q - k), part, bits});
                }
                at[w] = steps;
                got[w] = need[steps];
            }
        }
    }

    // writes one record (empty: the record of spare rows and entries of zero)
    void write(const Plan &p, const Record &rec, const SweepQuad *empty, SweepQuad *r) const {
        const Triangle &A = p.A;
        const int G = 1 << p.lg;
        memcpy(r, empty, (size_t)p.quads * 32 * sizeof(SweepQuad));
        const bool last = !(rec.bits & (1u << 16));
        for (int lane = 0; lane < rec.here * G; lane++) {
            const int row = order[rec.k + (lane >> p.lg)], g = lane & (G - 1), n = A.len(row), e0 = A.begin(row);
            r[lane].v[0] = (uint32_t)(row - b0);
            if (last) {
                if (p.exported[row]) r[lane].v[1] = (uint32_t)p.place[row];
                if (A.has_diag(row)) memcpy(&r[lane].v[2], A.vals + (size_t)(A.rptr[row + 1] - 1) * A.es, A.es);
            }
            for (int h = 0; h < 2 * p.lines; h++) {
                const int j = g + (rec.part * 2 * p.lines + h) * G;
                if (j >= n) break;
                const uint32_t num = number(p, A.cind[e0 + j]);
                SweepQuad &v = r[32 * (1 + h / 2) + lane];
                if (A.es == 4) {
                    v.v[2 * (h & 1)] = num * 4;
                    memcpy(&v.v[2 * (h & 1) + 1], A.vals + (size_t)(e0 + j) * 4, 4);
                } else {
                    memcpy(&v.v[2 * (h & 1)], A.vals + (size_t)(e0 + j) * 8, 8);
                    uint32_t &o = r[32 * (1 + p.lines) + lane].v[h / 2];
                    o = h & 1 ? (o & 0xffffu) | num << 16 : (o & 0xffff0000u) | num;
                }
            }
        }
        for (int k = 0; k < 32; k++) r[k].v[0] |= rec.bits;
    }

    std::vector<SweepQuad> empty_record(const Plan &p) const {
        const uint32_t zero = (uint32_t)(b1 - b0 + (int)imports.size()), spare = zero + 1;
        std::vector<SweepQuad> r((size_t)p.quads * 32, SweepQuad{{0u, 0u, 0u, 0u}});
        for (int k = 0; k < 32; k++) r[k] = SweepQuad{{spare, ~0u, 0u, 0u}};
        if (p.A.es == 4)
            for (int k = 32; k < 32 * (1 + p.lines); k++) r[k] = SweepQuad{{zero * 4, 0u, zero * 4, 0u}};
        else
            for (int k = 32 * (1 + p.lines); k < 32 * p.quads; k++)
                for (int h = 0; h < 4; h++) r[k].v[h] = zero | zero << 16;
        return r;
    }
};

}  // namespace

SweepPlan build_sweep_plan(const int *rptr, const int *cind, const void *vals, int es, int n, const SweepLimits &lim,
                           const int *level_hint) {
    SweepPlan s;
    s.n = n;
    const Triangle A{rptr, cind, (const unsigned char *)vals, es, n};
    std::vector<int> level(n, 0);
    bool lower = true;  // every row reads earlier rows only
    int reach = 0;      // how far back
    int nlev = 0;       // levels of the dependencies
    for (int i = 0; i < n; i++) {
        int lv = 0;
        for (int j = A.begin(i), e = j + A.len(i); j < e; j++) {
            const int c = cind[j];
            if (c >= i) lower = false;
            else reach = std::max(reach, i - c);
            if (level_hint && level_hint[c] >= level_hint[i]) throw SetupError{"level hint violates a dependency"};
            if (c < i) lv = std::max(lv, level[c] + 1);
        }
        level[i] = lv;
        nlev = std::max(nlev, lv + 1);
        s.nlev = std::max(s.nlev, (level_hint ? level_hint[i] : lv) + 1);
        s.nnz_off += A.len(i);
    }
    // the rows level by level for the kernels that go that way
    auto by_levels = [&]() -> const TriSchedule & {
        s.levels.reset(new TriSchedule(build_tri_schedule(rptr, cind, n, TRI_LD, 2 * kTriThreads / lim.lanes, 1 << 20, level_hint)));
        return *s.levels;
    };
    const bool one_cta = cta_fits(n, es, s.nlev, lim.smem);
    if (n == 0 || (!lower && !level_hint)) {  // (not a lower triangle)
        by_levels();
        s.one_cta = one_cta;
        return s;
    }
    {
        std::vector<int> count(s.nlev, 0);
        for (int i = 0; i < n; i++)
            s.max_level_rows = std::max(s.max_level_rows, ++count[level_hint ? level_hint[i] : level[i]]);
    }
    // the steps follow the dependencies themselves where rows read earlier rows
    // only (chunks of rows: fewer levels than chunks), else the hint
    if (!lower) {
        level.assign(level_hint, level_hint + n);
        nlev = s.nlev;
    }

    // the rows level by level
    std::vector<int> level_ptr(nlev + 1, 0), by_level(n);
    for (int i = 0; i < n; i++) level_ptr[level[i] + 1]++;
    for (int l = 0; l < nlev; l++) level_ptr[l + 1] += level_ptr[l];
    {
        std::vector<int> at(level_ptr.begin(), level_ptr.end() - 1);
        for (int i = 0; i < n; i++) by_level[at[level[i]]++] = i;
    }
    // the shape: candidate block counts that fit the shared memory, each at its best
    std::vector<int> counts;
    for (int p = 1; p <= 4096; p *= 2) {
        counts.push_back(p);
        if (p < lim.sms * 2 / 3 && 2 * p > lim.sms * 2 / 3) counts.push_back(lim.sms * 2 / 3);
        if (p < lim.sms && 2 * p > lim.sms) counts.push_back(lim.sms);
    }
    std::vector<Shape> shapes(counts.size());
    const int64_t room = (lim.smem - sweep_fixed_smem(kSweepMaxWarps, 3)) / es;
    const double least = (double)n / std::max<int64_t>(room, 1);
    on_threads(threads_for((int)counts.size(), s.nnz_off + n), (int)counts.size(), [&](int k) {
        const int p = counts[k];
        if (p > std::max(1, n / 128) || (p > 1 && !lower) || p < least || (p > lim.sms && p > 8 * least)) return;
        const std::vector<int> row0 = cut_rows(rptr, n, p);
        int64_t most = 0;
        for (int b = 0; b < p; b++) {
            if (row0[b + 1] <= row0[b]) return;
            most = std::max<int64_t>(most, row0[b + 1] - row0[b] + std::min(reach, row0[b]) + 2);
        }
        if (most > std::min<int64_t>(room, kSweepMaxSlots)) return;
        shapes[k] = pick_shape(A, by_level, level_ptr, row0, reach, lim);
    });
    Shape sh;
    for (const Shape &q : shapes)
        if (q.blocks > 0 && q.cost < sh.cost) sh = q;
    // Few levels of many rows (colours, chunks, orders with short chains): a level is
    // work for more warps than a block has (k_tri_cta: 31) or for all SMs (k_tri).  us
    // by blocks / one CTA / all SMs: int 4,900 rows in two colours 12.0 / 6.7 / 8.0,
    // 45,000 rows in four 74 / - / 17; FP64 10,388 rows in 17 colours 116 / 104 / 496,
    // 98,769 rows in 83 chunks 182 / - / 1,895.
    const double by_blocks = sh.blocks ? sweep_us(sh, es, lim.integer) : 1e300;
    const double bias = one_cta ? kCostSpread : kCostMargin;
    if (by_blocks >= bias * spread_least_us(nlev, es) || (one_cta && by_blocks >= kCostMargin * cta_least_us(s.nlev, es))) {
        const TriSchedule &t = by_levels();
        const double cta = one_cta ? kCostMargin * cta_us(t, lim.lanes, es) : 1e300;
        const double spread = !one_cta && sh.blocks == 0 ? 0.0 : bias * spread_us(t, lim.lanes, es, lim.sms);
        s.one_cta = cta <= spread;
        if (std::min(cta, spread) <= by_blocks) return s;
        s.one_cta = false;
        s.levels.reset();
    }
    const int P = sh.blocks, W = sh.warps;
    s.lg = sh.lg;
    s.lines = sh.lines;
    s.virt = lim.lanes_log > sh.lg ? lim.lanes_log - sh.lg : 0;
    s.quads = 1 + s.lines + (es == 8);
    s.row0 = cut_rows(rptr, n, P);
    std::vector<unsigned char> exported(n, 0);
    if (P > 1)
        on_threads(threads_for(P, s.nnz_off), P, [&](int b) {
            for (int i = s.row0[b]; i < s.row0[b + 1]; i++)
                for (int j = A.begin(i), e = j + A.len(i); j < e; j++)
                    if (cind[j] < s.row0[b])
                        reinterpret_cast<std::atomic<unsigned char> *>(&exported[cind[j]])->store(1, std::memory_order_relaxed);
        });
    std::vector<int> sorted(n), place(n);
    {
        std::vector<int> at(s.row0.begin(), s.row0.end() - 1), block(n);
        for (int b = 0; b < P; b++) std::fill(block.begin() + s.row0[b], block.begin() + s.row0[b + 1], b);
        for (int i : by_level) {
            place[i] = at[block[i]]++;
            sorted[place[i]] = i;
        }
    }
    const Plan plan{A, level, sorted, place, exported, W, s.lg, s.lines, s.quads, reach};
    std::vector<Block> blocks(P);
    on_threads(threads_for(P, 2 * (s.nnz_off + n)), P, [&](int b) { blocks[b].build(plan, s.row0[b], s.row0[b + 1]); });
    s.imp_ptr.assign(1, 0);
    s.grp_ptr.assign(1, 0);
    s.stream.assign(1, 0);
    for (const Block &q : blocks) {
        for (int c : q.imports) s.imp_place.push_back(place[c]);
        s.imp_ptr.push_back((int)s.imp_place.size());
        s.grp.insert(s.grp.end(), q.grp.begin(), q.grp.end());
        s.grp_ptr.push_back((int)s.grp.size());
        s.steps.push_back(q.steps);
        s.max_slots = std::max(s.max_slots, q.b1 - q.b0 + (int)q.imports.size() + 2);
        for (const auto &w : q.records) s.stream.push_back(s.stream.back() + (int64_t)w.size());
    }
    const int64_t own = (int64_t)rptr[n] * (4 + es) + 4ll * n, most = std::max(lim.record_bytes, kSweepRecordShare * own);
    if (s.max_slots > kSweepMaxSlots || (int64_t)s.max_slots * es + sweep_fixed_smem(W, s.quads) > lim.smem ||
        s.stream.back() * s.quads * 512 > most) {
        by_levels();
        s.one_cta = one_cta;
        return s;
    }
    // the records, in pieces of a few hundred
    struct Piece {
        int block, warp, from, to;
    };
    std::vector<Piece> pieces;
    std::vector<std::vector<SweepQuad>> empty(P);
    for (int b = 0; b < P; b++) {
        empty[b] = blocks[b].empty_record(plan);
        for (int w = 0; w < W; w++)
            for (int k = 0, m = (int)blocks[b].records[w].size(); k < m; k += 256) pieces.push_back(Piece{b, w, k, std::min(m, k + 256)});
    }
    const size_t rec = (size_t)s.quads * 32;
    s.data.reset(new SweepQuad[(size_t)s.stream.back() * rec]);
    on_threads(threads_for((int)pieces.size(), s.stream.back() * 32), (int)pieces.size(), [&](int i) {
        const Piece &q = pieces[i];
        SweepQuad *out = s.data.get() + (size_t)s.stream[(size_t)q.block * W + q.warp] * rec;
        for (int k = q.from; k < q.to; k++)
            blocks[q.block].write(plan, blocks[q.block].records[q.warp][k], empty[q.block].data(), out + (size_t)k * rec);
    });
    s.blocks = P;
    s.warps = W;
    // warps that fetch imports: by the imports of a step (Poisson 128^3, levels 0
    // and 1 with 65 a step: 287 and 358 us with 4, 228 and 303 us with 8; levels
    // with fewer than 20 a step lose up to 2 % to the other warps' polling)
    int64_t steps = 0;
    for (int q : s.steps) steps += q;
    const double imports_a_step = (double)s.imp_place.size() / std::max<int64_t>(1, steps);
    s.importers = P == 1 ? 0 : imports_a_step >= 24 ? 8 : imports_a_step >= 6 ? 4 : 2;
    return s;
}

}  // namespace sagb
