#include "tri_cost.hpp"

#include <algorithm>
#include <functional>
#include <queue>

namespace sagb {

double cta_us(const TriSchedule &s, int lanes, int es) {
    const int rows = (kCtaThreads / 32 - 1) * (32 / lanes);  // of a pass
    int64_t passes = 0, rounds = 0;
    for (int l = 0; l < s.nlev; l++)
        for (int p = s.lvl_ptr[l]; p < s.lvl_ptr[l + 1]; p += rows, passes++) {
            int longest = 0;
            for (int q = p; q < std::min(s.lvl_ptr[l + 1], p + rows); q++) longest = std::max(longest, s.prp[q + 1] - s.prp[q]);
            rounds += (longest + 4 * lanes - 1) / (4 * lanes);
        }
    const double row = 0.04e-3 * s.n, entry = s.prp[s.n] * 1e-3;
    return es == 8 ? 2.1 + 0.06 * s.nlev + 0.54 * passes + 0.23 * rounds + 0.51 * entry
                   : 2.1 + 0.30 * s.nlev + 0.37 * passes + 0.08 * rounds + 0.17 * entry + row;
}

double spread_us(const TriSchedule &s, int lanes, int es, int ctas) {
    const double round = es == 8 ? 3.0 : 0.95, pass = 0.4, claim = 0.5;
    constexpr int kWarps = kTriThreads / 32;
    const int rows = 32 / lanes, batch = kTriBatch * lanes;
    std::vector<double> done(s.n, 0.0);  // when each row's value is there
    std::priority_queue<double, std::vector<double>, std::greater<double>> idle(std::greater<double>(),
                                                                                std::vector<double>(ctas, 0.0));
    double end = 0;
    for (int c = 0; c < s.nchunks(); c++) {
        double t = idle.top() + claim;
        idle.pop();
        for (int sub = s.chunk_lv[c]; sub < s.chunk_lv[c + 1]; sub++) {
            double warp[kWarps];
            std::fill(warp, warp + kWarps, t);
            const int p1 = s.sub_bound[sub + 1];
            int w = 0;
            for (int p = s.sub_bound[sub]; p < p1; p += rows, w = (w + 1) % kWarps) {
                const int q1 = std::min(p1, p + rows);
                int longest = 0;
                for (int q = p; q < q1; q++) longest = std::max(longest, s.prp[q + 1] - s.prp[q]);
                double now = warp[w] + pass;
                for (int j0 = 0; j0 < longest; j0 += batch) {
                    for (int q = p; q < q1; q++)
                        for (int j = s.prp[q] + j0; j < std::min(s.prp[q + 1], s.prp[q] + j0 + batch); j++) now = std::max(now, done[s.pci[j]]);
                    now += round;
                }
                for (int q = p; q < q1; q++) done[s.perm[q]] = now;
                warp[w] = now;
            }
            t = *std::max_element(warp, warp + kWarps);
        }
        idle.push(t);
        end = std::max(end, t);
    }
    return 4.0 + 0.93 * end;
}

}  // namespace sagb
