// Random sets of systems: every one is placed in some launch, each CTA at most `depth` at a
// time, and with true times unlike the estimates (at most T each) no CTA waits longer than
// (depth - 1) T for its group.
#include "resident_queues.h"

#include <cmath>
#include <cstdio>
#include <random>
#include <set>

int main() {
    std::mt19937 rng(11);
    auto uniform = [&] { return std::uniform_real_distribution<double>(0, 1)(rng); };
    double longest = 0;
    for (int run = 0; run < 300; ++run) {
        const int ctas = 8 + rng() % 141, depth = 1 + rng() % 8, most = 4 + rng() % 253, n = 1 + rng() % 600;
        std::vector<yg::ResidentJob> all;
        std::vector<double> truth;
        for (int i = 0; i < n; ++i) {
            all.push_back({1 + (int)(rng() % (1 + std::min(ctas - 1, (int)(rng() % 48)))), std::exp(6 * uniform())});
            truth.push_back(uniform() < 0.5 ? uniform() * 0.01 : 1.0);  // T = 1
        }
        std::sort(all.begin(), all.end(), [](const yg::ResidentJob &a, const yg::ResidentJob &b) { return a.cost > b.cost; });
        while (!all.empty()) {
            const yg::ResidentQueues q = yg::place_resident(all, ctas, depth, most);
            if (q.placed.empty() || (int)q.placed.size() > most) return std::printf("%zu jobs placed\n", q.placed.size()), 1;
            std::vector<std::vector<int>> cta_of(q.placed.size());
            std::vector<std::set<int>> ranks(q.placed.size());
            for (int c = 0; c < ctas; ++c) {
                if ((int)q.queue[c].size() > depth) return std::printf("queue of %zu\n", q.queue[c].size()), 1;
                for (size_t k = 0; k < q.queue[c].size(); ++k) {
                    if (k && q.queue[c][k].first <= q.queue[c][k - 1].first) return std::printf("queue out of order\n"), 1;
                    cta_of[q.queue[c][k].first].push_back(c);
                    ranks[q.queue[c][k].first].insert(q.queue[c][k].second);
                }
            }
            std::vector<double> free(ctas, 0.0);  // when each CTA ends the job before
            for (size_t i = 0; i < q.placed.size(); ++i) {
                const int G = all[q.placed[i]].ctas;
                if ((int)cta_of[i].size() != G || (int)ranks[i].size() != G || *ranks[i].rbegin() != G - 1)
                    return std::printf("a group of %d has %zu CTAs\n", G, cta_of[i].size()), 1;
                double start = 0, first = 1e300;
                for (int c : cta_of[i]) {
                    start = std::max(start, free[c]);
                    first = std::min(first, free[c]);
                }
                longest = std::max(longest, start - first);
                if (start - first > depth - 1 + 1e-9) return std::printf("a wait of %g jobs at depth %d\n", start - first, depth), 1;
                for (int c : cta_of[i]) free[c] = start + truth[q.placed[i]];
            }
            std::vector<yg::ResidentJob> rest;
            std::set<int> placed(q.placed.begin(), q.placed.end());
            for (size_t i = 0; i < all.size(); ++i)
                if (!placed.count((int)i)) rest.push_back(all[i]);
            all.swap(rest);
        }
    }
    std::printf("longest wait: %g jobs\n", longest);
    return 0;
}
