// Random launches of waiting kernels on several streams: whatever order the device starts
// the ready ones in, those at work never have more blocks than places, and all end.
#include "sm_turns.h"

#include <cstdio>
#include <cstdlib>
#include <random>

struct Launch {
    int blocks, stream;
    std::vector<int> after;  // launches it follows
    bool started = false, done = false;
};

int main() {
    std::mt19937 rng(7);
    long long shared = 0;
    for (int run = 0; run < 400; ++run) {
        const int places = 1 + rng() % 40, streams = 1 + rng() % 7, total = 120;
        yg::SmTurns<int> turns(places);  // an event is the launch's index
        std::vector<Launch> all;
        std::vector<int> last(streams, -1);
        int at_work = 0, ended = 0;
        while (ended < total) {
            std::vector<int> ready, running;
            for (int i = 0; i < (int)all.size(); ++i) {
                if (all[i].done) continue;
                if (all[i].started) { running.push_back(i); continue; }
                bool ok = true;
                for (int b : all[i].after) ok = ok && all[b].done;
                if (ok) ready.push_back(i);
            }
            const int what = rng() % 3;
            if (what == 0 && (int)all.size() < total) {
                Launch l;
                l.blocks = rng() % 3 ? 1 + rng() % places : 1 + rng() % (1 + places / 4);
                l.stream = rng() % streams;
                std::vector<yg::SmTurns<int>::Hold> before;
                const auto place = turns.take(l.blocks, l.stream, [&](int e) { return all[e].done; }, before);
                if ((int)place.size() != l.blocks) return std::printf("%d places of %d\n", (int)place.size(), l.blocks), 1;
                if (last[l.stream] >= 0) l.after.push_back(last[l.stream]);
                for (const auto &b : before) l.after.push_back(b->event);
                last[l.stream] = (int)all.size();
                turns.give(place, std::make_shared<yg::SmHold<int>>(yg::SmHold<int>{(uint64_t)l.stream, (int)all.size()}));
                all.push_back(l);
            } else if (what == 1 && !ready.empty()) {
                Launch &l = all[ready[rng() % ready.size()]];
                l.started = true;
                shared += at_work > 0;
                if ((at_work += l.blocks) > places) return std::printf("%d blocks at work on %d places\n", at_work, places), 1;
            } else if (!running.empty()) {
                Launch &l = all[running[rng() % running.size()]];
                l.done = true;
                at_work -= l.blocks;
                ++ended;
            } else if (ready.empty() && (int)all.size() == total) {
                return std::printf("none of %d launches can go on\n", total - ended), 1;
            }
        }
    }
    // halves fit beside one another, a stream keeps its own places
    yg::SmTurns<int> t(8);
    std::vector<yg::SmTurns<int>::Hold> before;
    auto never = [](int) { return false; };
    for (int round = 0; round < 3; ++round)
        for (uint64_t s = 1; s <= 2; ++s) {
            const auto p = t.take(4, s, never, before);
            if (!before.empty()) return std::printf("halves wait for one another\n"), 1;
            t.give(p, std::make_shared<yg::SmHold<int>>(yg::SmHold<int>{s, 0}));
        }
    t.take(5, 1, never, before);
    if (before.size() != 1 || before[0]->stream != 2) return std::printf("five of eight beside four do not wait\n"), 1;
    std::printf("%lld launches started beside others\n", shared);
    return shared > 1000 ? 0 : 1;
}
