// resident_queues.h -- which CTAs iterate on which systems of a batch, and in what order
// (host only, no CUDA).
#pragma once
#include <algorithm>
#include <cstddef>
#include <utility>
#include <vector>

namespace yg {

struct ResidentJob {
    int ctas;     // CTAs of its group
    double cost;  // estimated time: it orders the work, no more
};

struct ResidentQueues {
    std::vector<int> placed;                               // jobs of the launch, in the order of all queues
    std::vector<std::vector<std::pair<int, int>>> queue;   // per CTA: (index into placed, rank in its group)
};

// Places jobs (longest first) on `ctas` CTAs: the longest that the free CTAs can take
// starts first; when there is none, on to the next time at which CTAs become free.  All
// queues have the placed jobs in one order, so the first job that is not done always has
// all its CTAs.  A CTA may reach a job while another CTA of its group is still at the job
// before, which may have waited for a third: `depth` bounds these chains.  A job's depth
// is one more than that of the jobs before it in its CTAs' queues, so with jobs of at
// most T each a job of depth d has all its CTAs after (d - 1) T, whatever the estimates,
// and no CTA waits longer than (depth - 1) T for its group.  Jobs that find no place stay
// for the next launch.
inline ResidentQueues place_resident(const std::vector<ResidentJob> &jobs, int ctas, int depth, int most) {
    ResidentQueues out;
    out.queue.resize(ctas);
    std::vector<int> todo(jobs.size()), deep(ctas, 0);
    for (size_t i = 0; i < jobs.size(); ++i) todo[i] = (int)i;
    std::vector<double> until(ctas, 0.0);
    double now = 0;
    while (!todo.empty() && (int)out.placed.size() < most) {
        std::vector<int> free;
        for (int c = 0; c < ctas; ++c)
            if (until[c] <= now && deep[c] < depth) free.push_back(c);
        size_t k = 0;
        while (k < todo.size() && jobs[todo[k]].ctas > (int)free.size()) ++k;
        if (k == todo.size()) {
            double next = 1e300;
            for (int c = 0; c < ctas; ++c)
                if (until[c] > now && deep[c] < depth) next = std::min(next, until[c]);
            if (next == 1e300) break;
            now = next;
            continue;
        }
        const ResidentJob &j = jobs[todo[k]];
        int before = 0;
        for (int i = 0; i < j.ctas; ++i) before = std::max(before, deep[free[i]]);
        for (int i = 0; i < j.ctas; ++i) {
            until[free[i]] = now + j.cost;
            deep[free[i]] = before + 1;
            out.queue[free[i]].push_back({(int)out.placed.size(), i});
        }
        out.placed.push_back(todo[k]);
        todo.erase(todo.begin() + k);
    }
    return out;
}

}  // namespace yg
