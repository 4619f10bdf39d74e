// sm_turns.h -- who may hold the SMs of a device among kernels whose blocks wait for one
// another (host only, no CUDA).
//
// Two such kernels must never hold part of the SMs each while both wait for the rest.
// Every SM of the device is a place; a launch of k blocks (one per SM at most) takes k
// places and follows, on the device, the launches that held them last.  A place's
// launches therefore follow one another, so the kernels at work at any time have no more
// blocks than the device has SMs, and all of their blocks find room.  Launches that fit
// beside one another share the device.
#pragma once
#include <algorithm>
#include <cstdint>
#include <memory>
#include <vector>

namespace yg {

// One launch: its stream (a number of its own, never used again) and `event`, which the
// places share; released when no place holds the launch any more.
template <typename Event>
struct SmHold {
    uint64_t stream;
    Event event;
};

template <typename Event>
class SmTurns {
  public:
    using Hold = std::shared_ptr<SmHold<Event>>;

    explicit SmTurns(int places) : held_(places), since_(places, 0) {}
    int places() const { return (int)held_.size(); }

    // The places a launch of `blocks` blocks on `stream` takes: the stream's own first,
    // then those whose launch is done (done(event)), then those held longest.  before:
    // the launches it has to follow (none of its own stream, none that is done).
    template <typename Done>
    std::vector<int> take(int blocks, uint64_t stream, Done done, std::vector<Hold> &before) {
        const int n = places();
        std::vector<int> cost(n), place(n);
        const SmHold<Event> *last = nullptr;
        int last_cost = 0;
        for (int i = 0; i < n; ++i) {
            place[i] = i;
            const SmHold<Event> *h = held_[i].get();
            if (h && h->stream != stream && h != last) {
                last = h;
                last_cost = done(h->event) ? 1 : 2;
            }
            cost[i] = !h ? 1 : (h->stream == stream ? 0 : last_cost);
        }
        std::stable_sort(place.begin(), place.end(), [&](int a, int b) {
            return cost[a] != cost[b] ? cost[a] < cost[b] : (cost[a] == 2 && since_[a] < since_[b]);
        });
        place.resize(std::min(blocks, n));
        before.clear();
        for (int i : place)
            if (cost[i] == 2 && std::find(before.begin(), before.end(), held_[i]) == before.end()) before.push_back(held_[i]);
        return place;
    }

    // The launch that now holds them.
    void give(const std::vector<int> &place, const Hold &launch) {
        ++turn_;
        for (int i : place) {
            held_[i] = launch;
            since_[i] = turn_;
        }
    }

  private:
    std::vector<Hold> held_;
    std::vector<uint64_t> since_;
    uint64_t turn_ = 0;
};

}  // namespace yg
