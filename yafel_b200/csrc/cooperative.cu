// cooperative.cu -- launches of kernels whose blocks wait for one another (resident PCG,
// batches of resident systems, ILU(0)).
#include "internal.h"
#include "sm_turns.h"

#include <atomic>
#include <mutex>

namespace yg {

uint64_t new_stream_number() {
    static std::atomic<uint64_t> n{0};
    return ++n;
}

namespace {

struct Event {
    cudaEvent_t e = nullptr;
    std::vector<cudaEvent_t> *spare = nullptr;
    Event(cudaEvent_t e_, std::vector<cudaEvent_t> *s) : e(e_), spare(s) {}
    Event(Event &&o) : e(o.e), spare(o.spare) { o.e = nullptr; }
    Event(const Event &) = delete;
    ~Event() {
        if (e) spare->push_back(e);
    }
};

struct Device {
    std::mutex m;
    std::vector<cudaEvent_t> spare;  // events of launches that no place holds any more
    std::unique_ptr<SmTurns<Event>> turns;
    std::atomic<int> solving{0}, streaming{0};
};

Device &device_at(int device) {
    static auto *all = new Device[64];  // (never destroyed: contexts may outlive static objects)
    return all[device & 63];
}
Device &device_of(yg_context ctx) { return device_at(ctx->device); }

// Runs `launch`, of kernels of up to `blocks` blocks, in its turn.
template <typename Launch>
yg_status in_turn(yg_context ctx, int blocks, Launch launch) {
    Device &d = device_of(ctx);
    std::lock_guard<std::mutex> hold(d.m);
    if (!d.turns) d.turns.reset(new SmTurns<Event>(ctx->num_sms));
    std::vector<SmTurns<Event>::Hold> before;
    auto done = [](const Event &e) { return cudaEventQuery(e.e) == cudaSuccess; };
    const std::vector<int> place = d.turns->take(blocks, ctx->stream_number, done, before);
    cudaGetLastError();  // (not ready is no error)
    for (const auto &b : before) YG_CUDA(cudaStreamWaitEvent(ctx->stream, b->event.e, 0));
    cudaEvent_t e = nullptr;
    if (!d.spare.empty()) {
        e = d.spare.back();
        d.spare.pop_back();
    } else {
        YG_CUDA(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    }
    SmTurns<Event>::Hold mine(new SmHold<Event>{ctx->stream_number, Event(e, &d.spare)});
    YG_TRY(launch());
    YG_CUDA(cudaEventRecord(e, ctx->stream));
    d.turns->give(place, mine);
    return YG_OK;
}

}  // namespace

Beside::Beside(yg_context ctx, bool streams) : device_(ctx->device), streams_(streams) {
    ++device_at(device_).solving;
    if (streams_) ++device_at(device_).streaming;
}
Beside::~Beside() {
    --device_at(device_).solving;
    if (streams_) --device_at(device_).streaming;
}
int Beside::solving(yg_context ctx) { return device_of(ctx).solving; }
int Beside::streaming(yg_context ctx) { return device_of(ctx).streaming; }

yg_status launch_cooperative(yg_context ctx, const void *kern, int grid, int threads, size_t smem, void **args) {
    auto launch = [&]() -> yg_status {
        YG_CUDA(cudaLaunchCooperativeKernel(kern, dim3(grid), dim3(threads), args, smem, ctx->stream));
        YG_LAUNCHED(ctx);
        return YG_OK;
    };
    cudaStreamCaptureStatus cs;
    YG_CUDA(cudaStreamIsCapturing(ctx->stream, &cs));
    if (cs == cudaStreamCaptureStatusNone) return in_turn(ctx, grid, launch);
    ctx->captured_blocks = std::max(ctx->captured_blocks, grid);  // the replays take the turn (launch_graph)
    return launch();
}

yg_status launch_graph(yg_context ctx, cudaGraphExec_t exec, int blocks) {
    auto launch = [&]() -> yg_status {
        YG_CUDA(cudaGraphLaunch(exec, ctx->stream));
        return YG_OK;
    };
    return blocks > 0 ? in_turn(ctx, blocks, launch) : launch();
}

}  // namespace yg
