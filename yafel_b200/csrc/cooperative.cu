// cooperative.cu -- launches of kernels whose blocks wait for one another (resident PCG,
// batches of resident systems, ILU(0)).
#include "internal.h"
#include "sm_turns.h"

#include <atomic>
#include <chrono>
#include <mutex>
#include <thread>

namespace yg {

uint64_t new_stream_number() {
    static std::atomic<uint64_t> n{0};
    return ++n;
}

namespace {

using Clock = std::chrono::steady_clock;

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
    std::atomic<int> calls[3]{};  // in progress, by Beside::Kind
    // the two contexts whose calls ended last, the later one first
    std::mutex ended_m;
    struct {
        uint64_t stream = 0;
        Clock::time_point at{};
    } ended[2];
};

Device &device_of(yg_context ctx) {
    static auto *all = new Device[64];  // (never destroyed: contexts may outlive static objects)
    return all[ctx->device & 63];
}

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

Beside::Beside(yg_context ctx, Kind kind) : ctx_(ctx), kind_(kind) { ++device_of(ctx).calls[kind]; }
Beside::~Beside() {
    Device &d = device_of(ctx_);
    std::lock_guard<std::mutex> hold(d.ended_m);
    if (d.ended[0].stream != ctx_->stream_number) d.ended[1] = d.ended[0];
    d.ended[0] = {ctx_->stream_number, Clock::now()};
    --d.calls[kind_];
}
int Beside::streaming(yg_context ctx) { return device_of(ctx).calls[kStreams]; }
int Beside::not_wide(yg_context ctx) { return streaming(ctx) + device_of(ctx).calls[kNarrow]; }
bool Beside::others(yg_context ctx, int own) {
    Device &d = device_of(ctx);
    if (not_wide(ctx) + d.calls[kWide] > own) return true;
    std::lock_guard<std::mutex> hold(d.ended_m);
    const auto &last = d.ended[d.ended[0].stream == ctx->stream_number];
    return last.stream && Clock::now() - last.at < std::chrono::milliseconds(10);
}
void Beside::yield(yg_context ctx, double ms) {
    const auto end = Clock::now() + std::chrono::duration<double, std::milli>(ms);
    auto seen = Clock::now();
    for (auto now = seen; now < end && now - seen < std::chrono::microseconds(100); now = Clock::now()) {
        if (not_wide(ctx)) seen = now;  // (a program's next call follows the last one within microseconds)
        std::this_thread::sleep_for(std::chrono::microseconds(20));
    }
}

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
