// Copies between host memory and the device.
//
// Memory that is pinned already, or that is no plain host memory, is left to the driver, which copies it at the bus rate by
// itself (1024 x 1024 x 1024 product from pinned arrays: 254 us, 487 when it was staged like the rest).
//
// cudaMemcpy on pageable memory goes through the driver's staging buffer with one CPU thread: 17 - 18 GB/s measured, a
// third of what the bus takes (50 GB/s from pinned memory).  Here several threads copy pieces between the caller's memory and
// pinned buffers of this library while the pieces before them are on the bus.
//
// No transfer waits for another.  A lane is a pair of pinned buffers; there are kLanes of them per process and each belongs to
// one thread of one transfer at a time.  A large transfer that finds the helper threads free takes a lane for each of them, any
// other takes one and copies by itself, and one that finds no lane leaves the copy to the driver.  Lanes are made when they are
// first used, hold 2 x 512 KB, and are given back by tb_shutdown or when the process ends.
#include "common.h"
#include "copy_helpers.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <exception>
#include <functional>
#include <mutex>
#include <vector>

namespace tb {

namespace {

constexpr size_t kPiece = 512 * 1024;
constexpr size_t kThreadedFrom = 1024 * 1024;         // waking the helpers takes ~10 us, in which one thread copies 200 KB
constexpr int kLanes = 12;
constexpr int kDevices = 64;

struct Lane {
    char* buf[2] = {};
    cudaEvent_t last[2] = {};                           // behind the buffer's last copy, on whichever device that was
    cudaEvent_t ev[kDevices][2] = {};                   // (an event is recorded on the device it was made on)

    bool prepare(int device) {
        for (int b = 0; b < 2; ++b) {
            if (!buf[b] && cudaHostAlloc(reinterpret_cast<void**>(&buf[b]), kPiece, cudaHostAllocPortable) != cudaSuccess) return false;
            if (!ev[device][b] && cudaEventCreateWithFlags(&ev[device][b], cudaEventDisableTiming) != cudaSuccess) return false;
        }
        return true;
    }
    // the buffer's last copy has left it, or arrived in it
    cudaError_t settled(int b) { return last[b] ? cudaEventSynchronize(last[b]) : cudaSuccess; }
    cudaError_t record(int b, int device, cudaStream_t st) {
        last[b] = ev[device][b];
        return cudaEventRecord(last[b], st);
    }
    int free_all() {
        for (int b = 0; b < 2; ++b) {
            TB_CUDA(settled(b));
            last[b] = nullptr;
            for (auto& e : ev) {
                if (e[b]) TB_CUDA(cudaEventDestroy(e[b]));
                e[b] = nullptr;
            }
            if (buf[b]) TB_CUDA(cudaFreeHost(buf[b]));
            buf[b] = nullptr;
        }
        return 0;
    }
};
Lane g_lanes[kLanes];
Handout<kLanes> g_lane_handout;
std::mutex g_helpers_busy;

struct TakenLanes {
    int which[kLanes], n = 0;
    void take(int want) { n = g_lane_handout.take(want, which); }
    void give(int keep) {
        if (n > keep) g_lane_handout.give(which + keep, n - keep);
        n = std::min(n, keep);
    }
    ~TakenLanes() { give(0); }
};

// whether the driver copies from / to it directly: pinned, managed or device memory
bool needs_no_staging(const void* host) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, host) != cudaSuccess) { cudaGetLastError(); return false; }
    return a.type != cudaMemoryTypeUnregistered;
}

// The pieces of all spans, dealt to the threads in turn; a span that needs no staging is one piece, for the calling thread.  A buffer is written once the piece it held before -- this
// transfer's or an earlier one's -- has left it (its event).
//
// ready (optional): called on the calling thread, span by span in order, once every piece of a span has been handed to the
// stream.  after (optional, device -> host): an event per span that its copies wait for.
int transfer(const CopySpan* spans, int count, bool to_device, cudaStream_t st, const std::function<int(int)>* ready,
             const cudaEvent_t* after) {
    int device = 0;
    TB_CUDA(cudaGetDevice(&device));
    TB_CHECK(device < kDevices, "device ordinal %d out of range", device);
    // (a span that goes on where the last one ended is taken for the same memory: either way of copying is right for any)
    std::vector<char> direct(count);
    size_t total = 0;
    for (int k = 0; k < count; ++k) {
        const bool same = k > 0 && spans[k].host == static_cast<char*>(spans[k - 1].host) + spans[k - 1].bytes;
        direct[k] = same ? direct[k - 1] : needs_no_staging(spans[k].host);
        if (!direct[k]) total += spans[k].bytes;
    }
    std::unique_lock<std::mutex> helpers_lock(g_helpers_busy, std::defer_lock);
    TakenLanes lanes;
    const bool many = total >= kThreadedFrom && helpers_lock.try_lock();
    if (total > 0) lanes.take(many ? kHelperSlots : 1);
    for (int i = 0; i < lanes.n; ++i)
        if (!g_lanes[lanes.which[i]].prepare(device)) {
            cudaGetLastError();
            lanes.give(i);                              // (no pinned memory to be had: with the lanes there are, or none)
            break;
        }
    const int threads = lanes.n;
    if (threads == 0) std::fill(direct.begin(), direct.end(), (char)1);
    std::vector<std::atomic<int>> open(count);           // pieces of a span not handed over yet
    for (int k = 0; k < count; ++k) open[k] = direct[k] ? 1 : (int)((spans[k].bytes + kPiece - 1) / kPiece);
    int told = 0, told_rc = 0;                           // spans `ready` has been called for
    auto tell = [&]() {
        while (told < count && open[told].load(std::memory_order_acquire) == 0) {
            if (told_rc == 0) told_rc = (*ready)(told);
            ++told;
        }
    };
    cudaError_t err[kHelperSlots] = {};
    const std::function<void(int)> body = [&](int t) {
        auto ok = [&](cudaError_t e) { if (e != cudaSuccess && err[t] == cudaSuccess) err[t] = e; return e == cudaSuccess; };
        if (t > 0 && (t >= threads || !ok(cudaSetDevice(device)))) return;
        Lane* const lane = threads > 0 ? &g_lanes[lanes.which[t]] : nullptr;
        size_t before = 0;                              // the piece on its way in the other buffer (device -> host)
        char* before_at = nullptr;
        int b = 0, turn = 0;
        bool wait_for_stream = false;
        for (int k = 0; k < count; ++k) {
            if (direct[k]) {
                if (t != 0) continue;
                wait_for_stream = !to_device;
                if (!to_device && after && !ok(cudaStreamWaitEvent(st, after[k], 0))) return;
                if (!ok(cudaMemcpyAsync(to_device ? spans[k].dev : spans[k].host, to_device ? spans[k].host : spans[k].dev, spans[k].bytes,
                                        to_device ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost, st)))
                    return;
                open[k].fetch_sub(1, std::memory_order_release);
                if (ready) tell();
                continue;
            }
            for (size_t at = 0; at < spans[k].bytes; at += kPiece, ++turn) {
                if (turn % threads != t) continue;
                const size_t n = std::min(kPiece, spans[k].bytes - at);
                char *dev = static_cast<char*>(spans[k].dev) + at, *host = static_cast<char*>(spans[k].host) + at;
                if (!ok(lane->settled(b))) return;
                if (to_device) {
                    std::memcpy(lane->buf[b], host, n);
                    if (!ok(cudaMemcpyAsync(dev, lane->buf[b], n, cudaMemcpyHostToDevice, st))) return;
                    if (!ok(lane->record(b, device, st))) return;
                    open[k].fetch_sub(1, std::memory_order_release);
                    if (t == 0 && ready) tell();
                } else {
                    if (after && !ok(cudaStreamWaitEvent(st, after[k], 0))) return;
                    if (!ok(cudaMemcpyAsync(lane->buf[b], dev, n, cudaMemcpyDeviceToHost, st))) return;
                    if (!ok(lane->record(b, device, st))) return;
                    if (before_at) {
                        if (!ok(lane->settled(b ^ 1))) return;
                        std::memcpy(before_at, lane->buf[b ^ 1], before);
                    }
                    before_at = host; before = n;
                }
                b ^= 1;
            }
        }
        if (before_at && ok(lane->settled(b ^ 1))) std::memcpy(before_at, lane->buf[b ^ 1], before);
        if (wait_for_stream) ok(cudaStreamSynchronize(st));
    };
    if (threads > 1) helpers().run(body);
    else body(0);
    for (cudaError_t e : err) TB_CUDA(e);
    if (ready) tell();
    return told_rc;
}

// (these are called from C entry points)
int transfer_no_throw(const CopySpan* spans, int count, bool to_device, cudaStream_t st, const std::function<int(int)>* ready,
                      const cudaEvent_t* after) {
    try {
        return transfer(spans, count, to_device, st, ready, after);
    } catch (const std::exception& e) {
        set_error("host copy: %s", e.what());
        return -2;
    }
}

}  // namespace

int copy_h2d(const CopySpan* spans, int count, cudaStream_t st, const std::function<int(int)>* ready) {
    return transfer_no_throw(spans, count, true, st, ready, nullptr);
}
int copy_d2h(const CopySpan* spans, int count, cudaStream_t st, const cudaEvent_t* after) {
    return transfer_no_throw(spans, count, false, st, nullptr, after);
}
int copy_give_back() {
    std::lock_guard<std::mutex> lock(g_helpers_busy);
    helpers().stop();
    TakenLanes lanes;                                   // (one that a transfer of another thread holds stays)
    lanes.take(kLanes);
    for (int i = 0; i < lanes.n; ++i) TB_TRY(g_lanes[lanes.which[i]].free_all());
    return 0;
}

}  // namespace tb
