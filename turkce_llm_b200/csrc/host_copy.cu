// Copies between pageable host memory and the device.
//
// cudaMemcpy on pageable memory goes through the driver's staging buffer with one CPU thread: 17 - 18 GB/s measured, a
// third of what the bus takes (50 GB/s from pinned memory).  Here several threads copy pieces between the caller's memory and
// pinned buffers of this library while the pieces before them are on the bus.
//
// The helper threads and pinned buffers are one set per process, taken by one transfer at a time (a second caller waits,
// as it would for the bus).  They are made on the first large transfer, hold 2 x 512 KB per thread whatever the size of a
// transfer, and are given back by tb_shutdown or when the process ends.
#include "common.h"
#include "copy_helpers.h"

#include <algorithm>
#include <atomic>
#include <cstring>
#include <functional>
#include <mutex>
#include <vector>

namespace tb {

namespace {

constexpr int kCopyThreads = kHelperSlots;
constexpr size_t kPiece = 512 * 1024;
constexpr size_t kThreadedFrom = 1024 * 1024;         // waking the helpers takes ~10 us, in which one thread copies 200 KB

struct Staging {
    std::mutex busy;                                    // one transfer at a time
    int device = -1;                                    // the events belong to it; the pinned memory serves every device
    char* buf[kCopyThreads][2] = {};
    cudaEvent_t ev[kCopyThreads][2] = {};

    int prepare() {
        int dev = 0;
        TB_CUDA(cudaGetDevice(&dev));
        if (device >= 0 && device != dev) TB_TRY(drop_events());
        for (int t = 0; t < kCopyThreads; ++t)
            for (int b = 0; b < 2; ++b) {
                if (!buf[t][b]) TB_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&buf[t][b]), kPiece, cudaHostAllocPortable));
                if (!ev[t][b]) TB_CUDA(cudaEventCreateWithFlags(&ev[t][b], cudaEventDisableTiming));
            }
        device = dev;
        return 0;
    }
    int drop_events() {
        for (int t = 0; t < kCopyThreads; ++t)
            for (int b = 0; b < 2; ++b)
                if (ev[t][b]) {
                    TB_CUDA(cudaEventSynchronize(ev[t][b]));          // the buffer's last piece has left it
                    TB_CUDA(cudaEventDestroy(ev[t][b]));
                    ev[t][b] = nullptr;
                }
        return 0;
    }
    int give_back() {
        helpers().stop();
        TB_TRY(drop_events());
        for (int t = 0; t < kCopyThreads; ++t)
            for (int b = 0; b < 2; ++b) {
                if (buf[t][b]) TB_CUDA(cudaFreeHost(buf[t][b]));
                buf[t][b] = nullptr;
            }
        device = -1;
        return 0;
    }
};
Staging g_staging;

// The pieces of all spans, dealt to the threads in turn.  A buffer is written once the piece it held before -- this
// transfer's or an earlier one's -- has left it (its event).
//
// ready (optional): called on the calling thread, span by span in order, once every piece of a span has been handed to the
// stream.  after (optional, device -> host): an event per span that its copies wait for.
int transfer(const CopySpan* spans, int count, bool to_device, cudaStream_t st, const std::function<int(int)>* ready,
             const cudaEvent_t* after) {
    std::lock_guard<std::mutex> lock(g_staging.busy);
    TB_TRY(g_staging.prepare());
    Staging& g = g_staging;
    const int device = g.device;
    size_t total = 0;
    std::vector<std::atomic<int>> open(count);           // pieces of a span not handed over yet
    for (int k = 0; k < count; ++k) {
        total += spans[k].bytes;
        open[k] = (int)((spans[k].bytes + kPiece - 1) / kPiece);
    }
    int told = 0, told_rc = 0;                           // spans `ready` has been called for
    auto tell = [&]() {
        while (told < count && open[told].load(std::memory_order_acquire) == 0) {
            if (told_rc == 0) told_rc = (*ready)(told);
            ++told;
        }
    };
    const int threads = total >= kThreadedFrom ? kCopyThreads : 1;
    cudaError_t err[kCopyThreads] = {};
    const std::function<void(int)> body = [&](int t) {
        auto ok = [&](cudaError_t e) { if (e != cudaSuccess && err[t] == cudaSuccess) err[t] = e; return e == cudaSuccess; };
        if (t > 0 && !ok(cudaSetDevice(device))) return;
        size_t before = 0;                              // the piece on its way in the other buffer (device -> host)
        char* before_at = nullptr;
        int b = 0, turn = 0;
        for (int k = 0; k < count; ++k)
            for (size_t at = 0; at < spans[k].bytes; at += kPiece, ++turn) {
                if (turn % threads != t) continue;
                const size_t n = std::min(kPiece, spans[k].bytes - at);
                char *dev = static_cast<char*>(spans[k].dev) + at, *host = static_cast<char*>(spans[k].host) + at;
                if (!ok(cudaEventSynchronize(g.ev[t][b]))) return;
                if (to_device) {
                    std::memcpy(g.buf[t][b], host, n);
                    if (!ok(cudaMemcpyAsync(dev, g.buf[t][b], n, cudaMemcpyHostToDevice, st))) return;
                    if (!ok(cudaEventRecord(g.ev[t][b], st))) return;
                    open[k].fetch_sub(1, std::memory_order_release);
                    if (t == 0 && ready) tell();
                } else {
                    if (after && !ok(cudaStreamWaitEvent(st, after[k], 0))) return;
                    if (!ok(cudaMemcpyAsync(g.buf[t][b], dev, n, cudaMemcpyDeviceToHost, st))) return;
                    if (!ok(cudaEventRecord(g.ev[t][b], st))) return;
                    if (before_at) {
                        if (!ok(cudaEventSynchronize(g.ev[t][b ^ 1]))) return;
                        std::memcpy(before_at, g.buf[t][b ^ 1], before);
                    }
                    before_at = host; before = n;
                }
                b ^= 1;
            }
        if (before_at && ok(cudaEventSynchronize(g.ev[t][b ^ 1]))) std::memcpy(before_at, g.buf[t][b ^ 1], before);
    };
    if (threads > 1) helpers().run(body);
    else body(0);
    for (cudaError_t e : err) TB_CUDA(e);
    if (ready) tell();
    return told_rc;
}

}  // namespace

int copy_h2d(const CopySpan* spans, int count, cudaStream_t st, const std::function<int(int)>* ready) {
    return transfer(spans, count, true, st, ready, nullptr);
}
int copy_d2h(const CopySpan* spans, int count, cudaStream_t st, const cudaEvent_t* after) {
    return transfer(spans, count, false, st, nullptr, after);
}
int copy_give_back() {
    std::lock_guard<std::mutex> lock(g_staging.busy);
    return g_staging.give_back();
}

}  // namespace tb
