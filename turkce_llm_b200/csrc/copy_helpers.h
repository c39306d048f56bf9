// The threads that share a large host copy (host_copy.cu).  Standard C++ only: tested without a GPU
// (tests/test_copy_helpers_host.py).
#pragma once
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <functional>
#include <mutex>
#include <system_error>
#include <thread>

#include <unistd.h>

namespace tb {

constexpr int kHelperSlots = 4;                       // the caller and three helpers: 64 GB/s between them, more gained nothing

// One job at a time.  An object that lives as long as the process is never destroyed (helpers() below): a process forked from
// one with helpers holds std::thread objects whose threads it does not have, and would abort in their destructors.
class Helpers {
public:
    // body(0) on the calling thread, body(1 .. kHelperSlots - 1) on the helpers; returns when all are done
    void run(const std::function<void(int)>& body) {
        if (!start()) {                                 // no threads to be had: one after the other
            for (int t = 0; t < kHelperSlots; ++t) body(t);
            return;
        }
        {
            std::lock_guard<std::mutex> lock(m_);
            body_ = &body;
            left_ = kHelperSlots - 1;
            ++generation_;
        }
        wake_.notify_all();
        body(0);
        std::unique_lock<std::mutex> lock(m_);
        done_.wait(lock, [this] { return left_ == 0; });
        body_ = nullptr;
    }

    void stop() {
        if (!started_ || pid_ != getpid()) return;     // (a forked child has no helpers)
        {
            std::lock_guard<std::mutex> lock(m_);
            quit_ = true;
        }
        wake_.notify_all();
        for (std::thread& t : threads_) if (t.joinable()) t.join();
        started_ = false; quit_ = false;
    }

private:
    bool start() {
        if (started_) return pid_ == getpid();
        pid_ = getpid();
        const uint64_t seen = generation_;
        try {
            for (int i = 1; i < kHelperSlots; ++i) threads_[i] = std::thread([this, i, seen] { loop(i, seen); });
        } catch (const std::system_error&) {
            started_ = true;
            stop();
            return false;
        }
        started_ = true;
        return true;
    }
    // a helper waits for the next body for a tenth of a millisecond with open eyes, then asleep
    void loop(int index, uint64_t seen) {
        while (true) {
            const std::function<void(int)>* body;
            // (the way back of a product follows its way in by less than a sleeping thread takes to wake)
            const auto until = std::chrono::steady_clock::now() + std::chrono::microseconds(100);
            while (generation_.load(std::memory_order_acquire) == seen && !quit_.load(std::memory_order_relaxed) &&
                   std::chrono::steady_clock::now() < until) {}
            {
                std::unique_lock<std::mutex> lock(m_);
                wake_.wait(lock, [&] { return quit_ || generation_ != seen; });
                if (quit_) return;
                seen = generation_;
                body = body_;
            }
            (*body)(index);
            std::lock_guard<std::mutex> lock(m_);
            if (--left_ == 0) done_.notify_one();
        }
    }

    std::mutex m_;
    std::condition_variable wake_, done_;
    std::thread threads_[kHelperSlots];
    const std::function<void(int)>* body_ = nullptr;
    std::atomic<uint64_t> generation_{0};
    int left_ = 0;
    bool started_ = false;
    std::atomic<bool> quit_{false};
    pid_t pid_ = 0;
};

// N numbered things that are handed out without ever waiting for one.
template <int N>
class Handout {
public:
    // up to `want` of the free ones -> which[]; how many
    int take(int want, int* which) {
        std::lock_guard<std::mutex> lock(m_);
        int n = 0;
        for (int i = 0; i < N && n < want; ++i)
            if (!taken_[i]) { taken_[i] = true; which[n++] = i; }
        return n;
    }
    void give(const int* which, int n) {
        std::lock_guard<std::mutex> lock(m_);
        for (int i = 0; i < n; ++i) taken_[which[i]] = false;
    }

private:
    std::mutex m_;
    bool taken_[N] = {};
};

inline Helpers& helpers() {
    static Helpers* const h = new Helpers();
    return *h;
}

}  // namespace tb
