// memcpy by several threads, for the copies between pageable host arrays and
// pinned slots (host_copy.cu).  Host code only: a test runs it without a device.
#pragma once

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstddef>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <thread>

namespace umapb {

// memcpy by several threads.  One job at a time (callers hold 'owner').
class CopyThreads {
public:
    static constexpr size_t PART_BYTES = size_t(64) << 10;
    // Beside the caller: 'helpers' threads, started with the first copy.  first_job: for tests.
    explicit CopyThreads(int helpers, uint64_t first_job = 0) : helpers_(helpers), state_(first_job << JOB) {}
    std::mutex owner;
    std::atomic<bool> busy{false};   // set by the owner for a row of jobs: the threads stay awake between them

    void copy(char* dst, const char* src, size_t bytes) {
        start();
        dst_ = dst;
        src_ = src;
        bytes_ = bytes;
        const int parts = static_cast<int>((bytes + PART_BYTES - 1) / PART_BYTES);
        left_.store(parts, std::memory_order_relaxed);
        const uint64_t job = ((state_.load(std::memory_order_relaxed) >> JOB) + 1) & JOBS;
        state_.store(job << JOB | static_cast<uint64_t>(parts) << PARTS, std::memory_order_seq_cst);
        if (sleeping_.load(std::memory_order_seq_cst) > 0) {
            std::lock_guard<std::mutex> lock(mu_);
            cv_.notify_all();
        }
        work(job);
        while (left_.load(std::memory_order_acquire) > 0) std::this_thread::yield();
    }

private:
    // state_: job number, its parts, the next part to take -- in one word, so that a
    // thread late from the job before can take nothing of this one by mistake.
    static constexpr int JOB = 40, PARTS = 20;
    static constexpr uint64_t MASK = (uint64_t(1) << 20) - 1, JOBS = (uint64_t(1) << 24) - 1;   // (the job's number starts over)

    // Takes parts of job 'job' while it is the current one and has parts left.
    void work(uint64_t job) {
        uint64_t at = state_.load(std::memory_order_acquire);
        while ((at >> JOB) == job && (at & MASK) < ((at >> PARTS) & MASK)) {
            if (!state_.compare_exchange_weak(at, at + 1, std::memory_order_acq_rel)) continue;
            const size_t first = (at & MASK) * PART_BYTES;
            std::memcpy(dst_ + first, src_ + first, std::min(PART_BYTES, bytes_ - first));
            left_.fetch_sub(1, std::memory_order_release);
            at = state_.load(std::memory_order_acquire);
        }
    }
    void start() {
        if (started_) return;
        started_ = true;
        for (int i = 0; i < helpers_; ++i) {
            try {
                std::thread([this] { serve(); }).detach();
            } catch (const std::exception&) {
                break;   // fewer threads: the caller copies what they do not
            }
        }
    }
    void serve() {
        uint64_t done = state_.load(std::memory_order_acquire) >> JOB;   // the last job seen
        while (true) {
            // Awake between the jobs of one copy, which the bus paces (30 to 100 us), and
            // shortly after it (a call copies several arrays) -- not while a copy waits
            // for whatever is before it on its stream.
            int spin = 0;
            uint64_t job = state_.load(std::memory_order_acquire) >> JOB;
            while (job == done && ++spin < (busy.load(std::memory_order_relaxed) ? 1000 : 100)) {
                std::this_thread::yield();
                job = state_.load(std::memory_order_acquire) >> JOB;
            }
            if (job == done) {
                std::unique_lock<std::mutex> lock(mu_);
                sleeping_.fetch_add(1, std::memory_order_seq_cst);
                cv_.wait(lock, [&] { return state_.load(std::memory_order_seq_cst) >> JOB != done; });
                sleeping_.fetch_sub(1, std::memory_order_relaxed);
                continue;
            }
            done = job;
            work(job);
        }
    }
    const int helpers_;
    bool started_ = false;
    char* dst_ = nullptr;
    const char* src_ = nullptr;
    size_t bytes_ = 0;
    std::atomic<int> left_{0}, sleeping_{0};   // parts not copied yet; threads asleep
    std::atomic<uint64_t> state_;
    std::mutex mu_;
    std::condition_variable cv_;
};

}  // namespace umapb
