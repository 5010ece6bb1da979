// Copies between pageable host arrays and the device.
//
// The runtime moves pageable memory through a pinned buffer with one host
// thread, at 10 to 11 GB/s here (less into fresh pages, which the kernel clears
// one fault at a time), a fifth of the bus.  Arrays of COPY_MIN bytes and more
// go through pinned slots of our own instead, filled and emptied by a few
// threads while the bus moves the other slots: placing 10,000 new points among
// 100,000 (22 MB of host arrays) takes 4.1 ms instead of 6.4, the gradient over a
// graph of 2 million edges (18 MB) 1.0 instead of 1.3.
//
// The slots of a device are one copy's at a time; another thread that copies
// meanwhile takes the runtime's way.  They and the threads, which sleep
// between copies, last for the process: 8 MiB pinned per device used.
#include <cuda_runtime.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <thread>

#include "common.cuh"
#include "copy_threads.hpp"

namespace umapb {

namespace {

constexpr size_t COPY_MIN = size_t(1) << 20;
constexpr size_t SLOT_BYTES = size_t(2) << 20;
constexpr int SLOTS = 4;

// Bytes moved at a time.  The bus moves a piece only once it is there, and the
// helpers take some 100 us to wake, so a copy of few MB goes in pieces that the
// caller fills alone meanwhile; a larger one pays more for each piece than it
// gains.  us after 0.3 ms without copies, up / down, in pieces of 512 KB | 2 MB | the
// runtime's copy: 2 MB 128 / 166 | 289 / 366 | 209 / 144; 4 MB 221 / 222 | 399 / 371 | 410 /
// 263; 6.4 MB 320 / 344 | 485 / 293 | 610 / 399; 32 MB 1625 / 1252 | 1493 / 1060 | 3009 / 1957.
// Into fresh pages, where the faults decide: 2 MB 356 | 545 | 934, 6.4 MB 845 | 773 | 2863.
// Search of 30,011 points with 50 neighbours (3.6 MB up, twice 6 MB down into fresh
// arrays) 5.3 ms with 512 KB throughout, 4.9 with 2 MB, 4.65 so.
constexpr size_t PIECES_BELOW = size_t(5) << 20;
size_t piece_bytes(size_t bytes) { return bytes < PIECES_BELOW ? SLOT_BYTES / 4 : SLOT_BYTES; }
constexpr int MAX_THREADS = 4;   // the caller among them

CopyThreads& copy_threads() {
    const unsigned cores = std::thread::hardware_concurrency();
    static CopyThreads* t = new CopyThreads(std::min<int>(MAX_THREADS, cores > 1 ? static_cast<int>(cores) : 1) - 1);   // never destroyed: its threads may outlive main
    return *t;
}

struct Slots {
    char* slot[SLOTS] = {};
    cudaEvent_t moved[SLOTS] = {};   // the slot's last move over the bus
};

// The current device's slots, null where they cannot be had (copy_threads().owner held).
Slots* device_slots() {
    static std::map<int, Slots>* all = new std::map<int, Slots>();
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    Slots& s = (*all)[dev];
    for (int i = 0; i < SLOTS; ++i) {
        if (!s.slot[i] && cudaHostAlloc(reinterpret_cast<void**>(&s.slot[i]), SLOT_BYTES, cudaHostAllocPortable) != cudaSuccess) {
            s.slot[i] = nullptr;
            cudaGetLastError();
            return nullptr;
        }
        if (!s.moved[i] && cudaEventCreateWithFlags(&s.moved[i], cudaEventDisableTiming) != cudaSuccess) {
            s.moved[i] = nullptr;
            cudaGetLastError();
            return nullptr;
        }
    }
    return &s;
}

enum class Memory { pageable, device, other };
Memory memory_of(const void* p) {
    cudaPointerAttributes attr;
    if (cudaPointerGetAttributes(&attr, p) != cudaSuccess) {
        cudaGetLastError();
        return Memory::pageable;
    }
    return attr.type == cudaMemoryTypeDevice ? Memory::device
         : attr.type == cudaMemoryTypeUnregistered ? Memory::pageable : Memory::other;
}

void to_device(Slots& st, char* dst, const char* src, size_t bytes, cudaStream_t s) {
    const size_t piece = piece_bytes(bytes);
    int i = 0;
    for (size_t at = 0; at < bytes; at += piece, i = (i + 1) % SLOTS) {
        const size_t len = std::min(piece, bytes - at);
        UMAPB_CUDA(cudaEventSynchronize(st.moved[i]));
        copy_threads().copy(st.slot[i], src + at, len);
        UMAPB_CUDA(cudaMemcpyAsync(dst + at, st.slot[i], len, cudaMemcpyHostToDevice, s));
        UMAPB_CUDA(cudaEventRecord(st.moved[i], s));
    }
}

void to_host(Slots& st, char* dst, const char* src, size_t bytes, cudaStream_t s) {
    const size_t piece = piece_bytes(bytes);
    const size_t pieces = (bytes + piece - 1) / piece;
    auto move = [&](size_t c) {
        const size_t at = c * piece;
        UMAPB_CUDA(cudaMemcpyAsync(st.slot[c % SLOTS], src + at, std::min(piece, bytes - at), cudaMemcpyDeviceToHost, s));
        UMAPB_CUDA(cudaEventRecord(st.moved[c % SLOTS], s));
    };
    for (int i = 0; i < SLOTS; ++i) UMAPB_CUDA(cudaEventSynchronize(st.moved[i]));   // free of the copy before
    for (size_t c = 0; c < std::min<size_t>(pieces, SLOTS); ++c) move(c);
    for (size_t c = 0; c < pieces; ++c) {
        const size_t at = c * piece;
        UMAPB_CUDA(cudaEventSynchronize(st.moved[c % SLOTS]));
        copy_threads().copy(dst + at, st.slot[c % SLOTS], std::min(piece, bytes - at));
        if (c + SLOTS < pieces) move(c + SLOTS);
    }
}

}  // namespace

void copy_async(void* dst, const void* src, size_t bytes, cudaStream_t s) {
    if (bytes == 0) return;
    if (bytes >= COPY_MIN) {
        const Memory to = memory_of(dst), from = memory_of(src);
        const bool up = to == Memory::device && from == Memory::pageable;
        const bool down = to == Memory::pageable && from == Memory::device;
        if (up || down) {
            std::unique_lock<std::mutex> lock(copy_threads().owner, std::try_to_lock);
            Slots* st = lock.owns_lock() ? device_slots() : nullptr;
            if (st) {
                const double t0 = trace_enabled() ? host_ms() : 0.0;
                struct Awake {
                    Awake() { copy_threads().busy.store(true, std::memory_order_relaxed); }
                    ~Awake() { copy_threads().busy.store(false, std::memory_order_relaxed); }
                } awake;
                try {
                    if (up) to_device(*st, static_cast<char*>(dst), static_cast<const char*>(src), bytes, s);
                    else to_host(*st, static_cast<char*>(dst), static_cast<const char*>(src), bytes, s);
                } catch (...) {
                    cudaStreamSynchronize(s);   // nothing may still use the slots
                    cudaGetLastError();
                    throw;
                }
                if (trace_enabled()) trace_wait(up ? "copy to the device" : "copy to the host", t0, bytes, __FILE__, __LINE__);
                return;
            }
        }
    }
    UMAPB_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDefault, s));
}

}  // namespace umapb
