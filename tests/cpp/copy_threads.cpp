// The copy threads (copy_threads.hpp) by themselves.
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <ctime>
#include <string>
#include <vector>

#include "copy_threads.hpp"

static bool copies(int helpers, uint64_t first_job, size_t bytes, int times) {
    umapb::CopyThreads& t = *new umapb::CopyThreads(helpers, first_job);
    std::vector<char> from(bytes), to(bytes);
    for (int i = 0; i < times; ++i) {
        for (size_t b = 0; b < bytes; ++b) from[b] = static_cast<char>(b * 7 + i);
        t.copy(to.data(), from.data(), bytes);
        if (to != from) return false;
    }
    return true;
}

int main(int argc, char** argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "jobs") return !copies(std::atoi(argv[2]), std::strtoull(argv[3], nullptr, 0), 1000001, 6);
    if (what == "idle") {   // processor time of a copy that waits for the bus: the caller sleeps, the helpers have nothing to do
        umapb::CopyThreads& t = *new umapb::CopyThreads(3);
        std::vector<char> from(1 << 20), to(1 << 20);
        t.busy.store(true);
        t.copy(to.data(), from.data(), from.size());
        const std::clock_t start = std::clock();
        std::this_thread::sleep_for(std::chrono::milliseconds(500));
        std::printf("%.3f\n", static_cast<double>(std::clock() - start) / CLOCKS_PER_SEC);
        return 0;
    }
    return 2;
}
