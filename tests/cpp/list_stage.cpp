// A warp's lanes store their edges' entries (list_stage.cuh) one after another
// in different orders: the stage has to hold the same list every time.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <numeric>
#include <random>
#include <vector>

#include "list_stage.cuh"

int main(int argc, char** argv) {
    const int most = argc > 1 ? std::atoi(argv[1]) : 8;   // samples per edge
    std::mt19937 rng(7 + most);
    int wrong = 0;
    for (int trial = 0; trial < 2000; ++trial) {
        struct Lane {
            bool on;
            uint32_t off, draws, padding;
            int32_t head, target, sample[umapb::STAGE_SAMPLES];
        } lane[32];
        const int edges = 1 + static_cast<int>(rng() % 32);
        std::vector<int32_t> want;
        int32_t head = 1000;
        for (int l = 0; l < 32; ++l) {
            Lane& x = lane[l];
            x = Lane{};
            x.on = l < edges;
            x.off = static_cast<uint32_t>(want.size());
            if (!x.on) continue;
            x.draws = rng() % (most + 1);
            x.head = head;
            x.target = static_cast<int32_t>(0x80000000u | (100000u * (l + 1)));
            want.push_back(x.target);
            for (uint32_t i = 0; i < x.draws; ++i) {
                const int32_t k = static_cast<int32_t>(100000 * (l + 1) + 1 + i);
                if (i < umapb::STAGE_SAMPLES) x.sample[i] = k;
                want.push_back(i < umapb::STAGE_SAMPLES ? k : -1);   // later samples are not stored here
            }
            if (l + 1 == edges || rng() % 3 == 0) {   // the row ends
                x.padding = static_cast<uint32_t>(-want.size()) & 7u;
                want.insert(want.end(), x.padding, x.head);
                ++head;
            }
        }
        for (int way = 0; way < 6; ++way) {
            std::vector<int> order(32);
            std::iota(order.begin(), order.end(), 0);
            if (way == 1) std::reverse(order.begin(), order.end());
            if (way > 1) std::shuffle(order.begin(), order.end(), rng);
            std::vector<int32_t> stage(want.size() + 64, -7);
            for (int l : order) {
                const Lane& x = lane[l];
                umapb::stage_edge(stage.data() + x.off, x.on, x.target, x.sample, x.draws, x.padding, x.head);
            }
            for (size_t i = 0; i < stage.size(); ++i)
                wrong += i < want.size() ? want[i] != -1 && stage[i] != want[i] : stage[i] != -7;
        }
    }
    std::printf("%d\n", wrong);
    return wrong != 0;
}
