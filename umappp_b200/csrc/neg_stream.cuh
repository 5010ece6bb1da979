// The negative samples of one firing edge: a counter-based stream keyed by the
// seed with counter (head, tail, epoch, block), so that the samples depend
// neither on the launch shape nor on how epochs are split across calls.
#pragma once

#include "common.cuh"

namespace umapb {

struct NegStream {
    uint32_t c0, c1, c2, c3, k0, k1;
    Philox4 buf;
    int used;
    __device__ __forceinline__ NegStream(uint32_t h, uint32_t t, uint32_t epoch, uint32_t key0, uint32_t key1)
        : c0(h), c1(t), c2(epoch), c3(0), k0(key0), k1(key1), used(4) {}
    __device__ __forceinline__ uint32_t next() {
        if (used == 4) {
            // 7 rounds: the fewest for which Salmon et al. found Philox4x32 free
            // of BigCrush failures; negative samples only need uniform,
            // independent indices
            buf = philox4x32<7>(c0, c1, c2, c3++, k0, k1);
            used = 0;
        }
        // a select chain rather than buf.v[used]: a dynamically indexed array would live in local memory
        const uint32_t v = used == 0 ? buf.v[0] : used == 1 ? buf.v[1] : used == 2 ? buf.v[2] : buf.v[3];
        ++used;
        return v;
    }
    // Exactly uniform integer in [0, n) (Lemire, "Fast random integer generation
    // in an interval", ACM TOMACS 2019): multiply-shift with rejection.
    __device__ __forceinline__ int32_t bounded(uint32_t n) {
        uint64_t m = static_cast<uint64_t>(next()) * n;
        uint32_t l = static_cast<uint32_t>(m);
        if (l < n) {
            const uint32_t thr = (0u - n) % n;
            while (l < thr) {
                m = static_cast<uint64_t>(next()) * n;
                l = static_cast<uint32_t>(m);
            }
        }
        return static_cast<int32_t>(m >> 32);
    }
};

}  // namespace umapb
