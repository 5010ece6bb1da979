// How a lane of the list builder (sgd_lists.cu) stores one firing edge's
// entries in its warp's shared stage.  Also compiled for the host, where a test
// runs a warp's lanes one after another in any order.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define UMAPB_LANE __host__ __device__ __forceinline__
#else
#define UMAPB_LANE inline
#endif

namespace umapb {

constexpr int STAGE_SAMPLES = 8;   // samples stored here; an edge's later ones come at the epoch's end

// The target, the first of the edge's 'draws' samples, and 'padding' (< 8) times
// the head behind them all (the edge that ends its row; else 0).  A lane without
// an edge stores nothing.  Each entry has one lane that stores it, so the
// stores of a warp need no order: predicated ones, where eight unconditional
// ones a lane, sorted out by the order of the lanes' instructions, would rest on
// lanes running in step.
UMAPB_LANE void stage_edge(int32_t* out, bool on, int32_t target, const int32_t (&sample)[STAGE_SAMPLES], uint32_t draws,
                           uint32_t padding, int32_t head) {
    if (on) out[0] = target;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (uint32_t i = 0; i < STAGE_SAMPLES; ++i)
        if (i < draws) out[1 + i] = sample[i];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (uint32_t i = 0; i < 7; ++i)
        if (i < padding) out[draws + 1 + i] = head;
}

}  // namespace umapb
