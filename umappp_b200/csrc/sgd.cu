// optimize_layout on the device (include/umappp/optimize_layout.hpp:116-185).
//
// Rows.  The reference walks the heads in order and, for each head, its
// firing edges in CSR order: an attractive step that moves head and tail,
// then that edge's negative samples, which move the head only.  Here one
// thread (or a group of lanes, for layouts of more than four dimensions) takes
// the steps of one head's whole row in that order, from a flat list of the points the head
// meets in this epoch, which sgd_lists.cu has worked out ahead for a window of
// epochs: the schedule and the samples do not depend on the layout.  What is
// left is the chain that does: gather a point, take its step, move the head.
//
// Concurrency.  All rows of an epoch run at once (one launch per epoch), in a
// claim order fixed per epoch (epoch_order_kernel): chunks of rows of
// neighbouring index, rows that would end last ahead of them.  A row's head is
// kept in registers and its displacement is added to the embedding (vector
// atomic add) after every firing edge, or every eight entries (the relay
// kernel); tails move by vector atomic adds.  Measured on a
// 1,000,000-point mixture against the serial reference's edge cross-entropy:
// splitting a hub's row into concurrently processed pieces, or publishing the
// head's move only at the end of a long row, leaves the layout about 1-1.5 %
// tighter than the reference's; whole rows with the head published after each
// firing edge come within about 0.3 %, and so do the relays' at 5,000 and 40,000
// points.
#include <cub/cub.cuh>

#include <algorithm>
#include <cfloat>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "per_device.hpp"
#include "pow_pos.cuh"
#include "stages.cuh"
#include "umap_grad.cuh"

namespace umapb {

namespace {

constexpr int SCHED_BLOCK = 256;
constexpr int MAX_DIM = 64;

template <typename T>
struct FloatLimits;
template <>
struct FloatLimits<float> {
    static __device__ __forceinline__ float epsilon() { return FLT_EPSILON; }
};
template <>
struct FloatLimits<double> {
    static __device__ __forceinline__ double epsilon() { return DBL_EPSILON; }
};

// One schedule step of an edge at 'epoch' (optimize_layout.hpp:141-143,160-161,178-179).
template <typename T>
__device__ __forceinline__ bool schedule_step(T epoch, T eps, T epns, T& enext, T& enneg, int& nneg) {
    if (enext > epoch) return false;
    nneg = static_cast<int>((epoch - enneg) / epns);
    enext += eps;
    enneg += static_cast<T>(nneg) * epns;
    return true;
}

// Advances the schedule state by W epochs without any layout update.
template <typename T>
__global__ void sched_advance_kernel(int64_t nnz, const T* __restrict__ eps, T* __restrict__ enext, T* __restrict__ enneg,
                                     T rate, int e0, int W) {
    for (int64_t j = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; j < nnz; j += int64_t(gridDim.x) * blockDim.x) {
        const T ep = eps[j];
        const T epns = ep / rate;
        T en = enext[j], enn = enneg[j];
        for (int w = 0; w < W; ++w) {
            int nn;
            schedule_step<T>(static_cast<T>(e0 + w), ep, epns, en, enn, nn);
        }
        enext[j] = en;
        enneg[j] = enn;
    }
}

// Per-epoch totals of firing edges and negative samples drawn, from the schedule alone.
template <typename T>
__global__ void __launch_bounds__(SCHED_BLOCK) sched_totals_kernel(int64_t nnz, const T* __restrict__ eps,
                                                                   T* __restrict__ enext, T* __restrict__ enneg, T rate,
                                                                   int e0, int W,
                                                                   unsigned long long* __restrict__ totals) {
    typedef cub::BlockReduce<unsigned long long, SCHED_BLOCK> Reduce;
    __shared__ typename Reduce::TempStorage tmp;
    const int64_t j = static_cast<int64_t>(blockIdx.x) * SCHED_BLOCK + threadIdx.x;
    const bool valid = j < nnz;
    const T ep = valid ? eps[j] : T(1);
    const T epns = ep / rate;
    T en = valid ? enext[j] : T(0);
    T enn = valid ? enneg[j] : T(0);
    for (int w = 0; w < W; ++w) {
        int nn = 0;
        const bool fire = valid && schedule_step<T>(static_cast<T>(e0 + w), ep, epns, en, enn, nn);
        const int c = __syncthreads_count(fire);
        const unsigned long long negs = Reduce(tmp).Sum(fire && nn > 0 ? static_cast<unsigned long long>(nn) : 0ull);
        if (threadIdx.x == 0) {
            atomicAdd(&totals[2 * w], static_cast<unsigned long long>(c));
            atomicAdd(&totals[2 * w + 1], negs);
        }
        __syncthreads();
    }
    if (valid) {
        enext[j] = en;
        enneg[j] = enn;
    }
}

// ------------------------------------------------------------ row order --

// Rows per group of the claim order (row_order_key_kernel).
constexpr int ORDER_GROUP = 4096;
constexpr float RATE_UNIT = 256.0f;   // firing rates are summed as multiples of 1 / RATE_UNIT

// Firing rate of each row -- the sum of 1 / epochs_per_sample, the expected
// number of firing edges per epoch -- and their sum (in integers: the same
// whatever the order of the additions).
template <typename T>
__global__ void row_rate_kernel(int32_t n, const int64_t* __restrict__ ptr, const T* __restrict__ eps,
                                float* __restrict__ rate, unsigned long long* __restrict__ total) {
    unsigned long long sum = 0;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float r = 0.0f;
        for (int64_t j = ptr[i]; j < ptr[i + 1]; ++j) r += 1.0f / static_cast<float>(eps[j]);
        rate[i] = r;
        sum += static_cast<unsigned long long>(fminf(fmaxf(r, 0.0f), 1e9f) * RATE_UNIT);
    }
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0 && sum) atomicAdd(total, sum);
}

// Order key of each row, sorted ascending: groups of 'group' consecutive
// indices in index order, by descending rate within a group.  Rows in flight
// together then come from a narrow index range (the concurrency the layout's
// quality depends on), while the 32 rows a warp takes at once have similar
// lengths.  A row so long that, started in its own group's turn, it would
// still run when all other rows are done, goes to the last group from whose
// turn it ends in time: 'lanes' rows run at once, each lane for total / lanes
// in all, and group g starts after g / groups of that.  (Hubs are up to 50
// times the mean length: one taken in the last group's turn would decide the
// epoch's time.)
__global__ void row_order_key_kernel(int32_t n, const float* __restrict__ rate,
                                     const unsigned long long* __restrict__ total, int64_t lanes, int32_t group,
                                     uint64_t* __restrict__ key, int32_t* __restrict__ row) {
    const float span = static_cast<float>(static_cast<double>(*total) / (RATE_UNIT * static_cast<double>(lanes)));
    const int32_t groups = (n - 1) / group + 1;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float r = rate[i];
        const float slack = span > 0.0f ? fminf(fmaxf(1.0f - r / span, 0.0f), 1.0f) : 1.0f;   // of the epoch, after which it must have started
        const int32_t latest = static_cast<int32_t>(slack * static_cast<float>(groups));
        const uint32_t g = static_cast<uint32_t>(min(i / group, latest));
        key[i] = (static_cast<uint64_t>(g) << 32) | static_cast<uint64_t>(~__float_as_uint(fmaxf(r, 0.0f)));   // r >= 0: bits order as values
        row[i] = i;
    }
}

// Claim order of the epochs of a window (blockIdx.y): every chunk of
// ORDER_GROUP consecutive positions of the run's order sorted by descending
// number of entries in this epoch (equal counts, and counts of 4095 or more,
// in the run's order: a stable sort).  A chunk keeps its positions, so the
// rows in flight together still come from one index range, while the 32 rows
// a warp takes have nearly equal lists (and rows without entries come last).
constexpr int EPOCH_ORDER_THREADS = 512;
constexpr int EPOCH_ORDER_ITEMS = ORDER_GROUP / EPOCH_ORDER_THREADS;
__global__ void __launch_bounds__(EPOCH_ORDER_THREADS)
    epoch_order_kernel(const int32_t* __restrict__ run_order, int32_t n, bool sort, const ListSpan* __restrict__ span,
                       RowTask* __restrict__ tasks) {
    using Sort = cub::BlockRadixSort<uint32_t, EPOCH_ORDER_THREADS, EPOCH_ORDER_ITEMS, int32_t>;
    __shared__ typename Sort::TempStorage tmp;
    span += static_cast<int64_t>(blockIdx.y) * n;
    tasks += static_cast<int64_t>(blockIdx.y) * n;
    const int64_t first = static_cast<int64_t>(blockIdx.x) * ORDER_GROUP + threadIdx.x * EPOCH_ORDER_ITEMS;
    uint32_t key[EPOCH_ORDER_ITEMS];
    int32_t row[EPOCH_ORDER_ITEMS];
#pragma unroll
    for (int i = 0; i < EPOCH_ORDER_ITEMS; ++i) {   // blocked: item rank = position in the chunk
        const int64_t pos = first + i;
        row[i] = pos < n ? run_order[pos] : -1;
        key[i] = 4095u;   // past the end: last (and the stable sort keeps them behind rows without entries)
        if (pos < n) {
            const ListSpan sp = span[row[i]];
            key[i] = 4095u - min(sp.end - sp.start8 * LIST_ALIGN, 4095u);
        }
    }
    if (sort) Sort(tmp).Sort(key, row, 0, 12);
#pragma unroll
    for (int i = 0; i < EPOCH_ORDER_ITEMS; ++i) {
        if (first + i < n) {
            const ListSpan sp = span[row[i]];
            *reinterpret_cast<int4*>(tasks + first + i) =
                make_int4(row[i], static_cast<int>(sp.start8), static_cast<int>(sp.end - sp.start8 * LIST_ALIGN), 0);
        }
    }
}

// ---------------------------------------------------------- epoch kernels --

template <typename T>
struct StepParams {
    T a, b;
    T neg2ab;      // -2ab
    T gamma2b;     // 2 gamma b
    T alpha;
};

// clamp to [-4, 4] and floor to epsilon; a NaN gradient stays NaN, a NaN
// distance takes the floor, as the reference's comparisons have it
__device__ __forceinline__ float clamp4(float g) {
    asm("max.NaN.f32 %0, %0, 0fC0800000;\n\tmin.NaN.f32 %0, %0, 0f40800000;" : "+f"(g));
    return g;
}
__device__ __forceinline__ double clamp4(double g) {
    g = (g < -4.0) ? -4.0 : g;
    return (4.0 < g) ? 4.0 : g;
}
__device__ __forceinline__ float floor_eps(float d2) { return fmaxf(d2, FloatLimits<float>::epsilon()); }
__device__ __forceinline__ double floor_eps(double d2) {
    const double e = FloatLimits<double>::epsilon();
    return (e < d2) ? d2 : e;
}

// The gradient of one step (before the clamp) along every coordinate
// difference, optimize_layout.hpp:147-155 (attractive) and :170-176
// (repulsive): one power, one divide.
template <int NC>
__device__ __forceinline__ void step_gradient(double d2, bool attract, const double (&diff)[NC],
                                              const StepParams<double>& p, double (&g)[NC]) {
    const double q = pow_pos(d2, p.b);
    const double c = (attract ? p.neg2ab * q : p.gamma2b) / ((attract ? d2 : 0.001 + d2) * (p.a * q + 1.0));
#pragma unroll
    for (int j = 0; j < NC; ++j) g[j] = c * diff[j];
}

// FP32 layouts use the special-function unit's approximations (2^(b log2 d2)
// and a reciprocal; d2 is at least FLT_EPSILON, so no operand is subnormal):
// the step is stochastic and clamped, and the layout's cross-entropy was
// measured unchanged with libm's powf and IEEE division at a million points.
// A row is one chain of these steps, so the products are grouped to shorten
// it: after the power one fused multiply-add, the reciprocal and a product.
template <int NC>
__device__ __forceinline__ void step_gradient(float d2, bool attract, const float (&diff)[NC],
                                              const StepParams<float>& p, float (&g)[NC]) {
    float l, q, r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(d2));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(q) : "f"(l * p.b));
    const float e2 = attract ? d2 : 0.001f + d2, num = attract ? p.neg2ab : p.gamma2b;
    const float den = __fmaf_rn(e2 * p.a, q, e2);
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(den));
    const float c = num * (attract ? q : 1.0f) * r;
#pragma unroll
    for (int j = 0; j < NC; ++j) g[j] = c * diff[j];
}

// The transform's coefficients: the two written out apart (umap_grad.cuh).
template <typename T>
__device__ __forceinline__ T transform_coef(T d2, bool attract, const StepParams<T>& p) {
    constexpr bool fast = std::is_same<T, float>::value;
    return attract ? attract_dd2<fast>(d2, p.a, p.b, p.neg2ab) : repulse_dd2<fast>(d2, p.a, p.b, p.gamma2b, T(0.001));
}

// x + y z: fused for float layouts, separately rounded for double ones
__device__ __forceinline__ float madd(float x, float y, float z) { return __fmaf_rn(y, z, x); }
__device__ __forceinline__ double madd(double x, double y, double z) { return x + y * z; }

// Coherent device-scope load: ordered after this thread's own earlier atomic
// adds to the same address (per-location coherence), so a head re-read after
// its own publication sees it, plus whatever other threads have added.
__device__ __forceinline__ float ld_relaxed(const float* q) {
    float v;
    asm volatile("ld.relaxed.gpu.global.f32 %0, [%1];" : "=f"(v) : "l"(q) : "memory");
    return v;
}
__device__ __forceinline__ double ld_relaxed(const double* q) {
    double v;
    asm volatile("ld.relaxed.gpu.global.f64 %0, [%1];" : "=d"(v) : "l"(q) : "memory");
    return v;
}

// Vector and scalar adds to global memory where e is negative (predicated, not
// branched over: a chain of steps then stays one straight piece of code).
__device__ __forceinline__ void red_if_negative(int32_t e, float* q, float x) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %0, 0;\n\t@p red.relaxed.gpu.global.add.f32 [%1], %2;\n\t}" ::"r"(e),
                 "l"(q), "f"(x));
}
__device__ __forceinline__ void red_if_negative(int32_t e, double* q, double x) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %0, 0;\n\t@p red.relaxed.gpu.global.add.f64 [%1], %2;\n\t}" ::"r"(e),
                 "l"(q), "d"(x));
}
__device__ __forceinline__ void red_if_negative(int32_t e, float* q, float x, float y) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %0, 0;\n\t"
                 "@p red.relaxed.gpu.global.add.v2.f32 [%1], {%2, %3};\n\t}" ::"r"(e),
                 "l"(q), "f"(x), "f"(y));
}
__device__ __forceinline__ void red_if_negative(int32_t e, float* q, float x, float y, float z, float u) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.s32 p, %0, 0;\n\t"
                 "@p red.relaxed.gpu.global.add.v4.f32 [%1], {%2, %3, %4, %5};\n\t}" ::"r"(e),
                 "l"(q), "f"(x), "f"(y), "f"(z), "f"(u));
}

// A point as its lane group holds it: G lanes with NC coordinates each, lane g
// of the group the coordinates g, g + G, ...  G = 1: the whole point (dim = NC),
// read and added to as vectors where its size allows (the embedding is
// aligned to them, SgdEngine::run).
template <typename T, int NC, int G>
struct Point {
    T v[NC];
    __device__ __forceinline__ void load(const T* __restrict__ Y, int32_t k, int dim) {
        if constexpr (G == 1 && NC == 2 && sizeof(T) == 4) {
            const float2 q = __ldcg(reinterpret_cast<const float2*>(Y) + k);
            v[0] = q.x, v[1] = q.y;
        } else if constexpr (G == 1 && NC == 4 && sizeof(T) == 4) {
            const float4 q = __ldcg(reinterpret_cast<const float4*>(Y) + k);
            v[0] = q.x, v[1] = q.y, v[2] = q.z, v[3] = q.w;
        } else if constexpr (G == 1 && NC % 2 == 0) {
#pragma unroll
            for (int j = 0; j < NC / 2; ++j) {
                const double2 q = __ldcg(reinterpret_cast<const double2*>(Y) + static_cast<int64_t>(k) * (NC / 2) + j);
                v[2 * j] = q.x, v[2 * j + 1] = q.y;
            }
        } else {
            each(Y, k, dim, [](T& x, const T* q) { x = __ldcg(q); });
        }
    }
    __device__ __forceinline__ void reload(const T* Y, int32_t k, int dim) {
        each(Y, k, dim, [](T& x, const T* q) { x = ld_relaxed(q); });
    }
    // Adds the coordinates to point k where e is negative.
    __device__ __forceinline__ void add_if_negative(int32_t e, T* __restrict__ Y, int32_t k, int dim) const {
        T* q = Y + static_cast<int64_t>(k) * (G == 1 ? NC : dim);
        if constexpr (G == 1 && NC == 2 && sizeof(T) == 4) {
            red_if_negative(e, q, v[0], v[1]);
        } else if constexpr (G == 1 && NC == 4 && sizeof(T) == 4) {
            red_if_negative(e, q, v[0], v[1], v[2], v[3]);
        } else {
            const int g = threadIdx.x & (G - 1);
#pragma unroll
            for (int j = 0; j < NC; ++j) {
                const int c = g + j * G;
                red_if_negative(G == 1 || c < dim ? e : 0, q + c, v[j]);
            }
        }
    }
    template <class F>
    __device__ __forceinline__ void each(const T* Y, int32_t k, int dim, F f) {
        const T* row = Y + static_cast<int64_t>(k) * (G == 1 ? NC : dim);
        const int g = threadIdx.x & (G - 1);
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            if (G == 1) f(v[j], row + j);
            else if (g + j * G < dim) f(v[j], row + g + j * G);
            else v[j] = T(0);
        }
    }
};

// CH entries of a list, from an address aligned to them.
template <int CH>
struct Entries {
    int32_t e[CH];
    __device__ __forceinline__ void load(const int32_t* __restrict__ p) {
#pragma unroll
        for (int i = 0; i < CH; i += 4) {
            const int4 q = __ldg(reinterpret_cast<const int4*>(p + i));
            e[i] = q.x, e[i + 1] = q.y, e[i + 2] = q.z, e[i + 3] = q.w;
        }
    }
    __device__ __forceinline__ int32_t point(int i) const { return e[i] & INT32_MAX; }
};

// The first entries of a row's list, read ahead.
template <int CH>
struct ListHead {
    const int32_t* p;
    uint32_t cnt, chunks;
    Entries<CH> e0, e1;
    __device__ __forceinline__ void load(const int32_t* __restrict__ list, uint32_t start8, uint32_t count) {
        p = list + static_cast<int64_t>(start8) * LIST_ALIGN;
        cnt = count;
        chunks = (count + CH - 1) / CH;
        if (chunks) e0.load(p);
        if (chunks > 1) e1.load(p + CH);
    }
};

// One entry's step: moves head by its gradient at y (times rate); pull is the
// opposite move, the target's where the entry is one.
template <bool FIXED, typename T, int NC, int G>
__device__ __forceinline__ void take_step(Point<T, NC, G>& head, const Point<T, NC, G>& y, bool attract, T rate,
                                          const StepParams<T>& p, Point<T, NC, G>& pull) {
    T diff[NC], d2 = 0, grad[NC];
#pragma unroll
    for (int j = 0; j < NC; ++j) {
        diff[j] = head.v[j] - y.v[j];
        d2 = FIXED ? d2 + diff[j] * diff[j] : madd(d2, diff[j], diff[j]);
    }
    if constexpr (G > 1) {   // the group's lanes share the row
        const unsigned group = (G == 32 ? 0xffffffffu : (1u << G) - 1u) << (threadIdx.x & 31 & ~(G - 1));
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) d2 += __shfl_xor_sync(group, d2, o, G);
    }
    d2 = floor_eps(d2);
    if constexpr (FIXED) {
        const T cf = transform_coef(d2, attract, p);
#pragma unroll
        for (int j = 0; j < NC; ++j) grad[j] = cf * diff[j];
    } else {
        step_gradient(d2, attract, diff, p, grad);
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) {
        const T g = clamp4(grad[j]);
        head.v[j] = FIXED ? head.v[j] + rate * g : madd(head.v[j], rate, g);
        pull.v[j] = -(rate * g);
    }
}

// One row's list applied to its head, CH entries at a time: while CH steps
// run, the points of the next CH are gathered and the entries after those
// read.  The head's move is published at every firing edge, together with the
// edge's own pull on its tail, and a long row's head re-read after every 256
// entries, with the other rows' pulls on it.  (The head's move
// published once per 8 entries: 24.2 ms against 22.0 for a batch of 91,000
// points, 173.5 against 170.5 for a million; with the pulls kept in shared
// memory and added then, too: 25.7 and 177.)
// What bounds a row is the chain of its steps -- some 100 cycles each of
// dependent arithmetic -- so the steps are straight code of few instructions:
// the lists are padded with the head itself, and an entry equal to the head
// (padding, or a sample that hit it) takes a step of rate 0.
// FIXED (transform): only the head moves, it is not published, and the list's
// padding is not read.  A row without entries does nothing.
template <typename T, int NC, int G, int CH, bool FIXED>
struct RowWalk {
    Point<T, NC, G>& head;
    const int32_t h;
    const ListHead<CH>& l;
    T* __restrict__ Y;
    const int dim;
    const StepParams<T>& p;
    Point<T, NC, G> pub;

    __device__ __forceinline__ void gather(Point<T, NC, G> (&y)[CH], const Entries<CH>& e, uint32_t c) {
        if (c < l.chunks) {
#pragma unroll
            for (int i = 0; i < CH; ++i)
                if (!FIXED || c * CH + i < l.cnt) y[i].load(Y, e.point(i), dim);
        }
    }
    // Where e is negative.
    __device__ __forceinline__ void publish(int32_t e) {
        Point<T, NC, G> d;
#pragma unroll
        for (int j = 0; j < NC; ++j) {
            d.v[j] = head.v[j] - pub.v[j];
            pub.v[j] = e < 0 ? head.v[j] : pub.v[j];
        }
        d.add_if_negative(e, Y, h, dim);
    }
    // Chunk c's entries e at the points y; chunk c + 1 is gathered from en to
    // yn, and chunk c + 2 takes the place of e.
    __device__ __forceinline__ void chunk(uint32_t c, Entries<CH>& e, const Point<T, NC, G> (&y)[CH],
                                          const Entries<CH>& en, Point<T, NC, G> (&yn)[CH]) {
        gather(yn, en, c + 1);
        Entries<CH> far;
        if (c + 2 < l.chunks) far.load(l.p + (c + 2) * CH);
        if (!FIXED && c > 0 && c % (256 / CH) == 0) {
            publish(-1);
            head.reload(Y, h, dim);
            pub = head;
        }
#pragma unroll
        for (int i = 0; i < CH; ++i) {
            const T rate = (FIXED ? c * CH + i < l.cnt : e.e[i] != h) ? p.alpha : T(0);
            Point<T, NC, G> pull;
            take_step<FIXED>(head, y[i], e.e[i] < 0, rate, p, pull);
            if (!FIXED) {
                pull.add_if_negative(e.e[i], Y, e.point(i), dim);
                publish(e.e[i]);
            }
        }
        e = far;
    }
    __device__ __forceinline__ void run() {
        Entries<CH> e0 = l.e0, e1 = l.e1;
        Point<T, NC, G> y0[CH], y1[CH];
#pragma unroll
        for (int i = 0; i < CH; ++i) y0[i] = y1[i] = head;
        gather(y0, e0, 0);
        for (uint32_t c = 0; c < l.chunks; c += 2) {
            chunk(c, e0, y0, e1, y1);
            if (c + 1 < l.chunks) chunk(c + 1, e1, y1, e0, y0);
        }
        if (!FIXED && l.chunks) publish(-1);
    }
};

template <typename T, int NC, int G, int CH, bool FIXED>
__device__ __forceinline__ void walk_row(Point<T, NC, G>& head, int32_t h, const ListHead<CH>& l, T* __restrict__ Y,
                                         int dim, const StepParams<T>& p) {
    RowWalk<T, NC, G, CH, FIXED> w{head, h, l, Y, dim, p, head};
    w.run();
}

constexpr int ROW_BLOCK = 64;
constexpr int ROW_BLOCKS = 4;   // resident per SM

// One epoch: warps claim 32 / G rows at a time in the epoch's order, one claim
// ahead, and the next rows' first entries are read while the current rows run.
template <typename T, int NC, int G, int CH>
__global__ void __launch_bounds__(ROW_BLOCK, ROW_BLOCKS)
    sgd_rows_kernel(const RowTask* __restrict__ tasks, int32_t nrows, const int32_t* __restrict__ list,
                    T* __restrict__ Y, int dim, int* __restrict__ counter, const StepParams<T> p) {
    const int lane = threadIdx.x & 31;
    auto claim = [&](RowTask& r) {   // false: none left
        int32_t base = 0;
        if (lane == 0) base = atomicAdd(counter, 32 / G);
        base = __shfl_sync(0xffffffffu, base, 0);
        const int32_t i = base + lane / G;
        r = RowTask{0, 0, 0, 0};
        if (i < nrows) {
            const int4 q = __ldg(reinterpret_cast<const int4*>(tasks) + i);
            r = RowTask{q.x, static_cast<uint32_t>(q.y), static_cast<uint32_t>(q.z), 0};
        }
        return base < nrows;
    };
    RowTask cur, nxt;
    if (!claim(cur)) return;
    ListHead<CH> head_of_list;
    head_of_list.load(list, cur.start8, cur.count);
    while (true) {
        const bool more = claim(nxt);
        Point<T, NC, G> head;
        head.load(Y, cur.row, dim);
        walk_row<T, NC, G, CH, false>(head, cur.row, head_of_list, Y, dim, p);
        __syncwarp();
        if (!more) break;
        cur = nxt;
        head_of_list.load(list, cur.start8, cur.count);
    }
}

// ------------------------------------------ few rows in flight: the relay --
// Three warps work on the same rows ('share' of them, at most 32 / G), a chunk
// of CH entries of each at a time.  The first (fetch_rows) claims the rows in
// the epoch's order, reads their lists, gathers the points and leaves them in
// shared memory; the second (walk_chunk) takes the steps and does nothing
// else; the third (publish_rows) adds a chunk's moves to the embedding: every
// firing edge's pull on its tail, and the head's move.
// With few rows in flight an epoch takes as long as its longest row's chain of
// steps.  The dependent arithmetic of a step is 111 cycles (2-d float); in a
// warp that gathers and adds by itself it takes 205 with one row and 258 with
// 32, as a lone warp issues an instruction every 4-5 cycles and each add to
// global memory holds it up for some 40, active lanes or none.  Here it takes
// 142 with up to 8 rows, 227 with 32.  Where the SMs are full the three warps'
// instructions cost more than the chain (relay_rows()).
// About every RELOAD entries a head takes over the other rows' pulls on it.
constexpr int RELAY_WARPS = 3;
constexpr uint32_t RELOAD = 256;
// READY: points are there (fetching -> walking warp); DONE: steps are done
// (walking -> fetching and publishing warp).  Each for two buffers.
// START: the first chunk's kind is there, for the publishing warp.
enum RowBarrier { READY = 1, DONE = 3, START = 5 };

template <int ID, int WARPS>
__device__ __forceinline__ void row_sync() {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"n"(ID), "n"(32 * WARPS) : "memory");
}
template <int ID, int WARPS>
__device__ __forceinline__ void row_arrive() {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"n"(ID), "n"(32 * WARPS) : "memory");
}

// What the warps hand one another.  Chunk s has its points in buffer s % 2,
// which is filled again once the steps are done, and its moves in set s % 4,
// which chunk s + 4 uses: it is fetched after DONE of chunk s + 2, where the
// publishing warp arrives when it is done with chunk s + 1.
// A MEASURE chunk's publication finds out what others have added to the heads;
// the SHIFT chunk, three later, takes it over.
enum ChunkKind { CHUNK_NEXT, CHUNK_FIRST, CHUNK_MEASURE, CHUNK_SHIFT, CHUNK_STOP };
template <typename T, int NC, int CH>
struct RowMail {
    // a point or move with its entry: one access where they fit one
    static constexpr bool packed = NC * sizeof(T) < 16;
    struct alignas(NC * sizeof(T) > 4 ? 16 : 8) Packed {
        T v[NC];
        int32_t e;
    };
    struct alignas(16) Vector {
        T v[NC];
    };
    struct Split {
        Vector at[CH][32];
        int32_t e[CH][32];
    };
    struct Joint {
        Packed at[CH][32];
    };
    using Items = typename std::conditional<packed, Joint, Split>::type;
    template <int G>
    static __device__ __forceinline__ void put(Items& m, int i, int lane, const Point<T, NC, G>& y, int32_t e) {
        if constexpr (packed) {
            Packed q;
#pragma unroll
            for (int j = 0; j < NC; ++j) q.v[j] = y.v[j];
            q.e = e;
            m.at[i][lane] = q;
        } else {
            Vector q;
#pragma unroll
            for (int j = 0; j < NC; ++j) q.v[j] = y.v[j];
            m.at[i][lane] = q;
            m.e[i][lane] = e;
        }
    }
    template <int G>
    static __device__ __forceinline__ int32_t get(const Items& m, int i, int lane, Point<T, NC, G>& y) {
        const auto q = m.at[i][lane];
#pragma unroll
        for (int j = 0; j < NC; ++j) y.v[j] = q.v[j];
        if constexpr (packed) return q.e;
        else return m.e[i][lane];
    }
    struct Place {
        T v[NC];
    };
    Items point[2];          // the entries' points
    Items pull[2][2];        // [s / 2 % 2][s % 2] from here on: the pulls at firing edges, and their tails
    Place last[2][2][32];    // where the heads are in the end
    Place start[2][2][32];   // where they are first (CHUNK_FIRST)
    int32_t row[2][2][32];
    uint32_t edges[2][2][32];   // which entries are firing edges; bit 31: the row has entries here
    int kind[2][2];
    Place shift[32];         // what the heads take over
};

// One chunk's steps; false: there are no more.
template <int B, typename T, int NC, int G, int CH>
__device__ __forceinline__ bool walk_chunk(RowMail<T, NC, CH>& m, int half, Point<T, NC, G>& head, int32_t& h,
                                           const StepParams<T>& p, int lane) {
    row_sync<READY + B, 2>();
    const int kind = m.kind[half][B];
    if (kind == CHUNK_STOP) return false;
    if (kind == CHUNK_FIRST) {
        h = m.row[half][B][lane];
#pragma unroll
        for (int j = 0; j < NC; ++j) head.v[j] = m.start[half][B][lane].v[j];
    } else if (kind == CHUNK_SHIFT) {
#pragma unroll
        for (int j = 0; j < NC; ++j) head.v[j] += m.shift[lane].v[j];
    }
    Point<T, NC, G> y[CH];
    int32_t e[CH];
#pragma unroll
    for (int i = 0; i < CH; ++i) e[i] = RowMail<T, NC, CH>::get(m.point[B], i, lane, y[i]);
#pragma unroll
    for (int i = 0; i < CH; ++i) {
        Point<T, NC, G> pull;
        take_step<false>(head, y[i], e[i] < 0, e[i] != h ? p.alpha : T(0), p, pull);
        if (e[i] < 0) RowMail<T, NC, CH>::put(m.pull[half][B], i, lane, pull, e[i] & INT32_MAX);
    }
#pragma unroll
    for (int j = 0; j < NC; ++j) m.last[half][B][lane].v[j] = head.v[j];
    row_arrive<DONE + B, 3>();
    return true;
}

// The fetching warp's way along the lists of its rows, chunk by chunk.  Rows are
// claimed when the lists at hand are about to end, not earlier: a claimed row
// waits for the longest one before it.
template <typename T, int NC, int G, int CH>
struct RowCursor {
    const RowTask* __restrict__ tasks;
    const int32_t nrows;
    const int32_t* __restrict__ lists;
    int* __restrict__ counter;
    const int share;   // rows claimed at a time
    const int lane;
    // of the chunk last read
    Entries<CH> e;
    int32_t h = 0;
    bool on = false;          // the row has entries here
    int kind = CHUNK_FIRST;
    // of the rows at hand, and the next claim
    const int32_t* list = nullptr;
    uint32_t c = 0, chunks = 0, most = 0;
    int32_t base = 0;
    int4 task = make_int4(0, 0, 0, 0);
    bool claimed = false, fetched = false;

    __device__ __forceinline__ void claim() {
        if (lane == 0) base = atomicAdd(counter, share);
        claimed = true;
    }
    __device__ __forceinline__ void fetch() {
        base = __shfl_sync(0xffffffffu, base, 0);
        const int32_t i = base + lane / G;
        task = lane / G < share && i < nrows ? __ldg(reinterpret_cast<const int4*>(tasks) + i) : make_int4(0, 0, 0, 0);
        fetched = true;
    }
    __device__ __forceinline__ void read() {
        const uint32_t phase = c % (RELOAD / CH);
        kind = c < RELOAD / CH || (phase != 0 && phase != 3) ? CHUNK_NEXT : phase == 0 ? CHUNK_MEASURE : CHUNK_SHIFT;
        while (c >= most) {
            if (!claimed) claim();
            if (!fetched) fetch();
            if (base >= nrows) {
                kind = CHUNK_STOP;
                on = false;
                return;
            }
            h = task.x;
            list = lists + static_cast<int64_t>(static_cast<uint32_t>(task.y)) * LIST_ALIGN;
            chunks = (static_cast<uint32_t>(task.z) + CH - 1) / CH;
            most = __reduce_max_sync(0xffffffffu, chunks);
            c = 0;
            claimed = fetched = false;
            kind = CHUNK_FIRST;
        }
        if (claimed && !fetched) fetch();
        if (c + 3 >= most && !claimed) claim();
        on = c < chunks;
#pragma unroll
        for (int i = 0; i < CH; ++i) e.e[i] = h;
        if (on) e.load(list + c * CH);
        ++c;
    }
};

template <typename T, int NC, int G, int CH>
__device__ __forceinline__ void fetch_rows(RowMail<T, NC, CH>& m, const RowTask* __restrict__ tasks, int32_t nrows,
                                           const int32_t* __restrict__ lists, const T* __restrict__ Y, int dim,
                                           int* __restrict__ counter, int share, int lane) {
    RowCursor<T, NC, G, CH> ahead{tasks, nrows, lists, counter, share, lane};
    // the chunk whose points are being gathered
    Entries<CH> e;
    int32_t h;
    bool on;
    int kind;
    Point<T, NC, G> y[CH], head;
#pragma unroll
    for (int i = 0; i < CH; ++i)
#pragma unroll
        for (int j = 0; j < NC; ++j) y[i].v[j] = head.v[j] = T(0);
    auto gather = [&] {
        e = ahead.e, h = ahead.h, on = ahead.on, kind = ahead.kind;
        if (kind == CHUNK_STOP) return;
        if (on) {
#pragma unroll
            for (int i = 0; i < CH; ++i) y[i].load(Y, e.point(i), dim);
        }
        if (kind == CHUNK_FIRST) head.load(Y, h, dim);
        ahead.read();
    };
    int filled[2];   // the chunks' kinds
    auto fill = [&](int half, auto buffer) {
        constexpr int B = decltype(buffer)::value;
        filled[B] = kind;
        if (lane == 0) m.kind[half][B] = kind;
        if (kind != CHUNK_STOP) {
            uint32_t fires = on ? 1u << 31 : 0u;
#pragma unroll
            for (int i = 0; i < CH; ++i) {
                RowMail<T, NC, CH>::put(m.point[B], i, lane, y[i], e.e[i]);
                fires |= (static_cast<uint32_t>(e.e[i]) >> 31) << i;
            }
            m.edges[half][B][lane] = fires;
            if (kind == CHUNK_FIRST) {
                m.row[half][B][lane] = h;
#pragma unroll
                for (int j = 0; j < NC; ++j) m.start[half][B][lane].v[j] = head.v[j];
            }
        }
        row_arrive<READY + B, 2>();
    };
    using Zero = std::integral_constant<int, 0>;
    using One = std::integral_constant<int, 1>;
    // Once the steps of buffer B's chunk are done it is filled again, and the
    // points of the chunk after that are gathered.  False: the chunks end.
    int half = 0;
    auto turn = [&](auto buffer) {
        constexpr int B = decltype(buffer)::value;
        row_sync<DONE + B, 3>();
        if (filled[1 - B] == CHUNK_STOP) return false;
        fill(half ^ 1, buffer);
        if (kind != CHUNK_STOP) gather();
        return true;
    };
    ahead.read();
    gather();
    fill(0, Zero());
    row_arrive<START, 2>();
    if (kind == CHUNK_STOP) return;
    gather();
    fill(0, One());
    if (kind != CHUNK_STOP) gather();
    for (; turn(Zero()) && turn(One()); half ^= 1) {
    }
}

// Adds one chunk's moves; false: there are no more.
template <int B, typename T, int NC, int G, int CH>
__device__ __forceinline__ bool publish_chunk(RowMail<T, NC, CH>& m, int half, Point<T, NC, G>& pub, int32_t& h,
                                              T* __restrict__ Y, int dim, int lane) {
    const int kind = m.kind[half][B];   // written before DONE of the chunk before (or START)
    if (kind == CHUNK_STOP) return false;
    row_sync<DONE + B, 3>();
    if (kind == CHUNK_FIRST) {
        h = m.row[half][B][lane];
#pragma unroll
        for (int j = 0; j < NC; ++j) pub.v[j] = m.start[half][B][lane].v[j];
    } else if (kind == CHUNK_SHIFT) {
#pragma unroll
        for (int j = 0; j < NC; ++j) pub.v[j] += m.shift[lane].v[j];
    }
    const uint32_t edges = m.edges[half][B][lane];
    const bool on = edges >> 31;
    uint32_t left = edges & 0x7fffffffu;
    while (__any_sync(0xffffffffu, left)) {   // each lane's next firing edge
        Point<T, NC, G> pull;
        const int32_t tail = RowMail<T, NC, CH>::get(m.pull[half][B], left ? __ffs(left) - 1 : 0, lane, pull);
        pull.add_if_negative(left ? -1 : 0, Y, tail, dim);
        left &= left - 1;
    }
    Point<T, NC, G> move;
#pragma unroll
    for (int j = 0; j < NC; ++j) {
        const T at = m.last[half][B][lane].v[j];
        move.v[j] = at - pub.v[j];
        pub.v[j] = at;
    }
    move.add_if_negative(on ? -1 : 0, Y, h, dim);
    if (kind == CHUNK_MEASURE) {   // what is there beyond what was added from here
        Point<T, NC, G> now;
        if (on) now.reload(Y, h, dim);
#pragma unroll
        for (int j = 0; j < NC; ++j) m.shift[lane].v[j] = on ? now.v[j] - pub.v[j] : T(0);
    }
    return true;
}

// One epoch by relays.
template <typename T, int NC, int G, int CH>
__global__ void __launch_bounds__(32 * RELAY_WARPS, NC == 1 || G == 1 && NC * sizeof(T) < 16 ? 8 : 6)
    sgd_relay_kernel(const RowTask* __restrict__ tasks, int32_t nrows, const int32_t* __restrict__ list,
                    T* __restrict__ Y, int dim, int* __restrict__ counter, int share, const StepParams<T> p) {
    __shared__ RowMail<T, NC, CH> mail;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp == 0) {
        fetch_rows<T, NC, G, CH>(mail, tasks, nrows, list, Y, dim, counter, share, lane);
        return;
    }
    Point<T, NC, G> head;
    int32_t h = 0;
#pragma unroll
    for (int j = 0; j < NC; ++j) head.v[j] = T(0);
    if (warp == 1) {
        for (int half = 0; walk_chunk<0>(mail, half, head, h, p, lane) && walk_chunk<1>(mail, half, head, h, p, lane);
             half ^= 1) {
        }
        return;
    }
    row_sync<START, 2>();
    for (int half = 0; publish_chunk<0>(mail, half, head, h, Y, dim, lane) &&
                       publish_chunk<1>(mail, half, head, h, Y, dim, lane);
         half ^= 1) {
    }
}

// ------------------------------------------------------------ transform --
// Out-of-sample embedding (no counterpart in the reference: optimize_layout
// applied to points added to a finished layout).  Row i of the transform
// graph holds new point i's nearest reference points with their smoothed
// similarities; it is optimised like a row of optimize_layout
// (optimize_layout.hpp:136-180: schedule, attractive step, negative samples)
// except that only the new point moves: the reference points it is pulled to
// and the negative samples, drawn among the reference points, stay fixed.
// Rows then share nothing that changes, so one thread (or lane group) takes
// one row through all epochs of a window in one launch and the result does
// not depend on the launch shape.

// Initial position of every new point: the mean of its neighbours' reference
// positions weighted by the similarities (FP64 sums in edge order; plain mean
// if the weights sum to zero).
template <typename T>
__global__ void transform_init_kernel(int32_t nq, int dim, const int64_t* __restrict__ ptr,
                                      const int32_t* __restrict__ idx, const T* __restrict__ w,
                                      const T* __restrict__ Yref, T* __restrict__ Ynew) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x) {
        const int64_t r0 = ptr[i], r1 = ptr[i + 1];
        double ws = 0;
        for (int64_t j = r0; j < r1; ++j) ws += static_cast<double>(w[j]);
        const bool weighted = ws > 0;
        const double den = weighted ? ws : static_cast<double>(r1 - r0);
        for (int d = 0; d < dim; ++d) {
            double acc = 0;
            for (int64_t j = r0; j < r1; ++j) {
                const double wj = weighted ? static_cast<double>(w[j]) : 1.0;
                acc += wj * static_cast<double>(Yref[static_cast<size_t>(idx[j]) * dim + d]);
            }
            Ynew[static_cast<size_t>(i) * dim + d] = static_cast<T>(den > 0 ? acc / den : 0.0);
        }
    }
}

// The epochs [first, first + epochs) of every new point's row (lane group i: row i).
template <typename T, int NC, int G, int CH>
__global__ void __launch_bounds__(ROW_BLOCK, ROW_BLOCKS)
    transform_rows_kernel(int32_t nq, const ListSpan* __restrict__ span, const int32_t* __restrict__ list,
                          const T* __restrict__ Yref, T* __restrict__ Ynew, int dim, int first, int epochs, int total,
                          T lr, StepParams<T> p) {
    const int64_t i = (static_cast<int64_t>(blockIdx.x) * ROW_BLOCK + threadIdx.x) / G;
    const int32_t row = i < nq ? static_cast<int32_t>(i) : 0;
    Point<T, NC, G> head;
    head.load(Ynew, row, dim);
    for (int e = 0; e < epochs; ++e) {
        const T ef = static_cast<T>(first + e);
        // alpha as in the layout's epochs (optimize_layout.hpp:132-133)
        p.alpha = static_cast<T>(static_cast<double>(lr) * (1.0 - static_cast<double>(ef / static_cast<T>(total))));
        const ListSpan sp = span[static_cast<int64_t>(e) * nq + row];
        ListHead<CH> l;
        l.load(list, sp.start8, i < nq ? sp.end - sp.start8 * LIST_ALIGN : 0u);
        walk_row<T, NC, G, CH, true>(head, row, l, const_cast<T*>(Yref), dim, p);
    }
    if (i < nq) head.each(Ynew, row, dim, [](T& x, const T* q) { *const_cast<T*>(q) = x; });
}

// out, rows of 'to' coordinates, from in, rows of 'from' (the missing ones 0).
template <typename T>
__global__ void restride_kernel(size_t values, const T* __restrict__ in, int from, T* __restrict__ out, int to) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < values; i += size_t(gridDim.x) * blockDim.x) {
        const size_t row = i / to;
        const int c = static_cast<int>(i % to);
        out[i] = c < from ? in[row * from + c] : T(0);
    }
}

// Calls f with the coordinates per lane, lanes per row and entries in flight
// for a layout of 'dim' dimensions: one thread per row while the points in
// flight fit its registers, else the smallest group of lanes.
template <typename T, class F>
void for_dim(int dim, F f) {
    using std::integral_constant;
    auto go = [&](auto nc, auto g, auto ch) { f(nc, g, ch); };
    // gathers in flight per lane cover an L2 access: 8 float steps, 4 double ones
    constexpr int deep = sizeof(T) == 4 ? 8 : 4;
#define UMAPB_SHAPE(NC, G, CH) go(integral_constant<int, NC>(), integral_constant<int, G>(), integral_constant<int, CH>())
    if (dim == 1) UMAPB_SHAPE(1, 1, deep);
    else if (dim == 2) UMAPB_SHAPE(2, 1, deep);
    else if (dim == 4) UMAPB_SHAPE(4, 1, deep);
    else if (dim <= 8) UMAPB_SHAPE(1, 8, deep);
    else if (dim <= 16) UMAPB_SHAPE(1, 16, deep);
    else if (dim <= 32) UMAPB_SHAPE(1, 32, deep);
    else UMAPB_SHAPE(2, 32, deep);
#undef UMAPB_SHAPE
}

// UMAPB_CHECK_SCHEDULE=1: the lists' firing edges and negative samples are
// counted as they are written, and every run compares the counts with the
// schedule's own totals (sched_totals_kernel).
bool check_schedule() {
    const char* e = std::getenv("UMAPB_CHECK_SCHEDULE");
    return e && *e && *e != '0';
}

// Bytes of interaction lists held at once: at a million points ten epochs (the
// schedule state is read and written once a window: 126 ms a run with 2 GB, 135
// with 1 GB, 124 with 4 GB).  Windows of several epochs stay within an eighth
// above it, whatever the sample rate.  UMAPB_SGD_WINDOW_BYTES overrides it.
size_t window_bytes() {
    const char* e = std::getenv("UMAPB_SGD_WINDOW_BYTES");
    return e && *e ? static_cast<size_t>(std::max(1ll, std::atoll(e))) : size_t(1) << 31;
}

// Calls of at most this many epochs have their lists read ahead (SgdEngine::run).
constexpr int FEW_EPOCHS = 8;

// Rows in flight at once: at most n / window_div (a sliding window over the
// claim order), so that few rows run beside their neighbours with positions
// read before those neighbours' updates, in steps of 256; small layouts take
// min(n / 8, 32768).  At most 256 per SM: with eight gathers in flight each
// they keep the SM's gather rate (one point per cycle) busy, and more leave
// the longest rows a smaller share of it: a million points, 200 epochs take
// 131 ms with 256, 148 with 512, 139 with 192.
int64_t rows_in_flight(int32_t n, int window_div) {
    const int64_t most = int64_t(ROW_BLOCK * ROW_BLOCKS) * sm_count();
    if (window_div <= 0) return most;
    const int64_t w = std::max<int64_t>(1, std::max<int64_t>(n / window_div, std::min<int64_t>(n / 8, 32768)));
    return std::min(most, (w + 255) / 256 * 256);
}

// Blocks of an epoch kernel that are resident at once on the device.
template <class K>
int64_t resident_blocks(K kernel, int threads) {
    int r = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&r, kernel, threads, 0) != cudaSuccess || r < 1) {
        cudaGetLastError();
        r = 1;
    }
    return static_cast<int64_t>(r) * sm_count();
}

// Whether an epoch with this many rows in flight is run by relays: as long as
// its time is the longest rows' chains rather than what the SMs issue.  With more
// lanes per row a warp has fewer rows, and the relays that are resident (six to
// eight per SM) are out sooner.  ms for 15 neighbours, relays / single warps (epochs):
//   2 x f32 (50)  45,000 points 3.55 / 4.26, 70,000 4.82 / 4.51
//   5 x f32 (20)  45,000 1.65 / 2.48        10 x f32 (20)  45,000 2.84 / 2.91, 55,000 3.37 / 3.26
//   40 x f32 (30) 8,000 2.46 / 3.14, 12,000 3.44 / 3.34; (20) 45,000 7.57 / 5.00
//   2 x f64 (20)  45,000 2.84 / 4.16        5 x f64 (20)  45,000 3.84 / 4.69
//   10 x f64 (30) 20,000 5.57 / 6.60, 36,000 8.85 / 7.96
//   40 x f64 (30) 8,000 5.57 / 6.07, 12,000 8.05 / 6.46; (20) 45,000 18.3 / 10.3
// (an eighth of the points are in flight up to 262,144; 8 and fewer dimensions, and
// doubles of up to 4, would gain from relays beyond 6,144 rows: 55,000 x 5 f32 1.90 /
// 2.54, 100,000 x 2 f64 3.41 / 4.64.)
template <typename T, int G>
bool relay_rows(int64_t rows) {
    constexpr bool twice = sizeof(T) == 8;
    return rows <= (G == 32 ? (twice ? 1024 : 1536) : G == 16 && twice ? 3072 : 6144);
}

// Rows per relay: the fewest with which RELAY_BLOCKS per SM hold all rows (a
// relay's steps are faster with few rows, and it waits for the longest of
// them).  10,007 x 2 points, 500 epochs: 42.8 ms with 2, 43.7 with 4, 45.7 with
// 16, and 45.2 with 1, when there are more relays than run at once.
constexpr int RELAY_BLOCKS = 5;
template <int G>
int relay_share(int64_t rows) {
    int share = 1;
    while (share < 32 / G && rows > int64_t(RELAY_BLOCKS) * sm_count() * share) share *= 2;
    return share;
}

// Whether an epoch's rows are sorted by their entries.  Not where every row in
// flight has a relay of its own (up to some 5,900 points in up to 4 dimensions):
// there are no lists to match, and longest first puts an epoch's busiest rows,
// which pull on one another, side by side.  2,000 points, mean cross-entropy
// against the serial reference's (some 110 to 150 x 16 runs each, standard error
// 0.02 %): -0.52 % f64 and -0.54 % f32 sorted, -0.39 % both in the run's order (as
// before the lists: -0.40 %, 26 x 16 runs), for 6 % of the time (1,000 points, 500
// epochs 11.8 -> 12.5 ms).
template <typename T, int G>
bool sort_epoch(int64_t rows) { return !(relay_rows<T, G>(rows) && relay_share<G>(rows) == 1); }

template <typename T>
StepParams<T> step_params(double a, double b, double gamma) {
    StepParams<T> p{};
    p.a = static_cast<T>(a);
    p.b = static_cast<T>(b);
    p.neg2ab = T(-2) * p.a * p.b;
    p.gamma2b = T(2) * static_cast<T>(gamma) * p.b;
    return p;
}

ListStream list_stream(uint64_t seed, int32_t n) {
    ListStream st;
    st.k0 = static_cast<uint32_t>(seed) ^ RNG_NEGATIVE;
    st.k1 = static_cast<uint32_t>(seed >> 32);
    st.n = n;
    return st;
}

}  // namespace

template <typename T>
SgdEngine<T>::~SgdEngine() {
    for (cudaStream_t st : {epochs_stream_, lists_stream_}) {
        if (st) {
            cudaStreamSynchronize(st);
            stream_put(st);
        }
    }
}

template <typename T>
void SgdEngine<T>::setup(const DeviceEpochs<T>* ep, cudaStream_t s, int base_epoch) {
    ep_ = ep;
    base_epoch_ = base_epoch;
    const int64_t nnz = ep->nnz;
    const int32_t n = ep->n;
    enext_.allocate(nnz, s);
    enneg_.allocate(nnz, s);
    if (nnz) {
        UMAPB_CUDA(cudaMemcpyAsync(enext_.get(), ep->enext0.get(), nnz * sizeof(T), cudaMemcpyDeviceToDevice, s));
        UMAPB_CUDA(cudaMemcpyAsync(enneg_.get(), ep->enneg0.get(), nnz * sizeof(T), cudaMemcpyDeviceToDevice, s));
    }
    state_epoch_ = base_epoch_;
    order_.allocate(n, s);
    if (n > 0) {
        DevArray<uint64_t> key(n, s), key_sorted(n, s);
        DevArray<int32_t> row(n, s);
        DevArray<float> rate(n, s);
        DevArray<unsigned long long> total(1, s);
        total.zero(s);
        int32_t group = ORDER_GROUP;                       // UMAPB_SGD_ORDER_GROUP overrides it
        if (const char* e = std::getenv("UMAPB_SGD_ORDER_GROUP")) group = std::max(1, std::atoi(e));
        row_rate_kernel<T><<<grid_for(n, 256), 256, 0, s>>>(n, ep->ptr.get(), ep->eps.get(), rate.get(), total.get());
        UMAPB_LAUNCH_CHECK();
        row_order_key_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, rate.get(), total.get(), rows_in_flight(n, window_div),
                                                              group, key.get(), row.get());
        UMAPB_LAUNCH_CHECK();
        int end_bit = 33;
        while (end_bit < 64 && (int64_t(1) << (end_bit - 32)) <= int64_t(n) / group + 1) ++end_bit;
        size_t tb = 0;
        UMAPB_CUDA(cub::DeviceRadixSort::SortPairs(nullptr, tb, key.get(), key_sorted.get(), row.get(), order_.get(), n,
                                                   0, end_bit, s));
        DevArray<unsigned char> temp(tb, s);
        UMAPB_CUDA(cub::DeviceRadixSort::SortPairs(temp.get(), tb, key.get(), key_sorted.get(), row.get(), order_.get(),
                                                   n, 0, end_bit, s));
    }
    lists_.setup(ep, true, s);
}

template <typename T>
void SgdEngine<T>::state_at(int epoch, T* enext, T* enneg, cudaStream_t s) {
    const int64_t nnz = ep_->nnz;
    if (nnz == 0) return;
    require(epoch >= base_epoch_, "schedule state requested before its starting epoch");
    UMAPB_CUDA(cudaMemcpyAsync(enext, ep_->enext0.get(), nnz * sizeof(T), cudaMemcpyDeviceToDevice, s));
    UMAPB_CUDA(cudaMemcpyAsync(enneg, ep_->enneg0.get(), nnz * sizeof(T), cudaMemcpyDeviceToDevice, s));
    if (epoch > base_epoch_) {
        sched_advance_kernel<T><<<grid_for(nnz, 256), 256, 0, s>>>(nnz, ep_->eps.get(), enext, enneg,
                                                                   ep_->negative_sample_rate, base_epoch_,
                                                                   epoch - base_epoch_);
        UMAPB_LAUNCH_CHECK();
    }
}

template <typename T>
void SgdEngine<T>::run(T* Y, int num_dim, int first, int last, double a, double b, double gamma, double learning_rate,
                       uint64_t seed, cudaStream_t s, float* ms_schedule, float* ms_sgd) {
    if (ms_schedule) *ms_schedule = 0;
    if (ms_sgd) *ms_sgd = 0;
    if (last <= first) return;
    require(num_dim >= 1 && num_dim <= MAX_DIM, "num_dim must be between 1 and 64");
    const int total = ep_->total_epochs;
    const int32_t n = ep_->n;
    StepParams<T> p = step_params<T>(a, b, gamma);
    ListStream stream = list_stream(seed, n);
    stream.inst_start = inst_start_;
    stream.num_inst = num_inst_;
    const T lr = static_cast<T>(learning_rate);
    const bool check = check_schedule();
    const int device = current_device();
    const int64_t rows = rows_in_flight(n, window_div);
    // Points are read and added to as vectors of up to 16 bytes: a layout of
    // three dimensions, and an array that is not aligned to them, is worked on
    // in a copy (three dimensions as four, the fourth 0: one access each
    // instead of three).
    const int stride = num_dim == 3 ? 4 : num_dim;
    const size_t values = static_cast<size_t>(n) * stride;
    const bool copied = stride != num_dim || reinterpret_cast<uintptr_t>(Y) % 16 != 0;
    DevArray<T> copy(copied ? values : 0, s);
    DevArray<T> before;   // the layout as it was: a call that fails leaves it so, and its epochs undone
    T* Yp = copied ? copy.get() : Y;
    bool sort = false;
    for_dim<T>(stride, [&](auto, auto g, auto) { sort = epoch_order && sort_epoch<T, decltype(g)::value>(rows); });
    const int E = last - first;
    DevArray<int> counters(E, s);
    DevArray<unsigned long long> totals(check ? 2 * static_cast<size_t>(E) : 0, s);
    // The lists of the next window are built on one stream while this one's
    // epochs run on the other, which goes first where both want a place.  When
    // the epochs fill the device the two take turns instead: the epochs'
    // gathers and the lists' shuffles and shared memory go through the same
    // queue of an SM, and at a million points both side by side take 1.1 ms an
    // epoch against 0.65 ms one after the other.
    const bool overlap = rows < int64_t(ROW_BLOCK * ROW_BLOCKS) * sm_count();
    if (!epochs_stream_) epochs_stream_ = stream_get(true);
    if (!lists_stream_) lists_stream_ = stream_get();
    cudaStream_t es = epochs_stream_, ls = overlap ? lists_stream_ : epochs_stream_;
    cudaEvent_t start = event_get(), finish = event_get(), ready = event_get(), done[2] = {event_get(), event_get()};
    // Also on the way out of a failed call, when the streams have been waited for:
    // the lists (2 GB at a million points) go back to the workspace cache, where
    // the next call's come from, rather than staying with a layout that is done.
    // (Read ahead for a program that runs a few epochs at a time, a window stays.)
    auto settle = [&] {
        if (ahead_.epochs > 0) lists_.release(ahead_.buffer ^ 1);
        else lists_.release();
        event_put(start);
        event_put(finish);
        event_put(ready);
        event_put(done[0]);
        event_put(done[1]);
    };
    try {
        UMAPB_CUDA(cudaEventRecord(start, s));
        // A window that the call before has begun, and where the schedule state stands
        ListWindow w = ahead_;
        const bool begun = w.epochs > 0 && w.seed == seed && w.first <= first && first < w.first + w.epochs &&
                           state_epoch_ == w.first + w.epochs && !check;
        int from = begun ? w.first + w.epochs : first;
        ahead_ = ListWindow();
        if (!begun) {
            if (w.epochs > 0) lists_.release(w.buffer);
            if (state_epoch_ != first) state_at(first, enext_.get(), enneg_.get(), s);
        }
        state_epoch_ = -1;   // until the call has succeeded
        // Calls of a few epochs, one after the other (a program that shows the layout
        // as it goes): every window is as long as two before it, and what is left of
        // it is kept.  (20 calls of one epoch, ms: a million points 16.6 without,
        // 300 points 2.0.)
        const bool few = !check && E <= FEW_EPOCHS;
        const int least = few && first == run_end_ ? std::min(2 * std::max(least_, E), MAX_WINDOW) : 0;
        run_end_ = -1;
        counters.zero(s);
        if (check) totals.zero(s);
        if (copied && n > 0) {
            restride_kernel<T><<<grid_for(values, 256), 256, 0, s>>>(values, Y, num_dim, Yp, stride);
            UMAPB_LAUNCH_CHECK();
        }
        UMAPB_CUDA(cudaEventRecord(ready, s));
        UMAPB_CUDA(cudaStreamWaitEvent(es, ready, 0));
        UMAPB_CUDA(cudaStreamWaitEvent(ls, ready, 0));
        const size_t bytes = overlap ? window_bytes() / 2 : window_bytes();   // of each buffer
        // epochs of the window from 'at' on: the call's, or beyond them as far as is read ahead
        auto window = [&](int at, int into) {
            const int fit = lists_.window_epochs(into, bytes);
            const int more = std::min(least, std::min(lists_.window_epochs(into, bytes / 2), total - at));   // (half a buffer at most)
            return std::min(fit, std::max(last - at, more));
        };
        bool used[2] = {false, false};   // by epochs of this call
        int buffer = begun ? w.buffer : 0;
        auto after = [&] { return overlap && used[buffer] ? buffer ^ 1 : buffer; };   // in turns one is enough
        if (from < last && !begun) lists_.prepare(from, window(from, buffer), enext_.get(), enneg_.get(), overlap, ls);
        for (int e0 = first; e0 < last;) {
            if (e0 == from) {
                buffer = after();
                // the buffer's last epochs are done with it
                if (overlap && used[buffer]) UMAPB_CUDA(cudaStreamWaitEvent(ls, done[buffer], 0));
                auto build = [&] {
                    return lists_.build(buffer, bytes, enext_.get(), enneg_.get(), stream,
                                        check ? totals.get() + 2 * (e0 - first) : nullptr, overlap, ls);
                };
                w = ListWindow{e0, 0, buffer, seed};
                try {
                    w.epochs = build();
                } catch (const Error& e) {
                    if (e.code != UMAPB_ERR_OOM || !used[buffer ^ 1]) throw;
                    // no memory for a second window beside the one whose epochs run: after it then
                    UMAPB_CUDA(cudaStreamSynchronize(es));
                    lists_.release(buffer ^ 1);
                    lists_.prepare(e0, window(e0, buffer), enext_.get(), enneg_.get(), overlap, ls);
                    w.epochs = build();
                }
                from = e0 + w.epochs;
                if (n > 0) {
                    epoch_order_kernel<<<dim3((n - 1) / ORDER_GROUP + 1, w.epochs), EPOCH_ORDER_THREADS, 0, ls>>>(
                        order_.get(), n, sort, lists_.spans(buffer), lists_.tasks(buffer));
                    UMAPB_LAUNCH_CHECK();
                }
                UMAPB_CUDA(cudaEventRecord(ready, ls));
                UMAPB_CUDA(cudaStreamWaitEvent(es, ready, 0));
            }
            used[buffer] = true;
            if (from < last) {
                if (!copied && before.size() == 0) {   // a later window may fail
                    before.allocate(values, es);
                    UMAPB_CUDA(cudaMemcpyAsync(before.get(), Y, values * sizeof(T), cudaMemcpyDeviceToDevice, es));
                }
                lists_.prepare(from, window(from, after()), enext_.get(), enneg_.get(), overlap, ls);
            }
            const int e1 = std::min(from, last);
            for (int e = e0; e < e1 && n > 0; ++e) {
                const T epoch_t = static_cast<T>(e);
                // alpha = lr * (1 - epoch / num_epochs) in the reference's types (optimize_layout.hpp:132-133)
                p.alpha = static_cast<T>(static_cast<double>(lr) * (1.0 - static_cast<double>(epoch_t / static_cast<T>(total))));
                for_dim<T>(stride, [&](auto nc, auto g, auto ch) {
                    constexpr int NC = decltype(nc)::value, G = decltype(g)::value, CH = decltype(ch)::value;
                    const RowTask* tasks = lists_.tasks(buffer) + static_cast<size_t>(e - w.first) * n;
                    if (relay_rows<T, G>(rows)) {
                        static PerDevice known;
                        const int64_t resident = known.get(
                            device, [] { return resident_blocks(sgd_relay_kernel<T, NC, G, CH>, 32 * RELAY_WARPS); });
                        const int share = relay_share<G>(rows);
                        const int64_t blocks = std::min((rows + share - 1) / share, resident);
                        sgd_relay_kernel<T, NC, G, CH><<<static_cast<unsigned>(blocks), 32 * RELAY_WARPS, 0, es>>>(
                            tasks, n, lists_.list(buffer), Yp, stride, counters.get() + (e - first), share, p);
                    } else {
                        static PerDevice known;
                        const int64_t resident = known.get(
                            device, [] { return resident_blocks(sgd_rows_kernel<T, NC, G, CH>, ROW_BLOCK); });
                        const int64_t blocks = std::min((rows * G + ROW_BLOCK - 1) / ROW_BLOCK, resident);
                        sgd_rows_kernel<T, NC, G, CH><<<static_cast<unsigned>(blocks), ROW_BLOCK, 0, es>>>(
                            tasks, n, lists_.list(buffer), Yp, stride, counters.get() + (e - first), p);
                    }
                });
                UMAPB_LAUNCH_CHECK();
            }
            UMAPB_CUDA(cudaEventRecord(done[buffer], es));
            e0 = e1;
        }
        UMAPB_CUDA(cudaStreamWaitEvent(s, done[buffer], 0));   // the last window's: the lists came before it
        if (copied && n > 0) {
            restride_kernel<T><<<grid_for(values, 256), 256, 0, s>>>(static_cast<size_t>(n) * num_dim, Yp, stride, Y, num_dim);
            UMAPB_LAUNCH_CHECK();
        }
        UMAPB_CUDA(cudaEventRecord(finish, s));
        UMAPB_CUDA(cudaEventSynchronize(finish));
        float ms = 0;
        UMAPB_CUDA(cudaEventElapsedTime(&ms, start, finish));
        if (ms_sgd) *ms_sgd = ms;
        state_epoch_ = from;
        if (from > last) ahead_ = w;
        run_end_ = last;
        least_ = least;
    } catch (...) {
        cudaGetLastError();
        cudaStreamSynchronize(ls);   // nothing may still use what is released on the way out
        cudaStreamSynchronize(es);
        if (before.size()) cudaMemcpyAsync(Y, before.get(), before.bytes(), cudaMemcpyDeviceToDevice, s);
        cudaStreamSynchronize(s);
        settle();
        throw;
    }
    settle();
    if (check) {
        std::vector<int64_t> want(2 * static_cast<size_t>(E));
        counts(first, last, want.data(), s);
        std::vector<unsigned long long> got(2 * static_cast<size_t>(E));
        UMAPB_CUDA(cudaMemcpyAsync(got.data(), totals.get(), got.size() * sizeof(unsigned long long),
                                   cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        for (int w = 0; w < E; ++w)
            require(static_cast<int64_t>(got[2 * w]) == want[2 * w] && static_cast<int64_t>(got[2 * w + 1]) == want[2 * w + 1],
                    "schedule self-check failed at epoch " + std::to_string(first + w), UMAPB_ERR_CUDA);
    }
}

template <typename T>
void SgdEngine<T>::counts(int first, int last, int64_t* out, cudaStream_t s) {
    const int64_t nnz = ep_->nnz;
    const int W = last - first;
    if (W <= 0) return;
    DevArray<T> en(nnz, s), enn(nnz, s);
    state_at(first, en.get(), enn.get(), s);
    DevArray<unsigned long long> totals(2 * static_cast<size_t>(W), s);
    totals.zero(s);
    if (nnz) {
        const int64_t nblocks = (nnz + SCHED_BLOCK - 1) / SCHED_BLOCK;
        sched_totals_kernel<T><<<static_cast<unsigned>(nblocks), SCHED_BLOCK, 0, s>>>(
            nnz, ep_->eps.get(), en.get(), enn.get(), ep_->negative_sample_rate, first, W, totals.get());
        UMAPB_LAUNCH_CHECK();
    }
    std::vector<unsigned long long> h(2 * static_cast<size_t>(W));
    UMAPB_CUDA(cudaMemcpyAsync(h.data(), totals.get(), h.size() * sizeof(unsigned long long), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    for (size_t i = 0; i < h.size(); ++i) out[i] = static_cast<int64_t>(h[i]);
}

// UMAPB_SGD_WINDOW_DIV: rows in flight at most max(n / this, min(n / 8, 32768))
// (default 12; 0: no cap).
template <typename T>
int SgdEngine<T>::default_window_div() {
    const char* e = std::getenv("UMAPB_SGD_WINDOW_DIV");
    const int x = e ? std::atoi(e) : -1;
    return (x >= 0 && x <= 1 << 20) ? x : 12;
}

// UMAPB_SGD_EPOCH_ORDER=0 keeps the run's claim order in every epoch.
template <typename T>
bool SgdEngine<T>::default_epoch_order() {
    const char* e = std::getenv("UMAPB_SGD_EPOCH_ORDER");
    return !(e && std::atoi(e) == 0);
}

template class SgdEngine<float>;
template class SgdEngine<double>;

template <typename T>
void transform_init(int32_t nq, int num_dim, const int64_t* ptr, const int32_t* idx, const T* w, const T* Yref,
                    T* Ynew, cudaStream_t s) {
    if (nq <= 0) return;
    transform_init_kernel<T><<<grid_for(nq, 128), 128, 0, s>>>(nq, num_dim, ptr, idx, w, Yref, Ynew);
    UMAPB_LAUNCH_CHECK();
}

template <typename T>
void transform_layout(const DeviceEpochs<T>& ep, int num_dim, const T* Yref, int32_t nref, T* Ynew, int32_t head0,
                      double a, double b, double gamma, double learning_rate, uint64_t seed, cudaStream_t s) {
    require(num_dim >= 1 && num_dim <= MAX_DIM, "num_dim must be between 1 and 64");
    require(nref >= 1, "the transform needs at least one reference point");
    const int32_t nq = ep.n;
    if (nq <= 0) return;
    const StepParams<T> p = step_params<T>(a, b, gamma);
    ListStream stream = list_stream(seed, nref);
    stream.head0 = head0;
    DevArray<T> en(std::max<int64_t>(ep.nnz, 1), s), enn(std::max<int64_t>(ep.nnz, 1), s);
    if (ep.nnz) {
        UMAPB_CUDA(cudaMemcpyAsync(en.get(), ep.enext0.get(), ep.nnz * sizeof(T), cudaMemcpyDeviceToDevice, s));
        UMAPB_CUDA(cudaMemcpyAsync(enn.get(), ep.enneg0.get(), ep.nnz * sizeof(T), cudaMemcpyDeviceToDevice, s));
    }
    // as in SgdEngine::run: vectors, so three dimensions and unaligned arrays go through copies
    const int stride = num_dim == 3 ? 4 : num_dim;
    DevArray<T> ref_copy, new_copy;
    auto vectors = [&](const T* from, int32_t n, DevArray<T>& to) -> const T* {
        if (stride == num_dim && reinterpret_cast<uintptr_t>(from) % 16 == 0) return from;
        const size_t values = static_cast<size_t>(n) * stride;
        to.allocate(values, s);
        restride_kernel<T><<<grid_for(values, 256), 256, 0, s>>>(values, from, num_dim, to.get(), stride);
        UMAPB_LAUNCH_CHECK();
        return to.get();
    };
    Yref = vectors(Yref, nref, ref_copy);
    T* Yp = const_cast<T*>(vectors(Ynew, nq, new_copy));
    InteractionLists<T> lists;
    lists.setup(&ep, false, s);
    const int last = ep.total_epochs;
    const size_t bytes = window_bytes();
    lists.prepare(0, std::min(lists.window_epochs(0, bytes), last), en.get(), enn.get(), false, s);
    for (int e0 = 0; e0 < last;) {
        const int W = lists.build(0, bytes, en.get(), enn.get(), stream, nullptr, false, s);
        if (e0 + W < last) lists.prepare(e0 + W, std::min(lists.window_epochs(0, bytes), last - e0 - W), en.get(), enn.get(), false, s);
        for_dim<T>(stride, [&](auto nc, auto g, auto ch) {
            constexpr int NC = decltype(nc)::value, G = decltype(g)::value, CH = decltype(ch)::value;
            const int64_t threads = static_cast<int64_t>(nq) * G;
            transform_rows_kernel<T, NC, G, CH><<<static_cast<unsigned>((threads + ROW_BLOCK - 1) / ROW_BLOCK), ROW_BLOCK,
                                                  0, s>>>(nq, lists.spans(0), lists.list(0), Yref, Yp, stride, e0, W, last,
                                                          static_cast<T>(learning_rate), p);
        });
        UMAPB_LAUNCH_CHECK();
        e0 += W;
    }
    if (Yp != Ynew) {
        const size_t values = static_cast<size_t>(nq) * num_dim;
        restride_kernel<T><<<grid_for(values, 256), 256, 0, s>>>(values, Yp, stride, Ynew, num_dim);
        UMAPB_LAUNCH_CHECK();
    }
}

template void transform_init<float>(int32_t, int, const int64_t*, const int32_t*, const float*, const float*, float*,
                                    cudaStream_t);
template void transform_init<double>(int32_t, int, const int64_t*, const int32_t*, const double*, const double*,
                                     double*, cudaStream_t);
template void transform_layout<float>(const DeviceEpochs<float>&, int, const float*, int32_t, float*, int32_t, double,
                                      double, double, double, uint64_t, cudaStream_t);
template void transform_layout<double>(const DeviceEpochs<double>&, int, const double*, int32_t, double*, int32_t,
                                       double, double, double, double, uint64_t, cudaStream_t);

}  // namespace umapb
