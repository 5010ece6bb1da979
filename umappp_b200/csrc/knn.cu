// Exact Euclidean k-nearest neighbours on the device (the role of the
// knncolle search called at include/umappp/initialize.hpp:140).
//
// Candidate search (CUDA cores): one thread per query; tiles of 32 reference
// points and 32 dimensions are staged in shared memory (queries transposed so
// each thread reads its own column without bank conflicts, points broadcast),
// squared distances are accumulated from coordinate differences, and each
// thread keeps a sorted register list of its KCAP best (distance, index)
// candidates (ties keep the smaller index, as points arrive in index order).
//
// Float data: the list holds k + 8 candidates in FP32; a second kernel rescores
// them in FP64 from the original coordinates and keeps the best k by
// (distance, index).  A query whose (k+8)-th FP32 candidate is not clear of
// its k-th FP64 distance by more than the FP32 error bound is recomputed by
// the FP64 kernel, so the result equals an FP64 brute force except for ties.
// Double data: the FP64 kernel directly, with multiply and add kept separate
// so the sums round exactly as a sequential FP64 loop.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "stages.cuh"

namespace umapb {

int& last_knn_redo_count() {
    static int count = 0;
    return count;
}

static float bits_to_float(unsigned int b) {
    float f;
    std::memcpy(&f, &b, sizeof(f));
    return f;
}

int64_t& last_knn_tiles_scanned() {
    static int64_t tiles = 0;
    return tiles;
}

float& last_knn_kernel_ms() {
    static float ms = 0.0f;
    return ms;
}

double& last_knn_tc_error() {
    static double worst = 0.0;
    return worst;
}

namespace {

constexpr int KNN_BLOCK = 128;  // queries per block

// The tensor-core candidate search is the default; UMAPB_KNN_TENSOR_CORES=0
// selects the CUDA-core search instead (used by the precision comparison).
bool use_tensor_cores() {
    const char* v = std::getenv("UMAPB_KNN_TENSOR_CORES");
    return !(v && v[0] == '0');
}
constexpr int PT = 32;          // points per tile
constexpr int CH = 32;          // dimensions per chunk

__device__ __forceinline__ void add_sq(float& acc, float d) { acc = fmaf(d, d, acc); }
__device__ __forceinline__ void add_sq(double& acc, double d) { acc = __dadd_rn(acc, __dmul_rn(d, d)); }

template <typename A>
struct Inf;
template <>
struct Inf<float> {
    static __device__ __forceinline__ float v() { return CUDART_INF_F; }
};
template <>
struct Inf<double> {
    static __device__ __forceinline__ double v() { return CUDART_INF; }
};

// Sorted insertion into a register list (bd ascending); entries equal to an
// existing distance go after it, so earlier (smaller) indices win ties.
template <typename A, int KCAP>
__device__ __forceinline__ void insert_sorted(A (&bd)[KCAP], int (&bi)[KCAP], A cd, int ci) {
#pragma unroll
    for (int i = KCAP - 1; i > 0; --i) {
        if (cd < bd[i - 1]) {
            bd[i] = bd[i - 1];
            bi[i] = bi[i - 1];
        } else if (cd < bd[i]) {
            bd[i] = cd;
            bi[i] = ci;
        }
    }
    if (cd < bd[0]) {
        bd[0] = cd;
        bi[0] = ci;
    }
}

// Brute-force candidate kernel.  T = storage type, A = accumulation type.
// If 'queries' is non-null the block's threads take their query ids from it
// (nq entries), else queries are 0..nq-1.  The candidates are the data rows
// [0, n) other than the query itself.
template <typename T, typename A, int KCAP>
__global__ void __launch_bounds__(KNN_BLOCK) knn_bruteforce_kernel(const T* __restrict__ data, int32_t n, int32_t dim,
                                                                   const int32_t* __restrict__ queries, int32_t nq,
                                                                   int32_t* __restrict__ cand_idx,
                                                                   A* __restrict__ cand_d2) {
    __shared__ A qs[CH][KNN_BLOCK];
    __shared__ A ps[PT][CH + 1];
    const int tid = threadIdx.x;
    const int32_t slot = blockIdx.x * KNN_BLOCK + tid;
    const bool active = slot < nq;
    const int32_t q = active ? (queries ? queries[slot] : slot) : 0;

    A bd[KCAP];
    int bi[KCAP];
#pragma unroll
    for (int i = 0; i < KCAP; ++i) {
        bd[i] = Inf<A>::v();
        bi[i] = -1;
    }

    for (int32_t base = 0; base < n; base += PT) {
        A acc[PT];
#pragma unroll
        for (int p = 0; p < PT; ++p) acc[p] = 0;
        for (int c0 = 0; c0 < dim; c0 += CH) {
            const int cw = min(CH, dim - c0);
            __syncthreads();
            // stage this block's queries (transposed) and the point tile
            for (int c = 0; c < cw; ++c) qs[c][tid] = active ? static_cast<A>(data[static_cast<size_t>(q) * dim + c0 + c]) : A(0);
            for (int e = tid; e < PT * CH; e += KNN_BLOCK) {
                const int p = e / CH, c = e % CH;
                const int32_t j = base + p;
                ps[p][c] = (j < n && c < cw) ? static_cast<A>(data[static_cast<size_t>(j) * dim + c0 + c]) : A(0);
            }
            __syncthreads();
            for (int c = 0; c < cw; ++c) {
                const A qv = qs[c][tid];
#pragma unroll
                for (int p = 0; p < PT; ++p) add_sq(acc[p], qv - ps[p][c]);
            }
        }
        if (active) {
#pragma unroll
            for (int p = 0; p < PT; ++p) {
                const int32_t j = base + p;
                if (j < n && j != q && acc[p] < bd[KCAP - 1]) insert_sorted<A, KCAP>(bd, bi, acc[p], j);
            }
        }
    }
    if (active) {
#pragma unroll
        for (int i = 0; i < KCAP; ++i) {
            cand_idx[static_cast<size_t>(slot) * KCAP + i] = bi[i];
            cand_d2[static_cast<size_t>(slot) * KCAP + i] = bd[i];
        }
    }
}

// Sorts 32 PER (distance, index) pairs held by a warp, pair e = 32 i + lane,
// ascending: a bitonic network, partners in the same lane or a shuffle away.
template <int PER>
__device__ __forceinline__ void warp_sort(double (&d)[PER], int (&id)[PER]) {
    const int lane = threadIdx.x & 31;
    auto less = [](double x, int xi, double y, int yi) {   // index -1 (no candidate) maps above every index
        return x < y || (x == y && static_cast<uint32_t>(xi) < static_cast<uint32_t>(yi));
    };
#pragma unroll
    for (int size = 2; size <= 32 * PER; size <<= 1) {
#pragma unroll
        for (int stride = size >> 1; stride > 0; stride >>= 1) {
            if (stride >= 32) {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const int o = i ^ (stride >> 5);
                    if (o > i) {
                        const bool up = ((32 * i + lane) & size) == 0;
                        if (less(d[o], id[o], d[i], id[i]) == up) {
                            const double x = d[i];
                            d[i] = d[o];
                            d[o] = x;
                            const int y = id[i];
                            id[i] = id[o];
                            id[o] = y;
                        }
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < PER; ++i) {
                    const double x = __shfl_xor_sync(0xffffffffu, d[i], stride);
                    const int y = __shfl_xor_sync(0xffffffffu, id[i], stride);
                    // the lower lane keeps the smaller of an ascending pair
                    const bool small = (((32 * i + lane) & size) == 0) == ((lane & stride) == 0);
                    if (small ? less(x, y, d[i], id[i]) : less(d[i], id[i], x, y)) {
                        d[i] = x;
                        id[i] = y;
                    }
                }
            }
        }
    }
}

// Squared distance of two rows, FP64, summed in coordinate order.
__device__ __forceinline__ double distance2(const float* __restrict__ x, const float* __restrict__ y, int32_t dim,
                                            bool vec4) {
    double s = 0;
    auto add = [&s](float u, float v) {
        const double diff = static_cast<double>(u) - static_cast<double>(v);
        s = __dadd_rn(s, __dmul_rn(diff, diff));
    };
    if (vec4) {   // rows of whole 16-byte vectors
#pragma unroll 4
        for (int d = 0; d < dim; d += 4) {
            const float4 u = __ldg(reinterpret_cast<const float4*>(x + d)), v = __ldg(reinterpret_cast<const float4*>(y + d));
            add(u.x, v.x);
            add(u.y, v.y);
            add(u.z, v.z);
            add(u.w, v.w);
        }
    } else {
#pragma unroll 4
        for (int d = 0; d < dim; ++d) add(__ldg(x + d), __ldg(y + d));
    }
    return s;
}

// FP64 rescoring of the FP32 candidates of every query: keeps the best k by
// (FP64 distance, index) and flags queries whose candidate set may miss a
// true neighbour (others = 0: never).  A query's results go to row 'slot', or
// q - out_row0.  A query's candidates are 'lists' lists of list_len entries
// (32 PER in all at most), each the nearest of its part of the points in
// ascending FP32 order.  One warp per query, a candidate (or PER) per lane:
// bound by the candidates' rows, read from L2 a row per lane.  (A thread per
// query with an insertion sort in local memory took 3.9 ms for a million
// queries of 24 candidates in 50 dimensions.)
constexpr int RESCORE_WARPS = 4;
template <int PER>
__global__ void __launch_bounds__(RESCORE_WARPS * 32)
    knn_rescore_kernel(const float* __restrict__ data, int32_t others, int32_t dim, int32_t k,
                       const int32_t* __restrict__ queries, int32_t nq, int lists, int list_len, int cand_by_slot,
                       int out_by_slot, int32_t out_row0, const int32_t* __restrict__ cand_idx, const float* __restrict__ cand_d2,
                       int32_t* __restrict__ out_idx, float* __restrict__ out_dist, double* __restrict__ out_dist64,
                       int32_t* __restrict__ redo, double* __restrict__ redo_kth, int32_t* __restrict__ redo_count,
                       const float* __restrict__ norms,
                       const unsigned int* __restrict__ norm_max_bits, double tc_rel,
                       unsigned int* __restrict__ tc_err_bits) {
    const int lane = threadIdx.x & 31;
    const int64_t slot64 = static_cast<int64_t>(blockIdx.x) * RESCORE_WARPS + (threadIdx.x >> 5);
    if (slot64 >= nq) return;   // whole warps
    const int32_t slot = static_cast<int32_t>(slot64);
    const int32_t q = queries ? queries[slot] : slot;     // the query's data row (output row)
    const int ncand = lists * list_len;
    const size_t first = static_cast<size_t>(cand_by_slot ? slot : q) * ncand;   // its candidates
    const float* xq = data + static_cast<size_t>(q) * dim;
    const bool vec4 = dim % 4 == 0 && reinterpret_cast<uintptr_t>(data) % 16 == 0;
    const double scale = norms ? static_cast<double>(norms[q]) + static_cast<double>(__uint_as_float(*norm_max_bits)) : 0.0;
    const double err_scale = norms && tc_err_bits ? 1.0 / (scale + 1e-300) : 0.0;
    double d64[PER];
    int id[PER];
    float worst = 0.0f;   // largest |FP32 candidate distance - FP64 distance| / (|q|^2 + max |r|^2)
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = 32 * i + lane;
        id[i] = c < ncand ? cand_idx[first + c] : -1;
        d64[i] = CUDART_INF;
        if (id[i] >= 0) {
            d64[i] = distance2(xq, data + static_cast<size_t>(id[i]) * dim, dim, vec4);
            if (err_scale > 0.0)
                worst = fmaxf(worst, static_cast<float>(fabs(static_cast<double>(cand_d2[first + c]) - d64[i]) * err_scale));
        }
    }
    warp_sort<PER>(d64, id);
    // Certainty check: every point outside the candidate lists has an FP32
    // distance >= the last FP32 value of its list.  FP32 squared distances from
    // differences carry relative error below (dim + 2) * 2^-24 (plus the
    // rounding of the inputs, which is exact here); if the k-th FP64 distance
    // could exceed the true distance of such a point, the query is recomputed
    // in FP64.  For tensor-core candidates (norms given) the FP32 values are
    // |q|^2 + |r|^2 - 2 q.r with an absolute error below tc_rel * (|q|^2 + max |r|^2).
    float last32 = CUDART_INF_F;
    for (int l = 0; l < lists; ++l) last32 = fminf(last32, cand_d2[first + (l + 1) * list_len - 1]);
    double kth = 0;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const double v = __shfl_sync(0xffffffffu, d64[i], (k - 1) & 31);
        if (i == (k - 1) >> 5) kth = v;
    }
    const double rel = (dim + 2) * 1.2e-7 * 2.0;
    const bool full_list = lists == 1 && others <= ncand;   // every candidate point is in the list
    const bool certain = norms ? static_cast<double>(last32) - tc_rel * scale > kth * (1.0 + 1e-12) + 1e-300
                               : static_cast<double>(last32) * (1.0 - rel) > kth * (1.0 + rel);
    if (lane == 0 && !full_list && !certain) {
        const int32_t r = atomicAdd(redo_count, 1);
        redo[r] = out_by_slot ? slot : q;   // a slot when the output is by slot, else the data row
        if (redo_kth) redo_kth[r] = kth;    // k points are at least as near as that
    }
    if (err_scale > 0.0) {
        for (int o = 16; o > 0; o >>= 1) worst = fmaxf(worst, __shfl_xor_sync(0xffffffffu, worst, o));
        if (lane == 0 && worst > 0.0f) atomicMax(tc_err_bits, __float_as_uint(worst));
    }
    const size_t orow = static_cast<size_t>(out_by_slot ? slot : q - out_row0) * k;
#pragma unroll
    for (int i = 0; i < PER; ++i) {
        const int c = 32 * i + lane;
        if (c < k) {
            out_idx[orow + c] = id[i];
            const double dd = sqrt(d64[i]);
            out_dist[orow + c] = static_cast<float>(dd);
            if (out_dist64) out_dist64[orow + c] = dd;
        }
    }
}

unsigned rescore_grid(int32_t nq) { return static_cast<unsigned>((nq + RESCORE_WARPS - 1) / RESCORE_WARPS); }
template <int KCAP>
constexpr int per_lane() { return (KCAP + 31) / 32; }

// Writes the first k entries of FP64 candidate lists (sqrt of squared distance).
// Output row of entry 'slot': out_rows[slot] if given, else the query's data row.
template <typename T, int KCAP>
__global__ void knn_emit_f64_kernel(int32_t nq, const int32_t* __restrict__ queries, const int32_t* __restrict__ out_rows,
                                    int32_t k, const int32_t* __restrict__ cand_idx, const double* __restrict__ cand_d2,
                                    int32_t* __restrict__ out_idx, T* __restrict__ out_dist,
                                    double* __restrict__ out_dist64) {
    const int32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= nq) return;
    const int32_t q = out_rows ? out_rows[slot] : queries ? queries[slot] : slot;
    for (int c = 0; c < k; ++c) {
        out_idx[static_cast<size_t>(q) * k + c] = cand_idx[static_cast<size_t>(slot) * KCAP + c];
        const double dd = sqrt(cand_d2[static_cast<size_t>(slot) * KCAP + c]);
        out_dist[static_cast<size_t>(q) * k + c] = static_cast<T>(dd);
        if (out_dist64) out_dist64[static_cast<size_t>(q) * k + c] = dd;
    }
}

// FP64 search of the queries (data rows 'queries') among the data rows [0, n);
// results go to the queries' own rows, or to rows out_rows[slot] if given.
template <typename T, int KCAP>
void run_f64(const T* data, int32_t n, int32_t dim, int32_t k, const int32_t* queries, int32_t nq, int32_t* out_idx,
             T* out_dist, double* out_dist64, cudaStream_t s, const int32_t* out_rows = nullptr) {
    if (nq <= 0) return;
    DevArray<int32_t> ci(static_cast<size_t>(nq) * KCAP, s);
    DevArray<double> cd(static_cast<size_t>(nq) * KCAP, s);
    knn_bruteforce_kernel<T, double, KCAP><<<(nq + KNN_BLOCK - 1) / KNN_BLOCK, KNN_BLOCK, 0, s>>>(
        data, n, dim, queries, nq, ci.get(), cd.get());
    UMAPB_LAUNCH_CHECK();
    knn_emit_f64_kernel<T, KCAP><<<(nq + 127) / 128, 128, 0, s>>>(nq, queries, out_rows, k, ci.get(), cd.get(), out_idx,
                                                                  out_dist, out_dist64);
    UMAPB_LAUNCH_CHECK();
}

// FP64 search of queries whose lists are as long as k asks for.
void run_f64_lists(const float* data, int32_t n, int32_t dim, int32_t k, const int32_t* queries, int32_t nq,
                   const int32_t* out_rows, int32_t* out_idx, float* out_dist, double* out_dist64, cudaStream_t s) {
    if (k <= 16) run_f64<float, 16>(data, n, dim, k, queries, nq, out_idx, out_dist, out_dist64, s, out_rows);
    else if (k <= 32) run_f64<float, 32>(data, n, dim, k, queries, nq, out_idx, out_dist, out_dist64, s, out_rows);
    else if (k <= 64) run_f64<float, 64>(data, n, dim, k, queries, nq, out_idx, out_dist, out_dist64, s, out_rows);
    else run_f64<float, 128>(data, n, dim, k, queries, nq, out_idx, out_dist, out_dist64, s, out_rows);
}

// ---- uncertain queries ----
// A query whose candidates leave its k-th neighbour open: what they do tell is a
// distance within which k points lie (kth).  All points that may be that near are
// collected -- by FP32 differences, with their rounding in the bound -- and rescored
// in FP64.  Where the tensor cores' bound certifies nothing (data far from the
// origin, or one far outlier) that is every query: 20,000 x 20 points with an
// offset of 1000, k = 15, 30 and 60: 4.0, 5.5 and 8.9 ms in all (the FP64 search of
// every query, a list per thread: 7.2, 22.5 and 112.7; candidates by FP32
// differences on CUDA cores in the first place: 18.0 and 85.6 for 30 and 60).
// Collected are up to 128 points per query (256 for more than 56 neighbours);
// queries with more of them, ties mostly, are searched in FP64.
constexpr int32_t WITHIN_PLACES = 1 << 23;   // of the queries taken at a time (64 MB)

// Thread = query, blockIdx.y = stretch of the points.
template <int LIST>
__global__ void __launch_bounds__(KNN_BLOCK)
    knn_within_kernel(const float* __restrict__ data, int32_t n, int32_t dim, const int32_t* __restrict__ queries,
                      int32_t nq, const double* __restrict__ kth, int32_t stretch, int32_t* __restrict__ list,
                      int32_t* __restrict__ count) {
    __shared__ float qs[CH][KNN_BLOCK];
    __shared__ float ps[PT][CH + 1];
    const int tid = threadIdx.x;
    const int32_t slot = blockIdx.x * KNN_BLOCK + tid;
    const bool active = slot < nq;
    const int32_t q = active ? queries[slot] : 0;
    float bound = -1.0f;
    if (active) {
        const double d2 = kth[slot];
        const double rel = (dim + 2) * 1.2e-7 * 2.0;   // as in the certainty check
        // (the addition: squares of differences below 1e-19 lose bits)
        if (d2 < CUDART_INF) bound = __double2float_ru(d2 * (1.0 + rel) + 1e-36);
        else if (blockIdx.y == 0) atomicAdd(&count[slot], LIST + 1);   // fewer than k candidates
    }
    const int32_t first = blockIdx.y * stretch;   // (a multiple of PT)
    const int32_t last = static_cast<int32_t>(min(static_cast<int64_t>(n), static_cast<int64_t>(first) + stretch));
    for (int32_t base = first; base < last; base += PT) {
        float acc[PT];
#pragma unroll
        for (int p = 0; p < PT; ++p) acc[p] = 0;
        for (int c0 = 0; c0 < dim; c0 += CH) {
            const int cw = min(CH, dim - c0);
            __syncthreads();
            if (dim > CH || base == first)
                for (int c = 0; c < cw; ++c) qs[c][tid] = data[static_cast<size_t>(q) * dim + c0 + c];
            for (int e = tid; e < PT * CH; e += KNN_BLOCK) {
                const int p = e / CH, c = e % CH;
                const int32_t j = base + p;
                ps[p][c] = (j < last && c < cw) ? data[static_cast<size_t>(j) * dim + c0 + c] : 0.0f;
            }
            __syncthreads();
            for (int c = 0; c < cw; ++c) {
                const float qv = qs[c][tid];
#pragma unroll
                for (int p = 0; p < PT; ++p) add_sq(acc[p], qv - ps[p][c]);
            }
        }
#pragma unroll
        for (int p = 0; p < PT; ++p) {
            const int32_t j = base + p;
            if (acc[p] <= bound && j < last && j != q) {
                const int at = atomicAdd(&count[slot], 1);
                if (at < LIST) list[static_cast<size_t>(slot) * LIST + at] = j;
            }
        }
    }
}

// The queries with more points within reach than their lists hold.
__global__ void knn_crowded_kernel(int32_t nq, int32_t places, const int32_t* __restrict__ count, const int32_t* __restrict__ queries,
                                   int32_t row0, int32_t* __restrict__ crowded, int32_t* __restrict__ rows,
                                   int32_t* __restrict__ num) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < nq; i += gridDim.x * blockDim.x) {
        if (count[i] > places) {
            const int32_t at = atomicAdd(num, 1);
            crowded[at] = queries[i];
            rows[at] = queries[i] - row0;
        }
    }
}

// An array that a search does without where memory is short (false).
template <typename T>
bool allocate_if_possible(DevArray<T>& a, size_t n, cudaStream_t s) {
    try {
        a.allocate(n, s);
    } catch (const Error& e) {
        if (e.code != UMAPB_ERR_OOM) throw;
        return false;
    }
    return true;
}

// Exact search of 'nq' queries (data rows) among the data rows [0, n), k of
// which are known to lie within kth; results to rows query - row0.  False,
// with nothing done, where there is no memory for it.
template <int LIST>
bool run_within_lists(const float* data, int32_t n, int32_t dim, int32_t k, const int32_t* queries, int32_t nq,
                const double* kth, int32_t row0, int32_t* out_idx, float* out_dist, double* out_dist64, cudaStream_t s) {
    const int32_t batch = std::min(nq, WITHIN_PLACES / LIST);
    DevArray<int32_t> list, count, crowded, rows, num;
    DevArray<float> unused;   // the rescoring's FP32 distances
    const size_t places = static_cast<size_t>(batch) * LIST;
    if (!allocate_if_possible(list, places, s) || !allocate_if_possible(unused, places, s) ||
        !allocate_if_possible(count, batch, s) || !allocate_if_possible(crowded, batch, s) ||
        !allocate_if_possible(rows, batch, s) || !allocate_if_possible(num, 1, s))
        return false;
    for (int32_t at = 0; at < nq; at += batch) {
        const int32_t m = std::min(batch, nq - at);
        const int32_t* q = queries + at;
        UMAPB_CUDA(cudaMemsetAsync(list.get(), 0xff, list.bytes(), s));
        count.zero(s);
        num.zero(s);
        // stretches so that the device is filled four times over
        const int32_t blocks = (m + KNN_BLOCK - 1) / KNN_BLOCK, tiles = (n - 1) / PT + 1;
        const int32_t parts = std::min(tiles, std::max(1, 4 * 4 * sm_count() / blocks));
        const int32_t stretch = (tiles + parts - 1) / parts * PT;
        knn_within_kernel<LIST><<<dim3(blocks, (tiles - 1) / (stretch / PT) + 1), KNN_BLOCK, 0, s>>>(data, n, dim, q, m, kth + at,
                                                                                         stretch, list.get(), count.get());
        UMAPB_LAUNCH_CHECK();
        knn_rescore_kernel<LIST / 32><<<rescore_grid(m), RESCORE_WARPS * 32, 0, s>>>(
            data, 0, dim, k, q, m, 1, LIST, 1, 0, row0, list.get(), unused.get(), out_idx, out_dist, out_dist64,
            nullptr, nullptr, nullptr, nullptr, nullptr, 0.0, nullptr);
        UMAPB_LAUNCH_CHECK();
        knn_crowded_kernel<<<grid_for(m, 256), 256, 0, s>>>(m, LIST, count.get(), q, row0, crowded.get(), rows.get(), num.get());
        UMAPB_LAUNCH_CHECK();
        int32_t nc = 0;
        UMAPB_CUDA(cudaMemcpyAsync(&nc, num.get(), sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        if (nc > 0) run_f64_lists(data, n, dim, k, crowded.get(), nc, rows.get(), out_idx, out_dist, out_dist64, s);
    }
    return true;
}

// The uncertain queries of a search: kth (null: unknown) as above; results to
// rows out_rows[i], which are queries[i] - row0 (null: queries[i]).
void search_again(const float* data, int32_t n, int32_t dim, int32_t k, const int32_t* queries, int32_t nq,
                  const double* kth, int32_t row0, const int32_t* out_rows, int32_t* out_idx, float* out_dist,
                  double* out_dist64, cudaStream_t s) {
    const bool done = kth && (k <= 56 ? run_within_lists<128>(data, n, dim, k, queries, nq, kth, row0, out_idx, out_dist, out_dist64, s)
                                      : run_within_lists<256>(data, n, dim, k, queries, nq, kth, row0, out_idx, out_dist, out_dist64, s));
    if (!done) run_f64_lists(data, n, dim, k, queries, nq, out_rows, out_idx, out_dist, out_dist64, s);
}

__global__ void norm_max_kernel(int32_t n, const float* __restrict__ norms, unsigned int* __restrict__ out) {
    unsigned int m = 0;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        m = max(m, __float_as_uint(norms[i]));    // non-negative floats order like their bits
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_down_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// Tolerance of the tensor-core squared distances, relative to |q|^2 + |r|^2:
// 3xTF32 products (about 3 * 2^-22), FP32 accumulation over up to 64 terms and
// the final FP32 additions stay below 2^-17.
constexpr double TC_REL_BOUND = 1.0 / 131072.0;

__global__ void iota_kernel(int32_t count, int32_t first, int32_t* __restrict__ out) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) out[i] = first + i;
}

// The rows [lo, hi) of shard 'index' of 'count' equal contiguous ranges of the data rows.
void shard_row_range(int32_t n, KnnShard shard, int32_t& lo, int32_t& hi) {
    lo = static_cast<int32_t>(static_cast<int64_t>(n) * shard.index / shard.count);
    hi = static_cast<int32_t>(static_cast<int64_t>(n) * (shard.index + 1) / shard.count);
}

// Few points with 25 to 56 neighbours: the CUDA-core search, whose cost grows
// with n x dim, against the tensor cores' fixed one (tree, operands, two passes).
// ms, CUDA / tensor cores, 30 neighbours: 150 x 2 points 0.25 / 0.41, 600 x 2 0.72 /
// 0.66, 1,000 x 2 0.83 / 0.89; 300 x 20 0.47 / 0.66, 800 x 20 0.90 / 0.98; 300 x 50 0.59 /
// 0.66, 500 x 50 0.84 / 0.77; 128 x 100 0.57 / 0.51.  (Beyond 56 neighbours, with
// lists of 128, the tensor cores are ahead from 100 points on: 0.50 / 0.47 for 150 x 2.)
bool few_points(int32_t n, int32_t dim, int kcap) { return kcap == 64 && n < 1100 - 12 * static_cast<int64_t>(dim); }

// With a shard (count > 1) the search covers only the shard's queries, whose
// data rows go to *rows (*nrows of them); out_idx / out_dist are written at
// those rows only.
template <int KCAP>
void run_f32(const float* data, int32_t n, int32_t dim, int32_t k, int32_t* out_idx, float* out_dist,
             double* out_dist64, cudaStream_t s, KnnShard shard = KnnShard(), DevArray<int32_t>* rows = nullptr,
             int32_t* nrows = nullptr) {
    const bool sharded = shard.count > 1;
    DevArray<float> norms;
    DevArray<unsigned int> norm_max(1, s);
    bool tc = use_tensor_cores() && knn_tc_supported(dim, KCAP) && !few_points(n, dim, KCAP);
    // candidates: by data row (tensor-core search, unsharded brute force) or by
    // slot of the shard's row list (sharded brute force)
    DevArray<int32_t> ci;
    DevArray<float> cd;
    DevArray<int32_t> tree_rows;
    int32_t nq = n;
    const int32_t* queries = nullptr;
    bool by_slot = false;
    if (sharded) *nrows = -1;
    if (tc) {
        DevArray<int> err(1, s);
        err.zero(s);
        // unsharded: the rows in tree order, so that the rescoring walks the
        // queries with nearby ones together (their candidates share L2 lines)
        try {
            ci.allocate(static_cast<size_t>(n) * KCAP, s);
            cd.allocate(static_cast<size_t>(n) * KCAP, s);
            norms.allocate(((n + 127) / 128) * 128, s);
            tc = knn_tc_candidates(data, n, dim, KCAP, ci.get(), cd.get(), norms.get(), err.get(), s, shard, rows, nrows,
                                   sharded ? nullptr : &tree_rows);
        } catch (const Error& e) {
            // Beyond 32 candidates the CUDA-core search, which needs no operands, does
            // where memory is short: of the shard's rows in the tree, the same that
            // another process finds with more memory, or not at all.
            if (e.code != UMAPB_ERR_OOM || KCAP <= 32 || (sharded && *nrows < 0)) throw;
            tc = false;
            ci.release();
            cd.release();
            norms.release();
        }
        int h_err = 0;
        UMAPB_CUDA(cudaMemcpyAsync(&h_err, err.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        if (h_err != DEV_OK) fail(UMAPB_ERR_DEVICE_TIMEOUT, "tensor-core kNN: a pipeline wait gave up");
        if (tc) {
            norm_max.zero(s);
            norm_max_kernel<<<grid_for(n, 256, 1024), 256, 0, s>>>(n, norms.get(), norm_max.get());
            UMAPB_LAUNCH_CHECK();
            if (sharded) {
                nq = *nrows;
                queries = rows->get();
            } else if (tree_rows.get()) {
                queries = tree_rows.get();   // nq = n; candidates and output by data row
            }
        }
    }
    if (!tc) {
        if (sharded) {   // CUDA-core candidates by slot
            if (*nrows < 0) {   // contiguous data rows
                int32_t lo, hi;
                shard_row_range(n, shard, lo, hi);
                *nrows = hi - lo;
                rows->allocate(std::max<int32_t>(hi - lo, 1), s);
                if (hi > lo) {
                    iota_kernel<<<grid_for(hi - lo, 256), 256, 0, s>>>(hi - lo, lo, rows->get());
                    UMAPB_LAUNCH_CHECK();
                }
            }
            nq = *nrows;
            queries = rows->get();
            by_slot = true;
        }
        ci.allocate(static_cast<size_t>(std::max(nq, 1)) * KCAP, s);
        cd.allocate(static_cast<size_t>(std::max(nq, 1)) * KCAP, s);
        if (nq > 0) {
            knn_bruteforce_kernel<float, float, KCAP><<<(nq + KNN_BLOCK - 1) / KNN_BLOCK, KNN_BLOCK, 0, s>>>(
                data, n, dim, queries, nq, ci.get(), cd.get());
            UMAPB_LAUNCH_CHECK();
        }
    }
    DevArray<int32_t> redo(std::max(nq, 1), s), redo_count(1, s);
    DevArray<double> redo_kth;
    allocate_if_possible(redo_kth, std::max(nq, 1), s);
    redo_count.zero(s);
    DevArray<unsigned int> tc_err(1, s);
    tc_err.zero(s);
    if (nq > 0) {
        knn_rescore_kernel<per_lane<KCAP>()><<<rescore_grid(nq), RESCORE_WARPS * 32, 0, s>>>(
            data, n - 1, dim, k, queries, nq, 1, KCAP, by_slot ? 1 : 0, 0, 0, ci.get(), cd.get(), out_idx, out_dist,
            out_dist64, redo.get(), redo_kth.get(), redo_count.get(), tc ? norms.get() : nullptr, norm_max.get(),
            TC_REL_BOUND, tc_err.get());
    }
    UMAPB_LAUNCH_CHECK();
    int32_t nredo = 0;
    unsigned int err_bits = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&nredo, redo_count.get(), sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(&err_bits, tc_err.get(), sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    last_knn_redo_count() = nredo;
    last_knn_tc_error() = tc ? static_cast<double>(bits_to_float(err_bits)) : 0.0;
    if (nredo > 0) {
        search_again(data, n, dim, k, redo.get(), nredo, redo_kth.get(), 0, nullptr, out_idx, out_dist, out_dist64, s);
    }
}

__global__ void row_norms_kernel(const float* __restrict__ data, int32_t n, int32_t dim, float* __restrict__ norms) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double s = 0;
        for (int d = 0; d < dim; ++d) {
            const double v = data[static_cast<size_t>(i) * dim + d];
            s += v * v;
        }
        norms[i] = static_cast<float>(s);
    }
}

__global__ void shift_indices_kernel(int32_t* __restrict__ idx, size_t count, int32_t delta) {
    for (size_t t = blockIdx.x * size_t(blockDim.x) + threadIdx.x; t < count; t += size_t(gridDim.x) * blockDim.x)
        idx[t] += delta;
}

// Batched tensor-core search with FP64 rescoring; instances holding uncertain
// queries are recomputed whole by the per-instance search.
template <int KCAP>
void run_f32_batched(const float* data, const std::vector<int32_t>& inst, int32_t dim, int32_t k, int32_t* out_idx,
                     float* out_dist, cudaStream_t s) {
    const int ninst = static_cast<int>(inst.size()) - 1;
    const int32_t n = inst[ninst];
    DevArray<int32_t> ci(static_cast<size_t>(n) * KCAP, s);
    DevArray<float> cd(static_cast<size_t>(n) * KCAP, s);
    DevArray<int> err(1, s);
    err.zero(s);
    knn_tc_candidates_batched(data, inst, dim, KCAP, ci.get(), cd.get(), err.get(), s);
    int h_err = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&h_err, err.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    if (h_err != DEV_OK) fail(UMAPB_ERR_DEVICE_TIMEOUT, "tensor-core kNN: a pipeline wait gave up");
    DevArray<float> norms(n, s);
    DevArray<unsigned int> norm_max(1, s);
    norm_max.zero(s);
    row_norms_kernel<<<grid_for(n, 256), 256, 0, s>>>(data, n, dim, norms.get());
    UMAPB_LAUNCH_CHECK();
    norm_max_kernel<<<grid_for(n, 256, 1024), 256, 0, s>>>(n, norms.get(), norm_max.get());
    UMAPB_LAUNCH_CHECK();
    DevArray<int32_t> redo(n, s), redo_count(1, s);
    redo_count.zero(s);
    DevArray<unsigned int> tc_err(1, s);
    tc_err.zero(s);
    knn_rescore_kernel<per_lane<KCAP>()><<<rescore_grid(n), RESCORE_WARPS * 32, 0, s>>>(
        data, n - 1, dim, k, nullptr, n, 1, KCAP, 0, 0, 0, ci.get(), cd.get(), out_idx, out_dist, nullptr, redo.get(),
        nullptr, redo_count.get(), norms.get(), norm_max.get(), TC_REL_BOUND, tc_err.get());
    UMAPB_LAUNCH_CHECK();
    int32_t nredo = 0;
    unsigned int err_bits = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&nredo, redo_count.get(), sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaMemcpyAsync(&err_bits, tc_err.get(), sizeof(unsigned int), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    last_knn_redo_count() = nredo;
    last_knn_tc_error() = static_cast<double>(bits_to_float(err_bits));
    if (nredo > 0) {
        std::vector<int32_t> rq(nredo);
        UMAPB_CUDA(cudaMemcpyAsync(rq.data(), redo.get(), nredo * sizeof(int32_t), cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        std::vector<char> mark(ninst, 0);
        for (int32_t q : rq) mark[std::upper_bound(inst.begin(), inst.end(), q) - inst.begin() - 1] = 1;
        for (int i = 0; i < ninst; ++i) {
            if (!mark[i]) continue;
            const int32_t start = inst[i], len = inst[i + 1] - inst[i];
            run_f64<float, KCAP>(data + static_cast<size_t>(start) * dim, len, dim, k, nullptr, len,
                                 out_idx + static_cast<size_t>(start) * k, out_dist + static_cast<size_t>(start) * k,
                                 nullptr, s);
            shift_indices_kernel<<<grid_for(static_cast<size_t>(len) * k, 256), 256, 0, s>>>(
                out_idx + static_cast<size_t>(start) * k, static_cast<size_t>(len) * k, start);
            UMAPB_LAUNCH_CHECK();
        }
    }
}

}  // namespace

template <typename T>
void knn_exact_batched(const T* data, const std::vector<int32_t>& inst, int32_t dim, int32_t k, int32_t* out_idx,
                       T* out_dist, cudaStream_t s) {
    const int ninst = static_cast<int>(inst.size()) - 1;
    require(ninst >= 1, "at least one instance is needed");
    require(k >= 1 && k <= 120, "num_neighbors must be in [1, 120] for the device search");
    for (int i = 0; i < ninst; ++i) {
        require(inst[i + 1] - inst[i] > k, "every instance needs more observations than num_neighbors");
    }
    if constexpr (std::is_same<T, float>::value) {
        const int kcap = (k + 8 <= 16) ? 16 : (k + 8 <= 24) ? 24 : 32;
        if (k + 8 <= 32 && use_tensor_cores() && knn_tc_supported(dim, kcap)) {
            if (kcap == 16) run_f32_batched<16>(data, inst, dim, k, out_idx, out_dist, s);
            else if (kcap == 24) run_f32_batched<24>(data, inst, dim, k, out_idx, out_dist, s);
            else run_f32_batched<32>(data, inst, dim, k, out_idx, out_dist, s);
            return;
        }
    }
    for (int i = 0; i < ninst; ++i) {
        const int32_t start = inst[i], len = inst[i + 1] - inst[i];
        knn_exact<T>(data + static_cast<size_t>(start) * dim, len, dim, k, out_idx + static_cast<size_t>(start) * k,
                     out_dist + static_cast<size_t>(start) * k, s);
        shift_indices_kernel<<<grid_for(static_cast<size_t>(len) * k, 256), 256, 0, s>>>(
            out_idx + static_cast<size_t>(start) * k, static_cast<size_t>(len) * k, start);
        UMAPB_LAUNCH_CHECK();
    }
}

template void knn_exact_batched<float>(const float*, const std::vector<int32_t>&, int32_t, int32_t, int32_t*, float*,
                                       cudaStream_t);
template void knn_exact_batched<double>(const double*, const std::vector<int32_t>&, int32_t, int32_t, int32_t*,
                                        double*, cudaStream_t);

template <typename T>
void knn_exact_shard(const T* data, int32_t n, int32_t dim, int32_t k, KnnShard shard, int32_t* out_idx, T* out_dist,
                     DevArray<int32_t>& rows, int32_t& nrows, cudaStream_t s) {
    require(n >= 2, "the neighbour search needs at least two observations");
    require(dim >= 1, "data_dim must be positive");
    require(k >= 1 && k < n, "num_neighbors must be in [1, num_obs)");
    require(k <= 120, "num_neighbors above 120 is not supported by the device search");
    require(shard.count >= 1 && shard.index >= 0 && shard.index < shard.count, "shard must be in [0, num_shards)");
    if (shard.count == 1) {
        knn_exact<T>(data, n, dim, k, out_idx, out_dist, s);
        rows.allocate(n, s);
        iota_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, 0, rows.get());
        UMAPB_LAUNCH_CHECK();
        nrows = n;
        return;
    }
    if constexpr (std::is_same<T, float>::value) {
        if (k + 8 <= 16) run_f32<16>(data, n, dim, k, out_idx, out_dist, nullptr, s, shard, &rows, &nrows);
        else if (k + 8 <= 24) run_f32<24>(data, n, dim, k, out_idx, out_dist, nullptr, s, shard, &rows, &nrows);
        else if (k + 8 <= 32) run_f32<32>(data, n, dim, k, out_idx, out_dist, nullptr, s, shard, &rows, &nrows);
        else if (k + 8 <= 64) run_f32<64>(data, n, dim, k, out_idx, out_dist, nullptr, s, shard, &rows, &nrows);
        else run_f32<128>(data, n, dim, k, out_idx, out_dist, nullptr, s, shard, &rows, &nrows);
    } else {
        int32_t lo, hi;
        shard_row_range(n, shard, lo, hi);
        nrows = hi - lo;
        rows.allocate(std::max<int32_t>(nrows, 1), s);
        if (nrows > 0) {
            iota_kernel<<<grid_for(nrows, 256), 256, 0, s>>>(nrows, lo, rows.get());
            UMAPB_LAUNCH_CHECK();
            if (k <= 16) run_f64<double, 16>(data, n, dim, k, rows.get(), nrows, out_idx, out_dist, nullptr, s);
            else if (k <= 32) run_f64<double, 32>(data, n, dim, k, rows.get(), nrows, out_idx, out_dist, nullptr, s);
            else if (k <= 64) run_f64<double, 64>(data, n, dim, k, rows.get(), nrows, out_idx, out_dist, nullptr, s);
            else run_f64<double, 128>(data, n, dim, k, rows.get(), nrows, out_idx, out_dist, nullptr, s);
        }
    }
}

template void knn_exact_shard<float>(const float*, int32_t, int32_t, int32_t, KnnShard, int32_t*, float*,
                                     DevArray<int32_t>&, int32_t&, cudaStream_t);
template void knn_exact_shard<double>(const double*, int32_t, int32_t, int32_t, KnnShard, int32_t*, double*,
                                      DevArray<int32_t>&, int32_t&, cudaStream_t);

// Ranges the references are split into for nq queries: enough that the query
// tiles' CTAs fill the device twice over, as many as four lists of KCAP
// candidates go through one rescoring; 0 where the references are too few for
// the tensor-core search to pay (10 and 500 queries, 10 and 50 dimensions: 512
// references 0.24 and 0.27 ms against 0.18 and 0.31 on CUDA cores, 1024 0.23 and
// 0.28 against 0.25 and 0.49; 100,000 references and 10,000 queries 2.9 against
// 30 ms; with up to 8 neighbours in 3 dimensions 20,000 queries against 1,100
// references 0.48 against 0.41, 3,000 0.53 against 0.61).
static int query_lists(int32_t nref, int32_t nq, int32_t dim, int kcap) {
    if (nref < 1024 || (kcap == 16 && nref < 1536 - 10 * static_cast<int64_t>(dim))) return 0;
    const int64_t tiles = (static_cast<int64_t>(nq) + 127) / 128;
    int lists = 1;
    while (lists < 4 && 2 * lists * kcap <= 128 && tiles * lists < 2 * sm_count()) lists *= 2;
    return lists;
}

__global__ void add_offset_kernel(int32_t count, const int32_t* __restrict__ src, int32_t add,
                                  int32_t* __restrict__ dst) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) dst[i] = src[i] + add;
}

// Float queries against reference rows: FP32 candidates, FP64 rescoring and
// certification, FP64 search of the uncertain queries.  rows[slot] = nref +
// slot are the queries' data rows; results are written by slot.
// The candidates come from the tensor-core search (knn_tc.cu: every query tile
// against all references, a query tile's references split over several CTAs
// with a list each) where it takes the data, else from the brute-force kernel.
template <int KCAP>
void run_query_f32(const float* data, int32_t nref, int32_t nq, int32_t dim, int32_t k, const int32_t* rows,
                   int32_t* out_idx, float* out_dist, cudaStream_t s) {
    const int lists = query_lists(nref, nq, dim, KCAP);
    DevArray<int32_t> ci;
    DevArray<float> cd;
    DevArray<float> norms;
    DevArray<unsigned int> norm_max(1, s);
    bool tc = use_tensor_cores() && lists > 0 && knn_tc_supported(dim, KCAP);
    if (tc) {
        DevArray<int> err(1, s);
        err.zero(s);
        try {
            ci.allocate(static_cast<size_t>(nq) * lists * KCAP, s);
            cd.allocate(static_cast<size_t>(nq) * lists * KCAP, s);
            norms.allocate(static_cast<size_t>(nref) + nq, s);
            tc = knn_tc_query_candidates(data, nref, nq, dim, KCAP, lists, ci.get(), cd.get(), norms.get(), err.get(), s);
        } catch (const Error& e) {
            if (e.code != UMAPB_ERR_OOM) throw;   // the CUDA-core search needs no operands, and one list
            tc = false;
            ci.release();
            cd.release();
            norms.release();
        }
        int h_err = 0;
        UMAPB_CUDA(cudaMemcpyAsync(&h_err, err.get(), sizeof(int), cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        if (h_err != DEV_OK) fail(UMAPB_ERR_DEVICE_TIMEOUT, "tensor-core kNN: a pipeline wait gave up");
        if (tc) {
            norm_max.zero(s);
            norm_max_kernel<<<grid_for(nref + nq, 256, 1024), 256, 0, s>>>(nref + nq, norms.get(), norm_max.get());
            UMAPB_LAUNCH_CHECK();
        }
    }
    if (!tc) {
        ci.reserve(static_cast<size_t>(nq) * KCAP, s);
        cd.reserve(static_cast<size_t>(nq) * KCAP, s);
        knn_bruteforce_kernel<float, float, KCAP><<<(nq + KNN_BLOCK - 1) / KNN_BLOCK, KNN_BLOCK, 0, s>>>(
            data, nref, dim, rows, nq, ci.get(), cd.get());
        UMAPB_LAUNCH_CHECK();
    }
    DevArray<int32_t> redo(nq, s), redo_count(1, s);
    DevArray<double> redo_kth;
    allocate_if_possible(redo_kth, nq, s);
    redo_count.zero(s);
    auto rescore = [&](auto per) {
        knn_rescore_kernel<decltype(per)::value><<<rescore_grid(nq), RESCORE_WARPS * 32, 0, s>>>(
            data, nref, dim, k, rows, nq, tc ? lists : 1, KCAP, 1, 1, 0, ci.get(), cd.get(), out_idx, out_dist, nullptr,
            redo.get(), redo_kth.get(), redo_count.get(), tc ? norms.get() : nullptr, norm_max.get(), TC_REL_BOUND, nullptr);
        UMAPB_LAUNCH_CHECK();
    };
    if (tc && lists * KCAP > 32 * per_lane<KCAP>()) rescore(std::integral_constant<int, 4>());
    else rescore(std::integral_constant<int, per_lane<KCAP>()>());
    int32_t nredo = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&nredo, redo_count.get(), sizeof(int32_t), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    last_knn_redo_count() = nredo;
    if (nredo > 0) {   // redo holds slots: their data rows are nref + slot
        DevArray<int32_t> redo_rows(nredo, s);
        add_offset_kernel<<<grid_for(nredo, 256), 256, 0, s>>>(nredo, redo.get(), nref, redo_rows.get());
        UMAPB_LAUNCH_CHECK();
        search_again(data, nref, dim, k, redo_rows.get(), nredo, redo_kth.get(), nref, redo.get(), out_idx, out_dist,
                     nullptr, s);
    }
}

template <typename T>
void knn_query(const T* data, int32_t nref, int32_t nq, int32_t dim, int32_t k, int32_t* out_idx, T* out_dist,
               cudaStream_t s) {
    require(nref >= 1, "the search needs at least one reference point");
    require(dim >= 1, "data_dim must be positive");
    require(nq >= 0, "the number of query points must not be negative");
    require(k >= 1 && k <= nref, "num_neighbors must be in [1, number of reference points]");
    require(k <= 120, "num_neighbors above 120 is not supported by the device search");
    require(static_cast<int64_t>(nref) + nq <= INT32_MAX, "too many points for 32-bit indices");
    if (nq == 0) return;
    DevArray<int32_t> rows(nq, s);
    iota_kernel<<<grid_for(nq, 256), 256, 0, s>>>(nq, nref, rows.get());
    UMAPB_LAUNCH_CHECK();
    if constexpr (std::is_same<T, float>::value) {
        if (k + 8 <= 16) run_query_f32<16>(data, nref, nq, dim, k, rows.get(), out_idx, out_dist, s);
        else if (k + 8 <= 24) run_query_f32<24>(data, nref, nq, dim, k, rows.get(), out_idx, out_dist, s);
        else if (k + 8 <= 32) run_query_f32<32>(data, nref, nq, dim, k, rows.get(), out_idx, out_dist, s);
        else if (k + 8 <= 64) run_query_f32<64>(data, nref, nq, dim, k, rows.get(), out_idx, out_dist, s);
        else run_query_f32<128>(data, nref, nq, dim, k, rows.get(), out_idx, out_dist, s);
    } else {
        DevArray<int32_t> slots(nq, s);
        iota_kernel<<<grid_for(nq, 256), 256, 0, s>>>(nq, 0, slots.get());
        UMAPB_LAUNCH_CHECK();
        if (k <= 16) run_f64<double, 16>(data, nref, dim, k, rows.get(), nq, out_idx, out_dist, nullptr, s, slots.get());
        else if (k <= 32) run_f64<double, 32>(data, nref, dim, k, rows.get(), nq, out_idx, out_dist, nullptr, s, slots.get());
        else if (k <= 64) run_f64<double, 64>(data, nref, dim, k, rows.get(), nq, out_idx, out_dist, nullptr, s, slots.get());
        else run_f64<double, 128>(data, nref, dim, k, rows.get(), nq, out_idx, out_dist, nullptr, s, slots.get());
    }
}

template void knn_query<float>(const float*, int32_t, int32_t, int32_t, int32_t, int32_t*, float*, cudaStream_t);
template void knn_query<double>(const double*, int32_t, int32_t, int32_t, int32_t, int32_t*, double*, cudaStream_t);

template <typename T>
void knn_exact(const T* data, int32_t n, int32_t dim, int32_t k, int32_t* out_idx, T* out_dist, cudaStream_t s,
               double* out_dist_f64) {
    require(n >= 2, "the neighbour search needs at least two observations");
    require(dim >= 1, "data_dim must be positive");
    require(k >= 1 && k < n, "num_neighbors must be in [1, num_obs)");
    require(k <= 120, "num_neighbors above 120 is not supported by the device search");
    if constexpr (std::is_same<T, float>::value) {
        if (k + 8 <= 16) {
            run_f32<16>(data, n, dim, k, out_idx, out_dist, out_dist_f64, s);
        } else if (k + 8 <= 24) {
            run_f32<24>(data, n, dim, k, out_idx, out_dist, out_dist_f64, s);
        } else if (k + 8 <= 32) {
            run_f32<32>(data, n, dim, k, out_idx, out_dist, out_dist_f64, s);
        } else if (k + 8 <= 64) {
            run_f32<64>(data, n, dim, k, out_idx, out_dist, out_dist_f64, s);
        } else {
            run_f32<128>(data, n, dim, k, out_idx, out_dist, out_dist_f64, s);
        }
    } else {
        if (k <= 16) {
            run_f64<double, 16>(data, n, dim, k, nullptr, n, out_idx, out_dist, out_dist_f64, s);
        } else if (k <= 32) {
            run_f64<double, 32>(data, n, dim, k, nullptr, n, out_idx, out_dist, out_dist_f64, s);
        } else if (k <= 64) {
            run_f64<double, 64>(data, n, dim, k, nullptr, n, out_idx, out_dist, out_dist_f64, s);
        } else {
            run_f64<double, 128>(data, n, dim, k, nullptr, n, out_idx, out_dist, out_dist_f64, s);
        }
    }
}

template void knn_exact<float>(const float*, int32_t, int32_t, int32_t, int32_t*, float*, cudaStream_t, double*);
template void knn_exact<double>(const double*, int32_t, int32_t, int32_t, int32_t*, double*, cudaStream_t, double*);

}  // namespace umapb
