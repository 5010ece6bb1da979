// Initial layouts on the device.
//
// spectral_init (include/umappp/spectral_init.hpp:171-207): connectivity
// check, then the top num_dim + 1 eigenvectors of the shifted normalised
// Laplacian I + D^-1/2 W D^-1/2 (built in FP64 exactly as :38-78), of which
// the last num_dim are scaled to a maximum magnitude of 'scale' (:126-137).
// The reference obtains them with irlba; here a thick-restart Lanczos
// iteration (Wu and Simon, SIAM J. Matrix Anal. Appl. 22(2), 2000) runs its
// sparse products, Gram-Schmidt reorthogonalisation (two passes, FP64) and
// Ritz-vector updates on the device; only the small projected eigenproblem
// (ncv x ncv, ncv <= 64) is solved on the host by cyclic Jacobi.  Eigenvectors
// are signed so that their largest-magnitude entry is positive.
//
// random_init (:209-225): uniform on (-scale, scale) from Philox4x32-10.
// Jitter (:190-204): Box-Muller normals from Philox4x32-10.
#include <algorithm>
#include <cmath>
#include <vector>

#include "stages.cuh"

namespace umapb {

namespace {

template <typename T>
__global__ void degree_sqrt_kernel(int32_t n, const int64_t* __restrict__ ptr, const T* __restrict__ w,
                                   double* __restrict__ sums) {
    for (int32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < n; c += gridDim.x * blockDim.x) {
        double s = 0;
        for (int64_t p = ptr[c]; p < ptr[c + 1]; ++p) s += static_cast<double>(w[p]);
        sums[c] = sqrt(s);
    }
}

// One warp per row: rows differ in length by a factor of a hundred.
template <typename T>
__global__ void laplacian_values_kernel(int32_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                                        const T* __restrict__ w, const double* __restrict__ sums,
                                        double* __restrict__ lap) {
    const int64_t warps = static_cast<int64_t>(gridDim.x) * (blockDim.x >> 5);
    for (int64_t c = static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5); c < n; c += warps) {
        for (int64_t p = ptr[c] + (threadIdx.x & 31); p < ptr[c + 1]; p += 32) {
            lap[p] = __dmul_rn(__ddiv_rn(__ddiv_rn(-static_cast<double>(w[p]), sums[idx[p]]), sums[c]), -1.0);
        }
    }
}

// ---- Lanczos steps ----
// One step is three launches without a host read: every block owns a stretch
// of rows, so a product's rows go into the block's part of the next dot
// products at once, and a sum over blocks is taken by every block of the next
// launch for itself (the same bits everywhere).
//   step_product    v_j = x / |x| (its norm's partial sums given), w = A v_j,
//                   partial dots of w with v_0 .. v_j
//   step_project    w -= V h, then the partial dots again (first pass) or the
//                   partial squared norm (second pass)
// At 20,000 points a step takes 31 us; a row per thread and a launch for each
// vector operation, with two host reads, took 140 us (76 of them the product:
// its longest row is 300 edges).
constexpr int STEP_BLOCK = 512;
constexpr int STEP_WARPS = STEP_BLOCK / 32;
constexpr int MAX_BASIS = 64;

__device__ __forceinline__ double warp_sum(double x) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Sums of the blocks' partials of column c (nblk of them), by one warp.
__device__ __forceinline__ double sum_partials(const double* __restrict__ partial, int c, int nblk) {
    double s = 0;
    for (int b = threadIdx.x & 31; b < nblk; b += 32) s += partial[static_cast<size_t>(c) * nblk + b];
    return warp_sum(s);
}

// This block's rows of an n-vector.
__device__ __forceinline__ void block_rows(int32_t n, int32_t& r0, int32_t& r1) {
    r0 = static_cast<int32_t>(static_cast<int64_t>(n) * blockIdx.x / gridDim.x);
    r1 = static_cast<int32_t>(static_cast<int64_t>(n) * (blockIdx.x + 1) / gridDim.x);
}

// partial[c][block] = the block's part of V[:, c] . w, c < ncol; w's rows of
// this block are complete.
__device__ __forceinline__ void partial_dots(int32_t n, int32_t r0, int32_t r1, const double* V, int ncol,
                                             const double* w, double* __restrict__ partial) {
    const int lane = threadIdx.x & 31;
    for (int c = threadIdx.x >> 5; c < ncol; c += STEP_WARPS) {
        const double* v = V + static_cast<size_t>(c) * n;
        double s = 0;
        for (int32_t i = r0 + lane; i < r1; i += 32) s += v[i] * w[i];
        s = warp_sum(s);
        if (lane == 0) partial[static_cast<size_t>(c) * gridDim.x + blockIdx.x] = s;
    }
}

// x: v_j itself (norm2 null: then it is column j already), or a vector whose
// squared norm's partials are norm2; it is scaled to unit length (to zero if it
// is zero) and becomes column j, its norm *beta.  w = (I + D^-1/2 W D^-1/2) v_j.
__global__ void __launch_bounds__(STEP_BLOCK, 2)
    step_product_kernel(int32_t n, const int64_t* __restrict__ ptr, const int32_t* __restrict__ idx,
                        const double* __restrict__ lap, const double* __restrict__ x, const double* __restrict__ norm2,
                        double* V, int j, double* w, double* __restrict__ partial, double* __restrict__ beta) {
    __shared__ double scale;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t r0, r1;
    block_rows(n, r0, r1);
    double* vj = V + static_cast<size_t>(j) * n;
    if (warp == 0) {
        double f = 1.0;
        if (norm2) {
            const double nrm = sqrt(sum_partials(norm2, 0, gridDim.x));
            f = nrm > 0 ? 1.0 / nrm : 0.0;
            if (blockIdx.x == 0 && lane == 0) *beta = nrm;
        }
        if (lane == 0) scale = f;
    }
    __syncthreads();
    const double f = scale;
    if (norm2)
        for (int32_t i = r0 + threadIdx.x; i < r1; i += STEP_BLOCK) vj[i] = x[i] * f;
    for (int32_t c = r0 + warp; c < r1; c += STEP_WARPS) {
        double s = 0;
        for (int64_t p = ptr[c] + lane; p < ptr[c + 1]; p += 32) s += lap[p] * (x[idx[p]] * f);
        s = warp_sum(s);
        if (lane == 0) w[c] = x[c] * f + s;
    }
    __syncthreads();
    partial_dots(n, r0, r1, V, j + 1, w, partial);
}

// The dots alone (a fresh direction after an invariant subspace).
__global__ void __launch_bounds__(STEP_BLOCK, 2)
    step_dots_kernel(int32_t n, const double* V, int ncol, const double* w, double* __restrict__ partial) {
    int32_t r0, r1;
    block_rows(n, r0, r1);
    partial_dots(n, r0, r1, V, ncol, w, partial);
}

// w -= V[:, :ncol] h, h the sums of 'partial'; then 'out' gets the partial dots
// of w (second = false) or of |w|^2.  *alpha: h of the last column.
__global__ void __launch_bounds__(STEP_BLOCK, 2)
    step_project_kernel(int32_t n, const double* V, int ncol, const double* __restrict__ partial, double* w,
                        double* __restrict__ out, bool second, double* __restrict__ alpha) {
    __shared__ double h[MAX_BASIS + 1];
    __shared__ double red[STEP_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int32_t r0, r1;
    block_rows(n, r0, r1);
    for (int c = warp; c < ncol; c += STEP_WARPS) {
        const double s = sum_partials(partial, c, gridDim.x);
        if (lane == 0) {
            h[c] = s;
            if (blockIdx.x == 0 && c == ncol - 1) *alpha = s;
        }
    }
    __syncthreads();
    double sq = 0;
    for (int32_t i = r0 + threadIdx.x; i < r1; i += STEP_BLOCK) {
        double s = w[i];
        for (int c = 0; c < ncol; ++c) s -= h[c] * V[static_cast<size_t>(c) * n + i];
        w[i] = s;
        sq += s * s;
    }
    if (!second) {
        __syncthreads();
        partial_dots(n, r0, r1, V, ncol, w, out);
        return;
    }
    sq = warp_sum(sq);
    if (lane == 0) red[warp] = sq;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0;
        for (int q = 0; q < STEP_WARPS; ++q) s += red[q];
        out[blockIdx.x] = s;
    }
}

// Column 'col' = w / |w| and *beta = |w|, the end of a basis.
__global__ void __launch_bounds__(STEP_BLOCK, 2)
    step_scale_kernel(int32_t n, const double* __restrict__ w, const double* __restrict__ norm2, double* __restrict__ col,
                      double* __restrict__ beta) {
    __shared__ double scale;
    int32_t r0, r1;
    block_rows(n, r0, r1);
    if (threadIdx.x < 32) {
        const double nrm = sqrt(sum_partials(norm2, 0, gridDim.x));
        if (threadIdx.x == 0) {
            scale = nrm > 0 ? 1.0 / nrm : 0.0;
            if (blockIdx.x == 0) *beta = nrm;
        }
    }
    __syncthreads();
    for (int32_t i = r0 + threadIdx.x; i < r1; i += STEP_BLOCK) col[i] = w[i] * scale;
}

constexpr int DOT_BLOCK = 256;

// partial[b * ncol + c] = sum over the rows of block b of V[:, c] * w
__global__ void __launch_bounds__(DOT_BLOCK) multi_dot_kernel(int32_t n, const double* __restrict__ V, int ncol,
                                                              const double* __restrict__ w,
                                                              double* __restrict__ partial) {
    __shared__ double red[DOT_BLOCK / 32];
    const int c = blockIdx.y;
    const double* v = V + static_cast<size_t>(c) * n;
    double s = 0;
    for (int32_t i = blockIdx.x * DOT_BLOCK + threadIdx.x; i < n; i += gridDim.x * DOT_BLOCK) s += v[i] * w[i];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int q = 0; q < DOT_BLOCK / 32; ++q) t += red[q];
        partial[static_cast<size_t>(blockIdx.x) * ncol + c] = t;
    }
}

__global__ void reduce_partials_kernel(int nblk, int ncol, const double* __restrict__ partial, double* __restrict__ h) {
    const int c = threadIdx.x;
    if (c >= ncol) return;
    double t = 0;
    for (int b = 0; b < nblk; ++b) t += partial[static_cast<size_t>(b) * ncol + c];
    h[c] = t;
}

__global__ void scale_vector_kernel(int32_t n, const double* __restrict__ x, double f, double* __restrict__ y) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) y[i] = x[i] * f;
}

// out[:, c] = V[:, :nrow] S[:, c] for c < ncol (S row-major nrow x ldS)
__global__ void ritz_vectors_kernel(int32_t n, const double* __restrict__ V, int nrow, const double* __restrict__ S,
                                    int ldS, int ncol, double* __restrict__ out) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        for (int c = 0; c < ncol; ++c) {
            double s = 0;
            for (int r = 0; r < nrow; ++r) s += V[static_cast<size_t>(r) * n + i] * S[r * ldS + c];
            out[static_cast<size_t>(c) * n + i] = s;
        }
    }
}

// Deterministic start vector: splitmix64 of (seed + (i + 1) * golden) mapped to [-0.5, 0.5).
__global__ void start_vector_kernel(int32_t n, uint64_t seed, double* __restrict__ v) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        uint64_t z = seed + 0x9E3779B97F4A7C15ULL * static_cast<uint64_t>(i + 1);
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        z ^= z >> 31;
        v[i] = static_cast<double>(z >> 11) * (1.0 / 9007199254740992.0) - 0.5;
    }
}

// Per column: largest magnitude (as ordered bits; non-negative doubles order
// like their bit patterns), then the first index attaining it.
__global__ void col_max_abs_kernel(int32_t n, const double* __restrict__ V, unsigned long long* __restrict__ best) {
    const int c = blockIdx.y;
    const double* v = V + static_cast<size_t>(c) * n;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        atomicMax(&best[c], static_cast<unsigned long long>(__double_as_longlong(fabs(v[i]))));
    }
}

__global__ void col_first_at_kernel(int32_t n, const double* __restrict__ V, const unsigned long long* __restrict__ best,
                                    int* __restrict__ where) {
    const int c = blockIdx.y;
    const double* v = V + static_cast<size_t>(c) * n;
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (static_cast<unsigned long long>(__double_as_longlong(fabs(v[i]))) == best[c]) atomicMin(&where[c], i);
    }
}

__global__ void max_abs_kernel(int32_t n, const double* __restrict__ V, int first_col, int ncol,
                               unsigned long long* __restrict__ out) {
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < int64_t(n) * ncol; t += int64_t(gridDim.x) * blockDim.x) {
        const int c = static_cast<int>(t / n);
        const int32_t i = static_cast<int32_t>(t % n);
        const double a = fabs(V[static_cast<size_t>(first_col + c) * n + i]);
        atomicMax(out, static_cast<unsigned long long>(__double_as_longlong(a)));
    }
}

template <typename T>
__global__ void write_embedding_kernel(int32_t n, int num_dim, const double* __restrict__ U, const double* __restrict__ sign,
                                       double expansion, T* __restrict__ Y) {
    for (int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; t < int64_t(n) * num_dim; t += int64_t(gridDim.x) * blockDim.x) {
        const int32_t c = static_cast<int32_t>(t / num_dim);
        const int d = static_cast<int>(t % num_dim);
        Y[t] = static_cast<T>(U[static_cast<size_t>(d + 1) * n + c] * sign[d + 1] * expansion);
    }
}

template <typename T>
__global__ void jitter_kernel(size_t ntotal, T* __restrict__ Y, double sd, uint32_t k0, uint32_t k1) {
    const size_t npairs = (ntotal + 1) / 2;
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < npairs; i += size_t(gridDim.x) * blockDim.x) {
        const Philox4 r = philox4x32_10(static_cast<uint32_t>(i), static_cast<uint32_t>(i >> 32), 0, 0, k0, k1);
        double u1 = u64_to_unit_double(r.v[0], r.v[1]);
        const double u2 = u64_to_unit_double(r.v[2], r.v[3]);
        if (u1 <= 0) u1 = 1.0 / 9007199254740992.0;
        const double rad = sqrt(-2.0 * log(u1));
        const double th = 6.283185307179586476925286766559 * u2;
        Y[2 * i] = static_cast<T>(static_cast<double>(Y[2 * i]) + rad * cos(th) * sd);
        if (2 * i + 1 < ntotal) Y[2 * i + 1] = static_cast<T>(static_cast<double>(Y[2 * i + 1]) + rad * sin(th) * sd);
    }
}

template <typename T>
__global__ void random_init_kernel(size_t ntotal, T* __restrict__ Y, T mult, T shift, uint32_t k0, uint32_t k1) {
    for (size_t i = blockIdx.x * size_t(blockDim.x) + threadIdx.x; i < ntotal; i += size_t(gridDim.x) * blockDim.x) {
        const Philox4 r = philox4x32_10(static_cast<uint32_t>(i), static_cast<uint32_t>(i >> 32), 0, 0, k0, k1);
        T u;
        if constexpr (std::is_same<T, float>::value) {
            u = u32_to_unit_float(r.v[0]);
        } else {
            u = u64_to_unit_double(r.v[0], r.v[1]);
        }
        Y[i] = u * mult - shift;   // (-scale, scale), spectral_init.hpp:217-223
    }
}

// Cyclic Jacobi for a symmetric m x m matrix (row-major, destroyed): evals in
// decreasing order, evecs row-major with column i = eigenvector i.
void jacobi_eigen(int m, std::vector<double>& A, std::vector<double>& evals, std::vector<double>& evecs) {
    std::vector<double> V(static_cast<size_t>(m) * m, 0.0);
    for (int i = 0; i < m; ++i) V[i * m + i] = 1;
    for (int sweep = 0; sweep < 100; ++sweep) {
        double off = 0, total = 0;
        for (int i = 0; i < m; ++i)
            for (int j = 0; j < m; ++j) {
                const double a = A[i * m + j] * A[i * m + j];
                total += a;
                if (i != j) off += a;
            }
        if (off == 0 || off <= 1e-30 * total) break;
        for (int p = 0; p < m; ++p) {
            for (int q = p + 1; q < m; ++q) {
                const double apq = A[p * m + q];
                if (apq == 0) continue;
                const double theta = (A[q * m + q] - A[p * m + p]) / (2 * apq);
                const double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1));
                const double c = 1 / std::sqrt(t * t + 1), s = t * c;
                for (int k = 0; k < m; ++k) {
                    const double akp = A[k * m + p], akq = A[k * m + q];
                    A[k * m + p] = c * akp - s * akq;
                    A[k * m + q] = s * akp + c * akq;
                }
                for (int k = 0; k < m; ++k) {
                    const double apk = A[p * m + k], aqk = A[q * m + k];
                    A[p * m + k] = c * apk - s * aqk;
                    A[q * m + k] = s * apk + c * aqk;
                }
                for (int k = 0; k < m; ++k) {
                    const double vkp = V[k * m + p], vkq = V[k * m + q];
                    V[k * m + p] = c * vkp - s * vkq;
                    V[k * m + q] = s * vkp + c * vkq;
                }
            }
        }
    }
    std::vector<int> order(m);
    for (int i = 0; i < m; ++i) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return A[x * m + x] > A[y * m + y]; });
    evals.assign(m, 0);
    evecs.assign(static_cast<size_t>(m) * m, 0);
    for (int i = 0; i < m; ++i) {
        evals[i] = A[order[i] * m + order[i]];
        for (int k = 0; k < m; ++k) evecs[k * m + i] = V[k * m + order[i]];
    }
}

// Lanczos workspace and steps on the device.
struct LanczosDevice {
    int32_t n;
    int ncv;
    cudaStream_t s;
    const int64_t* ptr;
    const int32_t* idx;
    const double* lap;
    DevArray<double> V, h, partial, tmp;
    DevArray<double> w[2], dots[2], norm2, coef;   // coef: per step, alpha of both passes and beta
    int nblk, steps_blk;
    int cur = 0;               // w[cur]: the last step's vector, its squared norm in norm2

    LanczosDevice(int32_t n_, int ncv_, const int64_t* p, const int32_t* i, const double* l, cudaStream_t st)
        : n(n_), ncv(ncv_), s(st), ptr(p), idx(i), lap(l) {
        V.allocate(static_cast<size_t>(n) * (ncv + 1), s);
        h.allocate(1, s);
        nblk = static_cast<int>(std::min<int64_t>((n + 1023) / 1024, 256));
        partial.allocate(nblk, s);
        tmp.allocate(static_cast<size_t>(n) * (ncv + 1), s);
        steps_blk = static_cast<int>(std::min<int64_t>((n + STEP_WARPS - 1) / STEP_WARPS, 2 * sm_count()));
        for (int b = 0; b < 2; ++b) {
            w[b].allocate(n, s);
            dots[b].allocate(static_cast<size_t>(steps_blk) * (ncv + 1), s);
        }
        norm2.allocate(steps_blk, s);
        coef.allocate(3 * (static_cast<size_t>(ncv) + 1), s);
    }
    double* col(int c) const { return V.get() + static_cast<size_t>(c) * n; }
    // coefficients of step j: h of column j in the two passes, norm of what is left
    double* alpha1(int j) const { return coef.get() + 3 * j; }

    // w[cur] made orthogonal to columns [0, ncol) (dots[0] given), its norm in norm2
    void project(int ncol, int j) {
        for (int pass = 0; pass < 2; ++pass) {
            step_project_kernel<<<steps_blk, STEP_BLOCK, 0, s>>>(n, V.get(), ncol, dots[pass].get(), w[cur].get(),
                                                                 pass ? norm2.get() : dots[1].get(), pass != 0,
                                                                 alpha1(j) + pass);
            UMAPB_LAUNCH_CHECK();
        }
    }
    // Steps [j, ncv).  ready: column j is there; else it is w[cur], to be scaled.
    void steps(int j, bool ready) {
        for (; j < ncv; ++j, ready = false) {
            const double* x = ready ? col(j) : w[cur].get();
            cur ^= 1;
            step_product_kernel<<<steps_blk, STEP_BLOCK, 0, s>>>(n, ptr, idx, lap, x, ready ? nullptr : norm2.get(), V.get(),
                                                                 j, w[cur].get(), dots[0].get(),
                                                                 j > 0 ? alpha1(j - 1) + 2 : alpha1(ncv));
            UMAPB_LAUNCH_CHECK();
            project(j + 1, j);
        }
        step_scale_kernel<<<steps_blk, STEP_BLOCK, 0, s>>>(n, w[cur].get(), norm2.get(), col(ncv), alpha1(ncv - 1) + 2);
        UMAPB_LAUNCH_CHECK();
    }
    // After step j: a fresh direction, orthogonal to columns [0, j], as w[cur].
    void fresh(int j, uint64_t seed) {
        start_vector_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, seed, w[cur].get());
        UMAPB_LAUNCH_CHECK();
        step_dots_kernel<<<steps_blk, STEP_BLOCK, 0, s>>>(n, V.get(), j + 1, w[cur].get(), dots[0].get());
        UMAPB_LAUNCH_CHECK();
        project(j + 1, ncv);   // its coefficients are not part of the projected matrix
    }
    double norm(const double* x) {
        multi_dot_kernel<<<dim3(nblk, 1), DOT_BLOCK, 0, s>>>(n, x, 1, x, partial.get());
        UMAPB_LAUNCH_CHECK();
        reduce_partials_kernel<<<1, 32, 0, s>>>(nblk, 1, partial.get(), h.get());
        UMAPB_LAUNCH_CHECK();
        double v = 0;
        UMAPB_CUDA(cudaMemcpyAsync(&v, h.get(), sizeof(double), cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        return std::sqrt(v);
    }
    void scale(const double* x, double f, double* y) {
        scale_vector_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, x, f, y);
        UMAPB_LAUNCH_CHECK();
    }
};

}  // namespace

template <typename T>
SpectralResult spectral_init(int32_t n, const int64_t* ptr, const int32_t* idx, const T* w, int num_dim, T* Y,
                             int extra_work, int max_iterations, double tol, double scale, bool jitter,
                             double jitter_sd, uint64_t seed, int* d_status, cudaStream_t s) {
    SpectralResult res;
    const int nev = num_dim + 1;
    require(num_dim >= 1 && nev <= 63, "num_dim must be between 1 and 62 for spectral initialisation");
    if (n <= 0 || nev > n) return res;
    if (count_components(n, ptr, idx, d_status, s) > 1) return res;     // :182-184

    int64_t nnz = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&nnz, ptr + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    DevArray<double> sums(n, s), lap(std::max<int64_t>(nnz, 1), s);
    degree_sqrt_kernel<T><<<grid_for(n, 256), 256, 0, s>>>(n, ptr, w, sums.get());
    UMAPB_LAUNCH_CHECK();
    laplacian_values_kernel<T><<<grid_for(static_cast<size_t>(n) * 32, 256), 256, 0, s>>>(n, ptr, idx, w, sums.get(), lap.get());
    UMAPB_LAUNCH_CHECK();

    int ncv = nev + std::max(extra_work, nev) + 8;
    if (ncv > n) ncv = n;
    if (ncv > 64) ncv = 64;
    LanczosDevice L(n, ncv, ptr, idx, lap.get(), s);
    const uint64_t start_seed = 5489u;
    start_vector_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, start_seed, L.col(0));
    UMAPB_LAUNCH_CHECK();
    {
        const double nrm = L.norm(L.col(0));
        L.scale(L.col(0), 1.0 / nrm, L.col(0));
    }

    std::vector<double> T_(static_cast<size_t>(ncv) * ncv, 0.0), Tc, theta, S;
    int k = 0;
    double beta_last = 0;
    bool converged = false;
    std::vector<double> Sdev_host;
    DevArray<double> Sdev(static_cast<size_t>(ncv) * ncv, s);
    const int restarts = std::max(max_iterations, 1);
    for (int restart = 0; restart < restarts; ++restart) {
        std::vector<double> coef(3 * static_cast<size_t>(ncv));
        bool ready = true;
        for (int j = k; j < ncv;) {
            L.steps(j, ready);
            UMAPB_CUDA(cudaMemcpyAsync(coef.data(), L.coef.get(), sizeof(double) * coef.size(), cudaMemcpyDeviceToHost, s));
            UMAPB_SYNC(s);
            for (ready = true; j < ncv && ready; ++j) {
                const double alpha = coef[3 * j] + coef[3 * j + 1];
                double beta = coef[3 * j + 2];
                T_[j * ncv + j] = alpha;
                if (!(beta > 1e-12 * (std::fabs(alpha) + 1e-300))) {
                    // invariant subspace: continue from a fresh direction orthogonal to the basis
                    // (a full basis leaves nothing to add)
                    L.fresh(j, start_seed + 7919u * static_cast<uint64_t>(j + 1) + 104729u * static_cast<uint64_t>(restart));
                    beta = 0;
                    ready = false;
                    if (j + 1 == ncv) {
                        step_scale_kernel<<<L.steps_blk, STEP_BLOCK, 0, s>>>(n, L.w[L.cur].get(), L.norm2.get(), L.col(ncv),
                                                                             L.alpha1(ncv));
                        UMAPB_LAUNCH_CHECK();
                    }
                }
                if (j + 1 < ncv) {
                    T_[j * ncv + j + 1] = beta;
                    T_[(j + 1) * ncv + j] = beta;
                }
                beta_last = beta;
            }
        }
        Tc = T_;
        jacobi_eigen(ncv, Tc, theta, S);
        const double tscale = std::fabs(theta[0]) > 0 ? std::fabs(theta[0]) : 1;
        bool ok = true;
        for (int i = 0; i < nev; ++i) {
            if (std::fabs(beta_last * S[(ncv - 1) * ncv + i]) > tol * tscale) ok = false;
        }
        // with a full basis (ncv == n) the projection is exact
        if (ncv == n) ok = true;
        res.restarts = restart + 1;
        const bool last = ok || restart == restarts - 1;
        int keep = last ? nev : nev + (ncv - nev) / 2;
        keep = std::min(keep, ncv - 1);
        if (keep < nev) keep = nev;
        UMAPB_CUDA(cudaMemcpyAsync(Sdev.get(), S.data(), sizeof(double) * S.size(), cudaMemcpyHostToDevice, s));
        ritz_vectors_kernel<<<grid_for(n, 256), 256, 0, s>>>(n, L.V.get(), ncv, Sdev.get(), ncv, keep, L.tmp.get());
        UMAPB_LAUNCH_CHECK();
        if (last) {
            converged = ok;
            for (int c = 0; c < nev && c < 64; ++c) res.evals[c] = theta[c];
            break;
        }
        // thick restart: Ritz vectors first, then the residual direction
        UMAPB_CUDA(cudaMemcpyAsync(L.col(keep), L.col(ncv), sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
        UMAPB_CUDA(cudaMemcpyAsync(L.V.get(), L.tmp.get(), sizeof(double) * n * keep, cudaMemcpyDeviceToDevice, s));
        std::fill(T_.begin(), T_.end(), 0.0);
        for (int c = 0; c < keep; ++c) {
            T_[c * ncv + c] = theta[c];
            const double coupling = beta_last * S[(ncv - 1) * ncv + c];
            T_[c * ncv + keep] = coupling;
            T_[keep * ncv + c] = coupling;
        }
        k = keep;
    }
    if (!converged) return res;   // :123-125

    // normalise and sign the nev Ritz vectors (in L.tmp)
    std::vector<double> sign(nev, 1.0);
    {
        DevArray<unsigned long long> best(nev, s);
        DevArray<int> where(nev, s);
        best.zero(s);
        UMAPB_CUDA(cudaMemsetAsync(where.get(), 0x7f, sizeof(int) * nev, s));
        for (int c = 0; c < nev; ++c) {
            const double nrm = L.norm(L.tmp.get() + static_cast<size_t>(c) * n);
            L.scale(L.tmp.get() + static_cast<size_t>(c) * n, 1.0 / nrm, L.tmp.get() + static_cast<size_t>(c) * n);
        }
        col_max_abs_kernel<<<dim3(grid_for(n, 256, 1024), nev), 256, 0, s>>>(n, L.tmp.get(), best.get());
        UMAPB_LAUNCH_CHECK();
        col_first_at_kernel<<<dim3(grid_for(n, 256, 1024), nev), 256, 0, s>>>(n, L.tmp.get(), best.get(), where.get());
        UMAPB_LAUNCH_CHECK();
        std::vector<int> hw(nev);
        UMAPB_CUDA(cudaMemcpyAsync(hw.data(), where.get(), sizeof(int) * nev, cudaMemcpyDeviceToHost, s));
        UMAPB_SYNC(s);
        for (int c = 0; c < nev; ++c) {
            const int32_t i = (hw[c] >= 0 && hw[c] < n) ? hw[c] : 0;
            double v = 0;
            UMAPB_CUDA(cudaMemcpyAsync(&v, L.tmp.get() + static_cast<size_t>(c) * n + i, sizeof(double),
                                       cudaMemcpyDeviceToHost, s));
            UMAPB_SYNC(s);
            sign[c] = (v < 0) ? -1.0 : 1.0;
        }
    }
    // scale to max |value| = scale over the kept columns (:128-131)
    DevArray<unsigned long long> mx(1, s);
    mx.zero(s);
    max_abs_kernel<<<grid_for(static_cast<size_t>(n) * num_dim, 256), 256, 0, s>>>(n, L.tmp.get(), 1, num_dim, mx.get());
    UMAPB_LAUNCH_CHECK();
    unsigned long long mbits = 0;
    UMAPB_CUDA(cudaMemcpyAsync(&mbits, mx.get(), sizeof(mbits), cudaMemcpyDeviceToHost, s));
    UMAPB_SYNC(s);
    double max_val;
    std::memcpy(&max_val, &mbits, sizeof(double));
    const double expansion = (max_val > 0 ? scale / max_val : 1);
    DevArray<double> dsign(nev, s);
    UMAPB_CUDA(cudaMemcpyAsync(dsign.get(), sign.data(), sizeof(double) * nev, cudaMemcpyHostToDevice, s));
    write_embedding_kernel<T><<<grid_for(static_cast<size_t>(n) * num_dim, 256), 256, 0, s>>>(
        n, num_dim, L.tmp.get(), dsign.get(), expansion, Y);
    UMAPB_LAUNCH_CHECK();
    if (jitter) {
        const size_t ntotal = static_cast<size_t>(n) * num_dim;
        jitter_kernel<T><<<grid_for((ntotal + 1) / 2, 256), 256, 0, s>>>(
            ntotal, Y, jitter_sd, static_cast<uint32_t>(seed) ^ RNG_JITTER, static_cast<uint32_t>(seed >> 32));
        UMAPB_LAUNCH_CHECK();
    }
    UMAPB_SYNC(s);
    res.ok = true;
    return res;
}

template <typename T>
void random_init(int32_t n, int num_dim, T* Y, uint64_t seed, double scale, cudaStream_t s) {
    const size_t ntotal = static_cast<size_t>(n) * num_dim;
    if (ntotal == 0) return;
    random_init_kernel<T><<<grid_for(ntotal, 256), 256, 0, s>>>(ntotal, Y, static_cast<T>(scale * 2),
                                                                static_cast<T>(scale),
                                                                static_cast<uint32_t>(seed) ^ RNG_RANDOM_INIT,
                                                                static_cast<uint32_t>(seed >> 32));
    UMAPB_LAUNCH_CHECK();
}

template SpectralResult spectral_init<float>(int32_t, const int64_t*, const int32_t*, const float*, int, float*, int, int,
                                             double, double, bool, double, uint64_t, int*, cudaStream_t);
template SpectralResult spectral_init<double>(int32_t, const int64_t*, const int32_t*, const double*, int, double*, int,
                                              int, double, double, bool, double, uint64_t, int*, cudaStream_t);
template void random_init<float>(int32_t, int, float*, uint64_t, double, cudaStream_t);
template void random_init<double>(int32_t, int, double*, uint64_t, double, cudaStream_t);

}  // namespace umapb
