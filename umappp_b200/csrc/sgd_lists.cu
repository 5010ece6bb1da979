// Interaction lists of the SGD epochs (sgd_lists.cuh).
//
// The schedule (include/umappp/optimize_layout.hpp:141-179: which edges fire,
// how many negative samples each draws) and the samples themselves do not
// depend on the layout, so they are worked out ahead of the epochs, in
// parallel over all edges, instead of inside the layout's serial chains.  The
// reference's Float_ arithmetic is kept exactly (this file is compiled with
// -fmad=false).
//
// One warp takes a segment of rows (about 288 edges, whole rows; a longer
// segment in chunks) through a whole window of epochs with the segment's state
// in shared memory: per epoch it compacts the firing edges into a queue, then
// takes the queue 32 edges at a time with all lanes busy -- schedule step,
// Philox draws, a scan that places every edge's entries (rows start at
// multiples of LIST_ALIGN), entries staged in shared memory and written out in
// order.  Bound by instruction issue, about 450 warp instructions per 32
// firing edges (the samples 130, the two sums that place the entries 35), and
// by the chains between them: at a million points, 200 epochs take 121 ms with
// six blocks per SM, 124 with five, 127 with five and one scan that carried
// the rows' starts along (85 instructions).  An edge per thread without the
// queue had 0.28 of the lanes busy in all of it.
#include <cub/cub.cuh>

#include <algorithm>

#include "list_stage.cuh"
#include "neg_stream.cuh"
#include "stages.cuh"

namespace umapb {

namespace {

constexpr int GEN_WARPS = 4;
// Blocks per SM, alone and beside epochs (which need half of the registers).
constexpr int GEN_BLOCKS = 6, GEN_BLOCKS_BESIDE = 3;
constexpr int STAGE = 512;   // entries staged per 32 firing edges (they have 6 each on average)
constexpr int LATE = 32;     // edges with more than STAGE_SAMPLES samples kept for the end of an epoch

// Edges of a segment's state kept in shared memory (9 KB per warp either way).
template <typename T>
constexpr int seg_edges() { return sizeof(T) == 4 ? 384 : 256; }
// Rows whose first edge falls in the same SEG_TARGET edges form a segment.
template <typename T>
constexpr int seg_target() { return seg_edges<T>() * 3 / 4; }

template <typename T>
struct alignas(16) GenWarp {
    T en[seg_edges<T>()], enn[seg_edges<T>()], ep[seg_edges<T>()], epns[seg_edges<T>()];
    int32_t stage[STAGE];
    uint16_t queue[seg_edges<T>()];
    uint32_t late_off[LATE], late_draws[LATE];
    uint16_t late_edge[LATE];
};

template <typename T>
struct GenArgs {
    const int64_t* ptr;
    const int32_t* heads;
    const int32_t* targets;
    const T* eps;
    T* enext;
    T* enneg;
    T rate;
    const int32_t* seg_row;
    int64_t nseg;
    int first, epochs;
    uint64_t* cap;              // sizing: [epoch][segment] entries, multiples of LIST_ALIGN
    const uint64_t* base;       // filling: the same, as offsets
    int32_t* list;
    ListSpan* span;
    int32_t nrows;
    ListStream stream;
    uint32_t key0[7], key1[7];  // the Philox key of each round
    unsigned long long* totals;
};

// First row r in [0, n] with ptr[r] >= s * target, for every s.
__global__ void segment_rows_kernel(int32_t n, const int64_t* __restrict__ ptr, int64_t nseg, int target,
                                    int32_t* __restrict__ seg_row) {
    for (int64_t s = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; s <= nseg; s += int64_t(gridDim.x) * blockDim.x) {
        int32_t lo = 0, hi = n;
        if (s == nseg) lo = n;   // the last segment takes the empty rows at the end
        while (lo < hi) {
            const int32_t mid = lo + (hi - lo) / 2;
            if (ptr[mid] < s * target) lo = mid + 1; else hi = mid;
        }
        seg_row[s] = lo;
    }
}

__device__ __forceinline__ uint32_t round_up(uint32_t x) { return (x + (LIST_ALIGN - 1)) & ~uint32_t(LIST_ALIGN - 1); }

// Inclusive sum over the lanes of a warp.
__device__ __forceinline__ uint32_t prefix_sum(uint32_t x) {
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)   // the shuffle's predicate: a lane with a source
        asm volatile("{\n\t.reg .pred p;\n\t.reg .u32 r;\n\t"
                     "shfl.sync.up.b32 r|p, %0, %1, 0, 0xffffffff;\n\t@p add.u32 %0, %0, r;\n\t}" : "+r"(x) : "r"(o));
    return x;
}

// Observation range of the instance that owns row h.
__device__ __forceinline__ void instance_range(int32_t h, const ListStream& p, int32_t& base, uint32_t& size) {
    base = 0;
    size = static_cast<uint32_t>(p.n);
    if (p.num_inst <= 1) return;
    int lo = 0, hi = p.num_inst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (p.inst_start[mid] <= h) lo = mid; else hi = mid - 1;
    }
    base = p.inst_start[lo];
    size = static_cast<uint32_t>(p.inst_start[lo + 1] - base);
}

// Philox4x32-7 (common.cuh) with the rounds' keys at hand.
template <typename T>
__device__ __forceinline__ Philox4 philox7(uint32_t c0, uint32_t c1, uint32_t c2, uint32_t c3, const GenArgs<T>& g) {
#pragma unroll
    for (int r = 0; r < 7; ++r) {
        const uint64_t p0 = static_cast<uint64_t>(0xD2511F53u) * c0, p1 = static_cast<uint64_t>(0xCD9E8D57u) * c2;
        c0 = static_cast<uint32_t>(p1 >> 32) ^ c1 ^ g.key0[r];
        c2 = static_cast<uint32_t>(p0 >> 32) ^ c3 ^ g.key1[r];
        c1 = static_cast<uint32_t>(p1);
        c3 = static_cast<uint32_t>(p0);
    }
    return Philox4{{c0, c1, c2, c3}};
}

// Samples [q, draws) of an edge, q a multiple of 4, to out[q..): the draws of
// NegStream::bounded without its rejections.  Returns whether one of them
// could be rejected (nsize in 2^32 per draw): the edge is then drawn again.
template <typename T>
__device__ __forceinline__ bool draw_from(uint32_t hid, uint32_t tid, uint32_t epoch, uint32_t q, uint32_t draws,
                                          int32_t nbase, uint32_t nsize, const GenArgs<T>& g, int32_t* out) {
    bool again = false;
    for (; q < draws; q += 4) {
        const Philox4 v = philox7(hid, tid, epoch, q >> 2, g);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint64_t x = static_cast<uint64_t>(v.v[i]) * nsize;
            if (q + i < draws) {
                again |= static_cast<uint32_t>(x) < nsize;
                out[q + i] = nbase + static_cast<int32_t>(x >> 32);
            }
        }
    }
    return again;
}

// All samples of an edge, with the rejections.
__device__ __forceinline__ void draw_all(uint32_t hid, uint32_t tid, uint32_t epoch, uint32_t draws, int32_t nbase,
                                      uint32_t nsize, uint32_t k0, uint32_t k1, int32_t* out) {
    NegStream rng(hid, tid, epoch, k0, k1);
    for (uint32_t q = 0; q < draws; ++q) out[q] = nbase + rng.bounded(nsize);
}

// FILL = false: cap = room for the segment's entries in every epoch of the
// window.  FILL = true: the entries, the rows' spans and the state at the end.
template <typename T, bool FILL>
__global__ void __launch_bounds__(GEN_WARPS * 32, GEN_BLOCKS) schedule_kernel(const __grid_constant__ GenArgs<T> g) {
    constexpr int SEG = seg_edges<T>();
    __shared__ GenWarp<T> slab[GEN_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    GenWarp<T>& w = slab[warp];
    // whole warps take segments, and there is no block-wide barrier
    for (int64_t s = static_cast<int64_t>(blockIdx.x) * GEN_WARPS + warp; s < g.nseg; s += int64_t(gridDim.x) * GEN_WARPS) {
        const int32_t r0 = g.seg_row[s], r1 = g.seg_row[s + 1];
        const int64_t j0 = g.ptr[r0], j1 = g.ptr[r1];
        // lane e keeps epoch e's position: entries placed so far, the last head, totals
        uint64_t base = 0, entries = 0, fired = 0, drawn = 0;
        uint32_t pos_of = 0;
        int32_t head_of = -1;
        if (FILL && lane < g.epochs) base = g.base[lane * g.nseg + s];
        for (int64_t c = j0; c < j1; c += SEG) {
            const int m = static_cast<int>(j1 - c < SEG ? j1 - c : SEG);
            for (int i = lane; i < m; i += 32) {
                const T ep = g.eps[c + i];
                w.en[i] = g.enext[c + i];
                w.enn[i] = g.enneg[c + i];
                w.ep[i] = ep;
                w.epns[i] = ep / g.rate;   // optimize_layout.hpp:160
            }
            for (int i = m + lane; i < (m + 127) / 128 * 128; i += 32) w.en[i] = T(CUDART_INF);   // never fires
            __syncwarp();
            for (int e = 0; e < g.epochs; ++e) {
                const T ef = static_cast<T>(g.first + e);
                int qn = 0;
                for (int i0 = 0; i0 < m; i0 += 128) {   // four edges per lane
                    const int i = i0 + 4 * lane;
                    T v[4];
                    if constexpr (sizeof(T) == 4) {
                        const float4 x = *reinterpret_cast<const float4*>(&w.en[i]);
                        v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
                    } else {
                        const double2 x = *reinterpret_cast<const double2*>(&w.en[i]);
                        const double2 y = *reinterpret_cast<const double2*>(&w.en[i + 2]);
                        v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
                    }
                    unsigned mask[4];
                    int at = qn;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        mask[k] = __ballot_sync(0xffffffffu, v[k] <= ef);
                        at += __popc(mask[k] & below);
                        qn += __popc(mask[k]);
                    }
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        if (v[k] <= ef) w.queue[at++] = static_cast<uint16_t>(i + k);
                }
                __syncwarp();
                uint64_t sum = 0;   // entries of this epoch (sizing), or samples drawn (filling, when counted)
                const uint64_t ebase = FILL ? __shfl_sync(0xffffffffu, base, e) : 0;
                uint32_t pos = FILL ? __shfl_sync(0xffffffffu, pos_of, e) : 0;
                // the stage holds the entries from 'origin', a multiple of LIST_ALIGN, on
                uint32_t origin = pos & ~uint32_t(LIST_ALIGN - 1);
                int nlate = 0;
                if (FILL && pos != origin) {   // a row of several chunks
                    if (lane < LIST_ALIGN) w.stage[lane] = g.list[ebase + origin + lane];
                    __syncwarp();
                }
                int32_t last = FILL ? __shfl_sync(0xffffffffu, head_of, e) : 0;
                const uint32_t epoch = static_cast<uint32_t>(g.first + e);
                ListSpan* spans = FILL ? g.span + static_cast<int64_t>(e) * g.nrows : nullptr;
                const int32_t* heads = FILL ? g.heads + c : nullptr;
                const int32_t* targets = FILL ? g.targets + c : nullptr;
                for (int q0 = 0; q0 < qn; q0 += 32) {
                    const bool on = q0 + lane < qn;
                    const int j = on ? w.queue[q0 + lane] : 0;
                    uint32_t draws = 0;
                    if (on) {   // optimize_layout.hpp:160-161,178-179
                        const T ep = w.ep[j], enn = w.enn[j], epns = w.epns[j];
                        const int nn = static_cast<int>((ef - enn) / epns);
                        w.en[j] += ep;
                        w.enn[j] = enn + static_cast<T>(nn) * epns;
                        draws = nn > 0 ? static_cast<uint32_t>(nn) : 0u;   // a negative count draws nothing
                    }
                    if (!FILL) {
                        if (on) sum += 1ull + draws;
                        continue;
                    }
                    sum += draws;
                    const int32_t h = on ? heads[j] : -2;
                    const int32_t t = on ? targets[j] : 0;
                    const uint32_t cnt = on ? draws + 1 : 0;
                    int32_t prev = __shfl_up_sync(0xffffffffu, h, 1);
                    if (lane == 0) prev = last;
                    // Placing 32 edges after one another, rows at multiples of
                    // LIST_ALIGN: a row starts where the one before it ends, which
                    // started at such a multiple too (or before this group, whose
                    // position is known), so its padding follows from the plain sums.
                    const bool opens = on && h != prev;
                    const uint32_t ahead = prefix_sum(cnt) - cnt;
                    const unsigned opened = __ballot_sync(0xffffffffu, opens) & below;
                    const uint32_t at_open = __shfl_sync(0xffffffffu, ahead, opened ? 31 - __clz(opened) : 0);
                    const uint32_t pad = opens ? ((opened ? at_open : 0u - pos) - ahead) & (LIST_ALIGN - 1) : 0u;
                    const uint32_t off = pos + ahead + prefix_sum(pad);
                    const uint32_t end = off + cnt;
                    const int32_t next = __shfl_down_sync(0xffffffffu, h, 1);
                    const bool ends = on && (lane == 31 || next != h);
                    ListSpan* sp = spans + h;
                    if (opens) sp->start8 = static_cast<uint32_t>(ebase / LIST_ALIGN) + off / LIST_ALIGN;
                    if (ends) sp->end = static_cast<uint32_t>(ebase) + end;
                    const int tail = min(qn - q0, 32) - 1;   // last lane in use
                    pos = __shfl_sync(0xffffffffu, end, tail);
                    last = __shfl_sync(0xffffffffu, h, tail);
                    const bool staged = round_up(pos) - origin <= STAGE;
                    const uint32_t hid = static_cast<uint32_t>(g.stream.head0 + h), tid = static_cast<uint32_t>(t);
                    int32_t nbase = 0;
                    uint32_t nsize = 0;
                    if (on) instance_range(h, g.stream, nbase, nsize);
                    bool again = false;
                    int32_t* out;
                    if (staged) {
                        out = w.stage + (off - origin);   // (without an edge: nothing is stored)
                        uint32_t low = 0xffffffffu;
                        int32_t k[STAGE_SAMPLES];
#pragma unroll
                        for (int q = 0; q < STAGE_SAMPLES; q += 4) {
                            const Philox4 v = philox7(hid, tid, epoch, q >> 2, g);
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const uint64_t x = static_cast<uint64_t>(v.v[i]) * nsize;
                                low = min(low, static_cast<uint32_t>(x));
                                k[q + i] = nbase + static_cast<int32_t>(x >> 32);
                            }
                        }
                        again = low < nsize;
                        // (the next 32 edges overwrite the padding where they continue the row)
                        stage_edge(out, on, t | LIST_ATTRACT, k, draws, ends ? (0u - end) & (LIST_ALIGN - 1) : 0u, h);
                    } else {   // many samples per edge: straight to the list
                        if (lane < LIST_ALIGN) g.list[ebase + origin + lane] = w.stage[lane];
                        __syncwarp();
                        out = g.list + (ebase + off);
                        if (on) {
                            out[0] = t | LIST_ATTRACT;
                            again = draw_from(hid, tid, epoch, 0, min(draws, uint32_t(STAGE_SAMPLES)), nbase, nsize, g, out + 1);
                        }
                        if (ends)
                            for (uint32_t i = end; i < round_up(end); ++i) out[i - off] = h;
                    }
                    // few edges draw more than 8: they wait until the epoch's end, when
                    // one pass takes them together (unless they are many, or rejected)
                    const unsigned more = __ballot_sync(0xffffffffu, draws > 8);
                    if (more || __any_sync(0xffffffffu, again)) {
                        __syncwarp();
                        const int few = __popc(more);
                        const bool wait = few <= 8 && nlate + few <= LATE;
                        if (draws > 8) {
                            if (wait) {
                                const int k = nlate + __popc(more & below);
                                w.late_off[k] = off;
                                w.late_draws[k] = again ? draws | 0x80000000u : draws;
                                w.late_edge[k] = static_cast<uint16_t>(j);
                            } else {
                                again |= draw_from(hid, tid, epoch, 8, draws, nbase, nsize, g, out + 1);
                            }
                        }
                        if (wait) nlate += few;
                        if (on && again && (draws <= 8 || !wait))
                            draw_all(hid, tid, epoch, draws, nbase, nsize, g.stream.k0, g.stream.k1, out + 1);
                    }
                    __syncwarp();
                    // whole blocks of LIST_ALIGN go out; the last, begun one (with its
                    // padding) stays, to be continued by the next 32 edges
                    const uint32_t upto = q0 + 32 < qn ? pos & ~uint32_t(LIST_ALIGN - 1) : round_up(pos);
                    if (staged) {
                        int4* to = reinterpret_cast<int4*>(g.list + (ebase + origin));
                        const int4* from = reinterpret_cast<const int4*>(w.stage);
                        for (uint32_t i = lane; i < (upto - origin) / 4; i += 32) to[i] = from[i];
                        const int32_t rest = lane < LIST_ALIGN && upto < pos ? w.stage[upto - origin + lane] : 0;
                        __syncwarp();
                        if (lane < LIST_ALIGN) w.stage[lane] = rest;
                    } else if (upto < pos && lane < LIST_ALIGN) {
                        w.stage[lane] = g.list[ebase + upto + lane];
                    }
                    origin = upto;
                    __syncwarp();
                }
                if (FILL && nlate) {
                    if (lane < nlate) {
                        const int64_t k = c + w.late_edge[lane];
                        const uint32_t draws = w.late_draws[lane] & 0x7fffffffu;
                        const int32_t h = g.heads[k];
                        const uint32_t hid = static_cast<uint32_t>(g.stream.head0 + h);
                        const uint32_t tid = static_cast<uint32_t>(g.targets[k]);
                        int32_t nbase;
                        uint32_t nsize;
                        instance_range(h, g.stream, nbase, nsize);
                        int32_t* out = g.list + (ebase + w.late_off[lane]) + 1;
                        bool again = w.late_draws[lane] >> 31;
                        again |= draw_from(hid, tid, epoch, 8, draws, nbase, nsize, g, out);
                        if (again) draw_all(hid, tid, epoch, draws, nbase, nsize, g.stream.k0, g.stream.k1, out);
                    }
                    __syncwarp();
                }
                if (!FILL || g.totals) {
                    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                    if (lane == e) {
                        entries += sum;
                        drawn += sum;
                        fired += static_cast<uint64_t>(qn);
                    }
                }
                if (FILL && lane == e) {
                    pos_of = pos;
                    head_of = last;
                }
                __syncwarp();
            }
            if (FILL) {
                for (int i = lane; i < m; i += 32) {
                    g.enext[c + i] = w.en[i];
                    g.enneg[c + i] = w.enn[i];
                }
            }
            __syncwarp();
        }
        if (lane < g.epochs) {
            if (!FILL) {
                // at most LIST_ALIGN - 1 entries of padding before each row that fires
                const uint64_t rows = static_cast<uint64_t>(r1 - r0);
                const uint64_t room = entries + (LIST_ALIGN - 1) * (rows < fired ? rows : fired);
                // a segment's positions are 32 bits: one beyond them makes the window's total refuse it
                g.cap[lane * g.nseg + s] = room > UINT32_MAX - LIST_ALIGN ? uint64_t(1) << 40
                                                                          : (room + LIST_ALIGN - 1) / LIST_ALIGN * LIST_ALIGN;
            } else if (g.totals) {
                atomicAdd(&g.totals[2 * lane], static_cast<unsigned long long>(fired));
                atomicAdd(&g.totals[2 * lane + 1], static_cast<unsigned long long>(drawn));
            }
        }
    }
}

template <typename T>
GenArgs<T> gen_args(const DeviceEpochs<T>& ep, const int32_t* seg_row, int64_t nseg, int first, int epochs) {
    GenArgs<T> g{};
    g.ptr = ep.ptr.get();
    g.heads = ep.heads.get();
    g.targets = ep.targets.get();
    g.eps = ep.eps.get();
    g.rate = ep.negative_sample_rate;
    g.seg_row = seg_row;
    g.nseg = nseg;
    g.first = first;
    g.epochs = epochs;
    g.nrows = ep.n;
    return g;
}

// Blocks for nseg segments: as many as are resident at once, each taking
// segment after segment.
unsigned gen_grid(int64_t nseg, bool beside_epochs) {
    const int per_sm = beside_epochs ? GEN_BLOCKS_BESIDE : GEN_BLOCKS;
    return static_cast<unsigned>(std::min<int64_t>((nseg + GEN_WARPS - 1) / GEN_WARPS, int64_t(sm_count()) * per_sm));
}

}  // namespace

template <typename T>
InteractionLists<T>::~InteractionLists() {
    if (sized_) {
        cudaEventSynchronize(sized_);   // the pinned word may still be written
        event_put(sized_);
    }
    pinned_put(total_);
}

template <typename T>
void InteractionLists<T>::setup(const DeviceEpochs<T>* ep, bool with_tasks, cudaStream_t s) {
    ep_ = ep;
    with_tasks_ = with_tasks;
    nseg_ = ep->n > 0 ? ep->nnz / seg_target<T>() + 1 : 0;
    if (nseg_ == 0) return;
    seg_row_.allocate(nseg_ + 1, s);
    segment_rows_kernel<<<grid_for(nseg_ + 1, 256), 256, 0, s>>>(ep->n, ep->ptr.get(), nseg_, seg_target<T>(),
                                                                 seg_row_.get());
    UMAPB_LAUNCH_CHECK();
}

template <typename T>
void InteractionLists<T>::release(int buffer) {
    list_[buffer].release();
    span_[buffer].release();
    tasks_[buffer].release();
}

template <typename T>
void InteractionLists<T>::release() {
    release(0);
    release(1);
    cap_.release();
    base_.release();
    temp_.release();
}

// Entries of a list allocated for a window's 'total': an eighth more, as windows
// of one run differ a little, within 'most' bytes -- and all of them where there
// is one buffer and the window takes half of it: in a run's first epochs fewer
// edges fire than later (0.73 of them in the first nine at a million points).
static uint64_t list_room(uint64_t total, double most, bool one_buffer) {
    const uint64_t all = static_cast<uint64_t>(std::max(0.0, most) / 4);
    return std::max(total, one_buffer && total >= all / 2 ? all : std::min(total + total / 8, all));
}

template <typename T>
int InteractionLists<T>::window_epochs(int buffer, size_t bytes) const {
    double entries = per_epoch_;
    if (entries == 0) {
        // no window yet: about 0.28 of the edges fire in an epoch (15 neighbours), with a
        // target and negative_sample_rate samples each, and rows are padded
        entries = (0.28 * (1.0 + std::max(0.0, static_cast<double>(ep_->negative_sample_rate))) + 0.17) *
                  static_cast<double>(std::max<int64_t>(ep_->nnz, 1));
    }
    // (a sixteenth above, once the entries are known: windows as long as the estimate's)
    double epochs = (per_epoch_ == 0 ? 1.0 : 1.0625) * static_cast<double>(bytes) / epoch_bytes(entries);
    if (full_grown(buffer, bytes)) epochs = std::min(epochs, list_[buffer].size() / entries);
    return static_cast<int>(std::min<double>(MAX_WINDOW, std::max(1.0, epochs)));
}

// Bytes of an epoch of so many entries: they, and each row's span and task.
template <typename T>
double InteractionLists<T>::epoch_bytes(double entries) const {
    return 4.0 * entries + static_cast<double>(sizeof(ListSpan) + sizeof(RowTask)) * ep_->n;
}

template <typename T>
void InteractionLists<T>::prepare(int first, int epochs, const T* enext, const T* enneg, bool beside_epochs,
                                  cudaStream_t s) {
    first_ = first;
    epochs_ = std::min(epochs, MAX_WINDOW);
    if (nseg_ == 0) return;
    int64_t cells = 0;
    size_t tb = 0;
    for (;; epochs_ = (epochs_ + 1) / 2) {
        cells = nseg_ * epochs_;
        if (cells >= INT32_MAX) {
            require(epochs_ > 1, "too many edges for the schedule's segments", UMAPB_ERR_OVERFLOW);
            continue;
        }
        try {
            cap_.reserve(cells + 1, s);
            base_.reserve(cells + 1, s);
            UMAPB_CUDA(cub::DeviceScan::ExclusiveSum(nullptr, tb, cap_.get(), base_.get(), static_cast<int>(cells + 1), s));
            temp_.reserve(tb, s);
            break;
        } catch (const Error& e) {
            cap_.release();
            base_.release();
            temp_.release();
            if (e.code != UMAPB_ERR_OOM || epochs_ == 1) throw;
        }
    }
    UMAPB_CUDA(cudaMemsetAsync(cap_.get() + cells, 0, sizeof(uint64_t), s));
    GenArgs<T> g = gen_args(*ep_, seg_row_.get(), nseg_, first_, epochs_);
    g.enext = const_cast<T*>(enext);   // read only while sizing
    g.enneg = const_cast<T*>(enneg);
    g.cap = cap_.get();
    schedule_kernel<T, false><<<gen_grid(nseg_, beside_epochs), GEN_WARPS * 32, 0, s>>>(g);
    UMAPB_LAUNCH_CHECK();
    UMAPB_CUDA(cub::DeviceScan::ExclusiveSum(temp_.get(), tb, cap_.get(), base_.get(), static_cast<int>(cells + 1), s));
    if (!total_) total_ = static_cast<uint64_t*>(pinned_get());
    if (!sized_) sized_ = event_get();
    UMAPB_CUDA(cudaMemcpyAsync(total_, base_.get() + cells, sizeof(uint64_t), cudaMemcpyDeviceToHost, s));
    UMAPB_CUDA(cudaEventRecord(sized_, s));
}

template <typename T>
int InteractionLists<T>::build(int buffer, size_t bytes, T* enext, T* enneg, const ListStream& stream,
                               unsigned long long* totals, bool beside_epochs, cudaStream_t s) {
    if (nseg_ == 0) return epochs_;
    DevArray<int32_t>& list = list_[buffer];
    while (true) {
        UMAPB_CUDA(cudaEventSynchronize(sized_));
        const uint64_t total = *total_;
        bool fits = total / LIST_ALIGN <= UINT32_MAX;
        per_epoch_ = static_cast<double>(std::max<uint64_t>(total, 1)) / epochs_;
        // (more samples or firing edges than the window's length was chosen for)
        const double most = 1.125 * static_cast<double>(bytes);
        if (epochs_ > 1 && (epoch_bytes(per_epoch_) * epochs_ > most ||
                            (total > list.size() && full_grown(buffer, bytes)))) {
            prepare(first_, std::min(epochs_ - 1, window_epochs(buffer, bytes)), enext, enneg, beside_epochs, s);
            continue;
        }
        if (fits) {
            try {
                if (total > list.size()) list.allocate(list_room(total, most - epoch_bytes(0) * epochs_, !beside_epochs), s);
                span_[buffer].reserve(static_cast<size_t>(epochs_) * ep_->n, s);
                if (with_tasks_) tasks_[buffer].reserve(static_cast<size_t>(epochs_) * ep_->n, s);
            } catch (const Error& e) {
                release(buffer);
                if (e.code != UMAPB_ERR_OOM || epochs_ == 1) throw;
                fits = false;
            }
        }
        if (fits) break;
        require(epochs_ > 1, "the epoch's interactions do not fit 32-bit offsets", UMAPB_ERR_OVERFLOW);
        prepare(first_, epochs_ / 2, enext, enneg, beside_epochs, s);
    }
    GenArgs<T> g = gen_args(*ep_, seg_row_.get(), nseg_, first_, epochs_);
    g.enext = enext;
    g.enneg = enneg;
    g.base = base_.get();
    g.list = list.get();
    g.span = span_[buffer].get();
    g.stream = stream;
    g.totals = totals;
    for (uint32_t r = 0; r < 7; ++r) {
        g.key0[r] = stream.k0 + r * 0x9E3779B9u;
        g.key1[r] = stream.k1 + r * 0xBB67AE85u;
    }
    // Rows that fire nothing keep an empty span.  (Not cleared by the segments' warps: the
    // rows without edges between two others are all one segment's.)
    UMAPB_CUDA(cudaMemsetAsync(span_[buffer].get(), 0, sizeof(ListSpan) * static_cast<size_t>(epochs_) * ep_->n, s));
    schedule_kernel<T, true><<<gen_grid(nseg_, beside_epochs), GEN_WARPS * 32, 0, s>>>(g);
    UMAPB_LAUNCH_CHECK();
    return epochs_;
}

template class InteractionLists<float>;
template class InteractionLists<double>;

}  // namespace umapb
