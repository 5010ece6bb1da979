// The epochs' work as flat lists (sgd_lists.cu): for every epoch of a window
// and every row, the points its head meets in the order of
// include/umappp/optimize_layout.hpp:136-180 -- a firing edge's target, marked
// by LIST_ATTRACT, then that edge's negative samples, edge after edge.
#pragma once

#include "common.cuh"

namespace umapb {

template <typename T>
struct DeviceEpochs;   // stages.cuh

constexpr int MAX_WINDOW = 32;                    // epochs per window: one lane keeps one epoch's position
constexpr int32_t LIST_ATTRACT = INT32_MIN;       // sign bit of an entry: a firing edge's target
constexpr int LIST_ALIGN = 8;                     // a row's entries of an epoch start at a multiple of this

// Entries of one row in one epoch: [start8 * LIST_ALIGN, end) of the window's
// list, 'end' kept modulo 2^32 (the count is the difference modulo 2^32).
struct ListSpan {
    uint32_t start8, end;
};

// One row of an epoch in claim order: 'count' entries from
// list[start8 * LIST_ALIGN].
struct alignas(16) RowTask {
    int32_t row;
    uint32_t start8, count;
    uint32_t unused;
};

// What the lists depend on besides the schedule itself.
struct ListStream {
    uint32_t k0, k1;               // Philox key of the negative samples
    int32_t head0 = 0;             // added to the row to give the stream's head counter
    int32_t n = 0;                 // negative samples are drawn from [0, n), or
    const int32_t* inst_start = nullptr;   // from the row's instance (num_inst + 1 boundaries)
    int32_t num_inst = 1;
};

// Builds the lists of consecutive windows of epochs and advances the schedule
// state: prepare() sizes a window, build() writes it into one of two buffers,
// so that a window's epochs can run (on another stream) while the next one is
// built.  All work is enqueued on the stream that is passed; a buffer is built
// into again only after what the stream has been made to wait for.
template <typename T>
class InteractionLists {
public:
    // with_tasks: the buffers also have room for the epochs' row tasks.
    void setup(const DeviceEpochs<T>* ep, bool with_tasks, cudaStream_t s);
    // Enqueues the sizing of the window [first, first + epochs) from the state
    // (enext, enneg) at 'first', which stays as it is.  beside_epochs: epochs
    // run on another stream meanwhile, so the launch leaves them room.  Fewer
    // epochs are sized where the device has no memory for more.
    void prepare(int first, int epochs, const T* enext, const T* enneg, bool beside_epochs, cudaStream_t s);
    // Waits for prepare(), then enqueues the window's lists (into 'buffer') and
    // the state at its end.  A window of several epochs is shortened and sized
    // again where it would take more than an eighth above 'bytes', or does not
    // fit the device.  totals (optional, 2 per epoch from the window's first):
    // [firing edges, negative samples].  Returns the epochs built.
    int build(int buffer, size_t bytes, T* enext, T* enneg, const ListStream& stream, unsigned long long* totals,
              bool beside_epochs, cudaStream_t s);
    // Epochs of a window that takes 'buffer' up to 'bytes', by the last window built.
    int window_epochs(int buffer, size_t bytes) const;
    const int32_t* list(int buffer) const { return list_[buffer].get(); }
    // Gives a buffer, or all memory, back to the workspace cache; prepare() and build() take it anew.
    void release(int buffer);
    void release();
    RowTask* tasks(int buffer) const { return tasks_[buffer].get(); }   // [epoch of the window][position]
    const ListSpan* spans(int buffer) const { return span_[buffer].get(); }   // [epoch of the window][row]
    InteractionLists() = default;
    InteractionLists(const InteractionLists&) = delete;
    InteractionLists& operator=(const InteractionLists&) = delete;
    ~InteractionLists();

private:
    const DeviceEpochs<T>* ep_ = nullptr;
    int64_t nseg_ = 0;
    int first_ = 0, epochs_ = 0;
    double per_epoch_ = 0;         // entries of an epoch of the last window
    double epoch_bytes(double entries) const;
    // A buffer that holds half of the bytes it may take is not grown for the next window: that is shortened.
    bool full_grown(int buffer, size_t bytes) const { return 8.0 * list_[buffer].size() >= static_cast<double>(bytes); }
    DevArray<int32_t> seg_row_;    // first row of each segment, nseg + 1
    DevArray<uint64_t> cap_, base_;
    DevArray<unsigned char> temp_;
    DevArray<int32_t> list_[2];
    DevArray<ListSpan> span_[2];
    DevArray<RowTask> tasks_[2];
    bool with_tasks_ = false;
    uint64_t* total_ = nullptr;    // pinned host word
    cudaEvent_t sized_ = nullptr;
};

}  // namespace umapb
