// Device memory that outlives a call: one buffer per device and stream, grown to the largest call on it.
#pragma once

#include "attn_common.cuh"

#include <mutex>
#include <vector>

namespace hipgpt {

// While it lives the calling thread may allocate, free and create although some stream is being captured (in the strictest mode a
// capture forbids that to every thread, and one that tries ends the capture): for calls on streams outside the capture.
class OutsideCapture {
public:
    OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    ~OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode_); }
    OutsideCapture(const OutsideCapture &) = delete;
    OutsideCapture &operator=(const OutsideCapture &) = delete;
private:
    cudaStreamCaptureMode mode_ = cudaStreamCaptureModeRelaxed;
};

inline bool being_captured(cudaStream_t st)
{
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    return cudaStreamIsCapturing(st, &cap) == cudaSuccess && cap != cudaStreamCaptureStatusNone;
}

// A call takes the lock (enter), gets a buffer and enqueues every kernel that touches it before it lets the lock go, so calls
// of several threads on one stream do not interleave.  Streams are told apart by their unique id: a handle may be
// reused after its stream has been destroyed, and the per-thread default stream has one handle for all threads.  At
// most kMostEntries buffers are kept; the one that was used longest ago goes first (cudaFree waits for its readers).
// During stream capture a buffer of the graph's own is used instead (stream-ordered allocation and release become nodes of the
// graph), so that a replay never refers to memory that a later, larger call has given back.
class StreamWorkspace {
public:
    // A second stream of the library beside the caller's, and events for work that goes to and fro between the two
    struct Side {
        cudaStream_t stream = nullptr;
        cudaEvent_t entered = nullptr, done[2] = {nullptr, nullptr}, taken[2] = {nullptr, nullptr};
    };

    class Lease {
    public:
        Lease() = default;
        Lease(const Lease &) = delete;
        Lease &operator=(const Lease &) = delete;
        ~Lease() { if (captured_) cudaFreeAsync(ptr_, st_); }
        uint8_t *get() const { return static_cast<uint8_t *>(ptr_); }
        const Side &side() const { return side_; }
    private:
        friend class StreamWorkspace;
        std::unique_lock<std::mutex> lock_;
        void *ptr_ = nullptr;
        cudaStream_t st_ = nullptr;
        bool captured_ = false;
        Side side_;
    };

    // with_side: not for a stream that is being captured
    int enter(cudaStream_t st, size_t need, Lease *out, bool with_side = false)
    {
        out->lock_ = std::unique_lock<std::mutex>(mu_);
        out->st_ = st;
        cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
        cudaError_t e = cudaStreamIsCapturing(st, &cap);
        if (e == cudaSuccess && cap == cudaStreamCaptureStatusActive) {
            e = cudaMallocAsync(&out->ptr_, need, st);
            if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaMallocAsync(%zu) during capture: %s", need, cudaGetErrorString(e));
            out->captured_ = true;
            return HIPGPT_OK;
        }
        int dev = 0;
        unsigned long long id = 0;
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaStreamGetId(st, &id);
        if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "workspace: %s", cudaGetErrorString(e));
        Entry *mine = nullptr;
        for (Entry &x : entries_) if (x.dev == dev && x.id == id) mine = &x;
        if (!mine) {
            const OutsideCapture outside;
            if (entries_.size() >= kMostEntries) {
                size_t oldest = 0;
                for (size_t i = 1; i < entries_.size(); ++i) if (entries_[i].used < entries_[oldest].used) oldest = i;
                give_back(entries_[oldest]);
                entries_.erase(entries_.begin() + (long)oldest);
            }
            entries_.push_back({dev, id, 0, nullptr, 0, {}});
            mine = &entries_.back();
        }
        mine->used = ++clock_;
        if (mine->cap < need) {
            const OutsideCapture outside;
            if (mine->buf) cudaFree(mine->buf);
            mine->buf = nullptr;
            mine->cap = 0;
            e = cudaMalloc(&mine->buf, need);
            if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "cudaMalloc(%zu): %s", need, cudaGetErrorString(e));
            mine->cap = need;
        }
        if (with_side) {
            e = make_side(mine->side);
            if (e != cudaSuccess) return fail(HIPGPT_ERR_CUDA, "second stream of a workspace: %s", cudaGetErrorString(e));
            out->side_ = mine->side;
        }
        out->ptr_ = mine->buf;
        return HIPGPT_OK;
    }

    void release()
    {
        std::lock_guard<std::mutex> lock(mu_);
        const OutsideCapture outside;
        for (Entry &x : entries_) give_back(x);
        entries_.clear();
    }

private:
    static constexpr size_t kMostEntries = 8;
    struct Entry { int dev; unsigned long long id, used; void *buf; size_t cap; Side side; };

    static cudaError_t make_side(Side &s)
    {
        if (s.taken[1]) return cudaSuccess;          // (the last to be made)
        const OutsideCapture outside;
        cudaError_t e = s.stream ? cudaSuccess : cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking);
        for (cudaEvent_t *ev : {&s.entered, &s.done[0], &s.done[1], &s.taken[0], &s.taken[1]})
            if (e == cudaSuccess && !*ev) e = cudaEventCreateWithFlags(ev, cudaEventDisableTiming);
        return e;
    }
    static void give_back(Entry &x)
    {
        int dev = x.dev;                             // an entry of another device is freed, and waited for, there
        cudaGetDevice(&dev);
        if (dev != x.dev) cudaSetDevice(x.dev);
        if (x.buf) cudaFree(x.buf);
        if (x.side.stream) cudaStreamDestroy(x.side.stream);
        for (cudaEvent_t ev : {x.side.entered, x.side.done[0], x.side.done[1], x.side.taken[0], x.side.taken[1]})
            if (ev) cudaEventDestroy(ev);
        if (dev != x.dev) cudaSetDevice(dev);
    }

    std::mutex mu_;
    unsigned long long clock_ = 0;
    std::vector<Entry> entries_;
};

}  // namespace hipgpt
