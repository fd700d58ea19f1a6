// hsr_scratch.h -- device scratch of the entry points that keep no plan (the
// Hessenberg reduction, its back-transform, the residuals).
#pragma once

#include <cuda_runtime.h>

namespace hsr {

// One growing device buffer of a host thread for one entry point.  A call holds
// it by a ScratchUse from before its first launch until after its last one.
//
// Outside a stream capture every call waits for the last one by an event, also
// on what looks like the same stream: a new stream can have the handle of one
// that was destroyed with its work still running (on the same stream the wait
// costs nothing on the device).  Inside one, a call gets memory that belongs to the graph (an
// allocation and a free node): the thread's buffer, which a later call may
// replace and the thread's end frees, never enters a graph, and replays need no
// order against direct calls.
//
// A thread's buffers keep their largest size until release_all
// (hsr_release_workspace) or its end.
struct Scratch {
    int device = -1;
    void *p = nullptr;
    size_t bytes = 0;
    cudaEvent_t ev = nullptr;
    bool used = false;
    Scratch *next;                                               // the thread's others
    static Scratch *&first() {
        static thread_local Scratch *f = nullptr;
        return f;
    }
    Scratch() : next(first()) { first() = this; }
    ~Scratch() {
        for (Scratch **s = &first(); *s; s = &(*s)->next)
            if (*s == this) {
                *s = next;
                break;
            }
        release();
    }
    Scratch(const Scratch &) = delete;
    Scratch &operator=(const Scratch &) = delete;
    static void release_all() {
        for (Scratch *s = first(); s; s = s->next) s->release();
    }
    void release() {
        if (p) cudaFree(p);
        if (ev) cudaEventDestroy(ev);
        p = nullptr;
        ev = nullptr;
        bytes = 0;
        used = false;
    }
};

class ScratchUse {
  public:
    // At least `want` bytes if they can be had, else at least `least`.
    ScratchUse(Scratch &s, size_t want, size_t least, int dev, cudaStream_t st) : s_(s), st_(st) {
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) {
            cudaGetLastError();
            return;
        }
        captured_ = cs != cudaStreamCaptureStatusNone;
        for (const size_t b : {want, least}) {
            if (captured_ ? cudaMallocAsync(&p_, b, st) == cudaSuccess : grow(b, dev)) {
                bytes_ = b;
                break;
            }
            cudaGetLastError();
            p_ = nullptr;
            if (want == least) break;
        }
        if (p_ && !captured_ && s.used && cudaStreamWaitEvent(st, s.ev, 0) != cudaSuccess) p_ = nullptr;
    }
    ~ScratchUse() {
        if (!p_) return;
        if (captured_) {
            cudaFreeAsync(p_, st_);
        } else if (cudaEventRecord(s_.ev, st_) == cudaSuccess) {
            s_.used = true;
        }
    }
    ScratchUse(const ScratchUse &) = delete;
    ScratchUse &operator=(const ScratchUse &) = delete;
    explicit operator bool() const { return p_ != nullptr; }
    size_t bytes() const { return bytes_; }                      // what was asked for and is there
    unsigned char *get() const { return static_cast<unsigned char *>(p_); }

  private:
    bool grow(size_t b, int dev) {
        if (s_.device != dev || b > s_.bytes) {
            s_.release();
            s_.device = dev;
            if (cudaMalloc(&s_.p, b) != cudaSuccess ||
                cudaEventCreateWithFlags(&s_.ev, cudaEventDisableTiming) != cudaSuccess) {
                s_.release();
                return false;
            }
            s_.bytes = b;
        }
        p_ = s_.p;
        return true;
    }
    Scratch &s_;
    cudaStream_t st_;
    void *p_ = nullptr;
    size_t bytes_ = 0;
    bool captured_ = false;
};

}  // namespace hsr
