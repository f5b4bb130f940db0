// hostcopy.h -- copies between pageable host memory and the device.
//
// cudaMemcpyAsync on pageable memory goes through the driver's own staging
// buffer on the calling thread, one copy at a time: a 768^2 x 800 host-buffer
// call (17.5 MB up, 9.4 MB down) spent 1.5 of its 2.1 ms there.  HostStager
// takes the pieces through page-locked slots of its own, filled and emptied by
// a few threads, so that host copies, transfers and kernels overlap:
// 1.2 ms.  Page-locked and managed buffers are copied directly.
#pragma once

#include <cuda_runtime.h>
#include <sys/types.h>

#include <cstddef>

namespace sarbp {

// Threads that share one memcpy at a time with the caller.  They start with
// the first copy of several pieces, spin for the next copy for a short while
// and then sleep.
class CopyThreads {
public:
    CopyThreads() = default;
    CopyThreads(const CopyThreads &) = delete;
    ~CopyThreads();
    void copy(char *dst, const char *src, size_t n);
    void zero(char *dst, size_t n, size_t piece);  // a piece to a thread
    // No copy follows soon: spinning threads sleep at once.
    void rest();

private:
    // Threads, lock and condition variable of the process that started them.
    // A forked child has none of the threads, and the lock and the condition
    // variable as the fork found them, so there it is left alone and never
    // freed, and the caller copies by itself.
    struct State;
    State *state();
    void run(char *dst, const char *src, size_t n, size_t piece);
    State *s_ = nullptr;
    pid_t pid_ = 0;
    bool tried_ = false;
};

class HostStager {
public:
    // Whether staging pays for a copy of n bytes at p (pageable, not small).
    static bool wants(const void *p, size_t n);
    // One session per host-buffer call; its end drops what a failed call left
    // in the slots and lets the threads sleep.
    class Session {
    public:
        explicit Session(HostStager *s) : s_(s) {}
        ~Session() {
            s_->abandon();
            s_->threads_.rest();
        }
        Session(const Session &) = delete;

    private:
        HostStager *s_;
    };
    // dst (device) <- src (host) on st; src has been read when this returns.
    cudaError_t upload(void *dst, const void *src, size_t n, cudaStream_t st);
    // dst (host) <- src (device) behind what st holds; complete after drain().
    // Both copy directly where no page-locked memory is to be had.
    cudaError_t download(void *dst, const void *src, size_t n, cudaStream_t st);
    cudaError_t drain();
    // Waits for the copies in flight and frees the slots.
    void release();

private:
    static constexpr size_t kSlotBytes = 2 << 20;
    static constexpr int kSlots = 8;  // 16 MB, from the first staged copy to the context's end
    struct Slot {
        cudaEvent_t ev = nullptr;
        bool busy = false;
        char *out = nullptr;  // destination of a download still in the slot
        size_t n = 0;
    };
    bool ready();
    cudaError_t acquire(int *slot);
    cudaError_t settle(Slot &s, int i);
    void abandon();  // drops downloads that a failed call left behind
    CopyThreads threads_;
    char *pin_ = nullptr;
    pid_t pid_ = 0;        // the process that locked the slots
    void *map_ = nullptr;  // the mapping that holds pin_
    size_t map_bytes_ = 0;
    Slot slots_[kSlots];
    int next_ = 0;
};

}  // namespace sarbp
