// hostcopy.cpp -- see hostcopy.h.
#include "hostcopy.h"

#include <unistd.h>

#include <algorithm>
#include <cstdint>
#include <cstring>

namespace sarbp {

namespace {
// One turn of a wait: a pause at first, then the core goes to whoever else
// wants it (other contexts' threads, or a copying thread that lost its core).
inline void relax(int turn) {
    if (turn >= 4096) {
        std::this_thread::yield();
        return;
    }
#if defined(__x86_64__)
    __builtin_ia32_pause();
#endif
}
}  // namespace

CopyThreads::~CopyThreads() {
    if (started_ && pid_ != getpid()) {  // a forked child has no such threads to join
        new std::vector<std::thread>(std::move(threads_));
        return;
    }
    {
        std::lock_guard<std::mutex> lk(mu_);
        stop_ = true;
        session_.store(false);
    }
    cv_.notify_all();
    for (std::thread &t : threads_) t.join();
}

void CopyThreads::begin() {
    if (!started_) {
        started_ = true;
        pid_ = getpid();
        // half of the cores at most, the caller among them (16 cores: 1.33 ms with 3
        // helpers, 1.23 with 5, 1.18 with 7)
        const int n = std::min(7, (int)std::thread::hardware_concurrency() / 2 - 1);
        for (int i = 0; i < n; ++i) {
            try {
                threads_.emplace_back(&CopyThreads::work, this);
            } catch (...) {  // no more threads: fewer share the copies
                break;
            }
        }
    }
    if (threads_.empty()) return;
    {
        std::lock_guard<std::mutex> lk(mu_);
        session_.store(true);
    }
    cv_.notify_all();
}

void CopyThreads::end() {
    if (!threads_.empty()) session_.store(false);
}

// Takes and copies pieces of generation gen until none is left.
bool CopyThreads::take(unsigned gen) {
    bool any = false;
    for (;;) {
        unsigned long long v = next_.load(std::memory_order_acquire);
        if ((unsigned)(v >> 32) != gen) return any;
        const unsigned i = (unsigned)v;
        if (i >= npieces_.load(std::memory_order_acquire)) return any;
        // (a changed generation fails the exchange, so dst_, src_ and n_ are
        // those of this copy until its last piece is done)
        if (!next_.compare_exchange_weak(v, v + 1, std::memory_order_acq_rel)) continue;
        const size_t o = (size_t)i * kPiece;
        std::memcpy(dst_ + o, src_ + o, std::min(kPiece, n_ - o));
        left_.fetch_sub(1, std::memory_order_release);
        any = true;
    }
}

void CopyThreads::work() {
    for (;;) {
        {
            std::unique_lock<std::mutex> lk(mu_);
            cv_.wait(lk, [&] { return stop_ || session_.load(); });
            if (stop_) return;
        }
        int idle = 0;
        while (session_.load(std::memory_order_relaxed)) {
            if (take((unsigned)(next_.load(std::memory_order_acquire) >> 32))) idle = 0;
            for (int k = 0; k < 32 && idle < 4096; ++k) relax(idle++);
            if (idle >= 4096) relax(idle);
        }
    }
}

void CopyThreads::copy(char *dst, const char *src, size_t n) {
    const size_t pieces = (n + kPiece - 1) / kPiece;
    if (threads_.empty() || pieces < 2) {
        std::memcpy(dst, src, n);
        return;
    }
    // no thread holds a piece here: the copy before ended with left_ == 0, and a
    // thread that still looks at its generation finds no piece left
    dst_ = dst;
    src_ = src;
    n_ = n;
    left_.store((unsigned)pieces, std::memory_order_relaxed);
    ++gen_;
    next_.store((unsigned long long)gen_ << 32 | 0xffffffffull, std::memory_order_relaxed);  // none yet
    npieces_.store((unsigned)pieces, std::memory_order_release);
    next_.store((unsigned long long)gen_ << 32, std::memory_order_release);
    take(gen_);
    for (int k = 0; left_.load(std::memory_order_acquire) != 0; k += k < 4096) relax(k);
}

bool HostStager::wants(const void *p, size_t n) {
    if (!p || n < (256 << 10)) return false;
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Makes slot i free: a download in it goes to its destination.
cudaError_t HostStager::settle(Slot &s, int i) {
    if (!s.busy) return cudaSuccess;
    cudaError_t e = cudaEventSynchronize(s.ev);
    if (e != cudaSuccess) return e;
    if (s.out) threads_.copy(s.out, pin_ + (size_t)i * kSlotBytes, s.n);
    s.out = nullptr;
    s.busy = false;
    return cudaSuccess;
}

cudaError_t HostStager::acquire(int *slot) {
    cudaError_t e = cudaSuccess;
    if (!pin_) {
        void *p = nullptr;
        if ((e = cudaMallocHost(&p, kSlotBytes * kSlots)) != cudaSuccess) return e;
        pin_ = static_cast<char *>(p);
    }
    Slot &s = slots_[next_];
    if (!s.ev && (e = cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = settle(s, next_)) != cudaSuccess) return e;
    *slot = next_;
    next_ = (next_ + 1) % kSlots;
    return cudaSuccess;
}

cudaError_t HostStager::upload(void *dst, const void *src, size_t n, cudaStream_t st) {
    for (size_t o = 0; o < n; o += kSlotBytes) {
        const size_t m = std::min(kSlotBytes, n - o);
        int i = 0;
        cudaError_t e = acquire(&i);
        if (e != cudaSuccess) return e;
        char *pin = pin_ + (size_t)i * kSlotBytes;
        threads_.copy(pin, static_cast<const char *>(src) + o, m);
        e = cudaMemcpyAsync(static_cast<char *>(dst) + o, pin, m, cudaMemcpyHostToDevice, st);
        if (e == cudaSuccess) e = cudaEventRecord(slots_[i].ev, st);
        if (e != cudaSuccess) return e;
        slots_[i].busy = true;
    }
    return cudaSuccess;
}

cudaError_t HostStager::download(void *dst, const void *src, size_t n, cudaStream_t st) {
    for (size_t o = 0; o < n; o += kSlotBytes) {
        const size_t m = std::min(kSlotBytes, n - o);
        int i = 0;
        cudaError_t e = acquire(&i);
        if (e != cudaSuccess) return e;
        e = cudaMemcpyAsync(pin_ + (size_t)i * kSlotBytes, static_cast<const char *>(src) + o, m,
                            cudaMemcpyDeviceToHost, st);
        if (e == cudaSuccess) e = cudaEventRecord(slots_[i].ev, st);
        if (e != cudaSuccess) return e;
        slots_[i].busy = true;
        slots_[i].out = static_cast<char *>(dst) + o;
        slots_[i].n = m;
    }
    return cudaSuccess;
}

cudaError_t HostStager::drain() {
    for (int k = 0; k < kSlots; ++k) {
        const int i = (next_ + k) % kSlots;  // oldest first
        if (!slots_[i].out) continue;        // uploads wait for their slot's next use
        cudaError_t e = settle(slots_[i], i);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void HostStager::abandon() {
    for (Slot &s : slots_) {
        if (!s.out) continue;
        cudaEventSynchronize(s.ev);
        s.out = nullptr;
        s.busy = false;
    }
}

void HostStager::release() {
    for (Slot &s : slots_) {
        if (s.busy) cudaEventSynchronize(s.ev);
        if (s.ev) cudaEventDestroy(s.ev);
        s = Slot{};
    }
    if (pin_) cudaFreeHost(pin_);
    pin_ = nullptr;
}

}  // namespace sarbp
