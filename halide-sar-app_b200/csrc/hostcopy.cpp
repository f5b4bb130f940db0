// hostcopy.cpp -- see hostcopy.h.
#include "hostcopy.h"

#include <sys/mman.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace sarbp {

namespace {
constexpr size_t kPiece = 128 << 10;
// How long a thread spins for the next copy before it sleeps: longer than the
// pauses between the copies of one call (768^2 x 800: 1.35 ms a call with 100
// us, 1.16 with 300 and with 1000), short against a call that computes for
// long.
constexpr std::chrono::microseconds kSpin(500);

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

struct CopyThreads::State {
    std::vector<std::thread> threads;
    std::mutex mu;
    std::condition_variable cv;
    bool stop = false;
    std::atomic<int> sleeping{0};
    std::atomic<bool> active{false};  // copies follow one another: spin for the next
    // the copy in hand: generation in the high half, next piece in the low one
    std::atomic<unsigned long long> next{0};
    std::atomic<unsigned> left{0};  // pieces not yet done
    std::atomic<unsigned> npieces{0};
    char *dst = nullptr;
    const char *src = nullptr;  // null: zeros
    size_t n = 0, piece = 0;
    unsigned gen = 0;

    bool available() const { return (unsigned)next.load() < npieces.load(); }

    // Takes and copies pieces until none is left.  A copy that has begun
    // meanwhile fails the exchange, so dst, src and n are those of the piece's
    // copy until its last piece is done.
    void take() {
        for (;;) {
            unsigned long long v = next.load(std::memory_order_acquire);
            const unsigned i = (unsigned)v;
            if (i >= npieces.load(std::memory_order_acquire)) return;
            if (!next.compare_exchange_weak(v, v + 1, std::memory_order_acq_rel)) continue;
            const size_t o = (size_t)i * piece, m = std::min(piece, n - o);
            if (src)
                std::memcpy(dst + o, src + o, m);
            else
                std::memset(dst + o, 0, m);
            left.fetch_sub(1, std::memory_order_release);
        }
    }

    void work() {
        for (;;) {
            take();
            const auto t0 = std::chrono::steady_clock::now();
            bool spin = true;
            for (int k = 0; spin && !available(); k += k < 4096) {
                relax(k);
                spin = active.load(std::memory_order_relaxed) &&
                       ((k & 63) || k == 0 || std::chrono::steady_clock::now() - t0 < kSpin);
            }
            if (spin) continue;
            std::unique_lock<std::mutex> lk(mu);
            sleeping.fetch_add(1);
            cv.wait(lk, [&] { return stop || available(); });
            sleeping.fetch_sub(1);
            if (stop) return;
        }
    }
};

CopyThreads::~CopyThreads() {
    if (!s_ || pid_ != getpid()) return;
    {
        std::lock_guard<std::mutex> lk(s_->mu);
        s_->stop = true;
        s_->active.store(false);
    }
    s_->cv.notify_all();
    for (std::thread &t : s_->threads) t.join();
    delete s_;
}

// The threads' state, or null where the caller copies alone.
CopyThreads::State *CopyThreads::state() {
    if (!tried_) {
        tried_ = true;
        // half of the cores at most, the caller among them (16 cores: 1.33 ms with 3
        // helpers, 1.23 with 5, 1.18 with 7)
        const int n = std::min(7, (int)std::thread::hardware_concurrency() / 2 - 1);
        if (n < 1 || !(s_ = new (std::nothrow) State)) return nullptr;
        pid_ = getpid();
        try {
            for (int i = 0; i < n; ++i) s_->threads.emplace_back(&State::work, s_);
        } catch (...) {  // no more threads: fewer share the copies
        }
    }
    return s_ && pid_ == getpid() && !s_->threads.empty() ? s_ : nullptr;
}

void CopyThreads::rest() {
    if (s_ && pid_ == getpid()) s_->active.store(false);
}

void CopyThreads::copy(char *dst, const char *src, size_t n) { run(dst, src, n, kPiece); }

void CopyThreads::zero(char *dst, size_t n, size_t piece) { run(dst, nullptr, n, piece); }

void CopyThreads::run(char *dst, const char *src, size_t n, size_t piece) {
    const size_t pieces = (n + piece - 1) / piece;
    State *s = pieces < 2 ? nullptr : state();
    if (!s) {
        if (src)
            std::memcpy(dst, src, n);
        else
            std::memset(dst, 0, n);
        return;
    }
    s->active.store(true);
    // no thread holds a piece here: the copy before ended with left == 0
    s->left.store((unsigned)pieces, std::memory_order_relaxed);
    ++s->gen;
    s->next.store((unsigned long long)s->gen << 32 | 0xffffffffull);  // none yet
    s->dst = dst;
    s->src = src;
    s->n = n;
    s->piece = piece;
    s->npieces.store((unsigned)pieces);
    s->next.store((unsigned long long)s->gen << 32);
    // a thread counts itself as sleeping before it looks for pieces a last time
    if (s->sleeping.load() > 0) {
        { std::lock_guard<std::mutex> lk(s->mu); }
        s->cv.notify_all();
    }
    s->take();
    for (int k = 0; s->left.load(std::memory_order_acquire) != 0; k += k < 4096) relax(k);
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

// The slots; false where there is no page-locked memory to be had (and in a
// forked child, which has no mapping of them).  A
// context's first call waits for the locking of 16 MB, so they are mapped in
// huge pages where the system has them and the threads touch the pages ahead
// of it: 1.2 ms, against 2.9 without the threads and 8 with cudaMallocHost
// (the first 768^2 x 800 call of a context 6 ms, as with the driver's own
// staging, against 8 and 20).
bool HostStager::ready() {
    if (pin_) return pid_ == getpid();
    constexpr size_t kHuge = 2 << 20, kBytes = kSlotBytes * kSlots;
    void *p = mmap(nullptr, kBytes + kHuge, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    if (p == MAP_FAILED) return false;
    char *at = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(p) + kHuge - 1) / kHuge * kHuge);
    madvise(at, kBytes, MADV_HUGEPAGE);
    // A fork would make the pages copies-on-write: the caller's next write to a
    // slot could go to a new page, the device's transfer to the old one.
    if (madvise(at, kBytes, MADV_DONTFORK) != 0) {
        munmap(p, kBytes + kHuge);
        return false;
    }
    threads_.zero(at, kBytes, kHuge);  // a page a thread, ahead of the locking
    if (cudaHostRegister(at, kBytes, cudaHostRegisterPortable) != cudaSuccess) {
        cudaGetLastError();
        munmap(p, kBytes + kHuge);
        return false;
    }
    pid_ = getpid();
    map_ = p;
    map_bytes_ = kBytes + kHuge;
    pin_ = at;
    return true;
}

cudaError_t HostStager::acquire(int *slot) {
    cudaError_t e = cudaSuccess;
    Slot &s = slots_[next_];
    if (!s.ev && (e = cudaEventCreateWithFlags(&s.ev, cudaEventDisableTiming)) != cudaSuccess) return e;
    if ((e = settle(s, next_)) != cudaSuccess) return e;
    *slot = next_;
    next_ = (next_ + 1) % kSlots;
    return cudaSuccess;
}

cudaError_t HostStager::upload(void *dst, const void *src, size_t n, cudaStream_t st) {
    if (!ready()) return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
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
    if (!ready()) return cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st);
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
    if (pin_ && pid_ == getpid()) {  // (a child may have other things mapped there)
        cudaHostUnregister(pin_);
        munmap(map_, map_bytes_);
    }
    pin_ = nullptr;
}

}  // namespace sarbp
