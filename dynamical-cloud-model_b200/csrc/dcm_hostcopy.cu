// dcm_hostcopy.cu -- see dcm_hostcopy.h.
#include "dcm_hostcopy.h"

#include <emmintrin.h>
#include <sched.h>
#include <unistd.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <new>
#include <thread>
#include <vector>

namespace dcm {
namespace {

constexpr int NBUF = 4;
constexpr size_t CHUNK = 4u << 20;
constexpr size_t SLICE = 256u << 10;
static_assert(CHUNK % SLICE == 0, "a slice lies in one chunk");
// shorter transfers are as fast through the driver
constexpr size_t MIN_BYTES = 2u << 20;

// A thread that finds nothing to do looks again for this long, then sleeps: a
// chunk's DMA takes 80 us, so in a running transfer nobody sleeps, but a
// download queued behind a kernel of milliseconds costs no core.
constexpr std::chrono::microseconds LOOK{300};

// the processors this process may run on
int processors() {
    cpu_set_t set;
    return sched_getaffinity(0, sizeof set, &set) == 0 ? CPU_COUNT(&set)
                                                       : (int)std::thread::hardware_concurrency();
}

class Patience {
public:
    bool over() {
        if (over_ || ++n_ % 64) return over_;
        const auto now = std::chrono::steady_clock::now();
        if (n_ == 64) until_ = now + LOOK;
        return over_ = now >= until_;
    }
    void reset() {
        n_ = 0;
        over_ = false;
    }

private:
    unsigned n_ = 0;
    bool over_ = false;
    std::chrono::steady_clock::time_point until_;
};

// between two looks at an event, then (events that a thread can sleep on cost an
// interrupt each: 69 MB went 3 % slower)
void doze() { std::this_thread::sleep_for(std::chrono::microseconds(50)); }

// pageable: the driver knows nothing about the address
bool pageable(const void* p) {
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
        cudaGetLastError();
        return true;
    }
    return a.type == cudaMemoryTypeUnregistered;
}

// Into a page-locked buffer, past the caches: the DMA that follows reads lines
// that are dirty in several cores' caches at a fraction of memory's rate.
void stream_copy(char* dst, const char* src, size_t n) {
    size_t o = 0;
    for (; o + 64 <= n; o += 64) {
        const __m128i a = _mm_loadu_si128((const __m128i*)(src + o)),
                      b = _mm_loadu_si128((const __m128i*)(src + o + 16)),
                      c = _mm_loadu_si128((const __m128i*)(src + o + 32)),
                      e = _mm_loadu_si128((const __m128i*)(src + o + 48));
        _mm_stream_si128((__m128i*)(dst + o), a);
        _mm_stream_si128((__m128i*)(dst + o + 16), b);
        _mm_stream_si128((__m128i*)(dst + o + 32), c);
        _mm_stream_si128((__m128i*)(dst + o + 48), e);
    }
    if (o < n) std::memcpy(dst + o, src + o, n - o);
    _mm_sfence();
}

// One transfer at a time.  The buffers hold the transfer's chunks in turn; a
// chunk is copied in slices, which the calling thread and the others take from
// one counter, so that the caller starts at once and the others help from when
// they have woken (up to a millisecond on an idle host).
class Copier {
public:
    // false in a child process, which has the object but none of its threads
    bool here() const { return owner_ == getpid(); }
    // false when the page-locked buffers cannot be had
    bool start() {
        if (started_) return true;
        for (char*& p : pin_)
            if (cudaHostAlloc(&p, CHUNK, cudaHostAllocPortable) != cudaSuccess) {
                cudaGetLastError();
                free_buffers();
                return false;
            }
        const int cpus = processors();
        try {
            for (int t = 1; t < std::min(8, cpus / 2); t++) threads_.emplace_back([this] { work(); });
        } catch (...) {  // fewer threads than asked for
        }
        started_ = true;
        return true;
    }
    ~Copier() {
        {
            std::lock_guard<std::mutex> l(m_);
            quit_ = true;
        }
        cv_.notify_all();
        for (std::thread& t : threads_) t.join();
        free_buffers();
    }

    cudaError_t transfer(char* dev, char* host, size_t n, bool down, cudaStream_t st) {
        cudaEvent_t ev[NBUF] = {};
        cudaError_t e = cudaSuccess;
        for (int q = 0; q < NBUF && e == cudaSuccess; q++)
            e = cudaEventCreateWithFlags(&ev[q], cudaEventDisableTiming);
        const long nch = (long)((n + CHUNK - 1) / CHUNK);
        auto bytes = [&](long c) { return std::min(CHUNK, n - (size_t)c * CHUNK); };
        auto slices = [&](long c) { return (long)((bytes(c) + SLICE - 1) / SLICE); };
        // the DMA of chunk c, from or to its buffer
        auto dma = [&](long c) {
            char *d = dev + (size_t)c * CHUNK, *p = pin_[c % NBUF];
            const cudaError_t r = down ? cudaMemcpyAsync(p, d, bytes(c), cudaMemcpyDeviceToHost, st)
                                       : cudaMemcpyAsync(d, p, bytes(c), cudaMemcpyHostToDevice, st);
            return r == cudaSuccess ? cudaEventRecord(ev[c % NBUF], st) : r;
        };
        host_ = host;
        n_ = n;
        down_ = down;
        base_ = open_.load(std::memory_order_relaxed);
        wake(true);  // the threads take a while to come
        if (down)
            for (long c = 0; c < std::min<long>(NBUF, nch) && e == cudaSuccess; c++) e = dma(c);
        long opened = 0, copied = 0;
        Patience patience;
        while (e == cudaSuccess && copied < nch) {
            // open the next chunk once its buffer's last DMA is done
            if (opened < nch && opened < copied + NBUF) {
                const bool wait = down || opened >= NBUF;
                cudaError_t r = wait ? cudaEventQuery(ev[opened % NBUF]) : cudaSuccess;
                // nothing else left to do for a while
                if (r == cudaErrorNotReady && copied == opened && patience.over()) doze();
                if (r == cudaSuccess) {
                    done_[opened % NBUF].store(0, std::memory_order_relaxed);
                    open_.fetch_add(slices(opened), std::memory_order_seq_cst);
                    opened++;
                    patience.reset();
                    if (asleep_.load(std::memory_order_seq_cst)) wake(true);
                    continue;
                }
                if (r != cudaErrorNotReady) e = r;
            }
            if (take()) {
                patience.reset();
                continue;
            }
            if (copied < opened &&
                done_[copied % NBUF].load(std::memory_order_acquire) == slices(copied)) {
                if (!down)
                    e = dma(copied);
                else if (copied + NBUF < nch)
                    e = dma(copied + NBUF);
                copied++;
            }
        }
        // every slice that was opened is copied before the arrays are let go
        for (; copied < opened; copied++)
            while (done_[copied % NBUF].load(std::memory_order_acquire) < slices(copied))
                if (!take()) std::this_thread::yield();
        wake(false);
        // the buffers are free for the next transfer, on any stream
        for (cudaEvent_t x : ev) {
            if (!x) continue;
            cudaError_t r;
            for (Patience look; (r = cudaEventQuery(x)) == cudaErrorNotReady;)
                if (look.over()) doze();
            if (e == cudaSuccess) e = r;
            cudaEventDestroy(x);
        }
        if (e == cudaErrorNotReady) e = cudaErrorUnknown;  // never "not taken"
        cudaGetLastError();  // the queries' "not ready"
        return e;
    }

private:
    // copies one open slice; false when there is none.  Slices are numbered
    // over all transfers, so that a thread that is late from one transfer
    // cannot mistake the next one's counter for open work.
    bool take() {
        long s = next_.load(std::memory_order_relaxed);
        do {
            if (s >= open_.load(std::memory_order_acquire)) return false;
        } while (!next_.compare_exchange_weak(s, s + 1, std::memory_order_acq_rel));
        const size_t o = (size_t)(s - base_) * SLICE, n = std::min(SLICE, n_ - o);
        const int buf = (int)(o / CHUNK % NBUF);
        char *p = pin_[buf] + o % CHUNK, *h = host_ + o;
        if (down_)
            std::memcpy(h, p, n);
        else
            stream_copy(p, h, n);
        done_[buf].fetch_add(1, std::memory_order_release);
        return true;
    }
    // a transfer is on (or over), for the threads that look and those that sleep
    void wake(bool on) {
        {
            std::lock_guard<std::mutex> l(m_);
            active_.store(on, std::memory_order_release);
            job_++;
        }
        if (on) cv_.notify_all();
    }
    void work() {
        unsigned long seen = 0;
        bool bored = false;  // found nothing for a while in a transfer that goes on
        for (;;) {
            {
                std::unique_lock<std::mutex> l(m_);
                // open work is looked for after asleep_ is set, and the opener
                // looks at asleep_ after opening: one of them sees the other
                if (bored) asleep_.fetch_add(1, std::memory_order_seq_cst);
                cv_.wait(l, [&] {
                    return quit_ || (job_ != seen && active_.load(std::memory_order_relaxed)) ||
                           next_.load(std::memory_order_relaxed) <
                               open_.load(std::memory_order_seq_cst);
                });
                if (bored) asleep_.fetch_sub(1, std::memory_order_seq_cst);
                if (quit_) return;
                seen = job_;
            }
            bored = false;
            for (Patience look; !bored && active_.load(std::memory_order_acquire);) {
                if (take()) {
                    look.reset();
                } else {
                    std::this_thread::yield();
                    bored = look.over();
                }
            }
        }
    }
    void free_buffers() {
        for (char*& p : pin_) {
            if (p) cudaFreeHost(p);
            p = nullptr;
        }
    }

    char* pin_[NBUF] = {};
    std::vector<std::thread> threads_;
    std::mutex m_;
    std::condition_variable cv_;
    const pid_t owner_ = getpid();
    bool started_ = false, quit_ = false, down_ = false;
    unsigned long job_ = 0;
    char* host_ = nullptr;
    size_t n_ = 0;
    long base_ = 0;                         // number of the transfer's first slice
    std::atomic<long> next_{0}, open_{0};   // slices taken, slices open
    std::atomic<long> done_[NBUF] = {};     // slices copied of a buffer's chunk
    std::atomic<bool> active_{false};
    std::atomic<int> asleep_{0};  // threads that sleep through a pause of a transfer
};

std::mutex g_copier_lock;  // one transfer at a time; the others take the driver's path
std::mutex g_count_lock;
int g_handles = 0;
// given back by the last handle only: a process that exits with handles leaves
// it, so that no exit handler waits for threads a fork did not copy
Copier* g_copier = nullptr;

// a transfer through the copier; cudaErrorNotReady: not taken
cudaError_t staged(char* dev, char* host, size_t n, bool down, cudaStream_t st) {
    std::unique_lock<std::mutex> l(g_copier_lock, std::try_to_lock);
    if (!l.owns_lock()) return cudaErrorNotReady;
    if (!g_copier) g_copier = new (std::nothrow) Copier();
    if (!g_copier || !g_copier->start()) return cudaErrorNotReady;
    return g_copier->transfer(dev, host, n, down, st);
}

}  // namespace

void hostcopy_retain() {
    std::lock_guard<std::mutex> l(g_count_lock);
    g_handles++;
}

void hostcopy_release() {
    std::lock_guard<std::mutex> l(g_count_lock);
    if (--g_handles > 0) return;
    if (g_copier && !g_copier->here()) {  // left as it is: there are no threads to join
        g_copier = nullptr;
        return;
    }
    std::lock_guard<std::mutex> c(g_copier_lock);
    delete g_copier;
    g_copier = nullptr;
}

cudaError_t hostcopy_h2d(void* dst, const void* src, size_t n, cudaStream_t st) {
    if (n >= MIN_BYTES) {
        // an error pending here (a refused launch) is the caller's to hear of;
        // what follows clears errors of its own
        const cudaError_t before = cudaGetLastError();
        if (before != cudaSuccess) return before;
    }
    if (n >= MIN_BYTES && pageable(src)) {
        const cudaError_t e =
            staged((char*)dst, const_cast<char*>((const char*)src), n, false, st);
        if (e != cudaErrorNotReady) return e;
    }
    return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
}

cudaError_t hostcopy_d2h(void* dst, const void* src, size_t n, cudaStream_t st) {
    if (n >= MIN_BYTES) {
        const cudaError_t before = cudaGetLastError();
        if (before != cudaSuccess) return before;
    }
    if (n >= MIN_BYTES && pageable(dst)) {
        const cudaError_t e = staged(const_cast<char*>((const char*)src), (char*)dst, n, true, st);
        if (e != cudaErrorNotReady) return e;
    }
    return cudaMemcpyAsync(dst, src, n, cudaMemcpyDeviceToHost, st);
}

}  // namespace dcm
