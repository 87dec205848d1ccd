// Copies between ordinary host memory and the device (host_staging.cuh).
//
// A copy from pageable memory goes through page-locked memory either way; the driver's own way costs a synchronous 17 us
// at 90 KB and 41 us at 0.5 MB, and one thread's memcpy (18 GB/s beyond the CPU's caches) bounds it for large operands,
// where the link takes 53 GB/s.  Here the calling thread moves piece after piece into the page-locked buffer and queues
// each piece's copy while it moves the next, and for large operands a few kept helper threads move pieces too (they make
// no CUDA calls; starting threads for one call cost 100 us each).  A download runs the same way backwards: the calling
// thread watches the pieces land, and whoever is free moves one out.
#include "host_staging.cuh"

#include <atomic>
#include <condition_variable>
#include <cstring>
#include <exception>
#include <new>
#include <thread>
#if defined(__SSE2__)
#include <emmintrin.h>
#endif

namespace t81b200 {

namespace {

constexpr int kMaxDevices = 64;
HostStaging g_staging[kMaxDevices];

constexpr size_t kPinnedMost = 96u << 20;      // larger calls are copied by the driver, from where the operands are
constexpr size_t kHelpedUp = 2u << 20, kHelpedDown = 1u << 20;  // below, waking helpers costs what they save
constexpr int kHelpers = 3;

inline void pause() {
#if defined(__x86_64__)
    __builtin_ia32_pause();
#else
    std::this_thread::yield();
#endif
}

// Copy into a page-locked buffer the device is about to read, with stores that go past the CPU's caches: lines that are
// still dirty in the caches of several cores reach the device at 8 GB/s.  dst is 16-byte aligned.
void copy_for_device(char *dst, const char *src, size_t bytes) {
#if defined(__SSE2__)
    size_t i = 0;
    for (; i + 64 <= bytes; i += 64) {
        const __m128i a = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i)), b = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 16));
        const __m128i c = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 32)), d = _mm_loadu_si128(reinterpret_cast<const __m128i *>(src + i + 48));
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i), a);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 16), b);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 32), c);
        _mm_stream_si128(reinterpret_cast<__m128i *>(dst + i + 48), d);
    }
    memcpy(dst + i, src + i, bytes - i);
    _mm_sfence();  // the stores are on their way to memory before anyone is told that the piece is there
#else
    memcpy(dst, src, bytes);
#endif
}

// Helper threads shared by all calls of the process, one job at a time; a call that finds them busy does without.  A job
// is a function that claims its own work, so nothing depends on how many helpers take part.  Nothing here allocates or throws (the
// callers are C entry points) but the start of a thread, which is caught.
class Helpers {
public:
    // Offers `work` (a function object that outlives end()) to the helpers; false when they are busy.
    template <typename F> bool begin(F &work) {
        if (!busy_.try_lock()) return false;
        std::lock_guard<std::mutex> lock(mu_);
        try {
            for (; count_ < kHelpers && count_ + 1 < (int)std::thread::hardware_concurrency(); ++count_) threads_[count_] = std::thread([this] { run(); });
        } catch (const std::exception &) {
            // no more threads to be had: those there are help
        }
        call_ = [](void *f) { (*static_cast<F *>(f))(); };
        work_ = &work;
        ++job_;
        wake_.notify_all();
        return true;
    }
    // Takes the job back and waits for the helpers that took part.
    void end() {
        {
            std::unique_lock<std::mutex> lock(mu_);
            work_ = nullptr;
            idle_.wait(lock, [this] { return active_ == 0; });
        }
        busy_.unlock();
    }
    void stop() {  // gives the threads back
        std::lock_guard<std::mutex> only(busy_);
        {
            std::lock_guard<std::mutex> lock(mu_);
            stopping_ = true;
            wake_.notify_all();
        }
        for (; count_ > 0; --count_) threads_[count_ - 1].join();
        stopping_ = false;
    }

private:
    void run() {
        uint64_t seen = 0;
        std::unique_lock<std::mutex> lock(mu_);
        for (;;) {
            wake_.wait(lock, [&] { return stopping_ || (work_ && job_ != seen); });
            if (stopping_) return;
            seen = job_;
            void (*const call)(void *) = call_;
            void *const work = work_;
            ++active_;
            lock.unlock();
            call(work);
            lock.lock();
            if (--active_ == 0) idle_.notify_all();
        }
    }
    std::mutex busy_, mu_;
    std::condition_variable wake_, idle_;
    std::thread threads_[kHelpers];
    int count_ = 0;
    void (*call_)(void *) = nullptr;
    void *work_ = nullptr;
    uint64_t job_ = 0;
    int active_ = 0;
    bool stopping_ = false;
};
Helpers &helpers() {
    // outlives every static destructor that might still copy
    alignas(Helpers) static unsigned char place[sizeof(Helpers)];
    static Helpers *h = new (place) Helpers;
    return *h;
}

enum { UP, DOWN };

int ensure_pinned(HostStaging &s, int way, size_t bytes, bool *fits) {
    *fits = false;
    if (bytes > kPinnedMost) return T81B200_OK;
    if (bytes > s.pinned_cap[way]) {
        if (s.pinned[way]) cudaFreeHost(s.pinned[way]);
        s.pinned[way] = nullptr;
        s.pinned_cap[way] = 0;
        const size_t want = (bytes + (1u << 20) - 1) >> 20 << 20;
        void *p = nullptr;
        if (cudaHostAlloc(&p, want, cudaHostAllocDefault) != cudaSuccess) {
            (void)cudaGetLastError();  // page-locked memory is short: the driver's way then
            return T81B200_OK;
        }
        s.pinned[way] = static_cast<char *>(p);
        s.pinned_cap[way] = want;
    }
    *fits = true;
    return T81B200_OK;
}

constexpr int kMostOperands = 3;
constexpr size_t kUpPiece = 512u << 10;
constexpr int kMostUpPieces = (int)(kPinnedMost / kUpPiece) + kMostOperands;

int cuda_status(cudaError_t e, const char *what) {
    return e == cudaSuccess ? T81B200_OK : fail(T81B200_ECUDA, "%s failed: %s", what, cudaGetErrorString(e));
}

}  // namespace

int host_staging(HostStaging **out) {
    int dev = 0;
    T81_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(T81B200_ELIMIT, "device index %d not supported", dev);
    *out = &g_staging[dev];
    return T81B200_OK;
}

int host_staging_ready(HostStaging &s) {
    // page-locked operands may still be written by copies on the default stream, behind which these calls have always stood
    T81_CUDA_TRY(cudaStreamSynchronize(cudaStreamLegacy));
    if (!s.stream) T81_CUDA_TRY(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking));
    for (cudaEvent_t &e : s.landed)
        if (!e) T81_CUDA_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
    return T81B200_OK;
}

int host_staging_buffer(HostStaging &s, int which, size_t bytes) {
    if (bytes <= s.dev_cap[which]) return T81B200_OK;
    if (s.dev[which]) cudaFree(s.dev[which]);
    s.dev[which] = nullptr;
    s.dev_cap[which] = 0;
    T81_CUDA_TRY(cudaMalloc(&s.dev[which], bytes));
    s.dev_cap[which] = bytes;
    return T81B200_OK;
}

int host_upload(HostStaging &s, const HostOperand *ops, int n) {
    if (n > kMostOperands) return fail(T81B200_ELIMIT, "host_upload: %d operands", n);
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += (ops[i].bytes + 255) / 256 * 256;
    bool fits;
    if (int rc = ensure_pinned(s, UP, total, &fits)) return rc;
    if (!fits) {
        cudaError_t status = cudaSuccess;
        for (int i = 0; i < n && status == cudaSuccess; ++i)
            if (ops[i].bytes) status = cudaMemcpyAsync(ops[i].device, ops[i].host, ops[i].bytes, cudaMemcpyHostToDevice, s.stream);
        if (status != cudaSuccess) cudaStreamSynchronize(s.stream);  // what was queued still reads the caller's memory
        return cuda_status(status, "copy to the device");
    }
    // piece j of operand i, numbered through: begins[i] is the number of the operand's first one
    const size_t piece = total < (4u << 20) ? kUpPiece / 2 : kUpPiece;
    size_t bases[kMostOperands];
    int begins[kMostOperands + 1] = {0}, pieces = 0;
    for (size_t i = 0, base = 0; i < (size_t)n; ++i) {
        bases[i] = base;
        base += (ops[i].bytes + 255) / 256 * 256;
        begins[i + 1] = pieces += (int)((ops[i].bytes + piece - 1) / piece);
    }
    std::atomic<bool> moved[kMostUpPieces];
    for (int i = 0; i < pieces; ++i) moved[i].store(false, std::memory_order_relaxed);
    auto at = [&](int i, char *&pinned, char *&device, const char *&host) {  // returns the piece's size
        int o = 0;
        while (i >= begins[o + 1]) ++o;
        const size_t off = (size_t)(i - begins[o]) * piece;
        pinned = s.pinned[UP] + bases[o] + off;
        device = static_cast<char *>(ops[o].device) + off;
        host = static_cast<const char *>(ops[o].host) + off;
        return ops[o].bytes - off < piece ? ops[o].bytes - off : piece;
    };
    std::atomic<int> next{0};
    auto move_one = [&]() {
        const int i = next.fetch_add(1, std::memory_order_relaxed);
        if (i >= pieces) return false;
        char *pinned, *device;
        const char *host;
        const size_t bytes = at(i, pinned, device, host);
        copy_for_device(pinned, host, bytes);
        moved[i].store(true, std::memory_order_release);
        return true;
    };
    auto move_all = [&]() { while (move_one()) {} };
    const bool helped = total >= kHelpedUp && helpers().begin(move_all);
    cudaError_t status = cudaSuccess;
    for (int queued = 0; queued < pieces;) {
        const bool more = move_one();
        for (; queued < pieces && moved[queued].load(std::memory_order_acquire); ++queued) {
            char *pinned, *device;
            const char *host;
            const size_t bytes = at(queued, pinned, device, host);
            if (status == cudaSuccess) status = cudaMemcpyAsync(device, pinned, bytes, cudaMemcpyHostToDevice, s.stream);
        }
        if (!more) pause();
    }
    if (helped) helpers().end();
    if (status != cudaSuccess) cudaStreamSynchronize(s.stream);  // what was queued still reads the page-locked buffer
    return cuda_status(status, "copy to the device");
}

int host_abandon(HostStaging &s, int code) {
    cudaStreamSynchronize(s.stream);
    return code;
}

int host_download(HostStaging &s, void *host, const void *device, size_t bytes) {
    bool fits;
    if (int rc = ensure_pinned(s, DOWN, bytes, &fits)) return rc;
    if (!fits) {
        T81_CUDA_TRY(cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, s.stream));
        T81_CUDA_TRY(cudaStreamSynchronize(s.stream));
        return T81B200_OK;
    }
    size_t piece = 256u << 10;
    while ((bytes + piece - 1) / piece > (size_t)HostStaging::kMaxPieces) piece *= 2;
    const int pieces = (int)((bytes + piece - 1) / piece);
    auto size_of = [&](int i) { return bytes - i * piece < piece ? bytes - i * piece : piece; };
    cudaError_t queued = cudaSuccess;
    int n = 0;
    for (; n < pieces; ++n) {
        queued = cudaMemcpyAsync(s.pinned[DOWN] + n * piece, static_cast<const char *>(device) + n * piece, size_of(n), cudaMemcpyDeviceToHost, s.stream);
        if (queued == cudaSuccess) queued = cudaEventRecord(s.landed[n], s.stream);
        if (queued != cudaSuccess) break;
    }
    if (queued != cudaSuccess) {
        cudaStreamSynchronize(s.stream);
        return cuda_status(queued, "copy from the device");
    }
    std::atomic<int> next{0}, landed{0};
    std::atomic<bool> give_up{false};
    auto move_one = [&](bool wait) {  // false: nothing (more) to move
        int i = next.load(std::memory_order_relaxed);
        for (;;) {
            if (i >= pieces || give_up.load(std::memory_order_relaxed)) return false;
            if (landed.load(std::memory_order_acquire) <= i) {
                if (!wait) return false;
                pause();
                i = next.load(std::memory_order_relaxed);
                continue;
            }
            if (next.compare_exchange_weak(i, i + 1)) break;
        }
        memcpy(static_cast<char *>(host) + i * piece, s.pinned[DOWN] + i * piece, size_of(i));
        return true;
    };
    auto move_all = [&]() { while (move_one(true)) {} };
    const bool helped = bytes >= kHelpedDown && helpers().begin(move_all);
    cudaError_t status = cudaSuccess;
    for (int seen = 0; seen < pieces;) {
        const cudaError_t e = cudaEventQuery(s.landed[seen]);
        if (e == cudaSuccess) landed.store(++seen, std::memory_order_release);
        else if (e != cudaErrorNotReady) {
            status = e;
            give_up.store(true);
            break;
        } else if (!move_one(false)) pause();
    }
    while (status == cudaSuccess && move_one(false)) {}
    if (helped) helpers().end();
    if (status != cudaSuccess) cudaStreamSynchronize(s.stream);
    return cuda_status(status, "copy from the device");
}

void release_elementwise_staging();  // elementwise.cu

}  // namespace t81b200

using namespace t81b200;

extern "C" int t81b200_release_staging(void) {
    if (int rc = check_device()) return rc;
    int cur = 0, count = 0;
    T81_CUDA_TRY(cudaGetDevice(&cur));
    T81_CUDA_TRY(cudaGetDeviceCount(&count));
    for (int d = 0; d < count && d < kMaxDevices; ++d) {
        HostStaging &s = g_staging[d];
        std::lock_guard<std::mutex> lock(s.mu);
        if (!s.stream && !s.pinned[UP] && !s.pinned[DOWN] && !s.dev[0] && !s.dev[1] && !s.dev[2] && !s.dev[3]) continue;
        T81_CUDA_TRY(cudaSetDevice(d));
        for (int i = 0; i < HostStaging::N_BUFFERS; ++i) {
            if (s.dev[i]) cudaFree(s.dev[i]);
            s.dev[i] = nullptr;
            s.dev_cap[i] = 0;
        }
        for (int way : {UP, DOWN}) {
            if (s.pinned[way]) cudaFreeHost(s.pinned[way]);
            s.pinned[way] = nullptr;
            s.pinned_cap[way] = 0;
        }
        for (cudaEvent_t &e : s.landed) { if (e) cudaEventDestroy(e); e = nullptr; }
        if (s.stream) cudaStreamDestroy(s.stream);
        s.stream = nullptr;
    }
    helpers().stop();
    T81_CUDA_TRY(cudaSetDevice(cur));
    release_elementwise_staging();
    T81_CUDA_TRY(cudaSetDevice(cur));
    return T81B200_OK;
}
