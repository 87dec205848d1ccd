// Copies between ordinary host memory and the device (host_staging.cuh).
//
// A copy from pageable memory goes through page-locked memory either way; the driver's own way costs a synchronous 17 us
// at 90 KB and 41 us at 0.5 MB, and one thread's memcpy (18 GB/s beyond the CPU's caches) bounds it for large operands,
// where the link takes 53 GB/s.  Here the calling thread moves piece after piece into the page-locked buffer while the
// earlier ones are on the link, and from kThreadedBytes on three more threads help; a download runs the same way
// backwards, a piece being moved out as soon as its event says that it has landed.
#include "host_staging.cuh"

#include <atomic>
#include <cstring>
#include <system_error>
#include <thread>

namespace t81b200 {

namespace {

constexpr int kMaxDevices = 64;
HostStaging g_staging[kMaxDevices];

constexpr size_t kPinnedMost = 96u << 20;      // larger calls are copied by the driver, from where the operands are
constexpr size_t kPiece = 512u << 10;
constexpr size_t kThreadedBytes = 4u << 20;    // below, starting threads (20 us each) costs what they save
constexpr int kHelpers = 3;

// Runs work() here and, for large copies, on helpers too; returns the first error any of them met.
template <typename F>
int with_helpers(size_t bytes, F &&work) {
    std::atomic<int> status{(int)cudaSuccess};
    auto guarded = [&]() {
        const cudaError_t e = work();
        int none = (int)cudaSuccess;
        if (e != cudaSuccess) status.compare_exchange_strong(none, (int)e);
    };
    std::thread helpers[kHelpers];
    int started = 0, dev = 0;
    if (bytes >= kThreadedBytes && cudaGetDevice(&dev) == cudaSuccess) {
        const int spare = (int)std::thread::hardware_concurrency() - 1;
        try {
            for (; started < kHelpers && started < spare; ++started)
                helpers[started] = std::thread([&, dev]() { if (cudaSetDevice(dev) == cudaSuccess) guarded(); });
        } catch (const std::system_error &) {
            // no more threads to be had: the others do the work
        }
    }
    guarded();
    for (int i = 0; i < started; ++i) helpers[i].join();
    return status.load();
}

int ensure_pinned(HostStaging &s, size_t bytes, bool *fits) {
    *fits = false;
    if (bytes > kPinnedMost) return T81B200_OK;
    if (bytes > s.pinned_cap) {
        if (s.pinned) cudaFreeHost(s.pinned);
        s.pinned = nullptr;
        s.pinned_cap = 0;
        const size_t want = (bytes + (1u << 20) - 1) >> 20 << 20;
        if (cudaHostAlloc(reinterpret_cast<void **>(&s.pinned), want, cudaHostAllocDefault) != cudaSuccess) {
            (void)cudaGetLastError();  // page-locked memory is short: the driver's way then
            s.pinned = nullptr;
            return T81B200_OK;
        }
        s.pinned_cap = want;
    }
    *fits = true;
    return T81B200_OK;
}

int cuda_status(int e, const char *what) {
    return e == (int)cudaSuccess ? T81B200_OK : fail(T81B200_ECUDA, "%s failed: %s", what, cudaGetErrorString((cudaError_t)e));
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
    size_t total = 0;
    for (int i = 0; i < n; ++i) total += (ops[i].bytes + 255) / 256 * 256;
    bool fits;
    if (int rc = ensure_pinned(s, total, &fits)) return rc;
    if (!fits) {
        for (int i = 0; i < n; ++i)
            if (ops[i].bytes) T81_CUDA_TRY(cudaMemcpyAsync(ops[i].device, ops[i].host, ops[i].bytes, cudaMemcpyHostToDevice, s.stream));
        return T81B200_OK;
    }
    std::atomic<size_t> next{0};  // pieces are numbered through the operands
    const int rc = with_helpers(total, [&]() {
        for (;;) {
            size_t piece = next.fetch_add(1), base = 0;
            int i = 0;
            for (; i < n; ++i) {
                const size_t pieces = (ops[i].bytes + kPiece - 1) / kPiece;
                if (piece < pieces) break;
                piece -= pieces;
                base += (ops[i].bytes + 255) / 256 * 256;
            }
            if (i == n) return cudaSuccess;
            const size_t at = piece * kPiece, bytes = ops[i].bytes - at < kPiece ? ops[i].bytes - at : kPiece;
            memcpy(s.pinned + base + at, static_cast<const char *>(ops[i].host) + at, bytes);
            const cudaError_t e = cudaMemcpyAsync(static_cast<char *>(ops[i].device) + at, s.pinned + base + at, bytes, cudaMemcpyHostToDevice, s.stream);
            if (e != cudaSuccess) return e;
        }
    });
    if (rc != (int)cudaSuccess) cudaStreamSynchronize(s.stream);  // what was queued still reads the page-locked buffer
    return cuda_status(rc, "copy to the device");
}

int host_download(HostStaging &s, void *host, const void *device, size_t bytes) {
    bool fits;
    if (int rc = ensure_pinned(s, bytes, &fits)) return rc;
    if (!fits) {
        T81_CUDA_TRY(cudaMemcpyAsync(host, device, bytes, cudaMemcpyDeviceToHost, s.stream));
        T81_CUDA_TRY(cudaStreamSynchronize(s.stream));
        return T81B200_OK;
    }
    // the uploads that used the buffer come before these copies in the stream
    size_t piece = kPiece / 2;
    while ((bytes + piece - 1) / piece > (size_t)HostStaging::kMaxPieces) piece *= 2;
    const int pieces = (int)((bytes + piece - 1) / piece);
    auto size_of = [&](int i) { return bytes - i * piece < piece ? bytes - i * piece : piece; };
    cudaError_t queued = cudaSuccess;
    int n = 0;
    for (; n < pieces; ++n) {
        queued = cudaMemcpyAsync(s.pinned + n * piece, static_cast<const char *>(device) + n * piece, size_of(n), cudaMemcpyDeviceToHost, s.stream);
        if (queued == cudaSuccess) queued = cudaEventRecord(s.landed[n], s.stream);
        if (queued != cudaSuccess) break;
    }
    std::atomic<int> next{0};
    const int rc = queued != cudaSuccess ? (int)queued : with_helpers(bytes, [&]() {
        for (;;) {
            const int i = next.fetch_add(1);
            if (i >= n) return cudaSuccess;
            const cudaError_t e = cudaEventSynchronize(s.landed[i]);
            if (e != cudaSuccess) return e;
            memcpy(static_cast<char *>(host) + i * piece, s.pinned + i * piece, size_of(i));
        }
    });
    if (rc != (int)cudaSuccess) cudaStreamSynchronize(s.stream);
    return cuda_status(rc, "copy from the device");
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
        if (!s.stream && !s.pinned && !s.dev[0] && !s.dev[1] && !s.dev[2] && !s.dev[3]) continue;
        T81_CUDA_TRY(cudaSetDevice(d));
        for (int i = 0; i < HostStaging::N_BUFFERS; ++i) {
            if (s.dev[i]) cudaFree(s.dev[i]);
            s.dev[i] = nullptr;
            s.dev_cap[i] = 0;
        }
        if (s.pinned) cudaFreeHost(s.pinned);
        s.pinned = nullptr;
        s.pinned_cap = 0;
        for (cudaEvent_t &e : s.landed) { if (e) cudaEventDestroy(e); e = nullptr; }
        if (s.stream) cudaStreamDestroy(s.stream);
        s.stream = nullptr;
    }
    T81_CUDA_TRY(cudaSetDevice(cur));
    release_elementwise_staging();
    T81_CUDA_TRY(cudaSetDevice(cur));
    return T81B200_OK;
}
