// Operands that live in ordinary host memory: device buffers, page-locked buffers on the way there and a stream, one set
// per device, grown on demand, kept between calls and given back by t81b200_release_staging.
#pragma once

#include <mutex>

#include "common.cuh"

namespace t81b200 {

struct HostStaging {
    std::mutex mu;  // held for a whole call
    enum { A, B, C, WORKSPACE, N_BUFFERS };
    void *dev[N_BUFFERS] = {nullptr};
    size_t dev_cap[N_BUFFERS] = {0};
    char *pinned[2] = {nullptr, nullptr};  // on the way up and down
    size_t pinned_cap[2] = {0, 0};
    cudaStream_t stream = nullptr;
    static constexpr int kMaxPieces = 64;
    cudaEvent_t landed[kMaxPieces] = {nullptr};
};

// The current device's set, with its stream made on first use (call with `mu` held); ready: behind what the default stream holds.
int host_staging(HostStaging **out);
int host_staging_ready(HostStaging &s);
int host_staging_buffer(HostStaging &s, int which, size_t bytes);

struct HostOperand {
    void *device;
    const void *host;
    size_t bytes;
};
// Queues the operands' copies to the device on s.stream, first to last.
int host_upload(HostStaging &s, const HostOperand *ops, int n);
// Ends a call that failed behind its upload: waits for the copies, which read the caller's or the page-locked memory; returns `code`.
int host_abandon(HostStaging &s, int code);
// Copies device memory to the host behind what s.stream holds; returns when it is there.
int host_download(HostStaging &s, void *host, const void *device, size_t bytes);

}  // namespace t81b200
