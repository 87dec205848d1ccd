// Shared pieces of the TMA-fed kernels: bounded mbarrier waits, 2-D tensor-map loads, and
// host-side tensor-map creation through the driver entry point (no link-time libcuda dependency).
#pragma once

#include <cuda.h>

#include "common.cuh"

namespace t81b200 {

constexpr uint32_t kSpinLimit = 1u << 20;  // polls of 3.9 us before a wait gives up and the kernel reports a status (2^24 took 66 s)

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// Bounded wait: false when the phase did not complete within the spin limit.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t spin = 0; spin < kSpinLimit; ++spin) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (spin > 1024) __nanosleep(64);
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// Untiled copy: both addresses and the size are multiples of 16 bytes.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

// The same bytes to L2 only.
__device__ __forceinline__ void bulk_prefetch(const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(src), "r"(bytes) : "memory");
}

// A tensor map on its way to where copies look it up (the first copy through it waits some hundred ns otherwise).
__device__ __forceinline__ void prefetch_map(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

struct Ring {
    int stage = 0;
    uint32_t phase = 0;
    __device__ __forceinline__ void advance(int stages) {
        if (++stage == stages) { stage = 0; phase ^= 1; }
    }
};

// ---- host: tensor maps through the driver entry point (no link-time libcuda dependency) ----

typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                  const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled() {
    // looked up once, whichever thread comes first: an autograd worker may make its first call beside the main thread's
    static const EncodeTiledFn fn = [] {
        void *ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool found = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
        return found ? reinterpret_cast<EncodeTiledFn>(ptr) : nullptr;
    }();
    return fn;
}

// Tensor map of `rank` dimensions; dims, strides (bytes, of dimensions 1 ..) and box as the driver wants them.
inline int make_map(CUtensorMap *map, CUtensorMapDataType dt, int rank, const void *ptr, const cuuint64_t *dims, const cuuint64_t *strides,
                    const cuuint32_t *box, CUtensorMapSwizzle swz) {
    EncodeTiledFn fn = encode_tiled();
    if (!fn) return fail(T81B200_ECUDA, "cuTensorMapEncodeTiled is not available from the driver");
    const cuuint32_t estr[3] = {1, 1, 1};
    for (int attempt = 0;; ++attempt) {
        const CUresult rc = fn(map, dt, (cuuint32_t)rank, const_cast<void *>(ptr), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swz,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (rc == CUDA_SUCCESS) return T81B200_OK;
        // a thread that has made no runtime call with an effect yet (an autograd worker) has no current context: bind it
        if (rc != CUDA_ERROR_INVALID_CONTEXT || attempt > 0) return fail(T81B200_ECUDA, "cuTensorMapEncodeTiled failed with code %d", (int)rc);
        T81_CUDA_TRY(cudaFree(nullptr));
    }
}

inline int make_map_2d(CUtensorMap *map, CUtensorMapDataType dt, const void *ptr, uint64_t inner, uint64_t outer,
                uint64_t row_stride_bytes, uint32_t box_inner, uint32_t box_outer, CUtensorMapSwizzle swz) {
    const cuuint64_t dims[2] = {inner, outer}, strides[1] = {row_stride_bytes};
    const cuuint32_t box[2] = {box_inner, box_outer};
    return make_map(map, dt, 2, ptr, dims, strides, box, swz);
}

}  // namespace t81b200
