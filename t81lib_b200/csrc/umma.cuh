// tcgen05 pieces shared by the tensor-core kernels: shared-memory and instruction descriptors, MMA issue, commits,
// TMEM allocation and reads — all in their cta_group::2 form, where a pair of CTAs (ranks 2i and 2i + 1 of a cluster)
// works on one 256-row tile: each CTA holds its own 128 rows of A, half of the columns of B and its own 128 rows of
// the accumulator; the even CTA issues the MMAs and owns the barriers the pair is ordered by.
#pragma once

#include "common.cuh"
#include "tma.cuh"

namespace t81b200 {

constexpr uint32_t kTmemCols = 512;

// kind::f16 instruction descriptor for a 256-row pair tile: fp32 accumulators, A and B both bf16 or both fp16,
// n columns; a_mn / b_mn: the operand's shared-memory tile is contiguous along M / N instead of K.
__host__ __device__ constexpr uint32_t umma_instr_desc(int n, bool f16, bool a_mn = false, bool b_mn = false) {
    return (1u << 4) | ((f16 ? 0u : 1u) << 7) | ((f16 ? 0u : 1u) << 10) | ((a_mn ? 1u : 0u) << 15) | ((b_mn ? 1u : 0u) << 16) |
           ((uint32_t)(n >> 3) << 17) | ((256u >> 4) << 24);
}

// A role whose bounded wait ran out: the code is recorded, and the CTA stays about a millisecond longer, so that copies and
// commits under way land before its shared memory goes to another one.
static __device__ __noinline__ void give_up(int *status, int code) {
    if ((threadIdx.x & 31) == 0) atomicCAS(status, 0, code);
    for (int i = 0; i < 10; ++i) __nanosleep(100000);
}

// True in one lane of a converged warp.  The loops of the issuing warps run on all 32 lanes (addresses and descriptors
// stay in uniform registers) and only the issue itself is guarded: under a plain `lane == 0` branch the compiler cannot
// know the operands to be uniform and every tcgen05 / TMA instruction pays for moving them (an operand atom of four
// MMAs took 385 ns to issue that way, against 270 ns of tensor time).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .b32 x;\n\t.reg .pred p;\n\t"
        "elect.sync x|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r));
    return r != 0;
}

// K-major SWIZZLE_128B descriptor: rows of 128 bytes (64 k), 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t umma_desc_k(uint32_t smem_addr) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) |
           ((uint64_t)2 << 61);
}

// acc[256 x n] (+)= A B^T for one k-step of 16.
__device__ __forceinline__ void umma_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this shared-memory offset in both CTAs of the pair once the MMAs issued so far are done.
__device__ __forceinline__ void umma_commit_pair(uint32_t bar, uint16_t pair_mask) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"(pair_mask)
                 : "memory");
}

// The same shared-memory address in the even CTA of the pair (the CTA's cluster rank sits in the top byte).
__device__ __forceinline__ uint32_t pair_leader(uint32_t addr) { return addr & 0xFEFFFFFFu; }

__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(pair_leader(bar)) : "memory");
}
// 2-D TMA load into this CTA's shared memory whose bytes are counted on the even CTA's barrier.
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(pair_leader(bar))
        : "memory");
}

// Whole warp, both CTAs of the pair.
__device__ __forceinline__ void tmem_alloc_pair(uint32_t slot) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(slot), "r"(kTmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free_pair(uint32_t tmem) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
}

// 32 columns of this warp's 32 lanes: v[i] of lane l = accumulator (row l of the warp's quarter, column i).
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
          "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
          "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// 16 columns the other way; the caller waits (tcgen05.wait::st) before anyone reads them.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
          "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}
// Eight columns in two steps: what `v` holds may be read past the wait only, which is for every load before it.  The first step names
// registers as written that the load fills later, and the second takes and gives back the same ones, so that every use of `v` comes
// behind the wait.  What the language does not promise is that no copy of them is made in between: `v` is an array that only
// these two touch until then, in straight-line code, and the tests compare every column of the sums.
__device__ __forceinline__ void tmem_ld8_start(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_ld8_wait(uint32_t (&v)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(v[0]), "+r"(v[1]), "+r"(v[2]), "+r"(v[3]), "+r"(v[4]), "+r"(v[5]), "+r"(v[6]), "+r"(v[7])
                 :: "memory");
}
// tmem_ld32 for 8 columns.
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tma_store_2d(const CUtensorMap *map, uint32_t src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%2, %3}], [%1];"
                 ::"l"(map), "r"(src), "r"(x), "r"(y)
                 : "memory");
}

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// ---- a tile whose contraction is split over S pairs of a cluster ----
// 32-column block b of the accumulator is finished by slice b % S; each other slice owns one 16 KB slot per block
// ([column][128 rows] fp32) in that CTA's shared memory.
__device__ __forceinline__ uint32_t partial_slot(int b, int S, int from, int to) { return (uint32_t)((b / S) * (S - 1) + (from < to ? from : from - 1)); }

// v[i] (column i of the block) of this thread's row -> the slot at `dst` in the CTA of that cluster rank.
__device__ __forceinline__ void push_partial(const uint32_t (&v)[32], uint32_t dst, uint32_t to_rank) {
    asm("mapa.shared::cluster.u32 %0, %0, %1;" : "+r"(dst) : "r"(to_rank));
#pragma unroll
    for (int i = 0; i < 32; ++i) asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(dst + (uint32_t)i * 512u), "r"(v[i]) : "memory");
}

// v (this slice's own sums of block b) += the other slices' slots, in slice order whoever finishes the block.
__device__ __forceinline__ void fold_partials(uint32_t (&v)[32], const uint8_t *slots, int b, int S, int slice, uint32_t lane_row) {
    float sum[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) sum[i] = 0.0f;
    for (int s = 0; s < S; ++s) {
        const float *src = reinterpret_cast<const float *>(slots + (size_t)partial_slot(b, S, s, slice) * 16384) + lane_row;
#pragma unroll
        for (int i = 0; i < 32; ++i) sum[i] += s == slice ? __uint_as_float(v[i]) : src[i * 128];
    }
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(sum[i]);
}

// ---- host ----
// Clusters of `splits` CTA pairs (one CTA per SM) that the device runs at a time: clusters do not straddle GPCs, so
// fewer fit than the SM count suggests (74, 33, 22 and 15 for 1 to 4 splits on a B200).
int resident_pair_clusters(int splits);
// Token-major planes of a (tokens, K) or (K, tokens) operand in scratch memory, rows of K rounded up to 8 elements:
// 16-bit types are copied bit for bit (planes == 1), fp32 becomes two or three bf16 planes.
int stage_planes(const void *B, int dtype, int layout, int64_t ld, int64_t tokens, int64_t K, int planes, void *scratch, cudaStream_t st);

}  // namespace t81b200
