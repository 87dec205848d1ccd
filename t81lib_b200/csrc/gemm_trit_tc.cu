// TRIT-mode matmul on the 5th-generation tensor cores (tcgen05): more activation rows than the streaming kernel takes.
//
//   D[o][t] = sum_k T[o][k] * x[t][k]       o: output feature (256 per CTA pair, 128 per CTA)
//                                            t: token          (up to 256 per tile)
// A pair of CTAs (cta_group::2) works on one tile: each expands its own 128 weight rows into bf16 / fp16 operands in
// its shared memory and loads half of the tile's activation rows by TMA; the even CTA issues the MMAs, which read both
// halves, and each CTA keeps its 128 accumulator rows in TMEM (2 x 256 fp32 columns, double-buffered across tiles).
// Measured against the one-CTA 128 x 256 kernel before it (bf16, weights in limbs there and in codes here):
// 4096 x 14336 x 16384 tokens 958 -> 1506 TFLOP/s in a long run under the power cap, 9216 x 3072 x 2048 109 -> 84 us, 14336 x 4096 x 80
// 40.9 -> 19.2 us.
// What bounds the kernel is shared-memory bandwidth: a 64-deep step writes and reads 16 KB of expanded weights per CTA
// and writes and reads the activations, against 512 clocks of MMA at 256 tokens.  Halving the activation share is what
// the pair is for: a single CTA with a 128 x 256 tile needs 768 clocks of shared memory per 512 of MMA.
//
// Weights come in two formats (template FMT), both brought by bulk copies in 192-column chunks:
//   0  packed limbs: a lane takes four limbs (rows 8 apart), packed bf16 FMAs expand them to {-1, 0, +1} (common.cuh);
//   1  the decode-stream layout (pack_t2.cu): one word is 8 columns of 2 rows, i.e. two 16-byte pieces of the operand
//      tile; a pair of trits is one shift and one AND (the 2-bit code IS the top of the 16-bit number +-2 or 0, in
//      bf16 and in fp16 alike; the factor 2 leaves with alpha).  The 32 lanes of a warp store 8 rows x 4 column runs
//      of 48: under the 128-byte swizzle every quarter of a warp store covers all banks once.
// 192 columns are four limbs and three 64-column operand atoms: the unit in which converters hand weights to the MMAs.
//
// Activations: 16-bit types as they are (A and B of one MMA have the same type), fp32 as bf16 planes (x = hi + lo, 16
// mantissa bits) that are multiplied with the same expanded weights, side by side or in turn (Mode).  Rows TMA cannot read
// (unaligned, the (K, N) layout, fp32) are first copied into token-major planes in the caller's workspace.
// All planes but the first have an accumulator of their own beside it, and the epilogue adds the two.  The tensor core cuts an
// accumulator off at every 16 columns instead of rounding it.  With the first plane alone little is cut (trits times 8-bit
// mantissas mostly fit); with small terms mixed in a bit is lost at every step.  Relative to the exact sums of trits and N(0, 1)
// values, one accumulator -> two: two planes 4096 x 14336 x 300 tokens 1.7e-5 -> 2.5e-6, at any size now (what 16 mantissa bits
// leave); three planes (all 24 bits, the gradients) 3.2e-5 -> 2.6e-7, 1537 x 2050 x 1000 5.1e-6 -> 4.9e-8, where fp32 on CUDA
// cores has 1.8e-6 and 6.6e-7.
//
// Few tiles (small matrices, short prompts): the contraction is split over S = 2 or 4 pairs of one cluster, whose
// partial sums meet in the finishing CTA's shared memory (a tile's 32-token blocks go round the S pairs), added in rank
// order: deterministic, no scratch memory.
//
// 14 warps per CTA:   0 TMA producer   1 MMA issuer (even CTA), TMEM allocation   2-5 epilogue   6-13 converters
// (two groups of four: a warp per 32 rows, the groups take alternate chunks).  Every mbarrier wait is bounded; on
// expiry the role records a status code and all roles fall through to the common teardown (TMEM is always released).
#include "common.cuh"
#include "launch_order.cuh"
#include "tma.cuh"
#include "umma.cuh"

#include <atomic>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <type_traits>

namespace t81b200 {

namespace {

constexpr int BM = 128;          // output features per CTA
constexpr int BK = 64;           // operand atom: 64 k = 128 bytes
constexpr int CHUNK = 192;       // columns converted at a time: 3 atoms
constexpr int A_ATOM_BYTES = BM * BK * 2;        // 16 KB
constexpr int A_CHUNK_BYTES = 3 * A_ATOM_BYTES;  // 48 KB
constexpr int A_MAX = 3, B_MAX = 12;             // ring slots that have barriers
constexpr int RAW_STAGES = 3;                    // packed weights of a chunk (128 rows): 8 KB of limbs, 6 KB of codes
// The two groups of converters take alternate chunks, so a slot's uses go from one to the other; the barrier that tells a chunk's arrival is
// one of its group's own three.  With a barrier per slot a group came to one whose use before had been the other's, and a wait that
// tells phases by parity passes at once if that use has not even landed: chunk 0's copy later than chunk 1's by the time chunk 1
// takes to expand (weights whose pages are not in the TLB).  The group then took whatever lay there and handed the slot back once
// too often, and nothing fitted together from there on: waits that ran out, wrong sums, a lost context.  (Four slots are as safe, but cost
// the activation ring a stage: 1463 tokens of 6384 by 3192, bf16, 50.7 and 59.7 us.)
constexpr int RAW_BARRIERS = 2 * RAW_STAGES;
constexpr int MAX_SPLITS = 4;                    // clusters of up to 8 CTAs
constexpr int NUM_THREADS = 14 * 32;
constexpr int EPILOGUE_WARP0 = 2, CONVERTER_WARP0 = 6;
constexpr int OUT_TOKENS = 32;                        // tokens per staged output block (one tcgen05.ld of 32 columns)
constexpr int OUT_STAGE_BYTES = OUT_TOKENS * BM * 2;  // [token][feature] block of a 16-bit output type: 8 KB
constexpr int BARRIER_BYTES = 512;
constexpr int SMEM_LIMIT = 227 * 1024;
template <int FMT> constexpr int kRawBytes = FMT == 1 ? 4 * 1536 : BM * 64;

enum { STATUS_OK = 0, STATUS_TIMEOUT_PRODUCER = 1, STATUS_TIMEOUT_MMA = 2, STATUS_TIMEOUT_EPILOGUE = 3, STATUS_TIMEOUT_CONVERTER = 4 };

__device__ int g_tc_status = 0;

struct TcParams {
    const uint8_t *A;
    const float *row_scale, *bias;
    void *C;
    int64_t c_row_stride, c_tok_stride;  // element strides of C along output features and tokens
    int64_t M, N, kl;
    int tiles32;             // FMT 1: 32-row tiles of the matrix
    int m_tiles, n_tiles;    // 256-row pair tiles, bn-token tiles
    int bn;                  // tokens per tile: a multiple of 32
    int n_atoms, n_chunks;
    int planes, plane_rows;  // activation planes and their row distance in the tensor map
    int b_rows;              // rows of activations that a CTA loads per atom
    int splits;              // pairs of a cluster that share a tile's contraction
    int a_stages, b_stages;
    int out_bytes;           // of staged output blocks beside the rings: two, or none
    int b_step;              // atoms behind one barrier of the activation ring: 1, or 3 (a whole chunk)
    int one_tile;            // no cluster has more than one tile: all warps but the first two finish it
    uint32_t idesc, idesc_rest;  // of the first product, and of the third plane's beside two in one
    uint32_t one_mask;       // FMT 0: bits of bf16 +-1 that stay (all for bf16, 0xBC00 per half for fp16)
    float alpha, beta;
    int n_out_maps;      // > 0: the epilogue stages output blocks in shared memory and stores them by TMA through
                         // this many tensor maps (the local C first, then the peers'); 0: per-element stores
    int n_peers;         // other GPUs that receive a copy of every output element
    void *peer_C[T81B200_MAX_PEERS];  // their C, same strides as the local one
    int c_vec;           // 1: tokens are contiguous in C (the (M, N) argument order) and 16-byte aligned per 32-token block:
                         // a thread's 32 tokens of one feature are one run of memory, moved with 128-bit accesses
};

// Tensor maps of the result, for the TMA-store epilogue: [0] the local C, then one per peer.
struct TcOutMaps {
    CUtensorMap m[1 + T81B200_MAX_PEERS];
};

// AND of a predicate over the 128 epilogue threads (named barrier 2); every one of them must call it.
__device__ __forceinline__ bool epilogue_all(bool pred) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.and.pred p, 2, 128, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"((uint32_t)pred)
        : "memory");
    return r != 0;
}

// Where a 32-token block is staged on its way to a TMA store, and which four warps share it.
struct OutStage {
    uint8_t *gen;      // [32 tokens][128 features] of a 16-bit type
    uint32_t smem;
    uint32_t barrier;  // named barrier of the 128 threads
    bool first;        // this thread issues the store
    bool reused;       // an earlier store may still be reading the buffer
};

// One element a lane and token, 32 features of a token side by side.  One address that moves on: a 64-bit product and a compare per
// element made a block 3500 clocks long, and short contractions twice as long (2444 tokens of 576 by 8064, fp32: 90.9 us, 38.9 now).
// OFTEN: whole blocks without a compare per token; the other forms' kernels go without that code (16-bit results that TMA writes lose 2 %
// to it).  BETA: there may be one.
template <typename CT, bool OFTEN, bool BETA>
__device__ __forceinline__ void store_rows(const TcParams &p, const uint32_t (&v)[32], CT *dst, float scale, float bias, int tokens) {
    auto next = [&](auto *&at) {
        at += p.c_tok_stride;
        asm("" : "+l"(at));  // 32 addresses worked out ahead take registers from the whole kernel
    };
    float y[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) y[i] = __uint_as_float(v[i]) * scale + bias;
    if (BETA && p.beta != 0.0f) {  // the old values are all fetched before the first store (the compiler cannot know the stores to miss them)
        const CT *was = dst;
#pragma unroll
        for (int i = 0; i < 32; ++i, next(was))
            if (i < tokens) y[i] += p.beta * to_float<CT>(*was);
    }
    if (OFTEN && tokens >= 32) {
#pragma unroll
        for (int i = 0; i < 32; ++i, next(dst)) *dst = from_float<CT>(y[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i, next(dst))
            if (i < tokens) *dst = from_float<CT>(y[i]);
    }
}

// One 32-token block of this thread's output feature: scale, bias, beta, store.
// ROWS: a 16-bit token-major C that TMA cannot write, without beta or peers.  A kernel of its own, since every form of the epilogue costs
// the others registers.  Blocks staged in shared memory and written as words took three times as long as storing the elements (1024
// tokens of 768 by 7885, bf16: 27.7 us, 17.6 now; 8192 of 2047 by 2048 57 and 52).
template <typename CT, bool ROWS>
__device__ __forceinline__ void emit_block(const TcParams &p, const TcOutMaps &omaps, const uint32_t (&v)[32], int row0, int64_t row,
                                           float scale, float bias, int tok0, const OutStage &out) {
    const bool row_ok = row < p.M;
    CT *crow = static_cast<CT *>(p.C) + row * p.c_row_stride;
    if constexpr (ROWS) {
        if (row_ok) store_rows<CT, true, false>(p, v, crow + (int64_t)tok0 * p.c_tok_stride, scale, bias, (int)(p.N - tok0));
        return;
    }
    if (p.n_out_maps > 0) {
        // 16-bit output, token-major C: stage [32 tokens][128 features] blocks in shared memory and let
        // TMA write them (whole 256-byte rows; the tensor map clips rows and tokens past the end)
        CT *dst = reinterpret_cast<CT *>(out.gen) + (int)(row - row0);
#pragma unroll
        for (int i = 0; i < 32; ++i) dst[i * BM] = from_float<CT>(__uint_as_float(v[i]) * scale + bias);
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        // two buffers in turn: past this barrier the other one, stored from a block ago, has been read
        if (out.reused && out.first) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        asm volatile("bar.sync %0, 128;" ::"r"(out.barrier) : "memory");
        if (out.first) {
            if (row0 < p.M && tok0 < p.N)
                for (int j = 0; j < p.n_out_maps; ++j) tma_store_2d(&omaps.m[j], out.smem, row0, tok0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    } else if (row_ok && p.c_vec && (int64_t)tok0 + 32 <= p.N) {
        // (M, N) argument order: the thread's 32 tokens are contiguous — whole 16-byte pieces, and with
        // beta the old values are all fetched before the first store
        constexpr int PER = 16 / (int)sizeof(CT);  // elements per 128-bit access
        uint4 *dst = reinterpret_cast<uint4 *>(crow + tok0);
        uint4 old[32 / PER];
        if (p.beta != 0.0f) {
#pragma unroll
            for (int q = 0; q < 32 / PER; ++q) old[q] = dst[q];
        }
#pragma unroll
        for (int q = 0; q < 32 / PER; ++q) {
            CT out[PER];
            const CT *was = reinterpret_cast<const CT *>(&old[q]);
#pragma unroll
            for (int e = 0; e < PER; ++e) {
                float y = __uint_as_float(v[q * PER + e]) * scale + bias;
                if (p.beta != 0.0f) y += p.beta * to_float<CT>(was[e]);
                out[e] = from_float<CT>(y);
            }
            dst[q] = *reinterpret_cast<const uint4 *>(out);
        }
    } else if (row_ok) {
        store_rows<CT, sizeof(CT) == 4, true>(p, v, crow + (int64_t)tok0 * p.c_tok_stride, scale, bias, (int)(p.N - tok0));
        // column-sharded Linear: the same elements go into every peer's result over NVLink
        for (int pj = 0; pj < p.n_peers; ++pj) {
            CT *prow = static_cast<CT *>(p.peer_C[pj]) + row * p.c_row_stride;
#pragma unroll 1  // a rare path: unrolled it costs the whole kernel 40 registers
            for (int i = 0; i < 32; ++i) {
                const int64_t tok = (int64_t)tok0 + i;
                if (tok < p.N) prow[tok * p.c_tok_stride] = crow[tok * p.c_tok_stride];
            }
        }
    }
}

// How the activation planes of a tile meet its weights.
//   ONE    one plane.
//   SIDE   up to 96 tokens: the first two planes side by side are the columns of one product, each CTA loads one of them, and the sums
//          of the second come out beside those of the first; a third plane is a product of its own that adds to the second's.  The
//          weights are read once for both planes, which is what bounds narrow products.
//   APART  128 tokens: a product per plane, the sums 128 columns apart.
//   WIDE   192 to 256, where no pair has a second tile: the same, 256 columns apart.
enum Mode { ONE, SIDE, APART, WIDE };

// 32 columns of a tile's sums; all planes but the first have theirs `rest` columns further.
template <Mode MODE>
__device__ __forceinline__ void load_sums(const TcParams &p, uint32_t taddr, uint32_t (&v)[32]) {
    tmem_ld32(taddr, v);
    if constexpr (MODE != ONE) {
        const uint32_t rest = MODE == SIDE ? (uint32_t)p.bn : (MODE == APART ? 128u : 256u);
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // eight at a time: a whole block beside v costs the kernel spills
            uint32_t small[8];
            tmem_ld8(taddr + rest + (uint32_t)(8 * q), small);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[8 * q + i] = __float_as_uint(__uint_as_float(v[8 * q + i]) + __uint_as_float(small[i]));
        }
    }
}

// One warp's share of a chunk (32 rows x 192 columns), read from the raw ring.
template <int FMT> struct RawChunk;
template <> struct RawChunk<0> { uint4 q[4]; };  // limb (lane % 4) of rows lane / 4 + 8 i
template <> struct RawChunk<1> { uint4 q[3]; };  // the lane's twelve words

template <int FMT>
__device__ __forceinline__ void read_chunk(const TcParams &p, const uint8_t *raw_stage, int rt, int c, int lane, RawChunk<FMT> &raw) {
    if constexpr (FMT == 1) {
        const uint4 *src = reinterpret_cast<const uint4 *>(raw_stage + rt * 1536 + lane * 48);
#pragma unroll
        for (int j = 0; j < 3; ++j) raw.q[j] = src[j];
    } else {
        const bool there = (int64_t)4 * c + (lane & 3) < p.kl;  // past the row's last limb: zero trits
        const uint4 *src = reinterpret_cast<const uint4 *>(raw_stage + rt * 2048) + lane;
#pragma unroll
        for (int i = 0; i < 4; ++i)
            raw.q[i] = there ? src[32 * i] : make_uint4(kZeroTryteWord, kZeroTryteWord, kZeroTryteWord, kZeroTryteWord);
    }
}

// Expands the share into the operand tile at `tile` (this warp's 32 rows of the chunk's first atom): K-major rows of
// 128 bytes, 16-byte piece cc of row r at (cc ^ (r & 7)) * 16.
template <int FMT>
__device__ __forceinline__ void expand_chunk(const RawChunk<FMT> &raw, uint8_t *tile, int lane, uint32_t one_mask) {
    const int g = lane >> 2, t = lane & 3;  // row within a group of 8; 48-column run
    uint32_t off[6];
#pragma unroll
    for (int m = 0; m < 6; ++m) {
        const int piece = 6 * t + m;
        off[m] = (uint32_t)(piece >> 3) * A_ATOM_BYTES + (uint32_t)g * 128u + (uint32_t)(((piece & 7) ^ g) << 4);
    }
    if constexpr (FMT == 1) {
        const uint32_t *w = reinterpret_cast<const uint32_t *>(&raw.q[0]);
#pragma unroll
        for (int gr = 0; gr < 2; ++gr)
#pragma unroll
            for (int m = 0; m < 6; ++m) {
                const uint32_t x = w[6 * gr + m];
                constexpr uint32_t k = 0xC000C000u;
                uint8_t *dst = tile + gr * 2048 + off[m];
                *reinterpret_cast<uint4 *>(dst) = make_uint4(x & k, (x << 4) & k, (x << 8) & k, (x << 12) & k);
                *reinterpret_cast<uint4 *>(dst + 1024) = make_uint4((x << 2) & k, (x << 6) & k, (x << 10) & k, (x << 14) & k);
            }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t o[24], nat[24];
            decode_limb(raw.q[i], o);
            // decode order -> natural order: pairs (trit 2m, trit 2m+1)
#pragma unroll
            for (int pr = 0; pr < 8; ++pr) {
                nat[3 * pr + 0] = __byte_perm(o[3 * pr], o[3 * pr + 1], 0x5410) & one_mask;
                nat[3 * pr + 1] = __byte_perm(o[3 * pr + 2], o[3 * pr], 0x7610) & one_mask;
                nat[3 * pr + 2] = __byte_perm(o[3 * pr + 1], o[3 * pr + 2], 0x7632) & one_mask;
            }
#pragma unroll
            for (int m = 0; m < 6; ++m)
                *reinterpret_cast<uint4 *>(tile + i * 1024 + off[m]) = make_uint4(nat[4 * m], nat[4 * m + 1], nat[4 * m + 2], nat[4 * m + 3]);
        }
    }
}

// ROWS: see emit_block.
template <typename CT, int FMT, Mode MODE, bool ROWS>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_trit_tc_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ TcOutMaps omaps, const __grid_constant__ TcParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *gen_base = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t b_atom_bytes = MODE == SIDE ? (uint32_t)p.b_rows * (BK * 2) : (uint32_t)p.bn * (BK * 2 / 2);  // this CTA's half of the tokens
    const uint32_t b_stage_bytes = b_atom_bytes * (uint32_t)p.b_step;
    const uint32_t b_off = (uint32_t)p.a_stages * A_CHUNK_BYTES;
    const uint32_t raw_off = b_off + (uint32_t)p.b_stages * b_stage_bytes;
    const uint32_t out_off = raw_off + RAW_STAGES * kRawBytes<FMT>;
    const uint32_t bars = base + out_off + (uint32_t)p.out_bytes;
    auto a_full = [&](int s) { return bars + 8u * s; };
    auto a_empty = [&](int s) { return bars + 8u * (A_MAX + s); };
    auto b_full = [&](int s) { return bars + 8u * (2 * A_MAX + s); };
    auto b_empty = [&](int s) { return bars + 8u * (2 * A_MAX + B_MAX + s); };
    auto acc_full = [&](int s) { return bars + 8u * (2 * A_MAX + 2 * B_MAX + s); };
    auto acc_empty = [&](int s) { return bars + 8u * (2 * A_MAX + 2 * B_MAX + 2 + s); };
    auto raw_full = [&](int s) { return bars + 8u * (2 * A_MAX + 2 * B_MAX + 4 + s); };
    auto raw_empty = [&](int s) { return bars + 8u * (2 * A_MAX + 2 * B_MAX + 4 + RAW_BARRIERS + s); };
    const uint32_t tmem_slot = bars + 8u * (2 * A_MAX + 2 * B_MAX + 4 + RAW_BARRIERS + RAW_STAGES);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int half = (int)(rank & 1u), slice = (int)(rank >> 1);

    if (threadIdx.x == 0) {
        for (int s = 0; s < A_MAX; ++s) { mbar_init(a_full(s), 8); mbar_init(a_empty(s), 1); }
        for (int s = 0; s < B_MAX; ++s) { mbar_init(b_full(s), 1); mbar_init(b_empty(s), 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(acc_full(s), 1); mbar_init(acc_empty(s), 8); }
        for (int s = 0; s < RAW_BARRIERS; ++s) mbar_init(raw_full(s), 1);
        for (int s = 0; s < RAW_STAGES; ++s) mbar_init(raw_empty(s), 4);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();  // barriers initialised (this CTA)
    const int total_tiles = p.m_tiles * p.n_tiles;
    const int n_clusters = (int)gridDim.x / (2 * p.splits), cluster_id = (int)blockIdx.x / (2 * p.splits);
    // this pair's share of the contraction, in chunks
    const int c0 = p.n_chunks * slice / p.splits, c1 = p.n_chunks * (slice + 1) / p.splits;
    const uint16_t pair_mask = (uint16_t)(3u << (rank & ~1u));

    // The producer's weight loads run two chunks ahead of the activations; the first two start right behind the wait for the kernel ahead,
    // for which the cluster has met already.
    Ring raw_fill, raw_told;
    bool fill_ok = true;
    int raw_tile = cluster_id, raw_c = c0;
    auto load_raw = [&]() {
        if (raw_tile >= total_tiles || !fill_ok) return;
        fill_ok = mbar_wait(raw_empty(raw_fill.stage), raw_fill.phase ^ 1);
        if (!fill_ok) return;
        const int row0 = ((raw_tile % p.m_tiles) * 2 + half) * BM;
        const uint32_t dst = base + raw_off + (uint32_t)raw_fill.stage * (uint32_t)kRawBytes<FMT>, bar = raw_full(raw_told.stage);
        if (elect_one()) {
            if constexpr (FMT == 1) {
                // the row tiles of a chunk are contiguous; past the matrix's last one nothing is loaded (those rows
                // of the result are not stored)
                int n = p.tiles32 - (row0 >> 5);
                n = n < 0 ? 0 : (n > 4 ? 4 : n);
                if (n > 0) {
                    mbar_arrive_expect_tx(bar, (uint32_t)n * 1536u);
                    bulk_load(dst, p.A + ((int64_t)raw_c * p.tiles32 + (row0 >> 5)) * 1536, (uint32_t)n * 1536u, bar);
                } else mbar_arrive(bar);
            } else {
                mbar_arrive_expect_tx(bar, (uint32_t)kRawBytes<FMT>);
                tma_load_2d(dst, &map_w, raw_c * 64, row0, bar);
            }
        }
        __syncwarp();
        raw_fill.advance(RAW_STAGES);
        raw_told.advance(RAW_BARRIERS);
        if (++raw_c >= c1) { raw_c = c0; raw_tile += n_clusters; }
    };

    // Launched with programmatic stream serialization: what touches no global memory overlaps the tail of the previous kernel, the tensor
    // maps, the accumulators' allocation and the meeting of the cluster among it (us, with the meeting behind the wait and before it: 51
    // tokens of 2592 by 624, bf16, 9.7 and 8.9, 80 of 4096 by 14336 19.2 and 19.1, 777 of 3001 by 1999, fp32, 22.3 and 22.0).  All
    // threads wait here: no bounded wait of another role runs out while the kernel ahead takes its time.
    if (threadIdx.x == 0) {
        prefetch_map(&map_x);
        if (FMT == 0) prefetch_map(&map_w);
        if (p.n_out_maps > 0) prefetch_map(&omaps.m[0]);
    }
    if (warp == 1) tmem_alloc_pair(tmem_slot);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();  // the other CTAs' barriers are initialised before anything arrives on them
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (warp == 0) {
        load_raw();
        load_raw();
    }
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(gen_base + (tmem_slot - base));
    // scale and bias of this thread's output row, fetched long before the epilogue (a microsecond from HBM)
    auto row_scale = [&](int64_t row) { return (row < p.M && p.row_scale ? __ldg(p.row_scale + row) : 1.0f) * p.alpha; };
    auto row_bias = [&](int64_t row) { return row < p.M && p.bias ? __ldg(p.bias + row) : 0.0f; };
    const int own_row = ((cluster_id % p.m_tiles) * 2 + half) * BM + (warp & 3) * 32 + lane;
    const float own_scale = p.one_tile ? row_scale(own_row) : 0.0f, own_bias = p.one_tile ? row_bias(own_row) : 0.0f;

    if (warp == 0) {
        // ---------------- TMA producer: this CTA's packed weights and its half of the activation rows ----------------
        Ring b;
        bool ok = fill_ok;
        for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
            const int row = (tile / p.m_tiles) * p.bn + (MODE == SIDE ? half * p.plane_rows : half * (p.bn / 2));
            for (int c = c0; c < c1 && ok; ++c) {
                load_raw();
                ok = fill_ok;
                const int a_end = 3 * c + 3 < p.n_atoms ? 3 * c + 3 : p.n_atoms;
                for (int a0 = 3 * c; a0 < a_end && ok; a0 += p.b_step) {
                    const int a1 = a0 + p.b_step < a_end ? a0 + p.b_step : a_end;
                    for (int pl = 0; pl < (MODE == APART || MODE == WIDE ? p.planes : 1); ++pl) {
                        ok = mbar_wait(b_empty(b.stage), b.phase ^ 1);
                        if (!ok) break;
                        if (elect_one()) {
                            if (half == 0) mbar_arrive_expect_tx(b_full(b.stage), 2 * (uint32_t)(a1 - a0) * b_atom_bytes);
                            uint32_t dst = base + b_off + (uint32_t)b.stage * b_stage_bytes;
                            for (int a = a0; a < a1; ++a, dst += b_atom_bytes) {
                                tma_load_2d_pair(dst, &map_x, a * BK, pl * p.plane_rows + row, b_full(b.stage));
                                if (MODE == SIDE && p.planes == 3) {  // boxes of half a tile: the rest of this CTA's plane, and half of the third
                                    const uint32_t half_bytes = (uint32_t)p.bn * (BK * 2 / 2);
                                    tma_load_2d_pair(dst + half_bytes, &map_x, a * BK, row + p.bn / 2, b_full(b.stage));
                                    tma_load_2d_pair(dst + 2 * half_bytes, &map_x, a * BK, 2 * p.plane_rows + (tile / p.m_tiles) * p.bn + half * (p.bn / 2), b_full(b.stage));
                                }
                            }
                        }
                        __syncwarp();
                        b.advance(p.b_stages);
                    }
                }
            }
        }
        // The last commits' arrivals come from the pair's issuing CTA, one by one; this CTA may not end before they have landed.
        for (int i = 0; i < p.b_stages && ok; ++i) {
            ok = mbar_wait(b_empty(b.stage), b.phase ^ 1);
            b.advance(p.b_stages);
        }
        const int fills = cluster_id < total_tiles ? ((total_tiles - 1 - cluster_id) / n_clusters + 1) * (c1 - c0) : 0;
        for (int i = fills; i < fills + p.a_stages && ok; ++i) ok = mbar_wait(a_empty(i % p.a_stages), ((uint32_t)(i / p.a_stages) & 1u) ^ 1u);
        if (!ok) give_up(&g_tc_status, STATUS_TIMEOUT_PRODUCER);
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (half == 0) {
            Ring a, b;
            bool ok = true;
            int it = 0;
            for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters, ++it) {
                const int buf = it & 1;
                ok = mbar_wait(acc_empty(buf), ((uint32_t)(it >> 1) & 1u) ^ 1u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tile = tmem_base + (uint32_t)buf * 256u;
                for (int c = c0; c < c1 && ok; ++c) {
                    ok = mbar_wait(a_full(a.stage), a.phase);
                    if (!ok) break;
                    const int atoms = p.n_atoms - 3 * c < 3 ? p.n_atoms - 3 * c : 3;
                    const uint32_t a_base = base + (uint32_t)a.stage * A_CHUNK_BYTES;
                    for (int j0 = 0; j0 < atoms && ok; j0 += p.b_step) {
                        const int j1 = j0 + p.b_step < atoms ? j0 + p.b_step : atoms;
                        for (int pl = 0; pl < (MODE == APART || MODE == WIDE ? p.planes : 1); ++pl) {
                            ok = mbar_wait(b_full(b.stage), b.phase);
                            if (!ok) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                            const uint32_t d_tmem = d_tile + (pl > 0 ? (MODE == APART ? 128u : 256u) : 0u);
                            const uint32_t accumulate = c > c0 || j0 > 0 || pl > 1 ? 1u : 0u;
                            if (elect_one()) {
                                uint64_t bd = umma_desc_k(base + b_off + (uint32_t)b.stage * b_stage_bytes);
                                uint64_t ad = umma_desc_k(a_base + (uint32_t)j0 * A_ATOM_BYTES);
                                for (int j = j0; j < j1; ++j, ad += A_ATOM_BYTES >> 4, bd += b_atom_bytes >> 4) {
#pragma unroll
                                    for (int k = 0; k < BK / 16; ++k)
                                        umma_pair(d_tmem, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), p.idesc, k == 0 && j == j0 ? accumulate : 1u);
                                }
                                if (MODE == SIDE && p.planes == 3) {
                                    bd = umma_desc_k(base + b_off + (uint32_t)b.stage * b_stage_bytes + (uint32_t)p.bn * (BK * 2));
                                    ad = umma_desc_k(a_base + (uint32_t)j0 * A_ATOM_BYTES);
                                    for (int j = j0; j < j1; ++j, ad += A_ATOM_BYTES >> 4, bd += b_atom_bytes >> 4) {
#pragma unroll
                                        for (int k = 0; k < BK / 16; ++k)
                                            umma_pair(d_tile + (uint32_t)p.bn, ad + (uint64_t)(2 * k), bd + (uint64_t)(2 * k), p.idesc_rest, 1u);
                                    }
                                }
                                umma_commit_pair(b_empty(b.stage), pair_mask);
                            }
                            __syncwarp();
                            b.advance(p.b_stages);
                        }
                    }
                    if (!ok) break;
                    if (elect_one()) umma_commit_pair(a_empty(a.stage), pair_mask);
                    __syncwarp();
                    a.advance(p.a_stages);
                }
                if (ok && elect_one()) umma_commit_pair(acc_full(buf), pair_mask);
                __syncwarp();
            }
            if (!ok) give_up(&g_tc_status, STATUS_TIMEOUT_MMA);
        }
    } else if (warp < CONVERTER_WARP0) {
        // ---------------- epilogue of all but one-tile launches, which are finished below ----------------
        const int quarter = warp & 3;  // TMEM lanes 32 * quarter .. + 31 are this warp's
        bool ok = true;
        int it = 0, out_count = 0;
        for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters, ++it) {
            const int buf = it & 1;
            // One decision for all four epilogue warps (tcgen05.ld is .aligned, and the staging path meets at named
            // barriers): every thread's bounded wait returns, then the 128 threads agree.
            const int row0 = ((tile % p.m_tiles) * 2 + half) * BM, n0 = (tile / p.m_tiles) * p.bn;
            const int64_t row = (int64_t)row0 + quarter * 32 + lane;
            const float scale = p.one_tile ? 0.0f : row_scale(row), bias = p.one_tile ? 0.0f : row_bias(row);
            ok = epilogue_all(mbar_wait(acc_full(buf), (uint32_t)(it >> 1) & 1u));
            if (!ok) break;
            if (p.one_tile) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
            for (int c = 0; c < p.bn / 32; ++c) {
                uint32_t v[32];
                load_sums<MODE>(p, tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(buf * 256 + c * 32), v);
                const uint32_t stage = out_off + (uint32_t)(out_count++ & 1) * OUT_STAGE_BYTES;
                emit_block<CT, ROWS>(p, omaps, v, row0, row, scale, bias, n0 + c * 32,
                               OutStage{gen_base + stage, base + stage, 2, threadIdx.x == EPILOGUE_WARP0 * 32, true});
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(acc_empty(buf));
        }
        if (!ok) give_up(&g_tc_status, STATUS_TIMEOUT_EPILOGUE);
    } else {
        // ---------------- converters ----------------
        const int rt = (warp - CONVERTER_WARP0) & 3, group = (warp - CONVERTER_WARP0) >> 2;
        const int span = c1 - c0, my_tiles = cluster_id < total_tiles ? (total_tiles - 1 - cluster_id) / n_clusters + 1 : 0;
        Ring a, raw;
        if (group == 1) { a.advance(p.a_stages); raw.advance(RAW_BARRIERS); }
        bool ok = true;
        // The groups take alternate chunks of the CTA's whole sequence.  Slots of the operand ring change hands where there are three: there a
        // group waits for the MMAs of the slot's last chunk, k - 3.  It has seen those of k - 5 end when it took its own last chunk, and MMAs
        // end in order, so those of k - 6, the slot's use before, have ended too, and the wait cannot be a whole use behind.
        int c = c0 + group;
        for (int left = my_tiles * span - group; left > 0; left -= 2) {
            while (c >= c1) c -= span;
            ok = __all_sync(0xffffffffu, mbar_wait(raw_full(raw.stage), raw.phase));
            if (!ok) break;
            RawChunk<FMT> words;
            const int slot = raw.stage < RAW_STAGES ? raw.stage : raw.stage - RAW_STAGES;
            read_chunk<FMT>(p, gen_base + raw_off + slot * kRawBytes<FMT>, rt, c, lane, words);
            __syncwarp();
            if (lane == 0) mbar_arrive(raw_empty(slot));
            ok = __all_sync(0xffffffffu, mbar_wait(a_empty(a.stage), a.phase ^ 1));
            if (!ok) break;
            expand_chunk<FMT>(words, gen_base + a.stage * A_CHUNK_BYTES + rt * 4096, lane, p.one_mask);
            // generic-proxy writes must be visible to the tensor core's async proxy
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(a_full(a.stage));
            a.advance(p.a_stages);
            a.advance(p.a_stages);
            raw.advance(RAW_BARRIERS);
            raw.advance(RAW_BARRIERS);
            c += 2;
        }
        if (!ok) give_up(&g_tc_status, STATUS_TIMEOUT_CONVERTER);
    }
    __syncwarp();

    if (p.one_tile) {
        // Three groups of four warps take the tile's 32-token blocks in turn; what they stage goes into the activation
        // ring, idle by now.  With splits > 1 the pairs of the cluster hold partial sums: block b is finished by slice
        // b % splits, the others write theirs into its shared memory first (the weight ring, idle once every CTA of
        // the cluster has its last MMA behind it).
        const int group = (warp - EPILOGUE_WARP0) >> 2, quarter = warp & 3, S = p.splits, blocks = p.bn / 32;
        const int row0 = ((cluster_id % p.m_tiles) * 2 + half) * BM, n0 = (cluster_id / p.m_tiles) * p.bn;
        const uint32_t lane_row = (uint32_t)(quarter * 32 + lane);
        const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
        __syncthreads();
        if (S > 1) cluster_barrier();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (S > 1) {
            if (warp >= EPILOGUE_WARP0)
                for (int b = group; b < blocks; b += 3) {
                    const int to = b % S;
                    if (to == slice) continue;
                    uint32_t v[32];
                    load_sums<MODE>(p, t_lane + (uint32_t)(b * 32), v);
                    push_partial(v, base + partial_slot(b, S, slice, to) * 16384u + lane_row * 4u, (uint32_t)(2 * to + half));
                }
            __syncthreads();
            cluster_barrier();
        }
        if (warp >= EPILOGUE_WARP0) {
            const bool first = quarter == 2 && lane == 0;
            for (int b = slice + S * group; b < blocks; b += 3 * S) {
                uint32_t v[32];
                load_sums<MODE>(p, t_lane + (uint32_t)(b * 32), v);
                if (S > 1) fold_partials(v, gen_base, b, S, slice, lane_row);
                const uint32_t stage = b_off + (uint32_t)b * OUT_STAGE_BYTES;
                emit_block<CT, ROWS>(p, omaps, v, row0, own_row, own_scale, own_bias, n0 + b * 32, OutStage{gen_base + stage, base + stage, (uint32_t)(2 + group), first, false});
            }
            if (first) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
        }
    } else if (threadIdx.x == EPILOGUE_WARP0 * 32) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every store has completed

    // ---------------- teardown: no CTA leaves while its peer may still arrive on its barriers or read its operands
    // (the producers have seen every commit) ----
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_free_pair(tmem_base);
    }
}

// Everything a launch needs to know about the sizes.
struct TcShape {
    Mode mode = ONE;
    int bn = 0, n_tiles = 0, splits = 1, a_stages = 2, b_stages = 2, b_step = 1, b_rows = 0, out_bytes = 0;
    size_t smem = 0;
    double cost = 0.0;  // pick_shape's estimate, in units of 1.7 ns
};

// Time of a 64-deep step of one product of n columns, in units of 1.7 ns, measured in tiles of 24 to 96 steps, one and three to a pair:
// up to 160 columns it is the weights' own time, through shared memory and out of it again.
double product_cost(int n) {
    constexpr double cost[8] = {115, 119, 122, 125, 130, 153, 169, 187};  // 32, 64, .. 256 columns
    return cost[n / 32 - 1];
}
Mode mode_of(int bn, int planes) { return planes == 1 ? ONE : (bn <= 96 ? SIDE : (bn <= 128 ? APART : WIDE)); }
// The same of a step of all planes.  Products of 128 tokens apart take turns without a gap; side by side, at 256 columns, they took
// 420 ns a step, since two stages are all that fits (1500 tokens of 9000 by 1200, fp32: 75 and 82 us).
double step_cost(Mode mode, int bn, int planes) {
    if (mode == ONE) return product_cost(bn);
    if (mode == APART) return planes * 98.0;
    if (mode == WIDE) return planes * product_cost(bn);
    return product_cost(2 * bn) + (planes == 3 ? product_cost(bn) : 0.0);
}

// Planes side by side against apart, at the width that each form is best at (us, fp32): 777 tokens of 3001 by 1999 26.9 -> 22.8, 300
// of 1000 by 9000 21.5 -> 17.0, 64 of 4096 by 14336 25.7 -> 21.8, 17 of 4096 by 4096 15.1 -> 13.9.
//
// Tile width and split: the smallest estimate, in step_cost's units.  Fitted to every width and split of 50 shapes from
// 512 x 528 x 256 to 14336 x 4096 x 4096: the steps; a tile 400 more; writing the last tiles out, 3 a token; sharing partial sums 1300
// and 3 a token (the steps' costs refitted since: 900 tokens of 3000 by 5000, bf16, 34.3 -> 26.2 us, 400 of 6000 by 3000 25.3 -> 23.4, 200 of 2000
// by 2000, fp32, 13.7 -> 12.8; 27 others as they were).  Several planes take two accumulators a tile, so tiles that follow one another in a pair are at most
// 128 tokens wide there (4096 x 4096 x 4096 in two planes 202 us, 208 at 256 tokens with one accumulator); wider ones only where
// no pair has a second tile (5530 x 11021 x 249: 83 us at 128 tokens, 66 at 256).  The widths between 128 and 192 are left out for several
// planes: tiles that follow one another have no room for the second accumulator there, and tiles alone have not been measured.
TcShape pick_shape(int64_t M, int64_t N, int64_t K, int planes, int raw_bytes, bool staged) {
    const int64_t m_tiles = (M + 255) / 256, chunks = (K + CHUNK - 1) / CHUNK, wide = (N + 255) / 256, narrow = (N + 127) / 128;
    const int64_t least = planes > 1 && wide > resident_pair_clusters(1) ? narrow : wide, most = (planes > 1 ? narrow : wide) + 8;
    TcShape best;
    double best_t = 1e30;
    for (int64_t want = least; want <= most && want <= (N + 31) / 32; ++want) {
        const int bn = (int)(((N + want - 1) / want + 31) / 32 * 32);
        const int64_t n_tiles = (N + bn - 1) / bn, tiles = m_tiles * n_tiles;
        for (int s = 1; s <= MAX_SPLITS; ++s) {
            const int resident = resident_pair_clusters(s);
            if (s > chunks || (s > 1 && tiles > resident)) continue;
            if (planes > 1 && bn > 128 && (bn < 192 || tiles > resident)) continue;
            const double atom = step_cost(mode_of(bn, planes), bn, planes);
            const double t = (double)((tiles + resident - 1) / resident) * (3.0 * (double)((chunks + s - 1) / s) * atom + 400.0) +
                             3.0 * bn + (s > 1 ? 1300.0 + 3.0 * bn : 0.0);
            if (t < best_t) { best_t = t; best.bn = bn; best.n_tiles = (int)n_tiles; best.splits = s; }
        }
    }
    best.cost = best_t;
    const bool alone = best.splits > 1 || m_tiles * best.n_tiles <= resident_pair_clusters(1);
    best.mode = mode_of(best.bn, planes);
    const int columns = best.mode == SIDE ? 2 * best.bn : best.bn;
    best.b_rows = (columns + (best.mode == SIDE && planes == 3 ? best.bn : 0)) / 2;
    best.a_stages = columns <= 96 ? 3 : 2;
    const int atom = best.b_rows * BK * 2;
    // Output blocks are staged beside the rings only where tiles follow one another and TMA writes them; what is left goes to the
    // activation ring (4096 tokens of 4096 by 4096, fp32: 191 -> 183 us with a fourth stage, 500 in bf16 20.6 -> 19.4).
    best.out_bytes = staged && !alone ? 2 * OUT_STAGE_BYTES : 0;
    const int fixed = RAW_STAGES * raw_bytes + best.out_bytes + BARRIER_BYTES + 1024, room = SMEM_LIMIT - fixed - best.a_stages * A_CHUNK_BYTES;
    // One barrier per chunk instead of one per step where two stages of a chunk fit (up to 224 columns) and the planes do not fill the time
    // between two barriers anyway (wide ones do better with a deeper ring: 200 against 220 us at 4096 x 4096 x 4096, fp32, 192
    // tokens).  With one plane: 192 tokens 408 -> 314 us at 14336 x 4096 x 4096; 256 columns in two stages 76 -> 81 at 9216 x 3072 x 2048.
    best.b_step = best.mode != WIDE && best.bn <= 224 && room >= 6 * atom ? 3 : 1;
    const int stage = atom * best.b_step, b = room / stage;
    best.b_stages = b > B_MAX ? B_MAX : b;
    best.smem = (size_t)best.a_stages * A_CHUNK_BYTES + (size_t)best.b_stages * stage + fixed;
    return best;
}

template <typename CT, int FMT, Mode MODE, bool ROWS>
int launch_tc(const TcShape &shape, const CUtensorMap &mw, const CUtensorMap &mx, const TcOutMaps &om, const TcParams &p, cudaStream_t st) {
    auto kern = gemm_trit_tc_kernel<CT, FMT, MODE, ROWS>;
    // the shared-memory limit is a per-device attribute of the function: set it once on every device
    static std::atomic<bool> configured[64];
    int dev = 0;
    T81_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
        T81_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
    }
    const int tiles = p.m_tiles * p.n_tiles;
    const int clusters = p.one_tile ? tiles : resident_pair_clusters(1);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * 2 * p.splits), 1, 1);
    cfg.blockDim = dim3(NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = shape.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(2 * p.splits);
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    T81_CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, mw, mx, om, p));
    return T81B200_OK;
}

template <int FMT, Mode MODE>
int launch_tc_ct(int c_dtype, bool rows, const TcShape &shape, const CUtensorMap &mw, const CUtensorMap &mx, const TcOutMaps &om, const TcParams &p, cudaStream_t st) {
    switch (c_dtype) {
        case T81B200_F32: return launch_tc<float, FMT, MODE, false>(shape, mw, mx, om, p, st);
        case T81B200_BF16: return rows ? launch_tc<__nv_bfloat16, FMT, MODE, true>(shape, mw, mx, om, p, st) : launch_tc<__nv_bfloat16, FMT, MODE, false>(shape, mw, mx, om, p, st);
        case T81B200_F16: return rows ? launch_tc<__half, FMT, MODE, true>(shape, mw, mx, om, p, st) : launch_tc<__half, FMT, MODE, false>(shape, mw, mx, om, p, st);
    }
    return fail(T81B200_EINVAL, "gemm_trit: unknown output dtype %d", c_dtype);
}

// Pre-pass for activations TMA cannot read in place: token-major rows of kpad elements in scratch memory.  16-bit
// values are copied bit for bit; fp32 values become PLANES bf16 planes, plane i = bf16(x - planes before it).
// Bound by memory: every element is read once and written once (PLANES x 2 bytes).
// An infinity is the first plane's alone (what is left of it is no number), and a value that would round to one is
// the largest bf16 number and the rest.
__device__ __forceinline__ float plane_of(float r) { return isinf(r) ? r : fminf(fmaxf(r, -3.38953139e38f), 3.38953139e38f); }
__device__ __forceinline__ float rest_of(float r, float plane) { return isinf(plane) ? 0.0f : r - plane; }

template <int PLANES>
__device__ __forceinline__ void store_planes(const float (&v)[4], __nv_bfloat16 *out, int64_t plane_elems) {
    __nv_bfloat162 a = __floats2bfloat162_rn(plane_of(v[0]), plane_of(v[1])), b = __floats2bfloat162_rn(plane_of(v[2]), plane_of(v[3]));
    *reinterpret_cast<uint2 *>(out) = make_uint2(bf162_bits(a), bf162_bits(b));
    float r[4] = {rest_of(v[0], __low2float(a)), rest_of(v[1], __high2float(a)), rest_of(v[2], __low2float(b)), rest_of(v[3], __high2float(b))};
#pragma unroll
    for (int pl = 1; pl < PLANES; ++pl) {  // finite from here on
        a = __floats2bfloat162_rn(r[0], r[1]);
        b = __floats2bfloat162_rn(r[2], r[3]);
        *reinterpret_cast<uint2 *>(out + pl * plane_elems) = make_uint2(bf162_bits(a), bf162_bits(b));
        r[0] -= __low2float(a); r[1] -= __high2float(a); r[2] -= __low2float(b); r[3] -= __high2float(b);
    }
}

// (N, K) layout: a thread moves WIDTH consecutive k of one token; whole 16- / 8-byte loads where the rows allow them.  Four, and eight
// of much 16-bit data: there rows elsewhere are read in words, which lie one element off those of the result where a row starts
// between two of them (8192 tokens of 2047: 17.5 us element by element, 13.4 so); no word reaches past the row.
template <typename T, int PLANES, int WIDTH>
__global__ void __launch_bounds__(256) stage_rows_kernel(const T *__restrict__ B, int64_t ldb, int64_t N, int64_t K, __nv_bfloat16 *__restrict__ out,
                                                         int64_t kpad, int64_t plane_elems, bool vec, bool release) {
    wait_for_kernel_ahead(release);
    const int64_t n = (int64_t)blockIdx.x * blockDim.y + threadIdx.y, k = ((int64_t)blockIdx.y * blockDim.x + threadIdx.x) * WIDTH;
    if (n >= N || k >= kpad) return;
    const T *src = B + n * ldb + k;
    __nv_bfloat16 *dst = out + n * kpad + k;
    if constexpr (PLANES == 0 && WIDTH == 4) {  // bit copy of a 16-bit type
        uint16_t e[4] = {0, 0, 0, 0};
        const uint16_t *s16 = reinterpret_cast<const uint16_t *>(src);
        if (vec && k + 4 <= K) *reinterpret_cast<uint2 *>(e) = *reinterpret_cast<const uint2 *>(src);
        else
#pragma unroll
            for (int i = 0; i < 4; ++i) if (k + i < K) e[i] = s16[i];
        *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(e);
    } else if constexpr (PLANES == 0) {
        const uint16_t *s16 = reinterpret_cast<const uint16_t *>(src);
        uint32_t w[4] = {0u, 0u, 0u, 0u};
        if (k + 8 > K) {
#pragma unroll
            for (int i = 0; i < 8; ++i)
                if (k + i < K) w[i >> 1] |= (uint32_t)s16[i] << (16 * (i & 1));
        } else if (vec) {
            const uint2 a = reinterpret_cast<const uint2 *>(src)[0], b = reinterpret_cast<const uint2 *>(src)[1];
            w[0] = a.x; w[1] = a.y; w[2] = b.x; w[3] = b.y;
        } else if (reinterpret_cast<uintptr_t>(src) % 4 == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = reinterpret_cast<const uint32_t *>(src)[i];
        } else {
            const uint32_t first = s16[0], last = s16[7];
            uint32_t mid[3];
#pragma unroll
            for (int i = 0; i < 3; ++i) mid[i] = reinterpret_cast<const uint32_t *>(s16 + 1)[i];
            w[0] = __byte_perm(first, mid[0], 0x5410);
            w[1] = __byte_perm(mid[0], mid[1], 0x5432);
            w[2] = __byte_perm(mid[1], mid[2], 0x5432);
            w[3] = __byte_perm(mid[2], last, 0x5432);
        }
        *reinterpret_cast<uint4 *>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
    } else {
        float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        if (vec && k + 4 <= K) *reinterpret_cast<float4 *>(v) = *reinterpret_cast<const float4 *>(src);
        else
#pragma unroll
            for (int i = 0; i < 4; ++i) if (k + i < K) v[i] = to_float<T>(src[i]);
        store_planes<PLANES>(v, dst, plane_elems);
    }
}

// (K, N) layout: 64 k x 32 n tiles through shared memory, so that the reads (along n) and the writes (along k) coalesce.
template <typename T, int PLANES>
__global__ void __launch_bounds__(256) stage_columns_kernel(const T *__restrict__ B, int64_t ldb, int64_t N, int64_t K, __nv_bfloat16 *__restrict__ out,
                                                            int64_t kpad, int64_t plane_elems) {
    __shared__ T tile[32][65];
    wait_for_kernel_ahead();
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
    const int64_t n0 = (int64_t)blockIdx.x * 32, k0 = (int64_t)blockIdx.y * 64;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int64_t k = k0 + ty + 8 * i, n = n0 + tx;
        tile[tx][ty + 8 * i] = n < N && k < K ? B[k * ldb + n] : from_float<T>(0.0f);
    }
    __syncthreads();
    const int kq = (threadIdx.x & 15) * 4;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int a = (threadIdx.x >> 4) + 16 * i;
        const int64_t n = n0 + a, k = k0 + kq;
        if (n >= N || k >= kpad) continue;
        __nv_bfloat16 *dst = out + n * kpad + k;
        if constexpr (PLANES == 0) {
            T e[4] = {tile[a][kq], tile[a][kq + 1], tile[a][kq + 2], tile[a][kq + 3]};
            *reinterpret_cast<uint2 *>(dst) = *reinterpret_cast<const uint2 *>(e);
        } else {
            const float v[4] = {to_float<T>(tile[a][kq]), to_float<T>(tile[a][kq + 1]), to_float<T>(tile[a][kq + 2]), to_float<T>(tile[a][kq + 3])};
            store_planes<PLANES>(v, dst, plane_elems);
        }
    }
}

template <typename T, int PLANES>
int launch_stage(const void *B, int layout, int64_t ldb, int64_t N, int64_t K, __nv_bfloat16 *out, int64_t kpad, cudaStream_t st) {
    const T *src = static_cast<const T *>(B);
    const int64_t plane_elems = N * kpad;
    if (layout == T81B200_LAYOUT_KN) {
        const dim3 grid((unsigned)((N + 31) / 32), (unsigned)((kpad + 63) / 64));
        if (grid.y > 65535u) return fail(T81B200_ELIMIT, "gemm_trit: K too large");
        T81_CUDA_TRY(launch_behind(stage_columns_kernel<T, PLANES>, grid, 256, 0, st, src, ldb, N, K, out, kpad, plane_elems));
    } else {
        const bool vec = reinterpret_cast<uintptr_t>(B) % (4 * sizeof(T)) == 0 && ldb % 4 == 0;
        // The product's CTAs wait beside this pass, or come as its blocks end.  The first is up to 3 % faster, except for many tokens of
        // contractions up to four chunks, whose tiles then load and store all at once (fp32, 600 features, us, released early and
        // late: 6000 tokens of 513 27.3 and 25.3, 9000 of 600 46.0 and 43.0).
        const bool release = K > 768 || N < 2000;
        auto launch = [&](auto width) -> int {
            constexpr int W = decltype(width)::value;
            // a row's pieces side by side, and as many rows of few pieces as 256 threads take
            const int64_t pieces = (kpad + W - 1) / W, across = pieces < 256 ? (pieces + 31) / 32 * 32 : 256;
            const dim3 block((unsigned)across, (unsigned)(256 / across)), grid((unsigned)((N + block.y - 1) / block.y), (unsigned)((pieces + 255) / 256));
            if (grid.y > 65535u) return fail(T81B200_ELIMIT, "gemm_trit: K too large");
            T81_CUDA_TRY(launch_behind(stage_rows_kernel<T, PLANES, W>, grid, block, 0, st, src, ldb, N, K, out, kpad, plane_elems, vec, release));
            return T81B200_OK;
        };
        // Eight k a thread are half the loads in flight and no shorter a chain, so up to 1.5 million elements four are faster, or up to a
        // third of that where four leave more than a tenth of the lanes idle (whole products, us, eight and four: 1000 tokens of 1023 by
        // 2048 features 13.36 and 12.78, 200 of 4095 by 4096 18.89 and 17.99, 3000 of 513 by 600 12.20 and 13.78).
        if constexpr (PLANES == 0) {
            const int64_t pieces = (kpad + 3) / 4, lanes = pieces < 256 ? (pieces + 31) / 32 * 32 : (pieces + 255) / 256 * 256;
            if (plane_elems > (10 * pieces >= 9 * lanes ? 3 << 19 : 1 << 19)) return launch(std::integral_constant<int, 8>{});
        }
        return launch(std::integral_constant<int, 4>{});
    }
    return T81B200_OK;
}

// 16-bit token-major rows that TMA can read where they are.
bool reads_in_place(const void *B, int b_dtype, int layout, int64_t ldb) {
    return b_dtype != T81B200_F32 && layout == T81B200_LAYOUT_NK && reinterpret_cast<uintptr_t>(B) % 16 == 0 && (ldb * 2) % 16 == 0;
}

int64_t scratch_row(int64_t K) { return (K + 7) & ~(int64_t)7; }

}  // namespace

int resident_pair_clusters(int splits) {
    static std::atomic<int> known[64][MAX_SPLITS + 1];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return sm_count() / (2 * splits + 1);
    int n = known[dev][splits].load(std::memory_order_relaxed);
    if (n > 0) return n;
    auto kern = gemm_trit_tc_kernel<__nv_bfloat16, 1, ONE, false>;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(2 * splits), 1, 1);
    cfg.blockDim = dim3(NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = SMEM_LIMIT;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.x = (unsigned)(2 * splits);
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
        (void)cudaGetLastError();
        n = sm_count() / (2 * splits + 1);
    }
    known[dev][splits].store(n, std::memory_order_relaxed);
    return n;
}

int stage_planes(const void *B, int dtype, int layout, int64_t ld, int64_t tokens, int64_t K, int planes, void *scratch, cudaStream_t st) {
    __nv_bfloat16 *out = static_cast<__nv_bfloat16 *>(scratch);
    const int64_t kpad = scratch_row(K);
    if (dtype != T81B200_F32) return launch_stage<__nv_bfloat16, 0>(B, layout, ld, tokens, K, out, kpad, st);
    return planes == 3 ? launch_stage<float, 3>(B, layout, ld, tokens, K, out, kpad, st) : launch_stage<float, 2>(B, layout, ld, tokens, K, out, kpad, st);
}

bool gemm_trit_tc_eligible(int64_t M, int64_t N, int64_t K) {
    return M >= 1 && N >= 1 && K >= 1 && M < (1ll << 31) && N < (1ll << 29) && K < (1ll << 31);
}

// Time of a launch without staging, for the choice between tiles and slices of the streaming kernel: the planner's figure and 5.6 us.  A
// launch, its set-up and last stores take 4.6 on average on top of the figure (648 products of 17 to 80 tokens, 256 to 6144 features of
// 256 to 8192, bf16, captured one behind the other: 3.8 to 6.3), but slices take 1.0 to 2.7 times their estimate, and the line is what
// decides: with 5.6 the slower of the two is taken for 3.8 % on average, with 5.5 sizes beside the line went from the faster one to
// the slower (64 tokens of 1536 by 1024: 8.9 -> 9.6 us); 4.0 would leave 1.4 %.
double gemm_trit_tc_estimate_us(int64_t M, int64_t N, int64_t K) { return 5.6 + 1.7e-3 * pick_shape(M, N, K, 1, kRawBytes<1>, true).cost; }

// Scratch bytes for the activations: none when they are read in place.  `planes`: bf16 planes of fp32 activations.
size_t gemm_trit_tc_scratch_most(int b_dtype, int64_t N, int64_t K, int planes) {
    return (size_t)(b_dtype == T81B200_F32 ? planes : 1) * N * scratch_row(K) * 2;
}
size_t gemm_trit_tc_scratch(const void *B, int b_dtype, int layout, int64_t ldb, int64_t N, int64_t K, int planes) {
    return reads_in_place(B, b_dtype, layout, ldb) ? 0 : gemm_trit_tc_scratch_most(b_dtype, N, K, planes);
}

int gemm_trit_tc_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_tc_status, sizeof v) != cudaSuccess) return T81B200_ECUDA;
    if (reset && v != 0) {
        const int zero = 0;
        if (cudaMemcpyToSymbol(g_tc_status, &zero, sizeof zero) != cudaSuccess) return T81B200_ECUDA;
    }
    return v;
}

// fmt 0: A holds packed limbs, 1: the decode-stream layout.  A is 16-byte aligned; the workspace holds
// gemm_trit_tc_scratch bytes for `fp32_planes` (2: 16 mantissa bits of fp32 activations, 3: all of them).
int gemm_trit_tc_launch(int fmt, int fp32_planes, const uint8_t *A, const float *row_scale, const void *B, int b_dtype, int layout,
                        int64_t ldb, const float *bias, void *C, int c_dtype, int64_t ldc, int64_t M, int64_t N,
                        int64_t K, float alpha, float beta, void *workspace, size_t workspace_bytes, cudaStream_t st,
                        int n_peers, void *const *peer_C) {
    const void *x_ptr = B;
    int64_t x_ld = ldb, x_rows = N;
    const int planes = b_dtype == T81B200_F32 ? fp32_planes : (b_dtype == T81B200_BF16X3 ? 3 : 1);
    x_rows = (int64_t)planes * N;
    if (!reads_in_place(B, b_dtype, layout, ldb)) {
        const size_t need = gemm_trit_tc_scratch_most(b_dtype, N, K, planes);
        if (!workspace || workspace_bytes < need || reinterpret_cast<uintptr_t>(workspace) % 16 != 0)
            return fail(T81B200_EWORKSPACE, "gemm_trit: %zu bytes of 16-byte aligned workspace needed, %zu given", need, workspace_bytes);
        if (int rc = stage_planes(B, b_dtype, layout, ldb, N, K, planes, workspace, st)) return rc;
        x_ptr = workspace; x_ld = scratch_row(K);
    }
    // TMA-store epilogue: 16-bit output, token-major C (features contiguous), no read-modify-write, and every
    // result 16-byte aligned with a 16-byte multiple as its row pitch
    bool tma_out = dtype_size(c_dtype) == 2 && layout == T81B200_LAYOUT_NK && beta == 0.0f && (ldc * 2) % 16 == 0 &&
                   reinterpret_cast<uintptr_t>(C) % 16 == 0;
    for (int i = 0; i < n_peers; ++i) tma_out = tma_out && reinterpret_cast<uintptr_t>(peer_C[i]) % 16 == 0;
    const TcShape shape = pick_shape(M, N, K, planes, fmt == 1 ? kRawBytes<1> : kRawBytes<0>, tma_out);
    const bool f16 = b_dtype == T81B200_F16;
    CUtensorMap mw, mx;
    memset(&mw, 0, sizeof mw);
    if (fmt == 0) {
        const int64_t row_bytes = (K + 47) / 48 * 16;
        if (int rc = make_map_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_UINT8, A, (uint64_t)row_bytes, (uint64_t)M, (uint64_t)row_bytes, 64, BM,
                                 CU_TENSOR_MAP_SWIZZLE_NONE))
            return rc;
    }
    if (int rc = make_map_2d(&mx, f16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, x_ptr, (uint64_t)K,
                             (uint64_t)x_rows, (uint64_t)x_ld * 2, BK, (uint32_t)(shape.mode == SIDE && planes == 2 ? shape.bn : shape.bn / 2), CU_TENSOR_MAP_SWIZZLE_128B))
        return rc;
    TcParams p;
    memset(&p, 0, sizeof p);
    p.A = A; p.row_scale = row_scale; p.bias = bias; p.C = C; p.M = M; p.N = N; p.kl = (K + 47) / 48;
    if (layout == T81B200_LAYOUT_NK) { p.c_row_stride = 1; p.c_tok_stride = ldc; }
    else { p.c_row_stride = ldc; p.c_tok_stride = 1; }
    p.tiles32 = (int)((M + 31) / 32);
    p.m_tiles = (int)((M + 255) / 256);
    p.n_tiles = shape.n_tiles;
    p.bn = shape.bn;
    p.n_atoms = (int)((K + BK - 1) / BK);
    p.n_chunks = (int)((K + CHUNK - 1) / CHUNK);
    p.planes = planes; p.plane_rows = (int)N; p.b_rows = shape.b_rows; p.out_bytes = shape.out_bytes;
    p.splits = shape.splits;
    p.a_stages = shape.a_stages; p.b_stages = shape.b_stages; p.b_step = shape.b_step;
    p.one_tile = shape.splits > 1 || p.m_tiles * p.n_tiles <= resident_pair_clusters(1) ? 1 : 0;
    p.idesc = umma_instr_desc(shape.mode == SIDE ? 2 * shape.bn : shape.bn, f16);
    p.idesc_rest = umma_instr_desc(shape.bn, f16);
    p.one_mask = f16 ? 0xBC00BC00u : 0xFFFFFFFFu;
    p.alpha = fmt == 1 ? 0.5f * alpha : alpha;
    p.beta = beta;
    p.n_peers = n_peers;
    for (int i = 0; i < n_peers; ++i) p.peer_C[i] = peer_C[i];
    p.c_vec = layout == T81B200_LAYOUT_KN && n_peers == 0 && reinterpret_cast<uintptr_t>(C) % 16 == 0 &&
                      (ldc * (int64_t)dtype_size(c_dtype)) % 16 == 0 ? 1 : 0;
    TcOutMaps om;
    memset(&om, 0, sizeof om);
    if (tma_out) {
        const CUtensorMapDataType dt = c_dtype == T81B200_BF16 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
        for (int i = 0; i <= n_peers; ++i) {
            void *dst = i == 0 ? C : peer_C[i - 1];
            if (int rc = make_map_2d(&om.m[i], dt, dst, (uint64_t)M, (uint64_t)N, (uint64_t)ldc * 2, BM, OUT_TOKENS,
                                     CU_TENSOR_MAP_SWIZZLE_NONE))
                return rc;
        }
        p.n_out_maps = 1 + n_peers;
    }
    const bool rows = !tma_out && dtype_size(c_dtype) == 2 && layout == T81B200_LAYOUT_NK && beta == 0.0f && n_peers == 0;
    auto launch = [&](auto mode) {
        constexpr Mode MODE = decltype(mode)::value;
        return fmt == 1 ? launch_tc_ct<1, MODE>(c_dtype, rows, shape, mw, mx, om, p, st) : launch_tc_ct<0, MODE>(c_dtype, rows, shape, mw, mx, om, p, st);
    };
    switch (shape.mode) {
        case SIDE: return launch(std::integral_constant<Mode, SIDE>{});
        case APART: return launch(std::integral_constant<Mode, APART>{});
        case WIDE: return launch(std::integral_constant<Mode, WIDE>{});
        default: return launch(std::integral_constant<Mode, ONE>{});
    }
}

}  // namespace t81b200

// ---- staging by itself: what several products of one operand share ------------------------

extern "C" int64_t t81b200_stage_rows_ld(int64_t width) { return (width + 7) & ~(int64_t)7; }

extern "C" size_t t81b200_stage_rows_bytes(int dtype, int64_t tokens, int64_t width) {
    if (tokens <= 0 || width <= 0) return 0;
    return (size_t)(dtype == T81B200_F32 ? 3 : 1) * tokens * t81b200_stage_rows_ld(width) * 2;
}

extern "C" int t81b200_stage_rows(const void *src, int dtype, int64_t ld, int64_t tokens, int64_t width, void *out, void *stream) {
    using namespace t81b200;
    if (tokens < 0 || width < 0 || ld < width) return fail(T81B200_EINVAL, "stage_rows: bad dimensions");
    if (dtype != T81B200_F32 && dtype != T81B200_BF16 && dtype != T81B200_F16) return fail(T81B200_EINVAL, "stage_rows: unknown dtype %d", dtype);
    if (int rc = check_device()) return rc;
    if (tokens == 0 || width == 0) return T81B200_OK;
    if (!src || !out) return fail(T81B200_EINVAL, "stage_rows: null pointer");
    if (reinterpret_cast<uintptr_t>(out) % 16 != 0) return fail(T81B200_EALIGN, "stage_rows: the output must be 16-byte aligned");
    return stage_planes(src, dtype, T81B200_LAYOUT_NK, ld, tokens, width, 3, out, static_cast<cudaStream_t>(stream));
}

// ---- entry point that allocates nothing -------------------------------------------------

namespace {

// Scratch for the staging pre-pass of t81b200_gemm_trit_static.  It is part of the loaded
// module: every GPU that loads the library holds these bytes until the process exits.
static __device__ __align__(256) unsigned char g_static_scratch[T81B200_STATIC_SCRATCH_BYTES];

// In host code `g_static_scratch` is only a handle for the runtime, not a device address;
// the address the kernels need is looked up once per device, with that device current.
void *g_static_scratch_ptr[64] = {nullptr};
std::mutex g_static_scratch_mu;

int static_scratch_address(void **out) {
    int dev = 0;
    T81_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return t81b200::fail(T81B200_ELIMIT, "gemm_trit_static: device index %d not supported", dev);
    std::lock_guard<std::mutex> lock(g_static_scratch_mu);
    if (!g_static_scratch_ptr[dev]) {
        void *ptr = nullptr;
        T81_CUDA_TRY(cudaGetSymbolAddress(&ptr, g_static_scratch));
        g_static_scratch_ptr[dev] = ptr;
    }
    *out = g_static_scratch_ptr[dev];
    return T81B200_OK;
}

}  // namespace

extern "C" int t81b200_gemm_trit_static(const uint8_t *A, const float *row_scale, const void *B, int b_dtype, int layout,
                                        int64_t ldb, const float *bias, void *C, int c_dtype, int64_t ldc, int64_t M,
                                        int64_t N, int64_t K, float alpha, float beta, void *stream) {
    if (int rc = t81b200::check_device()) return rc;
    const size_t need = t81b200_gemm_trit_workspace_bytes(b_dtype, layout, c_dtype, M, N, K);
    if (need > (size_t)T81B200_STATIC_SCRATCH_BYTES)
        return t81b200::fail(T81B200_ELIMIT,
                             "gemm_trit_static: this call needs %zu bytes of scratch, the built-in buffer holds %zu; "
                             "use t81b200_gemm_trit with a caller-provided workspace",
                             need, (size_t)T81B200_STATIC_SCRATCH_BYTES);
    void *scratch = nullptr;
    if (int rc = static_scratch_address(&scratch)) return rc;
    return t81b200_gemm_trit(A, row_scale, B, b_dtype, layout, ldb, bias, C, c_dtype, ldc, M, N, K, alpha, beta, scratch,
                             (size_t)T81B200_STATIC_SCRATCH_BYTES, stream);
}

