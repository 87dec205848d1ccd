// Transcoders between the packed-limb layout and the GGUF ternary block formats TQ1_0 and TQ2_0, on the device:
// the on-disk formats either side of the matmul path (t81/gguf.py:518-662 of the reference, which quantises from
// and dequantises to float arrays on the CPU).  Here the trits never leave their integer form: export reads packed
// limbs (+ the per-row scale) and writes blocks, import reads blocks and writes packed limbs (+ the blocks' scales).
//
// A block holds 256 consecutive weights of one row:
//   TQ2_0 (66 bytes): 64 bytes of 2-bit digits q = trit + 1 — byte j of each 32-byte half holds elements
//          j, 32 + j, 64 + j, 96 + j of that half's 128 elements at bits 0, 2, 4, 6 — then the fp16 scale d.
//   TQ1_0 (54 bytes): 32 bytes for elements 0..159 (byte j: elements j, 32 + j, ..., 128 + j as base-3 digits,
//          first element most significant), 16 bytes for elements 160..239 (byte j: 160 + j, 176 + j, ...),
//          4 bytes for elements 240..255 (byte j: 240 + j, 244 + j, 248 + j, 252 + j, then a zero digit), each
//          value v in 0..242 stored as ceil(v * 256 / 243); then the fp16 scale d.
// A weight's value is d * (q - 1).  Rows are padded with zero trits to a whole number of blocks.
//
// In the limb layout a row is a flat stream of tryte bytes, byte = t0 + 3 t1 + 9 t2 + 13: element e of a row sits
// in byte e / 3 as digit e % 3, whatever the limb boundaries (48 trits = 16 bytes).
#include "common.cuh"
#include "launch_order.cuh"

namespace t81b200 {

namespace {

constexpr int kBlock = 256;

__host__ __device__ constexpr int block_bytes(int format) { return format == T81B200_TQ2_0 ? 66 : 54; }

// Both directions work in runs of up to nine blocks of a row: 2304 elements, 768 trytes (three blocks are the least that
// end on a tryte; a row is cut into equal runs).  A warp takes one run at a time, turns it into one byte per digit
// (trit + 1) in shared memory, four digits to a word, and puts the other form together from there.  Trytes become digits
// by a table with a copy per lane (one look-up per tryte, no bank conflicts); a block's words of digits lie 76 words from
// the next block's, so that the items of a pass (13 words of payload a TQ1_0 block) meet few of each other's banks; where
// an item reads and writes is worked out once per warp, not once per run.  Global memory is touched in whole words
// (trytes) and halfwords (blocks start on even bytes), each byte once; buffers that start on odd addresses (`wide` false)
// are taken byte by byte.  Bound by instructions.
// 14336 x 4096 TQ1_0 out and back: 349 us byte at a time (one CTA per block), 100 us with three blocks a warp and digits
// by arithmetic, 61 us with twelve, 49 us now (27 out, 22 in); 65 MB cross memory (10 us).
constexpr int kRunBlocks = 9;
constexpr int kPieces = kRunBlocks / 3;        // 256 trytes each: eight per lane
constexpr int kBlockPitch = 76;                // words of digits from one block to the next
constexpr int kDigitWords = kRunBlocks * kBlockPitch;
constexpr int kWarps = 4;

__device__ __forceinline__ int digit_place(int word) { return word + (word >> 6) * (kBlockPitch - 64); }

// table[value * 32 + lane]: the three digits of a tryte, first element in the low byte; 27..31 read as the zero tryte.
__device__ __forceinline__ void fill_tryte_table(uint32_t *table, int tid, int threads) {
    for (int i = tid; i < 32 * 32; i += threads) {
        int d0, d1, d2;
        tryte_digits((uint32_t)(i >> 5), d0, d1, d2);
        table[i] = (uint32_t)(d0 | (d1 << 8) | (d2 << 16));
    }
}

// Four trytes -> their twelve digits in element order.  `column` = table + lane.
__device__ __forceinline__ void word_digits(uint32_t b, const uint32_t *column, uint32_t (&w)[3]) {
    if (b & 0xE0E0E0E0u) {  // not trytes: they read as zero
#pragma unroll
        for (int i = 0; i < 4; ++i)
            if ((b >> (8 * i)) & 0xE0u) b |= 0x1Fu << (8 * i);
    }
    const uint32_t e0 = column[(b & 31u) << 5], e1 = column[((b >> 8) & 31u) << 5], e2 = column[((b >> 16) & 31u) << 5], e3 = column[((b >> 24) & 31u) << 5];
    w[0] = __byte_perm(e0, e1, 0x4210);
    w[1] = __byte_perm(e1, e2, 0x5421);
    w[2] = __byte_perm(e2, e3, 0x6542);
}

// Twelve digits -> four trytes: d0 + 3 d1 + 9 d2 (the offset 13 is the three digits' own 1 + 3 + 9).
__device__ __forceinline__ uint32_t digits_word(uint32_t w0, uint32_t w1, uint32_t w2) {
    const uint32_t d0 = __byte_perm(__byte_perm(w0, w1, 0x0630), w2, 0x5210);
    const uint32_t d1 = __byte_perm(__byte_perm(w0, w1, 0x0741), w2, 0x6210);
    const uint32_t d2 = __byte_perm(__byte_perm(w0, w1, 0x0052), w2, 0x7410);
    return d0 + 3u * d1 + 9u * d2;
}

__device__ __forceinline__ uint32_t bytes_word(const uint8_t *p) { return (uint32_t)p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24; }

// Positions from `left` on (of `n` digits in w, left < n) become zero trits.
template <int WORDS>
__device__ __forceinline__ void clear_past(uint32_t (&w)[WORDS], int64_t left) {
#pragma unroll
    for (int i = 0; i < WORDS; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            if (4 * i + j >= left) w[i] = (w[i] & ~(0xFFu << (8 * j))) | (1u << (8 * j));
}

// Word k of a block's payload: the digit words it is made of, first + m * pitch.  TQ2_0: four; TQ1_0: five, or four and
// a zero digit for the last word.
template <int FORMAT>
__device__ __forceinline__ void digit_words(int k, int &first, int &pitch) {
    if constexpr (FORMAT == T81B200_TQ2_0) {
        first = (k >> 3) * 32 + (k & 7);
        pitch = 8;
    } else {
        first = k < 8 ? k : (k < 12 ? 32 + k : 60);
        pitch = k < 8 ? 8 : (k < 12 ? 4 : 1);
    }
}

template <int FORMAT>
__global__ void __launch_bounds__(kWarps * 32) packed_to_tq_kernel(const uint8_t *__restrict__ packed, const float *__restrict__ row_scale, int64_t rows,
                                                                   int64_t cols, int64_t row_bytes, uint8_t *__restrict__ blocks, int64_t blocks_per_row,
                                                                   int runs_per_row, int run_blocks, bool wide) {
    constexpr int kBytes = block_bytes(FORMAT), kWords = FORMAT == T81B200_TQ2_0 ? 16 : 13;  // words of a block's payload
    constexpr int kPasses = (kRunBlocks * kWords + 31) / 32, kHalves = kRunBlocks * kBytes / 2;
    __shared__ uint32_t table[32 * 32];
    __shared__ __align__(16) uint32_t digits[kWarps][kDigitWords];
    __shared__ __align__(16) uint8_t staged[kWarps][kRunBlocks * 66 + 2];
    __shared__ uint8_t nonzero[kWarps][kRunBlocks];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    fill_tryte_table(table, threadIdx.x, kWarps * 32);
    __syncthreads();
    uint32_t *q = digits[warp];
    // item lane + 32 i of a run: word k of block b
    int from[kPasses], pitch[kPasses], to[kPasses], block[kPasses];
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
        const int item = lane + 32 * i, b = item / kWords, k = item - b * kWords;
        digit_words<FORMAT>(k, from[i], pitch[i]);
        from[i] += b * kBlockPitch;
        to[i] = b * (kBytes / 2) + 2 * k;
        block[i] = b;
    }
    const int64_t total = rows * runs_per_row, stride = (int64_t)gridDim.x * kWarps;
    auto locate = [&](int64_t at, int64_t &row, int64_t &block0, int &n_blocks) {
        row = total < (1ll << 32) ? (int64_t)((uint32_t)at / (uint32_t)runs_per_row) : at / runs_per_row;
        block0 = (at - row * runs_per_row) * run_blocks;  // run_blocks is a multiple of 3
        const int64_t left = blocks_per_row - block0;
        n_blocks = (int)(left < run_blocks ? left : run_blocks);
    };
    for (int64_t at = (int64_t)blockIdx.x * kWarps + warp; at < total; at += stride) {
        int64_t row, block0;
        int n_blocks;
        locate(at, row, block0, n_blocks);
        uint2 in[kPieces];
        const int64_t byte0 = block0 * kBlock / 3 + lane * 8;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            in[i] = make_uint2(kZeroTryteWord, kZeroTryteWord);
            if (3 * i < n_blocks && byte0 + 256 * i < row_bytes) {  // limbs are 16 bytes: all eight or none
                const uint8_t *src = packed + row * row_bytes + byte0 + 256 * i;
                if (wide) in[i] = __ldg(reinterpret_cast<const uint2 *>(src));
                else in[i] = make_uint2(bytes_word(src), bytes_word(src + 4));
            }
        }
        const int n_pieces = (n_blocks + 2) / 3;
        __syncwarp();
        if (lane < kRunBlocks) nonzero[warp][lane] = 0;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            if (i >= n_pieces) break;
            uint32_t lo[3], hi[3];
            word_digits(in[i].x, table + lane, lo);
            word_digits(in[i].y, table + lane, hi);
            uint32_t w[6] = {lo[0], lo[1], lo[2], hi[0], hi[1], hi[2]};
            const int64_t e0 = block0 * kBlock + 768 * i + lane * 24;
            if (e0 + 24 > cols) clear_past<6>(w, cols - e0);
#pragma unroll
            for (int j = 0; j < 3; ++j) *reinterpret_cast<uint2 *>(q + digit_place(i * 192 + lane * 6 + 2 * j)) = make_uint2(w[2 * j], w[2 * j + 1]);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kPasses; ++i) {
            if (lane + 32 * i >= n_blocks * kWords) break;
            const uint32_t *blk = q + from[i];
            uint32_t v = 0, differs = 0;
            if constexpr (FORMAT == T81B200_TQ2_0) {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t x = blk[m * 8];
                    differs |= x ^ 0x01010101u;
                    v |= x << (2 * m);
                }
            } else {
                const bool last = pitch[i] == 1;  // four digits and a zero one
                uint32_t n = 0;  // base-3 numbers 0..242, byte by byte
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t x = blk[m * pitch[i]];
                    differs |= x ^ 0x01010101u;
                    n = 3u * n + x;
                }
                const uint32_t x = last ? 0x01010101u : blk[4 * pitch[i]];
                differs |= x ^ 0x01010101u;
                n = 3u * n + (last ? 0u : x);
                // ceil(256 n / 243) = (69045 n + 65000) >> 16, exact for all 243 values: byte 2 of each product
                uint32_t y[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) y[j] = __byte_perm(n, 0u, 0x4440 | j) * 69045u + 65000u;
                v = __byte_perm(__byte_perm(y[0], y[1], 0x0062), __byte_perm(y[2], y[3], 0x0062), 0x5410);
            }
            if (differs) nonzero[warp][block[i]] = 1;
            uint16_t *dst = reinterpret_cast<uint16_t *>(staged[warp]) + to[i];
            dst[0] = (uint16_t)v;
            dst[1] = (uint16_t)(v >> 16);
        }
        __syncwarp();
        // the scale of a block with no non-zero trit is 0, like the absmax of an all-zero block
        if (lane < n_blocks) {
            const float d = nonzero[warp][lane] ? (row_scale ? row_scale[row] : 1.0f) : 0.0f;
            *reinterpret_cast<uint16_t *>(staged[warp] + lane * kBytes + kBytes - 2) = __half_as_ushort(__float2half_rn(d));
        }
        __syncwarp();
        uint8_t *out = blocks + (row * blocks_per_row + block0) * kBytes;
        if (wide) {
#pragma unroll
            for (int i = 0; i < (kHalves + 31) / 32; ++i)
                if (lane + 32 * i < n_blocks * kBytes / 2) reinterpret_cast<uint16_t *>(out)[lane + 32 * i] = reinterpret_cast<const uint16_t *>(staged[warp])[lane + 32 * i];
        } else
            for (int i = lane; i < n_blocks * kBytes; i += 32) out[i] = staged[warp][i];
    }
}

template <int FORMAT>
__global__ void __launch_bounds__(kWarps * 32) tq_to_packed_kernel(const uint8_t *__restrict__ blocks, int64_t rows, int64_t cols, int64_t row_bytes,
                                                                   uint8_t *__restrict__ packed, float *__restrict__ block_scale, int64_t blocks_per_row,
                                                                   int runs_per_row, int run_blocks, bool wide) {
    constexpr int kBytes = block_bytes(FORMAT), kWords = FORMAT == T81B200_TQ2_0 ? 16 : 13, kHalves = kRunBlocks * kBytes / 2;
    constexpr int kPasses = (kRunBlocks * kWords + 31) / 32, kLoads = (kHalves + 31) / 32;
    __shared__ __align__(16) uint32_t digits[kWarps][kDigitWords];
    __shared__ __align__(16) uint8_t staged[kWarps][kRunBlocks * 66 + 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *q = digits[warp];
    int to[kPasses], pitch[kPasses], from[kPasses];
#pragma unroll
    for (int i = 0; i < kPasses; ++i) {
        const int item = lane + 32 * i, b = item / kWords, k = item - b * kWords;
        digit_words<FORMAT>(k, to[i], pitch[i]);
        to[i] += b * kBlockPitch;
        from[i] = b * (kBytes / 2) + 2 * k;
    }
    const int64_t total = rows * runs_per_row, stride = (int64_t)gridDim.x * kWarps;
    auto locate = [&](int64_t at, int64_t &row, int64_t &block0, int &n_blocks) {
        row = total < (1ll << 32) ? (int64_t)((uint32_t)at / (uint32_t)runs_per_row) : at / runs_per_row;
        block0 = (at - row * runs_per_row) * run_blocks;
        const int64_t left = blocks_per_row - block0;
        n_blocks = (int)(left < run_blocks ? left : run_blocks);
    };
    for (int64_t at = (int64_t)blockIdx.x * kWarps + warp; at < total; at += stride) {
        int64_t row, block0;
        int n_blocks;
        locate(at, row, block0, n_blocks);
        const uint8_t *in = blocks + (row * blocks_per_row + block0) * kBytes;
        __syncwarp();
        if (wide) {
            uint16_t h[kLoads];
#pragma unroll
            for (int i = 0; i < kLoads; ++i) h[i] = lane + 32 * i < n_blocks * kBytes / 2 ? __ldg(reinterpret_cast<const uint16_t *>(in) + lane + 32 * i) : (uint16_t)0;
#pragma unroll
            for (int i = 0; i < kLoads; ++i)
                if (lane + 32 * i < kHalves) reinterpret_cast<uint16_t *>(staged[warp])[lane + 32 * i] = h[i];
        } else
            for (int i = lane; i < n_blocks * kBytes; i += 32) staged[warp][i] = in[i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kPasses; ++i) {
            if (lane + 32 * i >= n_blocks * kWords) break;
            const uint16_t *src = reinterpret_cast<const uint16_t *>(staged[warp]) + from[i];
            const uint32_t x = (uint32_t)src[0] | ((uint32_t)src[1] << 16);
            uint32_t *blk = q + to[i];
            if constexpr (FORMAT == T81B200_TQ2_0) {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t d = (x >> (2 * m)) & 0x03030303u;
                    blk[m * 8] = d - (d & (d >> 1) & 0x01010101u);  // 3 reads as 2
                }
            } else {
                // digit m of a byte is the top of byte * 3^m (mod 256) * 3 (t81/gguf.py:629-637)
                uint32_t even = x & 0x00FF00FFu, odd = (x >> 8) & 0x00FF00FFu;
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    even *= 3u;
                    odd *= 3u;
                    if (m < 4 || pitch[i] != 1) blk[m * pitch[i]] = __byte_perm(even, odd, 0x7351);
                    even &= 0x00FF00FFu;
                    odd &= 0x00FF00FFu;
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int64_t byte0 = block0 * kBlock / 3 + 256 * i + lane * 8, e0 = block0 * kBlock + 768 * i + lane * 24;
            if (3 * i >= n_blocks || byte0 >= row_bytes) break;
            uint32_t w[6];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const uint2 d = *reinterpret_cast<const uint2 *>(q + digit_place(i * 192 + lane * 6 + 2 * j));
                w[2 * j] = d.x;
                w[2 * j + 1] = d.y;
            }
            if (e0 + 24 > cols) clear_past<6>(w, cols - e0);
            const uint32_t t0 = digits_word(w[0], w[1], w[2]), t1 = digits_word(w[3], w[4], w[5]);
            uint8_t *dst = packed + row * row_bytes + byte0;
            if (wide) *reinterpret_cast<uint2 *>(dst) = make_uint2(t0, t1);
            else
                for (int j = 0; j < 4; ++j) { dst[j] = (uint8_t)(t0 >> (8 * j)); dst[4 + j] = (uint8_t)(t1 >> (8 * j)); }
        }
        if (block_scale && lane < n_blocks)
            block_scale[row * blocks_per_row + block0 + lane] =
                __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t *>(staged[warp] + lane * kBytes + kBytes - 2)));
    }
}

// A few runs a warp: the tables are made once per CTA.
unsigned tq_grid(int64_t runs) {
    const int64_t ctas = (runs + kWarps - 1) / kWarps, most = (int64_t)sm_count() * 12;
    return (unsigned)(ctas < most ? ctas : most);
}

}  // namespace
}  // namespace t81b200

using namespace t81b200;

extern "C" int64_t t81b200_tq_bytes(int format, int64_t rows, int64_t cols) {
    if ((format != T81B200_TQ1_0 && format != T81B200_TQ2_0) || rows < 0 || cols < 0) return -1;
    return rows * ((cols + kBlock - 1) / kBlock) * block_bytes(format);
}

extern "C" int t81b200_packed_to_tq(const uint8_t *packed, const float *row_scale, int64_t rows, int64_t cols, int format,
                                    uint8_t *blocks, void *stream) {
    if (format != T81B200_TQ1_0 && format != T81B200_TQ2_0) return fail(T81B200_EINVAL, "tq: unknown block format %d", format);
    if (rows < 0 || cols < 0) return fail(T81B200_EINVAL, "tq: negative dimension");
    if (int rc = check_device()) return rc;
    if (rows == 0 || cols == 0) return T81B200_OK;
    if (!packed || !blocks) return fail(T81B200_EINVAL, "tq: null pointer");
    const int64_t bpr = (cols + kBlock - 1) / kBlock, row_bytes = (cols + 47) / 48 * 16;
    if (bpr > 65535 || rows >= (1ll << 31)) return fail(T81B200_ELIMIT, "tq: matrix too large for one call");
    const bool wide = reinterpret_cast<uintptr_t>(packed) % 8 == 0 && reinterpret_cast<uintptr_t>(blocks) % 2 == 0;
    const int64_t runs0 = (bpr + kRunBlocks - 1) / kRunBlocks;
    const int run_blocks = (int)(((bpr + runs0 - 1) / runs0 + 2) / 3 * 3);
    const int64_t runs = (bpr + run_blocks - 1) / run_blocks;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (format == T81B200_TQ2_0)
        packed_to_tq_kernel<T81B200_TQ2_0><<<tq_grid(rows * runs), kWarps * 32, 0, st>>>(packed, row_scale, rows, cols, row_bytes, blocks, bpr, (int)runs, run_blocks, wide);
    else
        packed_to_tq_kernel<T81B200_TQ1_0><<<tq_grid(rows * runs), kWarps * 32, 0, st>>>(packed, row_scale, rows, cols, row_bytes, blocks, bpr, (int)runs, run_blocks, wide);
    T81_LAUNCH_CHECK("packed_to_tq_kernel");
    return T81B200_OK;
}

extern "C" int t81b200_tq_to_packed(const uint8_t *blocks, int64_t rows, int64_t cols, int format, uint8_t *packed,
                                    float *block_scale, void *stream) {
    if (format != T81B200_TQ1_0 && format != T81B200_TQ2_0) return fail(T81B200_EINVAL, "tq: unknown block format %d", format);
    if (rows < 0 || cols < 0) return fail(T81B200_EINVAL, "tq: negative dimension");
    if (int rc = check_device()) return rc;
    if (rows == 0 || cols == 0) return T81B200_OK;
    if (!packed || !blocks) return fail(T81B200_EINVAL, "tq: null pointer");
    const int64_t bpr = (cols + kBlock - 1) / kBlock, row_bytes = (cols + 47) / 48 * 16;
    if (bpr > 65535 || rows >= (1ll << 31)) return fail(T81B200_ELIMIT, "tq: matrix too large for one call");
    const bool wide = reinterpret_cast<uintptr_t>(packed) % 8 == 0 && reinterpret_cast<uintptr_t>(blocks) % 2 == 0;
    const int64_t runs0 = (bpr + kRunBlocks - 1) / kRunBlocks;
    const int run_blocks = (int)(((bpr + runs0 - 1) / runs0 + 2) / 3 * 3);
    const int64_t runs = (bpr + run_blocks - 1) / run_blocks;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (format == T81B200_TQ2_0)
        tq_to_packed_kernel<T81B200_TQ2_0><<<tq_grid(rows * runs), kWarps * 32, 0, st>>>(blocks, rows, cols, row_bytes, packed, block_scale, bpr, (int)runs, run_blocks, wide);
    else
        tq_to_packed_kernel<T81B200_TQ1_0><<<tq_grid(rows * runs), kWarps * 32, 0, st>>>(blocks, rows, cols, row_bytes, packed, block_scale, bpr, (int)runs, run_blocks, wide);
    T81_LAUNCH_CHECK("tq_to_packed_kernel");
    note_weights_written(st);
    return T81B200_OK;
}
