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

namespace t81b200 {

namespace {

constexpr int kBlock = 256;

__host__ __device__ constexpr int block_bytes(int format) { return format == T81B200_TQ2_0 ? 66 : 54; }

// Both directions work in groups of three blocks: 768 elements, 256 trytes.  A warp takes one group at a time, turns it
// into one byte per digit (trit + 1) in shared memory with four trytes or four block bytes per arithmetic step — digits
// are small enough for byte- or halfword-wise sums in a 32-bit register — and puts the other form together from there.
// Global memory is touched in whole words (trytes) and halfwords (blocks start on even bytes), each byte once; buffers
// that start on odd addresses (`wide` false) are taken byte by byte.  The
// byte-at-a-time form (one CTA per block) took 349 us for 14336 x 4096 TQ1_0 out and back; 65 MB cross memory (10 us).
constexpr int kGroup = 3 * kBlock;
constexpr int kWarps = 8;

// Four trytes -> their twelve digits in element order.
__device__ __forceinline__ void word_digits(uint32_t b, uint32_t (&w)[3]) {
    const uint32_t bad = __vcmpgtu4(b, 0x1A1A1A1Au);  // not a tryte: reads as zero
    b = (b & ~bad) | (kZeroTryteWord & bad);
    uint32_t d0 = 0, d1 = 0, d2 = 0;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const uint32_t x = (b >> (8 * h)) & 0x00FF00FFu;
        const uint32_t e2 = ((x * 57u) >> 9) & 0x00030003u, r = x - 9u * e2;   // x / 9
        const uint32_t e1 = ((r * 11u) >> 5) & 0x00030003u;                    // r / 3
        d0 |= (r - 3u * e1) << (8 * h);
        d1 |= e1 << (8 * h);
        d2 |= e2 << (8 * h);
    }
    w[0] = __byte_perm(__byte_perm(d0, d1, 0x1040), d2, 0x3410);                // d0[0] d1[0] d2[0] d0[1]
    w[1] = __byte_perm(__byte_perm(d1, d2, 0x2051), __byte_perm(d0, d1, 0x0062), 0x5410);  // d1[1] d2[1] d0[2] d1[2]
    w[2] = __byte_perm(__byte_perm(d2, d0, 0x0072), __byte_perm(d1, d2, 0x0073), 0x5410);  // d2[2] d0[3] d1[3] d2[3]
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

template <int FORMAT>
__global__ void __launch_bounds__(kWarps * 32) packed_to_tq_kernel(const uint8_t *__restrict__ packed, const float *__restrict__ row_scale, int64_t rows,
                                                                   int64_t cols, int64_t row_bytes, uint8_t *__restrict__ blocks, int64_t blocks_per_row,
                                                                   int64_t groups_per_row, bool wide) {
    constexpr int kBytes = block_bytes(FORMAT), kWords = FORMAT == T81B200_TQ2_0 ? 16 : 13;  // digit words of a block's payload
    __shared__ __align__(16) uint32_t digits[kWarps][kGroup / 4];
    __shared__ __align__(16) uint8_t staged[kWarps][3 * 66 + 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *q = digits[warp];
    const int64_t total = rows * groups_per_row, stride = (int64_t)gridDim.x * kWarps;
    for (int64_t item = (int64_t)blockIdx.x * kWarps + warp; item < total; item += stride) {
        const int64_t row = item / groups_per_row, group = item - row * groups_per_row;
        // eight trytes a lane
        const int64_t byte0 = group * 256 + lane * 8, e0 = group * kGroup + lane * 24;
        uint2 in = make_uint2(kZeroTryteWord, kZeroTryteWord);
        if (byte0 < row_bytes) {  // limbs are 16 bytes: all eight or none
            const uint8_t *src = packed + row * row_bytes + byte0;
            if (wide) in = __ldg(reinterpret_cast<const uint2 *>(src));
            else in = make_uint2(bytes_word(src), bytes_word(src + 4));
        }
        uint32_t lo[3], hi[3];
        word_digits(in.x, lo);
        word_digits(in.y, hi);
        uint32_t w[6] = {lo[0], lo[1], lo[2], hi[0], hi[1], hi[2]};
        if (e0 + 24 > cols) clear_past<6>(w, cols - e0);
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2 *>(q + lane * 6 + 2 * i) = make_uint2(w[2 * i], w[2 * i + 1]);
        __syncwarp();
        const int n_blocks = (int)(blocks_per_row - 3 * group < 3 ? blocks_per_row - 3 * group : 3);
#pragma unroll
        for (int b = 0; b < 3; ++b) {
            uint32_t v = 0;
            bool nonzero = false;
            if (b < n_blocks && lane < kWords) {
                const uint32_t *blk = q + b * 64;  // words of four digits
                auto at = [&](int word) { const uint32_t x = blk[word]; nonzero |= x != 0x01010101u; return x; };
                if constexpr (FORMAT == T81B200_TQ2_0) {
                    const int half = lane >> 3, j = lane & 7;
#pragma unroll
                    for (int m = 0; m < 4; ++m) v |= at(half * 32 + 8 * m + j) << (2 * m);
                } else {
                    uint32_t n = 0;  // base-3 numbers 0..242, byte by byte
                    if (lane < 8) {
#pragma unroll
                        for (int m = 0; m < 5; ++m) n = 3u * n + at(8 * m + lane);
                    } else if (lane < 12) {
#pragma unroll
                        for (int m = 0; m < 5; ++m) n = 3u * n + at(40 + 4 * m + lane - 8);
                    } else {
#pragma unroll
                        for (int m = 0; m < 4; ++m) n = 3u * n + at(60 + m);
                        n = 3u * n;
                    }
#pragma unroll
                    for (int j = 0; j < 4; ++j) v |= ((((n >> (8 * j)) & 0xFFu) * 256u + 242u) / 243u) << (8 * j);
                }
                uint16_t *dst = reinterpret_cast<uint16_t *>(staged[warp] + b * kBytes) + lane * 2;
                dst[0] = (uint16_t)v;
                dst[1] = (uint16_t)(v >> 16);
            }
            // the scale of a block with no non-zero trit is 0, like the absmax of an all-zero block
            nonzero = __any_sync(0xffffffffu, nonzero);
            if (b < n_blocks && lane == 0) {
                const float d = nonzero ? (row_scale ? row_scale[row] : 1.0f) : 0.0f;
                *reinterpret_cast<uint16_t *>(staged[warp] + b * kBytes + kBytes - 2) = __half_as_ushort(__float2half_rn(d));
            }
        }
        __syncwarp();
        uint16_t *out = reinterpret_cast<uint16_t *>(blocks + (row * blocks_per_row + 3 * group) * kBytes);
        if (wide)
            for (int i = lane; i < n_blocks * kBytes / 2; i += 32) out[i] = reinterpret_cast<const uint16_t *>(staged[warp])[i];
        else
            for (int i = lane; i < n_blocks * kBytes; i += 32) reinterpret_cast<uint8_t *>(out)[i] = staged[warp][i];
    }
}

template <int FORMAT>
__global__ void __launch_bounds__(kWarps * 32) tq_to_packed_kernel(const uint8_t *__restrict__ blocks, int64_t rows, int64_t cols, int64_t row_bytes,
                                                                   uint8_t *__restrict__ packed, float *__restrict__ block_scale, int64_t blocks_per_row,
                                                                   int64_t groups_per_row, bool wide) {
    constexpr int kBytes = block_bytes(FORMAT), kWords = FORMAT == T81B200_TQ2_0 ? 16 : 13;
    __shared__ __align__(16) uint32_t digits[kWarps][kGroup / 4];
    __shared__ __align__(16) uint8_t staged[kWarps][3 * 66 + 2];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *q = digits[warp];
    const int64_t total = rows * groups_per_row, stride = (int64_t)gridDim.x * kWarps;
    for (int64_t item = (int64_t)blockIdx.x * kWarps + warp; item < total; item += stride) {
        const int64_t row = item / groups_per_row, group = item - row * groups_per_row;
        const int n_blocks = (int)(blocks_per_row - 3 * group < 3 ? blocks_per_row - 3 * group : 3);
        const uint16_t *in = reinterpret_cast<const uint16_t *>(blocks + (row * blocks_per_row + 3 * group) * kBytes);
        __syncwarp();
        if (wide)
            for (int i = lane; i < n_blocks * kBytes / 2; i += 32) reinterpret_cast<uint16_t *>(staged[warp])[i] = __ldg(in + i);
        else
            for (int i = lane; i < n_blocks * kBytes; i += 32) staged[warp][i] = reinterpret_cast<const uint8_t *>(in)[i];
        __syncwarp();
        for (int i = lane; i < 3 * kWords; i += 32) {
            const int b = i / kWords, k = i - b * kWords;
            if (b >= n_blocks) break;  // elements past the row: cleared below
            const uint16_t *src = reinterpret_cast<const uint16_t *>(staged[warp] + b * kBytes) + 2 * k;
            const uint32_t x = (uint32_t)src[0] | ((uint32_t)src[1] << 16);
            uint32_t *blk = q + b * 64;
            if constexpr (FORMAT == T81B200_TQ2_0) {
                const int half = k >> 3, j = k & 7;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    const uint32_t d = (x >> (2 * m)) & 0x03030303u;
                    blk[half * 32 + 8 * m + j] = d - (d & (d >> 1) & 0x01010101u);  // 3 reads as 2
                }
            } else {
                // digit m of a byte is the top of byte * 3^m (mod 256) * 3 (t81/gguf.py:629-637)
                uint32_t even = x & 0x00FF00FFu, odd = (x >> 8) & 0x00FF00FFu;
                const int pitch = k < 8 ? 8 : (k < 12 ? 4 : 1), first = k < 8 ? k : (k < 12 ? 40 + k - 8 : 60), n = k < 12 ? 5 : 4;
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    even *= 3u;
                    odd *= 3u;
                    if (m < n) blk[first + m * pitch] = ((even >> 8) & 0x00FF00FFu) | (odd & 0xFF00FF00u);
                    even &= 0x00FF00FFu;
                    odd &= 0x00FF00FFu;
                }
            }
        }
        __syncwarp();
        const int64_t byte0 = group * 256 + lane * 8, e0 = group * kGroup + lane * 24;
        if (byte0 < row_bytes) {
            uint32_t w[6];
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const uint2 d = *reinterpret_cast<const uint2 *>(q + lane * 6 + 2 * i);
                w[2 * i] = d.x;
                w[2 * i + 1] = d.y;
            }
            if (e0 + 24 > cols) clear_past<6>(w, cols - e0);
            const uint32_t t0 = digits_word(w[0], w[1], w[2]), t1 = digits_word(w[3], w[4], w[5]);
            uint8_t *dst = packed + row * row_bytes + byte0;
            if (wide) *reinterpret_cast<uint2 *>(dst) = make_uint2(t0, t1);
            else
                for (int i = 0; i < 4; ++i) { dst[i] = (uint8_t)(t0 >> (8 * i)); dst[4 + i] = (uint8_t)(t1 >> (8 * i)); }
        }
        if (block_scale && lane < n_blocks)
            block_scale[row * blocks_per_row + 3 * group + lane] =
                __half2float(__ushort_as_half(*reinterpret_cast<const uint16_t *>(staged[warp] + lane * kBytes + kBytes - 2)));
    }
}

// A few groups per warp: enough CTAs to fill the GPU, no more than are resident at a time.
unsigned tq_grid(int64_t groups) {
    const int64_t ctas = (groups + kWarps - 1) / kWarps, most = (int64_t)sm_count() * 8;
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
    const int64_t groups = (bpr + 2) / 3;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (format == T81B200_TQ2_0)
        packed_to_tq_kernel<T81B200_TQ2_0><<<tq_grid(rows * groups), kWarps * 32, 0, st>>>(packed, row_scale, rows, cols, row_bytes, blocks, bpr, groups, wide);
    else
        packed_to_tq_kernel<T81B200_TQ1_0><<<tq_grid(rows * groups), kWarps * 32, 0, st>>>(packed, row_scale, rows, cols, row_bytes, blocks, bpr, groups, wide);
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
    const int64_t groups = (bpr + 2) / 3;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (format == T81B200_TQ2_0)
        tq_to_packed_kernel<T81B200_TQ2_0><<<tq_grid(rows * groups), kWarps * 32, 0, st>>>(blocks, rows, cols, row_bytes, packed, block_scale, bpr, groups, wide);
    else
        tq_to_packed_kernel<T81B200_TQ1_0><<<tq_grid(rows * groups), kWarps * 32, 0, st>>>(blocks, rows, cols, row_bytes, packed, block_scale, bpr, groups, wide);
    T81_LAUNCH_CHECK("tq_to_packed_kernel");
    return T81B200_OK;
}
