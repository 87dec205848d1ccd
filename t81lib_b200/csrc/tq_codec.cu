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

// Both directions turn a run of up to 24 blocks into one byte per digit (trit + 1) in shared memory, four digits to a
// word, and put the other form together from there, a warp to a run.  A run is a piece of a row that starts on a limb
// (24 blocks are 128 limbs), or several short rows whole; its blocks are contiguous in memory.  On the limb side a lane
// has a limb (16 trytes, twelve words of digits: three 128-bit accesses), on the block side 16 bytes of payload (four
// words, read or written as one 128-bit access per digit), eight blocks to a pass; the four bytes at the end of a TQ1_0
// payload and the scales are done once a run, a lane to a block.  Global memory is touched in 128-bit words, the ends of a
// run's blocks in bytes.
// Bound by instructions, so each step is the one that takes the fewest: a tryte's place in the table is one PRMT (the byte
// lands above the lane's own column), a base-3 number is one multiply-add per digit on four bytes at once, and on the way
// in digit m of a byte x is floor(3^(m+1) x / 256) - 3 floor(3^m x / 256), with no masks between the digits.
// 14336 x 4096 TQ1_0, out and in: 33 us, 49 with runs of nine blocks, a look-up address of three instructions and one word of
// payload an item; 65 MB cross memory (10 us).  747 and 640 warp instructions a run of 16 blocks, issue slots 61 % and 69 % busy.
constexpr int kRunBlocks = 24;
constexpr int kBlockPitch = 76;  // words of digits from one block to the next: blocks of a pass on different banks
constexpr int kLimbSlots = (kRunBlocks * kBlock + 47) / 48 / 32;  // limbs a lane has of a run
constexpr int kWarps = 4;
constexpr int kMaxCtas = 6;      // per SM

// Shared memory of a warp whose runs hold up to `blocks` blocks: digits, then the blocks as they lie in global memory.
__host__ __device__ constexpr int digit_words(int blocks) { return blocks * kBlockPitch + 8; }
__host__ __device__ constexpr int warp_bytes(int blocks, int format) { return digit_words(blocks) * 4 + (blocks * block_bytes(format) + 47) / 16 * 16; }

// A run: blocks [24 piece, 24 piece + n) of each of `rows` rows from `row` on (several rows: all of their blocks).
struct Run {
    int64_t row;
    int piece, rows, n;
};
struct Runs {
    int64_t rows, limbs_per_row, blocks_per_row;
    uint32_t total, runs_per_row;
    int cols, rows_per_run, most;  // most: blocks of a run
};
template <bool SHORT>
__device__ __forceinline__ Run locate(const Runs &r, uint32_t at) {
    if (SHORT) {
        const int64_t row = (int64_t)at * r.rows_per_run, left = r.rows - row;
        return {row, 0, (int)(left < r.rows_per_run ? left : r.rows_per_run), (int)r.blocks_per_row};
    }
    const uint32_t row = r.runs_per_row == 1 ? at : at / r.runs_per_row;
    const int piece = (int)(at - row * r.runs_per_row), left = (int)r.blocks_per_row - piece * kRunBlocks;
    return {(int64_t)row, piece, 1, left < kRunBlocks ? left : kRunBlocks};
}

// Where word `word` of a row's digits lies.  What a row's last limb has beyond its n blocks lies behind them, where rows follow
// one another in the pad of the last block.
template <bool SHORT>
__device__ __forceinline__ int digit_place(int word, int n) {
    const int block = word >> 6;
    return word + (!SHORT || block < n ? block : n - 1) * (kBlockPitch - 64);
}

// Digits of a row from element `cols` on, up to the end of its limbs, become zero trits.
template <bool SHORT>
__device__ __forceinline__ void clear_past_end(uint32_t *q, const Runs &r, const Run &run, int lane) {
    const int e0 = run.piece * (kRunBlocks * kBlock), from = r.cols - e0, to = (int)r.limbs_per_row * 48 - e0;
    if (from == to || run.n * kBlock < from) return;
    for (int row = 0; row < run.rows; ++row) {
        uint8_t *d = reinterpret_cast<uint8_t *>(q + (SHORT ? row * run.n * kBlockPitch : 0));
        for (int e = from + lane; e < to; e += 32) d[digit_place<SHORT>(e >> 4 << 2, run.n) * 4 + (e & 15)] = 1;
    }
    __syncwarp();
}

// table[value * 64 + lane]: the three digits of a tryte, first element in the low byte; 27..31 read as the zero tryte.
constexpr int kTableWords = 32 * 64;
__device__ __forceinline__ void fill_tryte_table(uint32_t *table, int tid) {
    static_assert(kWarps * 32 == 128, "a value to four threads");
    int d0, d1, d2;
    tryte_digits((uint32_t)(tid >> 2), d0, d1, d2);
    const uint32_t d = (uint32_t)(d0 | (d1 << 8) | (d2 << 16));
    uint4 *to = reinterpret_cast<uint4 *>(table + (tid >> 2) * 64 + (tid & 3) * 8);
    to[0] = to[1] = make_uint4(d, d, d, d);
}

// Four trytes below 32 -> their twelve digits in element order.  `column` = 4 * lane.
__device__ __forceinline__ void word_digits(uint32_t b, const uint32_t *table, uint32_t column, uint32_t (&w)[12], int at) {
    const uint8_t *t = reinterpret_cast<const uint8_t *>(table);
    const uint32_t e0 = *reinterpret_cast<const uint32_t *>(t + __byte_perm(b, column, 0x5504)), e1 = *reinterpret_cast<const uint32_t *>(t + __byte_perm(b, column, 0x5514)),
                   e2 = *reinterpret_cast<const uint32_t *>(t + __byte_perm(b, column, 0x5524)), e3 = *reinterpret_cast<const uint32_t *>(t + __byte_perm(b, column, 0x5534));
    w[at] = __byte_perm(e0, e1, 0x4210);
    w[at + 1] = __byte_perm(e1, e2, 0x5421);
    w[at + 2] = __byte_perm(e2, e3, 0x6542);
}

// Bytes that are no trytes (above 31; the table has 27..31) read as zero trits.
__device__ __forceinline__ uint32_t only_trytes(uint32_t b) {
#pragma unroll
    for (int i = 0; i < 4; ++i)
        if ((b >> (8 * i)) & 0xE0u) b |= 0x1Fu << (8 * i);
    return b & 0x1F1F1F1Fu;
}

// Twelve digits -> four trytes d0 + 3 d1 + 9 d2 (the offset 13 is the three digits' own 1 + 3 + 9), each formed in the top
// byte of its sum: no sum of three digits carries out of its byte.
__device__ __forceinline__ uint32_t digits_word(uint32_t w0, uint32_t w1, uint32_t w2) {
    const uint32_t t0 = w0 * 0x01030900u, t1 = w1 * 0x03090000u + w0, t2 = w2 * 0x09000000u + w1 * 0x00000103u, t3 = w2 * 0x00010309u;
    return __byte_perm(__byte_perm(t0, t1, 0x0073), __byte_perm(t2, t3, 0x0073), 0x5410);
}

// 16 bytes of packed limbs from / to an address that is a multiple of `align` (16, 8 or 1).
__device__ __forceinline__ uint32_t bytes_word(const uint8_t *p) { return (uint32_t)p[0] | (uint32_t)p[1] << 8 | (uint32_t)p[2] << 16 | (uint32_t)p[3] << 24; }
__device__ __forceinline__ uint4 load_limb(const uint8_t *p, int align) {
    if (align == 16) return __ldg(reinterpret_cast<const uint4 *>(p));
    if (align == 8) {
        const uint2 a = __ldg(reinterpret_cast<const uint2 *>(p)), b = __ldg(reinterpret_cast<const uint2 *>(p) + 1);
        return make_uint4(a.x, a.y, b.x, b.y);
    }
    return make_uint4(bytes_word(p), bytes_word(p + 4), bytes_word(p + 8), bytes_word(p + 12));
}
__device__ __forceinline__ void store_limb(uint8_t *p, const uint4 &v, int align) {
    if (align == 16) *reinterpret_cast<uint4 *>(p) = v;
    else if (align == 8) {
        reinterpret_cast<uint2 *>(p)[0] = make_uint2(v.x, v.y);
        reinterpret_cast<uint2 *>(p)[1] = make_uint2(v.z, v.w);
    } else {
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        for (int i = 0; i < 16; ++i) p[i] = (uint8_t)(w[i >> 2] >> (8 * (i & 3)));
    }
}

// A run's blocks in shared memory start at the same distance from a 16-byte boundary as in global memory (`lead`; an odd
// address, where nothing wider than a byte fits, at 0).  vectors [from, to) of 16 bytes, counted from that boundary, lie
// inside the run.
struct Span {
    int lead, from, to, bytes;
    __device__ Span(const uint8_t *global, int bytes_) : bytes(bytes_) {
        const uintptr_t a = reinterpret_cast<uintptr_t>(global);
        lead = a & 1 ? 0 : (int)(a & 15);
        from = (lead + 15) >> 4;
        to = (lead + bytes) >> 4;
        if ((a & 1) || to < from) to = from = 0;  // byte by byte
    }
    // Bytes before and behind the vectors, less than 16 each: the one that is this lane's, or -1.
    __device__ __forceinline__ int edge(int lane) const {
        const int i = lane < 16 ? lane : to * 16 - lead + lane - 16;
        return to > from && i < (lane < 16 ? from * 16 - lead : bytes) ? i : -1;
    }
    // Where there are no vectors: every byte, f(offset in the run).
    template <typename F> __device__ __forceinline__ void bytewise(int lane, F &&f) const {
        if (to == from)
            for (int i = lane; i < bytes; i += 32) f(i);
    }
};

// 16 bytes `part` of a block's payload: the digit words of byte m of each base-3 number (or 2-bit field), first + m * pitch.
template <int FORMAT>
__device__ __forceinline__ void payload_part(int part, int &first, int &pitch) {
    if constexpr (FORMAT == T81B200_TQ2_0) {
        first = (part >> 1) * 32 + (part & 1) * 4;
        pitch = 8;
    } else {  // parts 0 to 2
        first = part < 2 ? 4 * part : 40;
        pitch = part < 2 ? 8 : 4;
    }
}

// ceil(256 n / 243) = (69045 n + 65000) >> 16, exact for all 243 values, of the four bytes of n: a product is 24 bits, two lie
// side by side in a 64-bit one.
__device__ __forceinline__ uint32_t base3_bytes(uint32_t n) {
    constexpr uint64_t round = 65000ull | 65000ull << 24;
    const uint64_t outer = (uint64_t)(n & 0xFF0000FFu) * 69045u + round, inner = (uint64_t)__byte_perm(n, 0u, 0x2441) * 69045u + round;
    return __byte_perm(__byte_perm((uint32_t)outer, (uint32_t)inner, 0x0062), __byte_perm((uint32_t)(inner >> 32), (uint32_t)(outer >> 32), 0x0051), 0x5410);
}

// Digit m of the four bytes of a word (TQ1_0), m = 0, 1, ... in turn.
struct Base3Digits {
    uint32_t even, odd, before;
    __device__ __forceinline__ explicit Base3Digits(uint32_t x) {
        even = x & 0x00FF00FFu;
        odd = __byte_perm(x, 0u, 0x4341);
        before = 0;
    }
    __device__ __forceinline__ uint32_t next(uint32_t power) {  // 3^(m + 1)
        const uint32_t n = __byte_perm(even * power, odd * power, 0x7351), digit = n - 3u * before;
        before = n;
        return digit;
    }
};

template <int FORMAT, bool SHORT>
__global__ void __launch_bounds__(kWarps * 32, kMaxCtas) packed_to_tq_kernel(const uint8_t *__restrict__ packed, const float *__restrict__ row_scale, const Runs r,
                                                                   uint8_t *__restrict__ blocks, int align) {
    constexpr int kBytes = block_bytes(FORMAT), kParts = FORMAT == T81B200_TQ2_0 ? 4 : 3, kDigits = FORMAT == T81B200_TQ2_0 ? 4 : 5;
    __shared__ __align__(16) uint32_t table[kTableWords];
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    fill_tryte_table(table, threadIdx.x);
    __syncthreads();
    uint32_t *q = reinterpret_cast<uint32_t *>(smem + warp * warp_bytes(r.most, FORMAT));
    uint8_t *staged = reinterpret_cast<uint8_t *>(q + digit_words(r.most));
    int first, pitch;
    payload_part<FORMAT>(lane & 3, first, pitch);
    const bool has_part = (lane & 3) < kParts;
    const uint4 *part_q = reinterpret_cast<const uint4 *>(q + (lane >> 2) * kBlockPitch + first);
    pitch >>= 2;
    // the lane's limbs of a run are 32 apart: six blocks
    uint32_t *limb_q[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) limb_q[j] = q + digit_place<false>(12 * lane + 4 * j, 0);
    uint4 in[kLimbSlots];
    auto fetch = [&](const Run &run) {
        const int slots = (run.n * 16 + 2) / 3, all = run.rows * slots, left = (int)r.limbs_per_row - run.piece * (kRunBlocks * 16 / 3);
        const uint8_t *src = packed + (run.row * r.limbs_per_row + run.piece * (kRunBlocks * 16 / 3)) * 16;
#pragma unroll
        for (int i = 0; i < kLimbSlots; ++i) {
            int limb = lane + 32 * i;
            bool exists = limb < all && limb < left;
            if (SHORT) {
                const int row = (int)((unsigned)limb / (unsigned)slots), s = limb - row * slots;
                exists = limb < all && s < left;
                limb = row * left + s;
            }
            in[i] = make_uint4(kZeroTryteWord, kZeroTryteWord, kZeroTryteWord, kZeroTryteWord);
            if (exists) in[i] = load_limb(src + 16 * limb, align);
        }
    };
    uint32_t at = blockIdx.x * kWarps + warp;
    Run next = locate<SHORT>(r, at);
    if (at < r.total) fetch(next);
    while (at < r.total) {
        const Run run = next;
        // limbs of a row of the run, counted to the end of its blocks (the last of them need not exist: zero trits)
        const int slots = (run.n * 16 + 2) / 3, all = run.rows * slots, n_blocks = run.rows * run.n;
        __syncwarp();  // the run before has been read
#pragma unroll
        for (int i = 0; i < kLimbSlots; ++i) {
            if (lane + 32 * i >= all) break;
            if ((in[i].x | in[i].y | in[i].z | in[i].w) & 0xE0E0E0E0u)
                in[i] = make_uint4(only_trytes(in[i].x), only_trytes(in[i].y), only_trytes(in[i].z), only_trytes(in[i].w));
            uint32_t w[12];
            word_digits(in[i].x, table, 4u * lane, w, 0);
            word_digits(in[i].y, table, 4u * lane, w, 3);
            word_digits(in[i].z, table, 4u * lane, w, 6);
            word_digits(in[i].w, table, 4u * lane, w, 9);
            const int row = SHORT ? (lane + 32 * i) / slots : 0, s = lane + 32 * i - row * slots;
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                uint32_t *to = SHORT ? q + row * run.n * kBlockPitch + digit_place<true>(12 * s + 4 * j, run.n) : limb_q[j] + i * 6 * kBlockPitch;
                *reinterpret_cast<uint4 *>(to) = make_uint4(w[4 * j], w[4 * j + 1], w[4 * j + 2], w[4 * j + 3]);
            }
        }
        const float scale = lane < n_blocks && row_scale ? row_scale[run.row + (SHORT ? lane / run.n : 0)] : 1.0f;
        at += gridDim.x * kWarps;
        if (at < r.total) {  // the next run's limbs come while this one's blocks are made
            next = locate<SHORT>(r, at);
            fetch(next);
        }
        __syncwarp();
        clear_past_end<SHORT>(q, r, run, lane);
        uint8_t *out = blocks + (run.row * r.blocks_per_row + run.piece * kRunBlocks) * kBytes;
        const Span span(out, n_blocks * kBytes);
        uint8_t *image = staged + span.lead;
        uint32_t differs = 0;  // which parts of the lane's own block hold a non-zero trit
        const uint4 *d = part_q;
        uint16_t *dst = reinterpret_cast<uint16_t *>(image + (lane >> 2) * kBytes + 16 * (lane & 3));
        for (int pass = 0; pass * 8 < n_blocks; ++pass, d += 2 * kBlockPitch, dst += 4 * kBytes) {
            bool nonzero = false;
            if (has_part && pass * 8 + (lane >> 2) < n_blocks) {
                uint32_t n[4] = {0, 0, 0, 0};
#pragma unroll
                for (int m = 0; m < kDigits; ++m) {
                    const uint4 x = d[(FORMAT == T81B200_TQ2_0 ? kDigits - 1 - m : m) * pitch];
                    constexpr uint32_t base = FORMAT == T81B200_TQ2_0 ? 4u : 3u;
                    n[0] = base * n[0] + x.x; n[1] = base * n[1] + x.y; n[2] = base * n[2] + x.z; n[3] = base * n[3] + x.w;
                }
                // a byte of ones only: 1 + 4 + 16 + 64, or 1 + 3 + 9 + 27 + 81
                constexpr uint32_t ones = FORMAT == T81B200_TQ2_0 ? 0x55555555u : 0x79797979u;
                nonzero = ((n[0] ^ ones) | (n[1] ^ ones) | (n[2] ^ ones) | (n[3] ^ ones)) != 0;
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t v = FORMAT == T81B200_TQ2_0 ? n[j] : base3_bytes(n[j]);
                    dst[2 * j] = (uint16_t)v;
                    dst[2 * j + 1] = (uint16_t)(v >> 16);
                }
            }
            const uint32_t votes = __ballot_sync(0xffffffffu, nonzero);
            if (lane >> 3 == pass) differs = votes >> (4 * (lane & 7)) & 15u;
        }
        if (lane < n_blocks) {
            uint16_t *tail = reinterpret_cast<uint16_t *>(image + lane * kBytes + kBytes - 2);
            if constexpr (FORMAT == T81B200_TQ1_0) {
                const uint4 x = *reinterpret_cast<const uint4 *>(q + lane * kBlockPitch + 60);
                const uint32_t n = 27u * x.x + 9u * x.y + 3u * x.z + x.w, v = base3_bytes(3u * n);  // the fifth digit is 0
                differs |= n ^ 0x28282828u;
                tail[-2] = (uint16_t)v;
                tail[-1] = (uint16_t)(v >> 16);
            }
            // the scale of a block with no non-zero trit is 0, like the absmax of an all-zero block
            tail[0] = __half_as_ushort(__float2half_rn(differs ? scale : 0.0f));
        }
        __syncwarp();
        for (int v = span.from + lane; v < span.to; v += 32)
            *reinterpret_cast<uint4 *>(out - span.lead + 16 * v) = *reinterpret_cast<const uint4 *>(staged + 16 * v);
        if (const int i = span.edge(lane); i >= 0) out[i] = image[i];
        span.bytewise(lane, [&](int i) { out[i] = image[i]; });
    }
}

template <int FORMAT, bool SHORT>
__global__ void __launch_bounds__(kWarps * 32, kMaxCtas) tq_to_packed_kernel(const uint8_t *__restrict__ blocks, const Runs r, uint8_t *__restrict__ packed,
                                                                   float *__restrict__ block_scale, int align) {
    constexpr int kBytes = block_bytes(FORMAT), kParts = FORMAT == T81B200_TQ2_0 ? 4 : 3;
    constexpr int kLoads = (kRunBlocks * kBytes / 16 + 31) / 32;
    extern __shared__ __align__(16) uint8_t smem[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t *q = reinterpret_cast<uint32_t *>(smem + warp * warp_bytes(r.most, FORMAT));
    uint8_t *staged = reinterpret_cast<uint8_t *>(q + digit_words(r.most));
    int first, pitch;
    payload_part<FORMAT>(lane & 3, first, pitch);
    const bool has_part = (lane & 3) < kParts;
    uint4 *part_q = reinterpret_cast<uint4 *>(q + (lane >> 2) * kBlockPitch + first);
    pitch >>= 2;
    const uint32_t *limb_q[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) limb_q[j] = q + digit_place<false>(12 * lane + 4 * j, 0);
    uint4 v[kLoads];
    uint8_t edge = 0;
    auto start = [&](const Run &run) { return blocks + (run.row * r.blocks_per_row + run.piece * kRunBlocks) * kBytes; };
    auto fetch = [&](const Run &run) {
        const uint8_t *in = start(run);
        const Span span(in, run.rows * run.n * kBytes);
#pragma unroll
        for (int i = 0; i < kLoads; ++i)
            if (span.from + lane + 32 * i < span.to) v[i] = __ldg(reinterpret_cast<const uint4 *>(in - span.lead + 16 * (span.from + lane + 32 * i)));
        if (const int i = span.edge(lane); i >= 0) edge = in[i];
    };
    uint32_t at = blockIdx.x * kWarps + warp;
    Run next = locate<SHORT>(r, at);
    if (at < r.total) fetch(next);
    while (at < r.total) {
        const Run run = next;
        const int n_blocks = run.rows * run.n;
        const int64_t block0 = run.row * r.blocks_per_row + run.piece * kRunBlocks;
        const uint8_t *in = start(run);
        const Span span(in, n_blocks * kBytes);
        uint8_t *image = staged + span.lead;
        __syncwarp();  // the run before has been read
        if (const int i = span.edge(lane); i >= 0) image[i] = edge;
        span.bytewise(lane, [&](int i) { image[i] = in[i]; });
#pragma unroll
        for (int i = 0; i < kLoads; ++i)
            if (span.from + lane + 32 * i < span.to) *reinterpret_cast<uint4 *>(staged + 16 * (span.from + lane + 32 * i)) = v[i];
        at += gridDim.x * kWarps;
        if (at < r.total) {  // the next run's blocks come while this one's limbs are made
            next = locate<SHORT>(r, at);
            fetch(next);
        }
        __syncwarp();
        uint4 *d = part_q;
        const uint8_t *src = image + (lane >> 2) * kBytes + 16 * (lane & 3);
        const uint32_t skew = reinterpret_cast<uintptr_t>(src) & 2, select = skew ? 0x5432 : 0x3210;  // 8 blocks further it is the same
        src -= skew;
        for (int pass = 0; pass * 8 < n_blocks; ++pass, d += 2 * kBlockPitch, src += 8 * kBytes) {
            if (!has_part || pass * 8 + (lane >> 2) >= n_blocks) continue;
            uint32_t word[5], x[4];
#pragma unroll
            for (int j = 0; j < 5; ++j) word[j] = reinterpret_cast<const uint32_t *>(src)[j];  // the last one: scale, or pad behind the image
#pragma unroll
            for (int j = 0; j < 4; ++j) x[j] = __byte_perm(word[j], word[j + 1], select);
            if constexpr (FORMAT == T81B200_TQ2_0) {
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    uint32_t y[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const uint32_t f = (x[j] >> (2 * m)) & 0x03030303u;
                        y[j] = f - (f & (f >> 1) & 0x01010101u);  // 3 reads as 2
                    }
                    d[m * 2] = make_uint4(y[0], y[1], y[2], y[3]);
                }
            } else {
                Base3Digits digit[4] = {Base3Digits(x[0]), Base3Digits(x[1]), Base3Digits(x[2]), Base3Digits(x[3])};
                uint32_t power = 1;
#pragma unroll
                for (int m = 0; m < 5; ++m) {
                    power *= 3;
                    d[m * pitch] = make_uint4(digit[0].next(power), digit[1].next(power), digit[2].next(power), digit[3].next(power));
                }
            }
        }
        if (lane < n_blocks) {
            const uint16_t *tail = reinterpret_cast<const uint16_t *>(image + lane * kBytes + kBytes - 2);
            if constexpr (FORMAT == T81B200_TQ1_0) {
                Base3Digits digit((uint32_t)tail[-2] | (uint32_t)tail[-1] << 16);
                const uint32_t d0 = digit.next(3), d1 = digit.next(9), d2 = digit.next(27), d3 = digit.next(81);
                *reinterpret_cast<uint4 *>(q + lane * kBlockPitch + 60) = make_uint4(d0, d1, d2, d3);
            }
            if (block_scale) block_scale[block0 + lane] = __half2float(__ushort_as_half(tail[0]));
        }
        __syncwarp();
        clear_past_end<SHORT>(q, r, run, lane);
        const int whole = (run.n * 16 + 2) / 3, left = (int)r.limbs_per_row - run.piece * (kRunBlocks * 16 / 3), slots = left < whole ? left : whole;
        uint8_t *dst = packed + (run.row * r.limbs_per_row + run.piece * (kRunBlocks * 16 / 3)) * 16;
#pragma unroll
        for (int i = 0; i < kLimbSlots; ++i) {
            const int limb = lane + 32 * i;  // the rows of a run follow one another in the limbs too
            if (limb >= run.rows * slots) break;
            const int row = SHORT ? limb / slots : 0, s = limb - row * slots;
            uint32_t w[12];
#pragma unroll
            for (int j = 0; j < 3; ++j) {
                const uint4 x = *reinterpret_cast<const uint4 *>(SHORT ? q + row * run.n * kBlockPitch + digit_place<true>(12 * s + 4 * j, run.n) : limb_q[j] + i * 6 * kBlockPitch);
                w[4 * j] = x.x; w[4 * j + 1] = x.y; w[4 * j + 2] = x.z; w[4 * j + 3] = x.w;
            }
            store_limb(dst + 16 * limb,
                       make_uint4(digits_word(w[0], w[1], w[2]), digits_word(w[3], w[4], w[5]), digits_word(w[6], w[7], w[8]), digits_word(w[9], w[10], w[11])), align);
        }
    }
}

// Rows of up to half a run share one, where enough runs are left to give every SM eight.  False: too many runs to count.
bool plan_runs(Runs &r, int64_t rows, int64_t cols) {
    r.rows = rows;
    r.blocks_per_row = (cols + kBlock - 1) / kBlock;
    r.limbs_per_row = (cols + 47) / 48;
    r.cols = (int)cols;
    const int64_t slots = (r.blocks_per_row * 16 + 2) / 3, blocks_fit = kRunBlocks / r.blocks_per_row, limbs_fit = 32 * kLimbSlots / slots;
    const int64_t fit = blocks_fit < limbs_fit ? blocks_fit : limbs_fit, spare = rows / ((int64_t)sm_count() * 8);
    const int64_t together = fit < spare ? fit : spare, pieces = (r.blocks_per_row + kRunBlocks - 1) / kRunBlocks;
    r.rows_per_run = (int)(together > 1 ? together : 1);
    r.runs_per_row = (uint32_t)pieces;
    r.most = (int)(r.rows_per_run * (r.blocks_per_row < kRunBlocks ? r.blocks_per_row : kRunBlocks));
    const int64_t total = r.rows_per_run > 1 ? (rows + r.rows_per_run - 1) / r.rows_per_run : rows * pieces;
    r.total = (uint32_t)total;
    return total < (1ll << 32) - (1 << 20);  // the walk's last step stays below 2^32
}

// As many CTAs as are resident together, by shared memory and by registers; more runs are walked through.
unsigned tq_grid(const Runs &r, int cta_bytes) {
    const int fit = 227 * 1024 / (cta_bytes + 1024);
    const uint32_t ctas = (r.total - 1) / kWarps + 1, most = (uint32_t)(sm_count() * (fit < kMaxCtas ? fit : kMaxCtas));
    return ctas < most ? ctas : most;
}

int limb_alignment(const void *p) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    return a % 16 == 0 ? 16 : (a % 8 == 0 ? 8 : 1);
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
    Runs runs;
    if ((cols + kBlock - 1) / kBlock > 65535 || rows >= (1ll << 31) || !plan_runs(runs, rows, cols)) return fail(T81B200_ELIMIT, "tq: matrix too large for one call");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool tq2 = format == T81B200_TQ2_0, together = runs.rows_per_run > 1;
    const auto kernel = tq2 ? (together ? packed_to_tq_kernel<T81B200_TQ2_0, true> : packed_to_tq_kernel<T81B200_TQ2_0, false>)
                            : (together ? packed_to_tq_kernel<T81B200_TQ1_0, true> : packed_to_tq_kernel<T81B200_TQ1_0, false>);
    const int bytes = kWarps * warp_bytes(runs.most, format);
    kernel<<<tq_grid(runs, bytes + kTableWords * 4), kWarps * 32, bytes, st>>>(packed, row_scale, runs, blocks, limb_alignment(packed));
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
    Runs runs;
    if ((cols + kBlock - 1) / kBlock > 65535 || rows >= (1ll << 31) || !plan_runs(runs, rows, cols)) return fail(T81B200_ELIMIT, "tq: matrix too large for one call");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool tq2 = format == T81B200_TQ2_0, together = runs.rows_per_run > 1;
    const auto kernel = tq2 ? (together ? tq_to_packed_kernel<T81B200_TQ2_0, true> : tq_to_packed_kernel<T81B200_TQ2_0, false>)
                            : (together ? tq_to_packed_kernel<T81B200_TQ1_0, true> : tq_to_packed_kernel<T81B200_TQ1_0, false>);
    const int bytes = kWarps * warp_bytes(runs.most, format);
    kernel<<<tq_grid(runs, bytes), kWarps * 32, bytes, st>>>(blocks, runs, packed, block_scale, limb_alignment(packed));
    T81_LAUNCH_CHECK("tq_to_packed_kernel");
    note_weights_written(st);
    return T81B200_OK;
}
