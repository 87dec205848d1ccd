// Passes over the weight of the ternary Linear's training step (t81/nn/linear.py:72-99 with t81/qat.py:12-57 of the reference), and
// the bias gradient:
//   absmax_ema_kernel       the running scale: candidate = max |w| over the whole weight, clamped to >= 1e-6, blended into the stored
//                           scale with momentum 0.99 (_update_training_scale) — one reduction, the blend done by the last CTA;
//   qat_quantize_t2_kernel  trit = Q(w / scale, threshold) with the reference's rule (clamp to [-1, 1], |.| >= threshold keeps the sign)
//                           straight into the decode-stream layout of the weight (forward) and of its transpose (input gradient), and
//                           the scale as a vector of row scales: no fp32 copy of the quantised weight is ever made;
//   qat_quantize_pack_kernel  the same quantiser into limbs, for callers of the C interface;
//   column_sums_kernel      the output gradient summed over the tokens.
// The first two read the weight once each (4 bytes per weight) and are bound by memory.
#include "common.cuh"
#include "launch_order.cuh"

namespace t81b200 {

namespace {

// state[0]: the running scale (in/out)   state[1]: max |w| of this call as float bits (scratch, zero between calls)
// state[2]: CTAs that have contributed (scratch, zero between calls)   state[3]: 1 once state[0] holds a scale
// VEC elements per load (16 bytes, four of them in flight per thread) over a weight without gaps between its rows, or
// single elements row by row.  Bound by memory: 14336 x 4096 fp32 (235 MB, more than L2) 39.7 us = 5.9 TB/s.
template <typename T, int VEC>
__global__ void __launch_bounds__(256) absmax_ema_kernel(const T *__restrict__ w, int64_t rows, int64_t cols, int64_t ld,
                                                         float momentum, float one_minus, float *__restrict__ state) {
    __shared__ float warp_max[8];
    float m = 0.0f;
    auto take = [&](float v) { const float a = fabsf(v); m = a > m ? a : m; };  // a NaN compares false and never becomes the maximum
    if constexpr (VEC > 1) {
        const int64_t n = rows * cols / VEC, stride = (int64_t)gridDim.x * 256;
        const uint4 *src = reinterpret_cast<const uint4 *>(w);
        int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
        auto take16 = [&](const uint4 &q) {
            const T *e = reinterpret_cast<const T *>(&q);
#pragma unroll
            for (int j = 0; j < VEC; ++j) take(to_float<T>(e[j]));
        };
        for (; i + 3 * stride < n; i += 4 * stride) {
            uint4 q[4];
#pragma unroll
            for (int u = 0; u < 4; ++u) q[u] = __ldg(src + i + u * stride);
#pragma unroll
            for (int u = 0; u < 4; ++u) take16(q[u]);
        }
        for (; i < n; i += stride) take16(__ldg(src + i));
        if (blockIdx.x == 0)
            for (int64_t j = n * VEC + threadIdx.x; j < rows * cols; j += 256) take(to_float<T>(w[j]));
    } else {
        for (int64_t r = blockIdx.x; r < rows; r += gridDim.x)
            for (int64_t c = threadIdx.x; c < cols; c += 256) take(to_float<T>(w[r * ld + c]));
    }
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) take(__shfl_down_sync(0xffffffffu, m, off));
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int j = 1; j < 8; ++j) m = warp_max[j] > m ? warp_max[j] : m;
        unsigned int *bits = reinterpret_cast<unsigned int *>(state + 1);
        unsigned int *ticket = reinterpret_cast<unsigned int *>(state + 2);
        atomicMax(bits, __float_as_uint(m));  // non-negative floats order like their bit patterns
        __threadfence();
        if (atomicAdd(ticket, 1u) == gridDim.x - 1) {
            // the last CTA blends and resets the scratch words for the next call
            __threadfence();
            float candidate = __uint_as_float(atomicExch(bits, 0u));
            candidate = candidate < 1e-6f ? 1e-6f : candidate;
            float scale = candidate;
            if (state[3] != 0.0f) {
                scale = __fadd_rn(__fmul_rn(state[0], momentum), __fmul_rn(candidate, one_minus));
                scale = scale < 1e-6f ? 1e-6f : scale;
            }
            state[0] = scale;
            state[3] = 1.0f;
            *ticket = 0u;
        }
    }
}

// One thread per output word: 12 weights -> 4 tryte bytes.
template <typename T>
__global__ void __launch_bounds__(256) qat_quantize_pack_kernel(const T *__restrict__ w, int64_t rows, int64_t cols, int64_t ld,
                                                                float thr, const float *__restrict__ scale_ptr,
                                                                uint8_t *__restrict__ packed, float *__restrict__ row_scale) {
    const float scale = *scale_ptr;
    const int64_t kl = (cols + 47) / 48, words_per_row = kl * 4, total = rows * words_per_row;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        const int64_t r = i / words_per_row, q = i - r * words_per_row;
        const T *row = w + r * ld;
        uint32_t word = 0;
#pragma unroll
        for (int t = 0; t < 4; ++t) {
            uint32_t tryte = 0, weight = 1;
#pragma unroll
            for (int d = 0; d < 3; ++d, weight *= 3) {
                const int64_t c = 12 * q + 3 * t + d;
                uint32_t digit = 1;
                if (c < cols) {
                    const float x = __fdiv_rn(to_float<T>(row[c]), scale);  // weight / scale, as the reference divides
                    // |clamp(x)| >= thr keeps sign(x): the clamp changes neither compare (thr <= 1), a zero stays zero
                    digit = (x >= thr && x > 0.0f) ? 2u : ((x <= -thr && x < 0.0f) ? 0u : 1u);
                }
                tryte += digit * weight;
            }
            word |= tryte << (8 * t);
        }
        reinterpret_cast<uint32_t *>(packed)[i] = word;
        if (row_scale && q == 0) row_scale[r] = scale;
    }
}

// The rule compares w / scale, rounded, with the threshold, and keeps zeros (t81/qat.py:12-25).  Rounded division is
// monotonic, so that is a comparison of |w| with the smallest value whose quotient reaches the threshold and is not
// zero: bisected over the floats' bit patterns, from within four ulp of thr * scale where that brackets it.  Under a scale that is
// not finite no quotient reaches anything (inf / inf is no number): the cut is no number then, and no weight reaches that.
__device__ float quotient_cut(float thr, float scale) {
    auto reaches = [&](uint32_t bits) {
        const float q = __fdiv_rn(__uint_as_float(bits), scale);
        return q >= thr && q > 0.0f;
    };
    const uint32_t guess = __float_as_uint(__fmul_rn(thr, scale));
    uint32_t lo = guess > 4u ? guess - 4u : 0u, hi = guess + 4u;  // lo: below the cut, hi: at or above it
    if (reaches(lo) || !reaches(hi)) { lo = 0u; hi = 0x7F800000u; }
    if (!reaches(hi)) return __uint_as_float(0x7FC00000u);
    while (hi - lo > 1u) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (reaches(mid)) hi = mid;
        else lo = mid;
    }
    return __uint_as_float(hi);
}

// Quantise straight into the decode-stream layout of the weight (forward product) and of its transpose (input
// gradient), in one pass over the weight.  A CTA takes 96 rows x 384 columns: six blocks of the weight's layout and half
// of twelve of the transpose's.  A warp takes 16 rows x 128 columns at a time, a lane four columns: whole 512-byte row
// pieces, 16 loads in flight per lane.
//   A trit y = -1, 0, +1 is a compare and a sign; its code in the layout is the 2-bit two's complement of y.  Fields that
//   hold y + 2 do not borrow from each other, and (y + 2) ^ 2 is that code: so a lane's share of a word is a float sum of
//   y * 4^place (eight fields in two bytes 16 bits apart: exact), turned to an integer, plus 0xAA in each byte, exclusive-or
//   the same.  Four instructions a weight for both layouts.
//   A word of the weight's layout is 8 columns of 2 rows (g, g + 8): two neighbouring lanes' shares; a word of the
//   transpose's is 8 rows of 2 columns (c, c + 8): those of two lanes 2 apart.  Each pair of lanes exchanges half its shares
//   and finishes the other half.
// Blocks are put together in shared memory and leave as contiguous runs.  The rows are taken last first: the scale's
// reduction has just read the weight front to back, and its end is still in L2.  14336 x 4096: 110 us with two ballots and
// ten bit operations a weight (issue-bound), 51 us this way, 39 behind that reduction; 264 MB cross memory (41 us).
template <bool VEC>
__global__ void __launch_bounds__(192) qat_quantize_t2_kernel(const float *__restrict__ w, int64_t rows, int64_t cols, int64_t ld, float thr,
                                                              const float *__restrict__ scale_ptr, uint8_t *__restrict__ t2,
                                                              uint8_t *__restrict__ t2_t, float *__restrict__ scale_out, int64_t n_scales) {
    __shared__ __align__(16) uint32_t fwd[6 * 384], trn[12 * 192];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float scale = *scale_ptr;
    for (int64_t i = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * 192 + tid; i < n_scales; i += (int64_t)gridDim.x * gridDim.y * 192) scale_out[i] = scale;
    const float cut = quotient_cut(thr, scale);
    const int64_t rb = gridDim.y - 1 - blockIdx.y, row0 = rb * 96, col0 = (int64_t)blockIdx.x * 384;
    const int wx = warp % 3, col8 = wx * 16 + (lane >> 1);  // this lane's group of eight columns in the CTA's 48
    const int64_t col = col0 + wx * 128 + lane * 4;
    const float *src = w + row0 * ld + col;
    // word q of the weight's layout goes to fwd_at + q * 48 (its row pair) + tile; half of the row pairs each
    const int odd = lane & 1, upper = (lane >> 1) & 1;
    const int fwd_at = (col8 / 24) * (3 * 384) + (col8 % 24 / 6) * 12 + col8 % 6 + odd * (4 * 48);
    const int trn_at = (wx * 4 + (lane >> 3)) * 192 + (8 * odd) * 12 + ((lane >> 2) & 1) * 6;
    for (int rs = warp / 3; rs < 6; rs += 2) {
        float4 v[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float *p = src + (int64_t)(16 * rs + r) * ld;
            v[r] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (row0 + 16 * rs + r < rows) {
                if constexpr (VEC) {
                    if (col < cols) v[r] = __ldg(reinterpret_cast<const float4 *>(p));
                } else {
                    if (col < cols) v[r].x = __ldg(p);
                    if (col + 1 < cols) v[r].y = __ldg(p + 1);
                    if (col + 2 < cols) v[r].z = __ldg(p + 2);
                    if (col + 3 < cols) v[r].w = __ldg(p + 3);
                }
            }
        }
        float fs[8], ts[4][4];  // shares: row pairs; columns x groups of four rows
#pragma unroll
        for (int i = 0; i < 8; ++i) fs[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
            for (int i = 0; i < 4; ++i) ts[c][i] = 0.0f;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float e[4] = {v[r].x, v[r].y, v[r].z, v[r].w};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float nz = fabsf(e[c]) >= cut ? 1.0f : 0.0f;
                const float y = __uint_as_float(__float_as_uint(nz) | (__float_as_uint(e[c]) & 0x80000000u));
                // fields of four: the first two of a parity at bits 6 and 2, odd ones 16 higher; the second of a pair 2 lower
                fs[r & 7] = fmaf(y, (float)(1 << ((c & 1 ? 22 : 6) - 4 * (c >> 1) - (r >> 3 ? 2 : 0))), fs[r & 7]);
                ts[c][r >> 2] = fmaf(y, (float)(1 << ((r & 1 ? 22 : 6) - 4 * ((r & 3) >> 1))), ts[c][r >> 2]);
            }
        }
        // every place taken (0xAA per byte), and every other one (0x88)
        auto part = [](float sum) { return (uint32_t)((int)sum + 0x00880088) ^ 0x00880088u; };
        auto codes = [](float sum) { return (uint32_t)((int)sum + 0x00AA00AA) ^ 0x00AA00AAu; };
        uint32_t *out = fwd + fwd_at + (rs >> 1) * 384 + 6 * (rs & 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t a = codes(fs[i]), b = codes(fs[4 + i]);
            const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? a : b, 1);
            out[i * 48] = odd ? (got << 8) | b : (a << 8) | got;
        }
        if (t2_t) {
            // fields 2 bits apart are this column's; the column 8 on takes the places between them
            const int group = 2 * rs + upper;  // eight rows: 0 .. 11
            uint32_t *to = trn + trn_at + (group / 6) * 12 + group % 6;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const uint32_t a = (part(ts[c][0]) << 8) | part(ts[c][1]), b = (part(ts[c][2]) << 8) | part(ts[c][3]);
                const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? a : b, 2);
                to[c * 24] = upper ? got | (b >> 2) : a | (got >> 2);
            }
        }
    }
    __syncthreads();
    // block (chunk, row tile) of the weight: chunks 2 blockIdx.x, + 1, row tiles 3 rb ..; of the transpose: chunk rb / 2, row tiles 12 blockIdx.x ..
    const int64_t tiles = (rows + 31) / 32, tiles_t = (cols + 31) / 32, chunks = (cols + 191) / 192;
    for (int ch = 0; ch < 2; ++ch) {
        const int64_t chunk = (int64_t)blockIdx.x * 2 + ch;
        if (chunk >= chunks) break;
        const int64_t left = tiles - rb * 3;
        const int n = (int)(left < 3 ? left : 3) * 96;
        uint4 *dst = reinterpret_cast<uint4 *>(t2 + (chunk * tiles + rb * 3) * 1536);
        for (int i = tid; i < n; i += 192) dst[i] = reinterpret_cast<const uint4 *>(fwd + ch * 1152)[i];
    }
    if (t2_t) {
        const int64_t left = tiles_t - (int64_t)blockIdx.x * 12;
        const int n = (int)(left < 12 ? left : 12) * 48;  // per block: 8 runs of 6 pieces
        uint8_t *out = t2_t + ((rb >> 1) * tiles_t + (int64_t)blockIdx.x * 12) * 1536 + (rb & 1) * 96;
        for (int i = tid; i < n; i += 192) *reinterpret_cast<uint4 *>(out + i / 6 * 192 + i % 6 * 16) = reinterpret_cast<const uint4 *>(trn)[i];
        // an odd number of 96-row parts: the last chunk's other half is past the matrix
        if (rb == gridDim.y - 1 && !(rb & 1))
            for (int i = tid; i < n; i += 192) *reinterpret_cast<uint4 *>(out + 96 + i / 6 * 192 + i % 6 * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
}

// Column sums of a token-major matrix (the bias gradient): 32 columns per CTA, 32 warps of it take every 32nd row, eight
// rows in flight; fp32 sums, folded in a fixed order.
template <typename T>
__global__ void __launch_bounds__(1024) column_sums_kernel(const T *__restrict__ g, int64_t tokens, int64_t cols, int64_t ld, float *__restrict__ out) {
    __shared__ float part[32][33];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t col = (int64_t)blockIdx.x * 32 + lane;
    float sum = 0.0f;
    if (col < cols) {
        int64_t t = warp;
        for (; t + 7 * 32 < tokens; t += 8 * 32) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = to_float<T>(g[(t + 32 * i) * ld + col]);
#pragma unroll
            for (int i = 0; i < 8; ++i) sum += v[i];
        }
        for (; t < tokens; t += 32) sum += to_float<T>(g[t * ld + col]);
    }
    part[warp][lane] = sum;
    __syncthreads();
    float v = part[lane][warp];  // warp = column now
#pragma unroll
    for (int off = 16; off >= 1; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (lane == 0 && (int64_t)blockIdx.x * 32 + warp < cols) out[(int64_t)blockIdx.x * 32 + warp] = v;
}

template <typename T>
void launch_absmax(const void *w, int64_t rows, int64_t cols, int64_t ld, float momentum, float one_minus, float *state, cudaStream_t st) {
    constexpr int kVec = 16 / (int)sizeof(T);
    const T *src = static_cast<const T *>(w);
    const int64_t cap = (int64_t)sm_count() * 8;
    if ((ld == cols || rows == 1) && reinterpret_cast<uintptr_t>(w) % 16 == 0) {
        int64_t blocks = (rows * cols + 256 * kVec * 4 - 1) / (256 * kVec * 4);
        blocks = blocks < 1 ? 1 : (blocks > cap ? cap : blocks);
        absmax_ema_kernel<T, kVec><<<(unsigned)blocks, 256, 0, st>>>(src, rows, cols, ld, momentum, one_minus, state);
    } else {
        const int64_t blocks = rows < 1 ? 1 : (rows > cap ? cap : rows);
        absmax_ema_kernel<T, 1><<<(unsigned)blocks, 256, 0, st>>>(src, rows, cols, ld, momentum, one_minus, state);
    }
}

}  // namespace
}  // namespace t81b200

using namespace t81b200;

extern "C" int t81b200_qat_update_scale(const void *w, int w_dtype, int64_t rows, int64_t cols, int64_t ld, float momentum,
                                        float *state, void *stream) {
    if (rows < 0 || cols < 0 || ld < cols) return fail(T81B200_EINVAL, "qat_update_scale: bad dimensions");
    if (!(momentum >= 0.0f && momentum <= 1.0f)) return fail(T81B200_EINVAL, "qat_update_scale: momentum must be in [0, 1]");
    if (int rc = check_device()) return rc;
    if (!state || ((rows > 0 && cols > 0) && !w)) return fail(T81B200_EINVAL, "qat_update_scale: null pointer");
    const float one_minus = (float)(1.0 - (double)momentum);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (w_dtype) {
        case T81B200_F32: launch_absmax<float>(w, rows, cols, ld, momentum, one_minus, state, st); break;
        case T81B200_BF16: launch_absmax<__nv_bfloat16>(w, rows, cols, ld, momentum, one_minus, state, st); break;
        case T81B200_F16: launch_absmax<__half>(w, rows, cols, ld, momentum, one_minus, state, st); break;
        default: return fail(T81B200_EINVAL, "qat_update_scale: unknown dtype %d", w_dtype);
    }
    T81_LAUNCH_CHECK("absmax_ema_kernel");
    return T81B200_OK;
}

extern "C" int t81b200_qat_quantize_pack(const void *w, int w_dtype, int64_t rows, int64_t cols, int64_t ld, float threshold,
                                         const float *scale, uint8_t *packed, float *row_scale, void *stream) {
    if (rows < 0 || cols < 0 || ld < cols) return fail(T81B200_EINVAL, "qat_quantize_pack: bad dimensions");
    if (!(threshold >= 0.0f && threshold <= 1.0f)) return fail(T81B200_EINVAL, "threshold must be between 0 and 1");
    if (int rc = check_device()) return rc;
    if (rows == 0 || cols == 0) return T81B200_OK;
    if (!w || !scale || !packed) return fail(T81B200_EINVAL, "qat_quantize_pack: null pointer");
    if (reinterpret_cast<uintptr_t>(packed) % 4 != 0) return fail(T81B200_EALIGN, "qat_quantize_pack: packed must be 4-byte aligned");
    const int64_t total = rows * ((cols + 47) / 48) * 4;
    int64_t blocks = (total + 255) / 256;
    const int64_t cap = (int64_t)sm_count() * 16;
    blocks = blocks > cap ? cap : blocks;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (w_dtype) {
        case T81B200_F32: qat_quantize_pack_kernel<float><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const float *>(w), rows, cols, ld, threshold, scale, packed, row_scale); break;
        case T81B200_BF16: qat_quantize_pack_kernel<__nv_bfloat16><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const __nv_bfloat16 *>(w), rows, cols, ld, threshold, scale, packed, row_scale); break;
        case T81B200_F16: qat_quantize_pack_kernel<__half><<<(unsigned)blocks, 256, 0, st>>>(static_cast<const __half *>(w), rows, cols, ld, threshold, scale, packed, row_scale); break;
        default: return fail(T81B200_EINVAL, "qat_quantize_pack: unknown dtype %d", w_dtype);
    }
    T81_LAUNCH_CHECK("qat_quantize_pack_kernel");
    note_weights_written(st);
    return T81B200_OK;
}

extern "C" int t81b200_qat_quantize_t2(const float *w, int64_t rows, int64_t cols, int64_t ld, float threshold, const float *scale, uint8_t *t2,
                                       uint8_t *t2_transposed, float *scale_out, int64_t n_scales, void *stream) {
    if (rows < 0 || cols < 0 || ld < cols || n_scales < 0) return fail(T81B200_EINVAL, "qat_quantize_t2: bad dimensions");
    if (!(threshold >= 0.0f && threshold <= 1.0f)) return fail(T81B200_EINVAL, "threshold must be between 0 and 1");
    if (int rc = check_device()) return rc;
    if (rows == 0 || cols == 0) return T81B200_OK;
    if (!w || !scale || !t2 || (n_scales > 0 && !scale_out)) return fail(T81B200_EINVAL, "qat_quantize_t2: null pointer");
    if (reinterpret_cast<uintptr_t>(t2) % 16 != 0 || reinterpret_cast<uintptr_t>(t2_transposed) % 16 != 0)
        return fail(T81B200_EALIGN, "qat_quantize_t2: the outputs must be 16-byte aligned");
    const dim3 grid((unsigned)((cols + 383) / 384), (unsigned)((rows + 95) / 96));
    if (cols > (1ll << 31) || grid.y > 65535u) return fail(T81B200_ELIMIT, "qat_quantize_t2: matrix too large for one call");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (reinterpret_cast<uintptr_t>(w) % 16 == 0 && ld % 4 == 0 && cols % 4 == 0)
        qat_quantize_t2_kernel<true><<<grid, 192, 0, st>>>(w, rows, cols, ld, threshold, scale, t2, t2_transposed, scale_out, n_scales);
    else
        qat_quantize_t2_kernel<false><<<grid, 192, 0, st>>>(w, rows, cols, ld, threshold, scale, t2, t2_transposed, scale_out, n_scales);
    T81_LAUNCH_CHECK("qat_quantize_t2_kernel");
    note_weights_written(st);
    return T81B200_OK;
}

extern "C" int t81b200_column_sums(const void *g, int dtype, int64_t tokens, int64_t cols, int64_t ld, float *out, void *stream) {
    if (tokens < 0 || cols < 0 || ld < cols) return fail(T81B200_EINVAL, "column_sums: bad dimensions");
    if (int rc = check_device()) return rc;
    if (cols == 0) return T81B200_OK;
    if (!out || (tokens > 0 && !g)) return fail(T81B200_EINVAL, "column_sums: null pointer");
    const unsigned blocks = (unsigned)((cols + 31) / 32);
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (dtype) {
        case T81B200_F32: column_sums_kernel<float><<<blocks, 1024, 0, st>>>(static_cast<const float *>(g), tokens, cols, ld, out); break;
        case T81B200_BF16: column_sums_kernel<__nv_bfloat16><<<blocks, 1024, 0, st>>>(static_cast<const __nv_bfloat16 *>(g), tokens, cols, ld, out); break;
        case T81B200_F16: column_sums_kernel<__half><<<blocks, 1024, 0, st>>>(static_cast<const __half *>(g), tokens, cols, ld, out); break;
        default: return fail(T81B200_EINVAL, "column_sums: unknown dtype %d", dtype);
    }
    T81_LAUNCH_CHECK("column_sums_kernel");
    return T81B200_OK;
}
