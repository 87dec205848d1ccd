// Quantisation-aware-training forward of the ternary Linear (t81/nn/linear.py:72-99 with t81/qat.py:12-57 of the
// reference), the two steps that touch every weight fused into two streaming kernels:
//   1. the running scale: candidate = max |w| over the whole weight, clamped to >= 1e-6, blended into the stored
//      scale with momentum 0.99 (_update_training_scale) — one reduction kernel, the blend done by the last CTA;
//   2. quantise + pack: trit = Q(w / scale, threshold) with the reference's rule (clamp to [-1, 1], |.| >= threshold
//      keeps the sign), written straight into the packed-limb layout, and the scale broadcast into a per-row
//      vector — so the forward product runs on the packed-trit matmul kernels with that vector as row scale and
//      no fp32 copy of the quantised weight is ever materialised (the reference builds quantized * scale in full).
// Both read the weight once (4 bytes per weight for fp32) and write 1/3 byte per weight: HBM-bound streams.
#include "common.cuh"

namespace t81b200 {

namespace {

// state[0]: the running scale (in/out)   state[1]: max |w| of this call as float bits (scratch, zero between calls)
// state[2]: CTAs that have contributed (scratch, zero between calls)   state[3]: 1 once state[0] holds a scale
// VEC elements per load (16 bytes, four of them in flight per thread) over a weight without gaps between its rows, or
// single elements row by row.  Bound by memory: 14336 x 4096 fp32 (235 MB, more than L2) 63 us = 3.7 TB/s.
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

// Quantise straight into the decode-stream layout of the weight (forward product) and of its transpose (input
// gradient), in one pass over the weight.  A CTA takes 96 rows x 192 columns: three blocks of the weight's layout and half of six
// of the transpose's.  Warp w owns columns 32 w .. + 31, a lane one column, and walks the 96 rows (whole 128-byte
// reads, eight rows ahead of use: with nothing in flight while eight rows are packed the pass took 90 us):
//   transpose: the lane's column is a row of it; eight rows in turn fill one half of a word (two bits each, at the
//              places the layout wants), the lane eight columns on supplies the other half;
//   weight:    two ballots per row hold 32 columns of it; lane r keeps those of row r of a 32-row tile and spreads its
//              four bytes of each to word positions with a table.
// Blocks are put together in shared memory and leave as contiguous runs (4.5 KB, and 96 bytes of the transpose).  The rows
// are taken last first: the scale's reduction has just read the weight front to back, and its end is still in L2.
__device__ __forceinline__ uint32_t spread_place(int c) { return (c & 1 ? 30u : 14u) - 4u * (uint32_t)(c >> 1); }  // of column c of eight, first row of the pair

// The rule compares w / scale, rounded, with the threshold, and keeps zeros (t81/qat.py:12-25).  Rounded division is
// monotonic, so that is a comparison of |w| with the smallest value whose quotient reaches the threshold and is not
// zero: bisected over the floats' bit patterns, from within four ulp of thr * scale where that brackets it.  (A division
// per weight in the unrolled loop below would not fit the instruction cache: 33 us for 4096 x 4096 instead of 14.)
__device__ float quotient_cut(float thr, float scale) {
    auto reaches = [&](uint32_t bits) {
        const float q = __fdiv_rn(__uint_as_float(bits), scale);
        return q >= thr && q > 0.0f;
    };
    const uint32_t guess = __float_as_uint(__fmul_rn(thr, scale));
    uint32_t lo = guess > 4u ? guess - 4u : 0u, hi = guess + 4u;  // lo: below the cut, hi: at or above it
    if (reaches(lo) || !reaches(hi)) { lo = 0u; hi = 0x7F800000u; }
    while (hi - lo > 1u) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (reaches(mid)) hi = mid;
        else lo = mid;
    }
    return __uint_as_float(hi);
}

__global__ void __launch_bounds__(192) qat_quantize_t2_kernel(const float *__restrict__ w, int64_t rows, int64_t cols, int64_t ld, float thr,
                                                              const float *__restrict__ scale_ptr, uint8_t *__restrict__ t2,
                                                              uint8_t *__restrict__ t2_t, float *__restrict__ scale_out, int64_t n_scales) {
    __shared__ uint32_t spread[256];
    __shared__ __align__(16) uint32_t fwd[3 * 384], trn[6 * 192];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const float scale = *scale_ptr;
    for (int64_t i = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) * 192 + tid; i < n_scales; i += (int64_t)gridDim.x * gridDim.y * 192) scale_out[i] = scale;
    for (int b = tid; b < 256; b += 192) {
        uint32_t v = 0;
        for (int c = 0; c < 8; ++c) v |= (uint32_t)((b >> c) & 1) << spread_place(c);
        spread[b] = v;
    }
    const float cut = quotient_cut(thr, scale);
    __syncthreads();
    const int64_t rb = gridDim.y - 1 - blockIdx.y, row0 = rb * 96, col = (int64_t)blockIdx.x * 192 + 32 * warp + lane;
    const bool col_ok = col < cols;
    const float *src = w + row0 * ld + col;
    const int gr = lane >> 4, g = lane & 7;
    auto load8 = [&](int first, float (&v)[8]) {
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = col_ok && first < 96 && row0 + first + i < rows ? __ldg(src + (int64_t)(first + i) * ld) : 0.0f;
    };
    float v[8];
    load8(0, v);
    uint32_t my_nz = 0, my_neg = 0;
#pragma unroll 4
    for (int og = 0; og < 12; ++og) {  // groups of eight rows of the weight = eight columns of the transpose
        float ahead[8];
        load8(8 * og + 8, ahead);
        uint32_t half = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const bool nz = fabsf(v[i]) >= cut;
            const bool neg = nz && v[i] < 0.0f;
            const uint32_t nz_mask = __ballot_sync(0xffffffffu, nz), neg_mask = __ballot_sync(0xffffffffu, neg);
            if (lane == 8 * (og & 3) + i) { my_nz = nz_mask; my_neg = neg_mask; }
            half |= ((neg ? 2u : 0u) | (nz ? 1u : 0u)) << spread_place(i);
        }
        if (t2_t) {
            // word 6 gr + og % 6 of lane 4 g + t, t = 2 * (rb % 2) + og / 6: two of a block's four runs are this CTA's
            const uint32_t word = half | (__shfl_down_sync(0xffffffffu, half, 8) >> 2);
            if (!(lane & 8)) trn[warp * 192 + (2 * g + og / 6) * 12 + 6 * gr + og % 6] = word;
        }
        if ((og & 3) == 3) {
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const uint32_t h = spread[(my_nz >> (8 * b)) & 0xFFu] | (spread[(my_neg >> (8 * b)) & 0xFFu] << 1);
                const uint32_t word = h | (__shfl_down_sync(0xffffffffu, h, 8) >> 2);
                const int kg = 4 * warp + b;
                if (!(lane & 8)) fwd[(og >> 2) * 384 + (4 * g + kg / 6) * 12 + 6 * gr + kg % 6] = word;
            }
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = ahead[i];
    }
    __syncthreads();
    // block (chunk, row tile) of the weight: chunk = blockIdx.x, row tiles 3 rb ..; of the transpose: chunk rb / 2, row tiles 6 blockIdx.x ..
    const int64_t tiles = (rows + 31) / 32, tiles_t = (cols + 31) / 32;
    {
        const int64_t left = tiles - rb * 3;
        const int n = (int)(left < 3 ? left : 3) * 96;
        uint4 *dst = reinterpret_cast<uint4 *>(t2 + ((int64_t)blockIdx.x * tiles + rb * 3) * 1536);
        for (int i = tid; i < n; i += 192) dst[i] = reinterpret_cast<const uint4 *>(fwd)[i];
    }
    if (t2_t) {
        const int64_t left = tiles_t - (int64_t)blockIdx.x * 6;
        const int n = (int)(left < 6 ? left : 6) * 48;  // per block: 8 runs of 6 pieces
        uint8_t *out = t2_t + ((rb >> 1) * tiles_t + (int64_t)blockIdx.x * 6) * 1536 + (rb & 1) * 96;
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
    const dim3 grid((unsigned)((cols + 191) / 192), (unsigned)((rows + 95) / 96));
    if (cols > (1ll << 31) || grid.y > 65535u) return fail(T81B200_ELIMIT, "qat_quantize_t2: matrix too large for one call");
    qat_quantize_t2_kernel<<<grid, 192, 0, static_cast<cudaStream_t>(stream)>>>(w, rows, cols, ld, threshold, scale, t2, t2_transposed, scale_out, n_scales);
    T81_LAUNCH_CHECK("qat_quantize_t2_kernel");
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
