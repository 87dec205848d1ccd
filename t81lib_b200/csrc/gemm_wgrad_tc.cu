// Weight gradient of the ternary Linear's training step (t81/nn/linear.py:72-80 through t81/qat.py:28-57 of the
// reference) on the tensor cores:
//
//   out[o][k] = slope(w[o][k]) * sum_t g[t][o] * x[t][k]        slope = 2 where |w / scale| < 0.5, else 0
//
// g (tokens, rows) and x (tokens, cols) are token-major, so both operands are contiguous along the output index and
// strided along the contraction: they are loaded as they lie (boxes of 64 columns, 128-byte swizzle) and
// read by tcgen05.mma as M- / N-major operands; nothing is transposed in memory.  One pair of CTAs (cta_group::2) per
// 256 x bn tile; each loads its own 128 columns of g and half of the tile's columns of x.
//
// 16-bit operands multiply as they are: products exact, accumulation fp32.  fp32 operands are staged as three bf16
// planes (x = p0 + p1 + p2 exactly, 24 mantissa bits) and the six plane products of weight 2^-16 and above are
// accumulated; the three left out lie below an fp32 ulp of the product.  The five small products have an accumulator of
// their own.  The tensor cores cut an accumulator off at every 16-token step instead of rounding it: 0.9e-9 of the result (root
// mean square) a token, 4.4e-6 over 4096 tokens in one piece, where fp32 sums on CUDA cores had 6e-7 for 16-bit operands and
// 1.1e-6 for fp32 ones.  So an accumulator takes a segment of the tokens only, and the epilogue warps add the segments up in
// registers, while the MMAs fill the other accumulator: 16-bit operands 64 tokens below 512 of them, 128 below 1024 and 192 from
// there on, fp32 ones 256; each the longest that is no further off than those sums were.  The results are 1.9e-7 to 2.9e-7 off at
// 4096 tokens.  A segment of 64 tokens costs 960 clocks, 500 of MMA: from an accumulator handed back to the next one full are 1300, and
// there are two.
//
// 14336 x 4096 x 4096 tokens in bf16, back to back: 365 us (390 to 400 with the weights in registers at the end of a tile); nothing is
// saturated: the rest are the ends of tiles and 13 waves of them for 12.1.  A pair tile takes 32 KB per CTA and 64 tokens of 16-bit operands.  The planes of
// fp32 operands are loaded together, once for all six products (2050 x 1537 x 1000 tokens: 64 us with a load per product,
// 56 us this way).  Tiles are walked in groups of eight row tiles so that what runs at a time shares its operands in L2.  The slope
// is applied in the epilogue, in the shared memory that the weights have come to (below).
#include "common.cuh"
#include "tma.cuh"
#include "umma.cuh"

#include <atomic>
#include <cstring>

namespace t81b200 {

namespace {

// A stage of the operand ring: per 64 columns of this CTA (two groups of g, bn / 128 of x) one box of all planes.
__host__ __device__ constexpr int token_step(int planes) { return planes == 1 ? 64 : 32; }
__host__ __device__ constexpr int group_bytes(int planes) { return planes * token_step(planes) * 128; }  // 8 KB, or 12 KB
constexpr int MAX_STAGES = 8;
constexpr int EPILOGUE_WARPS = 8;             // two per quarter of the rows: each takes every other 32-column block
constexpr int NUM_THREADS = (2 + EPILOGUE_WARPS) * 32;
constexpr int EPILOGUE_WARP0 = 2;
constexpr int MAX_SPLITS = 4;
constexpr int BLOCK_BYTES = 32 * 128;         // a block of the epilogue: 32 columns of a warp's 32 rows, fp32
constexpr int MOST_BLOCKS = 4;                // of a warp: 256 columns / 64
constexpr int MAX_SLOTS = 3;                  // blocks whose weights a warp has in shared memory or on their way there
constexpr int BARRIER_BYTES = 512;
constexpr int SMEM_LIMIT = 227 * 1024;

enum { WGRAD_STATUS_PRODUCER = 11, WGRAD_STATUS_MMA = 12, WGRAD_STATUS_EPILOGUE = 13 };
__device__ int g_wgrad_status = 0;

struct WgradParams {
    const float *w, *scale;
    float *out;
    int64_t rows, cols, ldw;
    int m_tiles, n_tiles, bn;
    int planes, token_steps;          // 1 or 3 planes (6 plane products); stages of tokens
    int segment, lead;                // token stages an accumulator takes before the epilogue adds it up; those of a tile's first two
    int splits, stages;
    uint32_t idesc;
    int slots;                        // blocks of weights a warp of the epilogue holds
    int vec;                          // TMA reads w and writes out
};

// Plane pair i of an fp32 product: planes of g and of x.
__device__ __forceinline__ void plane_pair(int i, int &a, int &b) {
    a = i == 2 || i == 3 ? 1 : (i == 5 ? 2 : 0);   // 0 0 1 1 0 2
    b = i == 1 || i == 3 ? 1 : (i == 4 ? 2 : 0);   // 0 1 0 1 2 0
}

// M- / N-major SWIZZLE_128B operand: 64-column groups `group` bytes apart, 8-token groups 1 KB apart.
__device__ __forceinline__ uint64_t umma_desc_mn(uint32_t smem_addr, uint32_t group) {
    return (uint64_t)((smem_addr >> 4) & 0x3FFF) | ((uint64_t)(group >> 4) << 16) | ((uint64_t)(1024 >> 4) << 32) |
           ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}

__device__ __forceinline__ void tma_load_3d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, int z, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(pair_leader(bar))
        : "memory");
}

// Tile number -> row and column tile: groups of eight row tiles, row fastest inside a group.
__device__ __forceinline__ void tile_at(const WgradParams &p, int tile, int &m, int &n) {
    const int group = 8 * p.n_tiles, first = tile / group * 8;
    const int height = p.m_tiles - first < 8 ? p.m_tiles - first : 8;
    const int r = tile - first * p.n_tiles;
    m = first + r % height;
    n = r / height;
}

// A block is 32 columns of a warp's 32 rows.  Its weights come into a slot of shared memory (rows of 128 bytes, 16-byte piece j of row
// r at (j ^ (r & 7)) * 16) long before the block's sums are there, the thread that has a row's sums turns them into the gradient in
// place, and the slot leaves as it came.  VEC: both ways one TMA box; otherwise, rows off 16-byte boundaries, a word a lane and row.
// Few tokens leave little beside this: with the weights in registers, half a block ahead, a tile took 7000 clocks to put out, 3800 this
// way (9472 x 4096, 64 to 511 tokens: 67 to 99 us, 60 to 78; 310 MB cross memory in 47).  Copies of the 16-byte pieces that hold an
// unaligned row, and stores of them, took longer than words do (512 tokens of 12402 by 2988: 151 us before, 124 in words, 160).
template <bool VEC>
__device__ __forceinline__ void load_block(const WgradParams &p, const CUtensorMap *map_w, uint32_t slot, uint32_t bar, int row0, int col0, int lane) {
    if constexpr (VEC) {
        if (lane == 0) {
            mbar_arrive_expect_tx(bar, BLOCK_BYTES);
            tma_load_2d(slot, map_w, col0, row0, bar);
        }
    } else {
        const int n = col0 + lane < p.cols ? (int)(p.rows - row0 < 32 ? p.rows - row0 : 32) : 0;
        const float *src = p.w + (int64_t)row0 * p.ldw + col0 + lane;
        const uint32_t dst = slot + (uint32_t)(lane & 3) * 4u;
#pragma unroll
        for (int r = 0; r < 32; ++r, src += p.ldw)
            if (r < n)
                asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + (uint32_t)r * 128u + (uint32_t)(((lane >> 2) ^ (r & 7)) << 4)), "l"(src) : "memory");
        asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
    }
}

// The weights in the slot have arrived: they become the gradient, which leaves for memory.  `refill` runs between the two, when the
// stores of the block before have had the most time to read their slot.
template <bool VEC, typename F>
__device__ __forceinline__ void emit_block(const WgradParams &p, const CUtensorMap *map_out, const float2 (&sum)[16], uint8_t *slot, int row0, int col0,
                                           int lane, float half_scale, F &&refill) {
    // |w / scale| < 0.5 exactly where |w| < scale / 2: two floats that differ do so by 2^-24 of their size or more,
    // and a quotient 2^-24 below one half does not round up to it
    auto sloped = [&](float v, float weight) { return v * (fabsf(weight) < half_scale ? 2.0f : 0.0f); };
    uint8_t *row = slot + lane * 128;
    const int turn = (lane & 7) << 4;
#pragma unroll
    for (int h = 0; h < 8; h += 4) {
        float4 w[4];  // all of them before the first store: the compiler cannot know the stores to miss them
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = *reinterpret_cast<const float4 *>(row + (((h + j) << 4) ^ turn));
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float2 a = sum[2 * (h + j)], b = sum[2 * (h + j) + 1];
            *reinterpret_cast<float4 *>(row + (((h + j) << 4) ^ turn)) = make_float4(sloped(a.x, w[j].x), sloped(a.y, w[j].y), sloped(b.x, w[j].z), sloped(b.y, w[j].w));
        }
    }
    if constexpr (VEC) {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
        refill();
        __syncwarp();
        if (lane == 0) {
            if (row0 < p.rows && col0 < p.cols) tma_store_2d(map_out, smem_u32(slot), col0, row0);
            asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
    } else {
        refill();
        __syncwarp();
        const int n = col0 + lane < p.cols ? (int)(p.rows - row0 < 32 ? p.rows - row0 : 32) : 0;
        float *out = p.out + (int64_t)row0 * p.cols + col0 + lane;
        const uint8_t *src = slot + (lane & 3) * 4;
#pragma unroll
        for (int r = 0; r < 32; ++r, out += p.cols)
            if (r < n) *out = *reinterpret_cast<const float *>(src + r * 128 + (((lane >> 2) ^ (r & 7)) << 4));
        __syncwarp();
    }
}

// sum += 32 columns of each of the warp's blocks, which lie 64 columns apart; eight columns are on their way while the eight before are
// added (the sums of a whole tile take most of a thread's registers).  SMALL: the products beside the large one, which say nothing where
// an operand is infinite (its other planes are zero).
template <bool SMALL>
__device__ __forceinline__ void add_blocks(uint32_t taddr, int blocks, float2 (&sum)[MOST_BLOCKS][16]) {
    uint32_t v[2][8];
    tmem_ld8_start(taddr, v[0]);
#pragma unroll
    for (int q = 0; q < 4 * MOST_BLOCKS; ++q) {
        if (q / 4 >= blocks) break;
        tmem_ld8_wait(v[q & 1]);
        if (q + 1 < 4 * MOST_BLOCKS && (q + 1) / 4 < blocks) tmem_ld8_start(taddr + (uint32_t)((q + 1) / 4 * 64 + (q + 1) % 4 * 8), v[(q + 1) & 1]);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float2 x = make_float2(__uint_as_float(v[q & 1][2 * i]), __uint_as_float(v[q & 1][2 * i + 1]));
            if (SMALL && !isfinite(x.x)) x.x = 0.0f;
            if (SMALL && !isfinite(x.y)) x.y = 0.0f;
            float2 &to = sum[q / 4][4 * (q % 4) + i];
            to = __fadd2_rn(to, x);
        }
    }
}

__device__ __forceinline__ void store_columns(uint32_t taddr, const float2 (&sum)[16]) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        uint32_t v[16];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            v[2 * i] = __float_as_uint(sum[8 * h + i].x);
            v[2 * i + 1] = __float_as_uint(sum[8 * h + i].y);
        }
        tmem_st16(taddr + 16u * h, v);
    }
}

template <bool VEC>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_wgrad_tc_kernel(const __grid_constant__ CUtensorMap map_g, const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                     const __grid_constant__ CUtensorMap map_out, const __grid_constant__ WgradParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *gen_base = smem_raw + (base - smem_u32(smem_raw));
    const uint32_t group = (uint32_t)group_bytes(p.planes), stage_bytes = (2u + (uint32_t)p.bn / 128u) * group;
    const uint32_t slot_off = (uint32_t)p.stages * stage_bytes, bars = base + slot_off + (uint32_t)(EPILOGUE_WARPS * p.slots * BLOCK_BYTES);
    auto full = [&](int s) { return bars + 8u * s; };
    auto empty = [&](int s) { return bars + 8u * (MAX_STAGES + s); };
    auto acc_full = [&](int s) { return bars + 8u * (2 * MAX_STAGES + s); };
    auto acc_empty = [&](int s) { return bars + 8u * (2 * MAX_STAGES + 2 + s); };
    auto slot_full = [&](int warp, int s) { return bars + 8u * (2 * MAX_STAGES + 4 + warp * MAX_SLOTS + s); };
    const uint32_t tmem_slot = bars + 8u * (2 * MAX_STAGES + 4 + EPILOGUE_WARPS * MAX_SLOTS);

    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int half = (int)(rank & 1u), slice = (int)(rank >> 1);

    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; ++s) { mbar_init(full(s), 1); mbar_init(empty(s), 1); }
        for (int s = 0; s < 2; ++s) { mbar_init(acc_full(s), 1); mbar_init(acc_empty(s), 2 * EPILOGUE_WARPS); }
        for (int s = 0; s < EPILOGUE_WARPS * MAX_SLOTS; ++s) mbar_init(slot_full(0, s), VEC ? 1 : 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 1) tmem_alloc_pair(tmem_slot);
    if (threadIdx.x == 0) {
        prefetch_map(&map_g);
        prefetch_map(&map_x);
        if (VEC) {
            prefetch_map(&map_w);
            prefetch_map(&map_out);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t *>(gen_base + (tmem_slot - base));

    const int total_tiles = p.m_tiles * p.n_tiles;
    const int n_clusters = (int)gridDim.x / (2 * p.splits), cluster_id = (int)blockIdx.x / (2 * p.splits);
    // this pair's share of the tokens, in stages
    const int s0 = (int)((int64_t)p.token_steps * slice / p.splits), s1 = (int)((int64_t)p.token_steps * (slice + 1) / p.splits);
    auto segment_end = [&](int begin) {
        const int end = begin + (begin - s0 < 2 * p.lead ? p.lead : p.segment);
        return end < s1 ? end : s1;
    };
    const int n_bufs = p.planes == 1 ? 2 : 1;  // fp32: the second buffer holds the small products
    const uint16_t pair_mask = (uint16_t)(3u << (rank & ~1u));
    const float half_scale = 0.5f * *p.scale;

    if (warp == 0) {
        Ring ring;
        bool ok = true;
        for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
            int m, n;
            tile_at(p, tile, m, n);
            const int o0 = (2 * m + half) * 128, k0 = n * p.bn + half * (p.bn / 2);
            for (int s = s0; s < s1; ++s) {
                ok = mbar_wait(empty(ring.stage), ring.phase ^ 1);
                if (!ok) break;
                const int t0 = s * token_step(p.planes);
                if (elect_one()) {
                    if (half == 0) mbar_arrive_expect_tx(full(ring.stage), 2 * stage_bytes);
                    uint32_t dst = base + (uint32_t)ring.stage * stage_bytes;
                    for (int b = 0; b < 2; ++b, dst += group) tma_load_3d_pair(dst, &map_g, o0 + 64 * b, t0, 0, full(ring.stage));
                    for (int b = 0; b < p.bn / 128; ++b, dst += group) tma_load_3d_pair(dst, &map_x, k0 + 64 * b, t0, 0, full(ring.stage));
                }
                __syncwarp();
                ring.advance(p.stages);
            }
        }
        // every commit has landed here before this CTA may end (they arrive one by one from the pair's issuing CTA)
        for (int i = 0; i < p.stages && ok; ++i) {
            ok = mbar_wait(empty(ring.stage), ring.phase ^ 1);
            ring.advance(p.stages);
        }
        if (!ok) give_up(&g_wgrad_status, WGRAD_STATUS_PRODUCER);
    } else if (warp == 1) {
        if (half == 0) {
            Ring ring;
            bool ok = true;
            int it = 0;
            // a segment of a tile after the other: `it` counts them
            int begin = s0;
            for (int tile = cluster_id; tile < total_tiles && ok; ++it) {
                const int end = segment_end(begin), buf = it % n_bufs;
                ok = mbar_wait(acc_empty(buf), ((uint32_t)(it / n_bufs) & 1u) ^ 1u);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d_tmem = tmem_base + (uint32_t)buf * 256u;
                for (int s = begin; s < end; ++s) {
                    ok = mbar_wait(full(ring.stage), ring.phase);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = umma_desc_mn(base + (uint32_t)ring.stage * stage_bytes, group);
                    const uint64_t bd = umma_desc_mn(base + (uint32_t)ring.stage * stage_bytes + 2 * group, group);
                    const uint32_t more = s != begin ? 1u : 0u;
                    if (elect_one()) {  // 16 tokens: two 1 KB groups
                        if (p.planes == 1) {
#pragma unroll
                            for (int k = 0; k < token_step(1) / 16; ++k)
                                umma_pair(d_tmem, ad + (uint64_t)(128 * k), bd + (uint64_t)(128 * k), p.idesc, k != 0 ? 1u : more);
                        } else {
                            constexpr uint64_t plane = token_step(3) * 128 >> 4;
#pragma unroll
                            for (int k = 0; k < token_step(3) / 16; ++k)
#pragma unroll
                                for (int i = 0; i < 6; ++i) {
                                    int pa, pb;
                                    plane_pair(i, pa, pb);
                                    umma_pair(d_tmem + (i == 0 ? 0u : 256u), ad + pa * plane + (uint64_t)(128 * k), bd + pb * plane + (uint64_t)(128 * k),
                                              p.idesc, k != 0 || i > 1 ? 1u : more);
                                }
                        }
                        umma_commit_pair(empty(ring.stage), pair_mask);
                    }
                    __syncwarp();
                    ring.advance(p.stages);
                }
                if (ok && elect_one()) umma_commit_pair(acc_full(buf), pair_mask);
                __syncwarp();
                begin = end;
                if (begin >= s1) { begin = s0; tile += n_clusters; }
            }
            if (!ok) give_up(&g_wgrad_status, WGRAD_STATUS_MMA);
        }
    }

    // ---- epilogue: two warps per quarter of the rows, each with every other 32-column block of the tile, or of its slice of it ----
    const bool epilogue = warp >= EPILOGUE_WARP0;
    const int ew = warp - EPILOGUE_WARP0, quarter = warp & 3, first = ew >> 2;
    const uint32_t t_lane = tmem_base + ((uint32_t)(quarter * 32) << 16);
    const int block0 = p.splits == 1 ? first : slice + p.splits * first, block_step = 2 * p.splits;
    // the warp's blocks in order, one slot after the other
    const uint32_t slot0 = slot_off + (uint32_t)(ew * p.slots * BLOCK_BYTES);
    struct Place { int row, col; };  // first row, and column of block 0
    auto place_of = [&](int tile) {
        int m, n;
        tile_at(p, tile, m, n);
        return Place{(2 * m + half) * 128 + quarter * 32, n * p.bn};
    };
    int ahead = p.slots, fetch_block = block0;  // blocks that may still be fetched
    Place place = place_of(cluster_id), next = place;
    bool in_next = false;  // where the fetches are; the last one of the next tile does not come before this tile's last block has left
    Ring fill, use;
    auto fetch = [&](bool has_next) {
        for (; ahead > 0; --ahead) {
            if (fetch_block >= p.bn / 32) {
                if (in_next || !has_next) return;
                in_next = true;
                fetch_block = block0;
            }
            load_block<VEC>(p, &map_w, base + slot0 + (uint32_t)(fill.stage * BLOCK_BYTES), slot_full(ew, fill.stage), in_next ? next.row : place.row,
                            (in_next ? next.col : place.col) + fetch_block * 32, lane);
            fill.advance(p.slots);
            fetch_block += block_step;
        }
    };
    // `freed`: the slot of the block before may be filled again once that block has been read
    auto put_out = [&](const float2 (&sum)[16], int block, bool freed, bool has_next) {
        const bool ok = __all_sync(0xffffffffu, mbar_wait(slot_full(ew, use.stage), use.phase));
        if (!ok) return false;
        emit_block<VEC>(p, &map_out, sum, gen_base + slot0 + use.stage * BLOCK_BYTES, place.row, place.col + block * 32, lane, half_scale, [&] {
            ahead += freed ? 1 : 0;
            fetch(has_next);
        });
        use.advance(p.slots);
        return true;
    };
    if (epilogue) {
        const int blocks = p.bn / 64;
        bool ok = true;
        int it = 0;
        bool freed = false;
        fetch(false);
        for (int tile = cluster_id; tile < total_tiles && ok; tile += n_clusters) {
            const bool has_next = tile + n_clusters < total_tiles;
            float2 sum[MOST_BLOCKS][16];
#pragma unroll
            for (int c = 0; c < MOST_BLOCKS; ++c)
#pragma unroll
                for (int i = 0; i < 16; ++i) sum[c][i] = make_float2(0.0f, 0.0f);
            for (int s = s0; s < s1; s = segment_end(s), ++it) {
                const int buf = it % n_bufs;
                ok = __all_sync(0xffffffffu, mbar_wait(acc_full(buf), (uint32_t)(it / n_bufs) & 1u));
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = t_lane + (uint32_t)(buf * 256 + first * 32);
                add_blocks<false>(acc, blocks, sum);
                if (p.planes > 1) add_blocks<true>(acc + 256u, blocks, sum);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(acc_empty(buf));
                if (s == s0 && has_next) next = place_of(tile + n_clusters);
            }
            if (!ok) break;
            if (p.splits > 1) {  // back to where the pairs of the cluster take them from
#pragma unroll
                for (int c = 0; c < MOST_BLOCKS; ++c)
                    if (c < blocks) store_columns(t_lane + (uint32_t)(first * 32 + 64 * c), sum[c]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                break;
            }
#pragma unroll
            for (int c = 0; c < MOST_BLOCKS; ++c)
                if (c < blocks && ok) {
                    ok = put_out(sum[c], first + 2 * c, freed, has_next);
                    freed = true;
                }
            place = next;
            in_next = false;
        }
        if (!ok) give_up(&g_wgrad_status, WGRAD_STATUS_EPILOGUE);
    }
    __syncwarp();

    if (p.splits > 1) {
        // one tile per cluster, its tokens shared by the pairs: 32-column block b is finished by slice b % splits, the others
        // push their partial sums into its operand ring (idle once every CTA has its last MMA behind it)
        const int S = p.splits, blocks = p.bn / 32;
        const uint32_t lane_row = (uint32_t)(quarter * 32 + lane);
        __syncthreads();
        cluster_barrier();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        if (epilogue)
            for (int b = first; b < blocks; b += 2)
                if (b % S != slice) {
                    uint32_t v[32];
                    tmem_ld32(t_lane + (uint32_t)(b * 32), v);
                    push_partial(v, base + partial_slot(b, S, slice, b % S) * 16384u + lane_row * 4u, (uint32_t)(2 * (b % S) + half));
                }
        __syncthreads();
        cluster_barrier();
        if (epilogue) {
            bool ok = true;
            for (int b = block0; b < blocks && ok; b += block_step) {
                uint32_t v[32];
                tmem_ld32(t_lane + (uint32_t)(b * 32), v);
                fold_partials(v, gen_base, b, S, slice, lane_row);
                float2 sums[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) sums[i] = make_float2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1]));
                ok = put_out(sums, b, b != block0, false);
            }
            if (!ok) give_up(&g_wgrad_status, WGRAD_STATUS_EPILOGUE);
        }
    }
    if (VEC && epilogue && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");  // every store has completed

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cluster_barrier();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        tmem_free_pair(tmem_base);
    }
}

int make_map_3d(CUtensorMap *map, CUtensorMapDataType dt, const void *ptr, uint64_t inner, uint64_t tokens, int planes, uint64_t ld_bytes) {
    const cuuint64_t dims[3] = {inner, tokens, (cuuint64_t)planes}, strides[2] = {ld_bytes, ld_bytes * tokens};
    const cuuint32_t box[3] = {64, (cuuint32_t)token_step(planes), (cuuint32_t)planes};
    return make_map(map, dt, 3, ptr, dims, strides, box, CU_TENSOR_MAP_SWIZZLE_128B);
}

template <bool VEC>
int launch_wgrad(const cudaLaunchConfig_t &cfg, const CUtensorMap &mg, const CUtensorMap &mx, const CUtensorMap &mw, const CUtensorMap &mo, const WgradParams &p) {
    // the shared-memory limit is a per-device attribute of the function: set it once on every device
    static std::atomic<bool> configured[64];
    int dev = 0;
    T81_CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || !configured[dev].load(std::memory_order_acquire)) {
        T81_CUDA_TRY(cudaFuncSetAttribute(gemm_wgrad_tc_kernel<VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_LIMIT));
        if (dev >= 0 && dev < 64) configured[dev].store(true, std::memory_order_release);
    }
    T81_CUDA_TRY(cudaLaunchKernelEx(&cfg, gemm_wgrad_tc_kernel<VEC>, mg, mx, mw, mo, p));
    return T81B200_OK;
}

// Scratch of one operand: none when it is 16-bit (or staged planes already) and TMA can read it where it is.
size_t operand_scratch(const void *p, int dtype, int64_t ld, int64_t tokens, int64_t width) {
    if (dtype != T81B200_F32 && reinterpret_cast<uintptr_t>(p) % 16 == 0 && (ld * 2) % 16 == 0) return 0;
    return (t81b200_stage_rows_bytes(dtype, tokens, width) + 255) / 256 * 256;
}

}  // namespace

int gemm_wgrad_status(int reset) {
    int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_wgrad_status, sizeof v) != cudaSuccess) return T81B200_ECUDA;
    if (reset && v != 0) {
        const int zero = 0;
        if (cudaMemcpyToSymbol(g_wgrad_status, &zero, sizeof zero) != cudaSuccess) return T81B200_ECUDA;
    }
    return v;
}

}  // namespace t81b200

using namespace t81b200;

extern "C" size_t t81b200_qat_weight_grad_workspace_bytes(const void *g, int g_dtype, int64_t ldg, const void *x, int x_dtype, int64_t ldx,
                                                          int64_t tokens, int64_t rows, int64_t cols) {
    if (tokens <= 0 || rows <= 0 || cols <= 0) return 0;
    return operand_scratch(g, g_dtype, ldg, tokens, rows) + operand_scratch(x, x_dtype, ldx, tokens, cols);
}

extern "C" int t81b200_qat_weight_grad(const void *g, int g_dtype, int64_t ldg, const void *x, int x_dtype, int64_t ldx, int64_t tokens, int64_t rows,
                                       int64_t cols, const float *w, int64_t ldw, const float *scale, float *out, void *workspace, size_t workspace_bytes,
                                       void *stream) {
    if (tokens < 0 || rows < 0 || cols < 0 || ldg < rows || ldx < cols || ldw < cols) return fail(T81B200_EINVAL, "qat_weight_grad: bad dimensions");
    auto wide = [](int d) { return d == T81B200_F32 || d == T81B200_BF16X3; };
    auto narrow = [](int d) { return d == T81B200_BF16 || d == T81B200_F16; };
    if (!(wide(g_dtype) && wide(x_dtype)) && !(narrow(g_dtype) && g_dtype == x_dtype))
        return fail(T81B200_EINVAL, "qat_weight_grad: operand dtypes %d and %d", g_dtype, x_dtype);
    if (int rc = check_device()) return rc;
    if (rows == 0 || cols == 0) return T81B200_OK;
    if (!w || !scale || !out || (tokens > 0 && (!g || !x))) return fail(T81B200_EINVAL, "qat_weight_grad: null pointer");
    if (rows >= (1ll << 30) || cols >= (1ll << 30) || tokens >= (1ll << 27)) return fail(T81B200_ELIMIT, "qat_weight_grad: dimensions too large");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (tokens == 0) {
        T81_CUDA_TRY(cudaMemsetAsync(out, 0, (size_t)rows * cols * 4, st));
        return T81B200_OK;
    }
    const size_t need_g = operand_scratch(g, g_dtype, ldg, tokens, rows), need_x = operand_scratch(x, x_dtype, ldx, tokens, cols);
    if (need_g + need_x > 0 && (!workspace || workspace_bytes < need_g + need_x || reinterpret_cast<uintptr_t>(workspace) % 256 != 0))
        return fail(T81B200_EWORKSPACE, "qat_weight_grad: %zu bytes of 256-byte aligned workspace needed, %zu given", need_g + need_x, workspace_bytes);
    if ((g_dtype == T81B200_BF16X3 && need_g) || (x_dtype == T81B200_BF16X3 && need_x)) return fail(T81B200_EALIGN, "qat_weight_grad: planes must be 16-byte aligned rows");
    WgradParams p;
    memset(&p, 0, sizeof p);
    p.planes = wide(g_dtype) ? 3 : 1;
    const CUtensorMapDataType dt = g_dtype == T81B200_F16 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT16 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16;
    CUtensorMap mg, mx;
    struct { const void *src; int dtype; int64_t ld, width; size_t need; char *scratch; CUtensorMap *map; } ops[2] = {
        {g, g_dtype, ldg, rows, need_g, static_cast<char *>(workspace), &mg}, {x, x_dtype, ldx, cols, need_x, static_cast<char *>(workspace) + need_g, &mx}};
    for (auto &o : ops) {
        if (o.need) {
            if (int rc = t81b200_stage_rows(o.src, o.dtype, o.ld, tokens, o.width, o.scratch, stream)) return rc;
            o.src = o.scratch;
            o.ld = t81b200_stage_rows_ld(o.width);
        }
        if (int rc = make_map_3d(o.map, dt, o.src, (uint64_t)o.width, (uint64_t)tokens, p.planes, (uint64_t)o.ld * 2)) return rc;
    }
    p.w = w; p.scale = scale; p.out = out; p.rows = rows; p.cols = cols; p.ldw = ldw;
    p.token_steps = (int)((tokens + token_step(p.planes) - 1) / token_step(p.planes));
    p.m_tiles = (int)((rows + 255) / 256);
    // 256- or 128-column tiles, tokens split over up to four pairs of a cluster while that fits the GPU at once: whichever
    // needs fewer steps one after the other (a 128-column step costs about 0.65 of a 256-column one, a split six of 64 tokens)
    const double per_step = p.planes == 1 ? 1.0 : 3.0;
    double best = 1e30;
    for (int bn = 256; bn >= 128; bn -= 128)
        for (int s = 1; s <= MAX_SPLITS; ++s) {
            const int64_t tiles = (int64_t)p.m_tiles * ((cols + bn - 1) / bn), resident = resident_pair_clusters(s);
            if (s > p.token_steps || (s > 1 && tiles > resident)) continue;
            const double t = (double)((tiles + resident - 1) / resident) * ((p.token_steps + s - 1) / s) * per_step * (bn == 256 ? 1.0 : 0.65) + (s > 1 ? 6.0 : 0.0);
            if (t < best) { best = t; p.bn = bn; p.splits = s; }
        }
    p.segment = p.planes > 1 ? 256 / token_step(3) : (tokens < 512 ? 1 : (tokens < 1024 ? 2 : 3));  // how long: see the top
    p.n_tiles = (int)((cols + p.bn - 1) / p.bn);
    const int stage = (2 + p.bn / 128) * group_bytes(p.planes);
    p.vec = cols % 4 == 0 && ldw % 4 == 0 && ldw < (1ll << 37) && reinterpret_cast<uintptr_t>(w) % 16 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0 ? 1 : 0;
    // Three slots a warp leave four stages of 16-bit operands, two leave five.  Few tokens are over before two have been read and filled
    // again, many want the stages (16-bit, us, two and three: 304 tokens of 2416 by 4965 35.2 and 30.9, 1104 of 12192 by 12476 405 and
    // 380, 4096 of 4096 by 14336 365 and 371; over eight layers, three against two: 0.88 to 1.0 at 700 tokens, 0.95 to 1.02 at 2048 and 2400, 0.97
    // to 1.06 at 2800, 0.91 to 1.07 at 4096, 1.01 to 1.25 at 6000); fp32 stages and rows that lanes copy word by word gain nothing from a third.
    p.slots = p.planes == 1 && p.vec && p.bn == 256 && tokens <= 2048 ? 3 : 2;
    const int fit = (SMEM_LIMIT - 1024 - EPILOGUE_WARPS * p.slots * BLOCK_BYTES - BARRIER_BYTES) / stage;
    p.stages = fit < MAX_STAGES ? fit : MAX_STAGES;
    p.idesc = umma_instr_desc(p.bn, g_dtype == T81B200_F16, true, true);
    CUtensorMap mw, mo;
    memset(&mw, 0, sizeof mw);
    memset(&mo, 0, sizeof mo);
    if (p.vec) {
        if (int rc = make_map_2d(&mw, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, w, (uint64_t)cols, (uint64_t)rows, (uint64_t)ldw * 4, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
        if (int rc = make_map_2d(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, out, (uint64_t)cols, (uint64_t)rows, (uint64_t)cols * 4, 32, 32, CU_TENSOR_MAP_SWIZZLE_128B)) return rc;
    }
    const int64_t tiles = (int64_t)p.m_tiles * p.n_tiles;
    const int64_t clusters = p.splits > 1 || tiles < resident_pair_clusters(1) ? tiles : resident_pair_clusters(1);
    // While the epilogue puts a tile out, the MMAs of the next one have two accumulators to go on with: an eighth of the tokens each
    // where that is more, which leaves the whole tile's sums within the same bound.
    const int eighth = (int)(tokens / 8) / token_step(p.planes);
    p.lead = p.planes == 1 && tiles > clusters && eighth > p.segment ? eighth : p.segment;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(clusters * 2 * p.splits), 1, 1);
    cfg.blockDim = dim3(NUM_THREADS, 1, 1);
    cfg.dynamicSmemBytes = (size_t)p.stages * stage + EPILOGUE_WARPS * p.slots * BLOCK_BYTES + BARRIER_BYTES + 1024;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)(2 * p.splits);
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    return p.vec ? launch_wgrad<true>(cfg, mg, mx, mw, mo, p) : launch_wgrad<false>(cfg, mg, mx, mw, mo, p);
}
