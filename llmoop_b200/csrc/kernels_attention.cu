// Paged-KV GQA attention for decode / verify / prefill-chunk lanes, plus the
// greedy arg-max.  Semantics: append_gqa_attention_bf16.comp.template:189-339
// (each lane's K,V are written at its tick, then it attends over the
// min(tick+1, capacity) most recent tokens; f32 online softmax; one bf16
// rounding at the end).  Because every lane's K,V are appended first and lanes
// of one stream carry increasing ticks, lane i sees exactly the tokens of
// lanes < i plus the committed context - the same result as the reference's
// serial per-lane execution, in one launch.
#include <atomic>

#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

namespace {

__device__ __forceinline__ size_t kv_token_offset(const KvLayer &kv, int slot, uint32_t token, int head, bool value) {
    // token is the ring index (tick % capacity)
    int logical_page = static_cast<int>(token / kv.page_tokens);
    int within = static_cast<int>(token % kv.page_tokens);
    int physical = kv.block_table[static_cast<size_t>(slot) * kv.pages_per_slot + logical_page];
    size_t half = static_cast<size_t>(kv.kv_heads) * kv.page_tokens * kv.head_width;
    return static_cast<size_t>(physical) * (2 * half) + (value ? half : 0) +
           (static_cast<size_t>(head) * kv.page_tokens + within) * kv.head_width;
}

constexpr float LOWEST = -3.4028234663852886e38f;

// ---- tiled attention -------------------------------------------------------------------------------------------
// A CTA serves ROW_WARPS x 16 query rows of one (stream, kv head) - row r is query head r % group of the stream's lane
// r / group, so the query heads that share a kv head share its K/V tiles - over one split of the context.  K and V
// tiles of 64 tokens go through two shared-memory stages (cp.async one tile ahead, the tokens' page offsets two tiles
// ahead), Q stays in registers; Q.K^T and P.V run on mma.sync bf16 with f32 sums.  The probabilities enter P.V as three
// bf16 terms, which hold all 24 bits of their f32 value, and the sums over the tiles are f32 multiply-adds: the error
// against 64 bits, before the final rounding, is 2.2e-7 to 3.9e-7 of the output (32 lanes at 550 tokens .. 713 at 8713),
// where scalar f32 products and sums leave 2.7e-7 to 1.2e-6, and two terms with one running sum left 1.6e-6 to 1.0e-5.
// TOKEN_WARPS warps share a row tile's context: each takes 64 / TOKEN_WARPS tokens of every tile with a softmax of its
// own, and they merge at the end.  Prefill chunks (many rows per stream) run 8 x 1 warps; verify and draft batches
// (few rows, many tokens) 1 or 2 x 4, where four warps per row tile hide the tile's latency.
// What bounds it: prefill the legacy tensor path (four MMAs per 16 x 8 x 16 of K and V), decode the KV bytes.
// (One scalar f32 product per thread and token, the form this replaced, took 4.8 ms per 8B layer for 713 lanes at an
// 8713-token context; this takes 0.70 ms, with two terms it took 0.55.)

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ void load_matrices_transposed(uint32_t (&r)[4], uint32_t address) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(address));
}
__device__ __forceinline__ uint32_t pack_bf16_rn(float lo, float hi) {
    const __nv_bfloat162 pair = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t *>(&pair);
}

constexpr int TILE = 64;
// 16-byte chunk `c` of a tile row, permuted with the row so that eight rows' equal chunks hit eight bank groups
template <int HD>
__device__ __forceinline__ uint32_t tile_chunk(int row, int c) {
    return static_cast<uint32_t>(row * (HD / 8) + ((c & ~7) | ((c ^ row) & 7))) * 16;
}

struct AttentionArgs {
    const uint16_t *q;
    uint16_t *out;
    KvLayer kv;
    LaneTable meta;
    int lanes, lanes_per_stream, q_heads, group, row_blocks;
    float scale;
    int split_tokens, max_splits;
    float *scratch;
    const AttentionBlock *blocks;  // ragged batches: what each block of rows covers; nullptr: lanes_per_stream lanes per stream
};

template <int HD, int ROW_WARPS, int TOKEN_WARPS>
constexpr size_t attention_smem() {
    constexpr size_t tiles = 2 * 2 * static_cast<size_t>(TILE) * HD * 2;
    constexpr size_t merge = TOKEN_WARPS > 1 ? static_cast<size_t>(ROW_WARPS) * TOKEN_WARPS * 16 * (HD + 4) * 4 : 0;
    return tiles > merge ? tiles : merge;
}

// The verify form of 32 rows takes two CTAs per SM (128 registers, 92 bytes of spills): it waits for its K and V more than
// it multiplies, and 32 streams x 8 kv heads x splits are several waves of one CTA per SM (44 -> 35 us per launch).
template <int HD, int ROW_WARPS, int TOKEN_WARPS>
__global__ void __launch_bounds__(ROW_WARPS *TOKEN_WARPS * 32, ROW_WARPS * TOKEN_WARPS == 8 && TOKEN_WARPS > 1 ? 2 : 1) attention_tile_kernel(const __grid_constant__ AttentionArgs a) {
    constexpr int THREADS = ROW_WARPS * TOKEN_WARPS * 32, ROWS = ROW_WARPS * 16;
    constexpr int TOKENS = TILE / TOKEN_WARPS;  // of a tile, per warp
    constexpr int K_STEPS = HD / 16, N_TILES = TOKENS / 8, D_TILES = HD / 8;
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ size_t token_offset[2][TILE];
    grid_launch_dependents();
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, j = lane & 3;
    const int row_warp = warp / TOKEN_WARPS, token_warp = warp % TOKEN_WARPS;
    // the blocks with the longest contexts (the last rows of a chunk) start first
    const int block = static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x), kv_head = blockIdx.y, split = blockIdx.z;
    int lane0, rows, row0;
    if (a.blocks != nullptr) {
        const AttentionBlock entry = a.blocks[block];
        lane0 = entry.first_lane;
        rows = entry.lanes * a.group;
        row0 = entry.index * ROWS;
    } else {
        const int stream = block / a.row_blocks;
        lane0 = stream * a.lanes_per_stream;
        rows = a.lanes_per_stream * a.group;
        row0 = (block - stream * a.row_blocks) * ROWS;
    }
    const int slot = a.meta.slot[lane0];
    if (slot < 0) return;
    const uint32_t capacity = a.kv.capacity;
    const int last_row = min(row0 + ROWS, rows) - 1;
    const uint32_t newest = a.meta.position[lane0 + last_row / a.group];
    const uint32_t tokens = min(newest + 1u, capacity), first_tick = newest + 1u - tokens;  // attended window of the newest lane
    const uint32_t begin = static_cast<uint32_t>(split) * a.split_tokens;
    if (begin >= tokens) return;
    const uint32_t end = min(begin + a.split_tokens, tokens);
    const int tiles = static_cast<int>((end - begin + TILE - 1) / TILE);

    // this thread's two rows (g and g + 8 of the warp's sixteen) and their Q fragments
    const int r_lo = row0 + row_warp * 16 + g, r_hi = r_lo + 8;
    const bool warp_active = row0 + row_warp * 16 < rows;
    uint32_t tick[2];
    uint32_t q_frag[K_STEPS][4];
    {
        const int rr[2] = {min(r_lo, rows - 1), min(r_hi, rows - 1)};
        const uint32_t *source[2];
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int l = lane0 + rr[h] / a.group;
            tick[h] = a.meta.position[l];
            source[h] = reinterpret_cast<const uint32_t *>(a.q + (static_cast<size_t>(l) * a.q_heads + kv_head * a.group + rr[h] % a.group) * HD) + j;
        }
#pragma unroll
        for (int s = 0; s < K_STEPS; s++) {
            q_frag[s][0] = source[0][s * 8];
            q_frag[s][1] = source[1][s * 8];
            q_frag[s][2] = source[0][s * 8 + 4];
            q_frag[s][3] = source[1][s * 8 + 4];
        }
    }
    // the oldest of the warp's rows: tiles that end at or before its tick need no causal mask
    const uint32_t oldest_tick = __reduce_min_sync(0xffffffffu, min(tick[0], tick[1]));

    auto offset_of = [&](int tile, int t) -> size_t {
        const uint32_t index = min(begin + static_cast<uint32_t>(tile) * TILE + t, end - 1);
        uint32_t ring = first_tick + index;
        if (ring >= capacity) ring %= capacity;
        return kv_token_offset(a.kv, slot, ring, kv_head, false);
    };
    const size_t value_half = static_cast<size_t>(a.kv.kv_heads) * a.kv.page_tokens * HD;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    constexpr uint32_t TILE_BYTES = TILE * HD * 2;
    auto request = [&](int tile) {
        const uint32_t k_tile = base + static_cast<uint32_t>(tile & 1) * 2 * TILE_BYTES, v_tile = k_tile + TILE_BYTES;
        constexpr int CHUNKS = HD / 8;
#pragma unroll
        for (int i = 0; i < TILE * CHUNKS / THREADS; i++) {
            const int index = threadIdx.x + i * THREADS, t = index / CHUNKS, c = index % CHUNKS;
            const uint16_t *source = a.kv.pool + token_offset[tile & 1][t] + c * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(k_tile + tile_chunk<HD>(t, c)), "l"(source) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(v_tile + tile_chunk<HD>(t, c)), "l"(source + value_half) : "memory");
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    float acc[D_TILES][4];
#pragma unroll
    for (int d = 0; d < D_TILES; d++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[d][i] = 0.0f;
    float row_max[2] = {-INFINITY, -INFINITY}, row_sum[2] = {0.0f, 0.0f};
    const float log2_scale = a.scale * 1.4426950408889634f;

    if (threadIdx.x < TILE) {
        token_offset[0][threadIdx.x] = offset_of(0, threadIdx.x);
        token_offset[1][threadIdx.x] = offset_of(tiles > 1 ? 1 : 0, threadIdx.x);
    }
    __syncthreads();
    request(0);
    for (int tile = 0; tile < tiles; tile++) {
        if (tile + 1 < tiles) request(tile + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        size_t next_offset = 0;
        if (threadIdx.x < TILE && tile + 2 < tiles) next_offset = offset_of(tile + 2, threadIdx.x);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const uint32_t k_tile = base + static_cast<uint32_t>(tile & 1) * 2 * TILE_BYTES, v_tile = k_tile + TILE_BYTES;
        const uint32_t tile_begin = begin + static_cast<uint32_t>(tile) * TILE + token_warp * TOKENS;  // this warp's first token
        if (warp_active && tile_begin < end) {
            float score[N_TILES][4];
#pragma unroll
            for (int n = 0; n < N_TILES; n++)
#pragma unroll
                for (int i = 0; i < 4; i++) score[n][i] = 0.0f;
#pragma unroll
            for (int s = 0; s < K_STEPS; s++) {
#pragma unroll
                for (int pair = 0; pair < N_TILES / 2; pair++) {
                    const int matrix = lane >> 3, t = token_warp * TOKENS + pair * 16 + (matrix >> 1) * 8 + (lane & 7);
                    uint32_t b[4];
                    load_matrices(b, k_tile + tile_chunk<HD>(t, s * 2 + (matrix & 1)));
                    mma_bf16(score[2 * pair], q_frag[s], b[0], b[1]);
                    mma_bf16(score[2 * pair + 1], q_frag[s], b[2], b[3]);
                }
            }
            // causal and ring limits: tick - capacity < token's tick <= tick
            const bool masked = tile_begin + TOKENS > end || first_tick + tile_begin + TOKENS - 1 > oldest_tick || newest >= capacity;
            if (masked) {
#pragma unroll
                for (int n = 0; n < N_TILES; n++)
#pragma unroll
                    for (int i = 0; i < 4; i++) {
                        const uint32_t index = tile_begin + n * 8 + 2 * j + (i & 1), token_tick = first_tick + index, own = tick[i >> 1];
                        if (index >= end || token_tick > own || token_tick + capacity <= own) score[n][i] = -INFINITY;
                    }
            }
            float factor[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                float largest = row_max[h];
#pragma unroll
                for (int n = 0; n < N_TILES; n++) largest = fmaxf(largest, fmaxf(score[n][2 * h], score[n][2 * h + 1]));
                largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 1));
                largest = fmaxf(largest, __shfl_xor_sync(0xffffffffu, largest, 2));
                const float reference = largest == -INFINITY ? 0.0f : largest;  // nothing visible yet
                factor[h] = exp2f((row_max[h] - reference) * log2_scale);
                row_max[h] = largest;
                const float shift = reference * log2_scale;
                float sum = 0.0f;
#pragma unroll
                for (int n = 0; n < N_TILES; n++)
#pragma unroll
                    for (int i = 0; i < 2; i++) {
                        const float p = exp2f(fmaf(score[n][2 * h + i], log2_scale, -shift));
                        score[n][2 * h + i] = p;
                        sum += p;
                    }
                row_sum[h] = row_sum[h] * factor[h] + sum;  // this thread's columns; added up over the four threads in the end
            }
            // p as three bf16 terms, the 24 bits of its f32 value; a tile's products add up from zero, of sixteen tokens the
            // smallest terms first, and join the row's sum by one multiply-add, which rounds to nearest where the tensor
            // core's running sum truncates.  Eight sums at a time hide the latency of the chain (713 lanes at 8713 tokens: two
            // 741 us, four 723, eight 697).
            uint32_t p[3][TOKENS / 16][4];
#pragma unroll
            for (int kt = 0; kt < TOKENS / 16; kt++)
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    float p0 = score[2 * kt + (i >> 1)][2 * (i & 1)], p1 = score[2 * kt + (i >> 1)][2 * (i & 1) + 1];
#pragma unroll
                    for (int term = 0; term < 3; term++) {
                        const uint32_t packed = pack_bf16_rn(p0, p1);
                        p[term][kt][i] = packed;
                        p0 -= bf16_lo(packed);
                        p1 -= bf16_hi(packed);
                    }
                }
            constexpr int PAIRS = 4;  // of eight output dims in flight
            static_assert(D_TILES % (2 * PAIRS) == 0, "the output dims are taken PAIRS pairs at a time");
#pragma unroll
            for (int first = 0; first < D_TILES; first += 2 * PAIRS) {
                float sums[2 * PAIRS][4] = {};
#pragma unroll
                for (int kt = 0; kt < TOKENS / 16; kt++) {
                    const int matrix = lane >> 3, t = token_warp * TOKENS + kt * 16 + (matrix & 1) * 8 + (lane & 7);
                    uint32_t b[PAIRS][4];
#pragma unroll
                    for (int pair = 0; pair < PAIRS; pair++) load_matrices_transposed(b[pair], v_tile + tile_chunk<HD>(t, first + pair * 2 + (matrix >> 1)));
#pragma unroll
                    for (int term = 2; term >= 0; term--)
#pragma unroll
                        for (int pair = 0; pair < PAIRS; pair++) {
                            mma_bf16(sums[2 * pair], p[term][kt], b[pair][0], b[pair][1]);
                            mma_bf16(sums[2 * pair + 1], p[term][kt], b[pair][2], b[pair][3]);
                        }
                }
#pragma unroll
                for (int d = 0; d < 2 * PAIRS; d++)
#pragma unroll
                    for (int i = 0; i < 4; i++) acc[first + d][i] = fmaf(acc[first + d][i], factor[i >> 1], sums[d][i]);
            }
        }
        // (this tile's offsets were last read before the barrier above, when it was requested)
        if (threadIdx.x < TILE && tile + 2 < tiles) token_offset[tile & 1][threadIdx.x] = next_offset;
        __syncthreads();  // the tile is read; its stage may be overwritten
    }
#pragma unroll
    for (int h = 0; h < 2; h++) {
        row_sum[h] += __shfl_xor_sync(0xffffffffu, row_sum[h], 1);
        row_sum[h] += __shfl_xor_sync(0xffffffffu, row_sum[h], 2);
    }

    // a finished row: the output itself, or the split's partial (unnormalised row, then maximum and sum)
    auto finish = [&](int r, int d, float x0, float x1, float maximum, float sum) {
        const size_t pair = static_cast<size_t>(lane0 + r / a.group) * a.q_heads + kv_head * a.group + r % a.group;
        if (a.max_splits == 1) {
            const float inverse = sum == 0.0f ? 0.0f : 1.0f / sum;
            *reinterpret_cast<uint32_t *>(a.out + pair * HD + d) = sum == 0.0f ? 0u : pack_bf16(x0 * inverse, x1 * inverse);
        } else {
            float *part = a.scratch + (pair * a.max_splits + split) * (HD + 2);
            *reinterpret_cast<float2 *>(part + d) = make_float2(x0, x1);
            if (d == 0) *reinterpret_cast<float2 *>(part + HD) = make_float2(maximum == -INFINITY ? LOWEST : maximum * a.scale, sum);
        }
    };
    if (TOKEN_WARPS == 1) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = h == 0 ? r_lo : r_hi;
            if (r >= rows) continue;
#pragma unroll
            for (int d = 0; d < D_TILES; d++) finish(r, d * 8 + 2 * j, acc[d][2 * h], acc[d][2 * h + 1], row_max[h], row_sum[h]);
        }
        return;
    }
    // merge the token warps of a row tile: [warp][row][HD + maximum, sum]
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    constexpr int STRIDE = HD + 4;
    float *const parts = reinterpret_cast<float *>(smem);
    if (warp_active) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
            float *row = parts + (warp * 16 + g + 8 * h) * STRIDE;
#pragma unroll
            for (int d = 0; d < D_TILES; d++) *reinterpret_cast<float2 *>(row + d * 8 + 2 * j) = make_float2(acc[d][2 * h], acc[d][2 * h + 1]);
            if (j == 0) *reinterpret_cast<float2 *>(row + HD) = make_float2(row_max[h], row_sum[h]);
        }
    }
    __syncthreads();
    for (int index = threadIdx.x; index < ROWS * (HD / 2); index += THREADS) {
        const int local = index / (HD / 2), d = (index % (HD / 2)) * 2, r = row0 + local;
        if (r >= rows) continue;
        const float *row = parts + ((local / 16) * TOKEN_WARPS * 16 + local % 16) * STRIDE;
        float maximum = -INFINITY;
#pragma unroll
        for (int w = 0; w < TOKEN_WARPS; w++) maximum = fmaxf(maximum, row[w * 16 * STRIDE + HD]);
        const float reference = maximum == -INFINITY ? 0.0f : maximum;
        float x0 = 0.0f, x1 = 0.0f, sum = 0.0f;
#pragma unroll
        for (int w = 0; w < TOKEN_WARPS; w++) {
            const float *part = row + w * 16 * STRIDE;
            const float weight = exp2f((part[HD] - reference) * log2_scale);
            sum = fmaf(part[HD + 1], weight, sum);
            x0 = fmaf(part[d], weight, x0);
            x1 = fmaf(part[d + 1], weight, x1);
        }
        finish(r, d, x0, x1, maximum, sum);
    }
}

// ---- attention in scalar f32 ---------------------------------------------------------------------------------------
// The form for layers whose attention output is quantised to FP8: there a last-bit change of a sum turns into a step of
// one part in sixteen wherever a value sits on a rounding boundary (and, behind it, into another choice of experts), so
// these layers keep the plain f32 order of additions - one product after the other, no split probabilities.
__device__ __forceinline__ uint4 load16(const void *address) { return *reinterpret_cast<const uint4 *>(address); }

// Two f32 sums in one register pair (fma.rn.f32x2 rounds each as fmaf does).
using float_pair = unsigned long long;
__device__ __forceinline__ float_pair pair_of(float lo, float hi) {
    float_pair out;
    asm("mov.b64 %0, {%1, %2};" : "=l"(out) : "f"(lo), "f"(hi));
    return out;
}
__device__ __forceinline__ float2 halves_of(float_pair v) {
    float2 out;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(out.x), "=f"(out.y) : "l"(v));
    return out;
}
__device__ __forceinline__ float_pair pair_fma(float_pair a, float_pair b, float_pair c) {
    float_pair out;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(out) : "l"(a), "l"(b), "l"(c));
    return out;
}

template <int HD, int GROUP, int QL>
struct AttentionF32 {
    static constexpr int Q = QL * GROUP, THREADS = 128;
    static constexpr int K_STRIDE = HD + 8;   // elements: 16-byte loads of eight consecutive rows hit distinct banks
    static constexpr int P_STRIDE = Q + 4;    // floats: so do 16-byte stores
    // scores: four queries x SCORE_TOKENS tokens per thread; a warp's threads share the queries
    static constexpr int SCORE_SETS = Q / 4, SCORE_THREADS = THREADS / SCORE_SETS < TILE ? THREADS / SCORE_SETS : TILE;  // per set of queries
    static constexpr int SCORE_TOKENS = TILE / SCORE_THREADS;
    // P.V: two output dims x VALUE_QUERIES queries per thread
    static constexpr int VALUE_SETS = THREADS / (HD / 2) < Q / 2 ? THREADS / (HD / 2) : Q / 2, VALUE_QUERIES = Q / VALUE_SETS;
    static_assert(Q % 4 == 0 && VALUE_QUERIES % 2 == 0, "queries are taken in pairs");
    struct Shared {
        uint16_t k[TILE * K_STRIDE];  // K rows
        uint16_t v[TILE * HD];        // V rows
        float q[HD * Q];              // [dim][query]
        float p[TILE * P_STRIDE];     // [token][query]: scores, then probabilities
        float row_max[Q], row_sum[Q], row_alpha[Q];
        uint32_t lane_tick[QL];
        size_t offset[TILE];          // of the tile's K rows in the pool
    };
};

// A CTA of 128 threads serves QL consecutive lanes of one stream x the GROUP query heads of one kv head (Q = QL*GROUP query
// vectors) over one split of the context, tile by tile (TILE tokens): K and V rows through cp.async, scores, online softmax
// per query, P.V.  Every score and every output dimension is one chain of f32 multiply-adds, over the head's dimensions and
// over the tokens in order; two queries share a packed instruction.  The FP32 pipe and the shared-memory loads of the
// operands bound it about equally: the queries are widened once, and a thread takes 4 queries x 2 tokens (scores) or 8
// queries x 2 dims (P.V), so that a load feeds four packed operations.  (One token, eight queries unpacked per product and
// one load per product before: 60 us for 24 lanes of 8 streams at a 1024-token context;
// this 31.)
// A batch may mix streams: each stream contributes `lanes_per_stream` consecutive lanes, and a CTA never spans two streams.
template <int HD, int GROUP, int QL>
__global__ void __launch_bounds__(128)
attention_f32_kernel(const uint16_t *__restrict__ q, KvLayer kv, LaneTable lanes_meta, int lanes, int lanes_per_stream,
                     int q_heads, float scale, int split_tokens, int max_splits, float *__restrict__ scratch, const AttentionBlock *__restrict__ ragged) {
    using Form = AttentionF32<HD, GROUP, QL>;
    constexpr int Q = Form::Q, THREADS = Form::THREADS;
    extern __shared__ __align__(16) uint8_t smem_raw[];
    typename Form::Shared &shared = *reinterpret_cast<typename Form::Shared *>(smem_raw);
    grid_launch_dependents();
    grid_dependency_wait();
    const int kv_head = blockIdx.x, split = blockIdx.y, group_slot = blockIdx.z, tid = threadIdx.x;

    // lanes of one stream are consecutive and every stream of the batch has `lanes_per_stream` of them
    const int groups_per_stream = (lanes_per_stream + QL - 1) / QL;
    const int stream_index = group_slot / groups_per_stream;
    int group_index = group_slot % groups_per_stream, lane0 = stream_index * lanes_per_stream + group_index * QL;
    if (ragged != nullptr) {
        const AttentionBlock entry = ragged[group_slot];
        group_index = entry.index;
        lane0 = entry.first_lane + entry.index * QL;
        lanes_per_stream = entry.lanes;
    }
    if (lane0 >= lanes) return;
    const int slot = lanes_meta.slot[lane0];
    if (slot < 0) return;
    const uint32_t capacity = kv.capacity;
    // the newest tick among this CTA's lanes bounds the context it has to look at
    uint32_t tick_of[QL], newest = 0;
#pragma unroll
    for (int i = 0; i < QL; i++) {
        const bool valid = lane0 + i < lanes && group_index * QL + i < lanes_per_stream;
        tick_of[i] = valid ? lanes_meta.position[lane0 + i] : 0xffffffffu;
        if (valid) newest = max(newest, tick_of[i]);
    }
    const uint32_t tokens = newest + 1u < capacity ? newest + 1u : capacity;  // attended window of the newest lane
    const uint32_t first_tick = newest + 1u - tokens;
    const uint32_t begin = static_cast<uint32_t>(split) * split_tokens;
    if (begin >= tokens) return;
    const uint32_t end = begin + split_tokens < tokens ? begin + split_tokens : tokens;
    if (tid < QL) {
#pragma unroll
        for (int i = 0; i < QL; i++)
            if (tid == i) shared.lane_tick[i] = tick_of[i];
    }

    auto offset_of = [&](uint32_t tile_begin) {  // of row tid of a tile (rows beyond the split repeat its last one)
        uint32_t ring = first_tick + min(tile_begin + static_cast<uint32_t>(tid), end - 1);
        if (ring >= capacity) ring %= capacity;
        return kv_token_offset(kv, slot, ring, kv_head, false);
    };
    const size_t value_half = static_cast<size_t>(kv.kv_heads) * kv.page_tokens * HD;
    const uint32_t k_address = static_cast<uint32_t>(__cvta_generic_to_shared(shared.k)), v_address = static_cast<uint32_t>(__cvta_generic_to_shared(shared.v));
    if (tid < TILE) shared.offset[tid] = offset_of(begin);
    for (int index = tid; index < Q * HD / 8; index += THREADS) {
        const int query = index % Q, piece = index / Q, lane = lane0 + query / GROUP;
        uint4 value = make_uint4(0, 0, 0, 0);
        if (lane < lanes && group_index * QL + query / GROUP < lanes_per_stream)
            value = load16(q + (static_cast<size_t>(lane) * q_heads + kv_head * GROUP + query % GROUP) * HD + piece * 8);
        const uint32_t words[4] = {value.x, value.y, value.z, value.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            shared.q[(piece * 8 + 2 * i) * Q + query] = bf16_lo(words[i]);
            shared.q[(piece * 8 + 2 * i + 1) * Q + query] = bf16_hi(words[i]);
        }
    }
    if (tid < Q) {
        shared.row_max[tid] = -3.4028234663852886e38f;
        shared.row_sum[tid] = 0.0f;
    }
    // P.V: this thread's dims and queries
    constexpr int VQ = Form::VALUE_QUERIES;
    const int value_set = tid / (HD / 2), value_dim = (tid % (HD / 2)) * 2;
    bool value_active = value_set < Form::VALUE_SETS;
    {
        bool any = false;
#pragma unroll
        for (int i = 0; i < QL; i++) any |= tick_of[i] != 0xffffffffu && i >= value_set * VQ / GROUP && i <= (value_set * VQ + VQ - 1) / GROUP;
        value_active &= any;
    }
    float_pair acc[2][VQ / 2];
#pragma unroll
    for (int i = 0; i < VQ / 2; i++) acc[0][i] = acc[1][i] = 0ull;

    for (uint32_t tile_begin = begin; tile_begin < end; tile_begin += TILE) {
        const int count = static_cast<int>(end - tile_begin < TILE ? end - tile_begin : TILE);
        __syncthreads();  // the previous tile is consumed (and the queries, offsets and row states are in place)
#pragma unroll
        for (int i = 0; i < TILE * (HD / 8) / THREADS; i++) {
            const int index = tid + i * THREADS, t = index / (HD / 8), piece = index % (HD / 8);
            const uint16_t *source = kv.pool + shared.offset[t] + piece * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(k_address + (t * Form::K_STRIDE + piece * 8) * 2), "l"(source) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(v_address + (t * HD + piece * 8) * 2), "l"(source + value_half) : "memory");
        }
        size_t next_offset = 0;
        if (tid < TILE && tile_begin + TILE < end) next_offset = offset_of(tile_begin + TILE);
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncthreads();
        if (tid < TILE && tile_begin + TILE < end) shared.offset[tid] = next_offset;
        // ---- scores
        {
            constexpr int ST = Form::SCORE_TOKENS;
            const int set = tid / Form::SCORE_THREADS, t0 = tid % Form::SCORE_THREADS;
            const bool active = set < Form::SCORE_SETS;
            float_pair score[ST][2];
#pragma unroll
            for (int i = 0; i < ST; i++) score[i][0] = score[i][1] = 0ull;
            if (active) {
                const float *queries = shared.q + set * 4;
#pragma unroll 4
                for (int piece = 0; piece < HD / 8; piece++) {
                    uint4 k[ST];
#pragma unroll
                    for (int i = 0; i < ST; i++)
                        k[i] = *reinterpret_cast<const uint4 *>(shared.k + (t0 + i * Form::SCORE_THREADS) * Form::K_STRIDE + piece * 8);
#pragma unroll
                    for (int d = 0; d < 8; d++) {
                        const ulonglong2 four = *reinterpret_cast<const ulonglong2 *>(queries + (piece * 8 + d) * Q);
#pragma unroll
                        for (int i = 0; i < ST; i++) {
                            const uint32_t word = d < 2 ? k[i].x : d < 4 ? k[i].y : d < 6 ? k[i].z : k[i].w;
                            const float value = (d & 1) ? bf16_hi(word) : bf16_lo(word);
                            const float_pair both = pair_of(value, value);
                            score[i][0] = pair_fma(four.x, both, score[i][0]);
                            score[i][1] = pair_fma(four.y, both, score[i][1]);
                        }
                    }
                }
#pragma unroll
                for (int i = 0; i < ST; i++) {
                    const int t = t0 + i * Form::SCORE_THREADS;
                    const uint32_t token_tick = first_tick + tile_begin + t;
                    const float2 first = halves_of(score[i][0]), second = halves_of(score[i][1]);
                    float out[4] = {first.x, first.y, second.x, second.y};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const uint32_t tick = shared.lane_tick[(set * 4 + j) / GROUP];
                        // causal + ring window of this lane: ticks in (tick - capacity, tick]
                        const bool visible = t < count && tick != 0xffffffffu && token_tick <= tick && token_tick + capacity > tick;
                        out[j] = visible ? out[j] * scale : -INFINITY;
                    }
                    *reinterpret_cast<float4 *>(shared.p + t * Form::P_STRIDE + set * 4) = make_float4(out[0], out[1], out[2], out[3]);
                }
            }
        }
        __syncthreads();
        // ---- online softmax: warp w handles queries w, w+4, ...
        {
            const int warp = tid >> 5, lane_id = tid & 31;
#pragma unroll
            for (int query = warp; query < Q; query += 4) {
                float *row = shared.p + query;
                const float s0 = row[lane_id * Form::P_STRIDE], s1 = row[(32 + lane_id) * Form::P_STRIDE];
                const float tile_max = warp_max(fmaxf(s0, s1));
                const float old_max = shared.row_max[query];
                const float next_max = fmaxf(old_max, tile_max);
                float p0 = 0.0f, p1 = 0.0f, alpha = 1.0f;
                if (next_max > -3.0e38f) {
                    alpha = expf(old_max - next_max);
                    p0 = s0 == -INFINITY ? 0.0f : expf(s0 - next_max);
                    p1 = s1 == -INFINITY ? 0.0f : expf(s1 - next_max);
                }
                const float tile_sum = warp_sum(p0 + p1);
                row[lane_id * Form::P_STRIDE] = p0;
                row[(32 + lane_id) * Form::P_STRIDE] = p1;
                __syncwarp();
                if (lane_id == 0) {
                    shared.row_alpha[query] = alpha;
                    shared.row_sum[query] = shared.row_sum[query] * alpha + tile_sum;
                    shared.row_max[query] = next_max;
                }
            }
        }
        __syncthreads();
        // ---- P.V
        if (value_active) {
            const float *row = shared.p + value_set * VQ;
            const uint16_t *values = shared.v + value_dim;
#pragma unroll
            for (int i = 0; i < VQ / 2; i++) {
                const float a0 = shared.row_alpha[value_set * VQ + 2 * i], a1 = shared.row_alpha[value_set * VQ + 2 * i + 1];
#pragma unroll
                for (int d = 0; d < 2; d++) {
                    const float2 sum = halves_of(acc[d][i]);
                    acc[d][i] = pair_of(sum.x * a0, sum.y * a1);
                }
            }
#pragma unroll 4
            for (int t = 0; t < count; t++) {
                const uint32_t word = *reinterpret_cast<const uint32_t *>(values + t * HD);
                const float_pair v0 = pair_of(bf16_lo(word), bf16_lo(word)), v1 = pair_of(bf16_hi(word), bf16_hi(word));
#pragma unroll
                for (int i = 0; i < VQ / 2; i++) {
                    const float_pair probabilities = *reinterpret_cast<const float_pair *>(row + t * Form::P_STRIDE + 2 * i);
                    acc[0][i] = pair_fma(probabilities, v0, acc[0][i]);
                    acc[1][i] = pair_fma(probabilities, v1, acc[1][i]);
                }
            }
        }
    }
    if (value_active) {
#pragma unroll
        for (int i = 0; i < VQ; i++) {
            const int query = value_set * VQ + i;
            if (shared.lane_tick[query / GROUP] == 0xffffffffu) continue;
            float *out = scratch + ((static_cast<size_t>(lane0 + query / GROUP) * q_heads + kv_head * GROUP + query % GROUP) * max_splits + split) * (HD + 2);
            const float2 first = halves_of(acc[0][i / 2]), second = halves_of(acc[1][i / 2]);
            *reinterpret_cast<float2 *>(out + value_dim) = (i & 1) ? make_float2(first.y, second.y) : make_float2(first.x, second.x);
        }
    }
    if (tid < Q && shared.lane_tick[tid / GROUP] != 0xffffffffu) {
        float *out = scratch + ((static_cast<size_t>(lane0 + tid / GROUP) * q_heads + kv_head * GROUP + tid % GROUP) * max_splits + split) * (HD + 2);
        out[HD] = shared.row_max[tid];
        out[HD + 1] = shared.row_sum[tid];
    }
}

// Log-sum-exp merge of the split partials of one (lane, q head) pair by one warp: thread s weighs split s, the weighted
// partials are added split by split in order, as are the sums.  (Every thread weighing every split for each of its dims, one
// load after the other: 9 us for 17 splits; this, the first rows requested along with the states, 3.3.)
__global__ void attention_f32_merge_kernel(const float *__restrict__ scratch, uint16_t *__restrict__ out, KvLayer kv,
                                           LaneTable lanes_meta, int lanes, int q_heads, int head_width, int split_tokens,
                                           int max_splits) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), thread = threadIdx.x & 31;
    if (pair >= lanes * q_heads) return;
    const int lane = pair / q_heads;
    if (lanes_meta.slot[lane] < 0) return;
    const uint32_t tick = lanes_meta.position[lane];
    const uint32_t tokens = tick + 1u < kv.capacity ? tick + 1u : kv.capacity;
    const int splits = min(static_cast<int>((tokens + split_tokens - 1) / split_tokens), max_splits), stride = head_width + 2;
    const float *base = scratch + static_cast<size_t>(pair) * max_splits * stride;
    constexpr int DIMS = 4, BATCH = 8;  // heads of at most 128; splits whose rows are in flight together
    float part[BATCH][DIMS];
    auto fetch = [&](int first) {
#pragma unroll
        for (int i = 0; i < BATCH; i++)
#pragma unroll
            for (int d = 0; d < DIMS; d++)
                if (first + i < splits && thread + 32 * d < head_width) part[i][d] = base[static_cast<size_t>(first + i) * stride + thread + 32 * d];
    };
    float2 state = make_float2(-3.4028234663852886e38f, 0.0f);
    if (thread < splits) state = *reinterpret_cast<const float2 *>(base + static_cast<size_t>(thread) * stride + head_width);
    fetch(0);
    float maximum = state.x;
    for (int s = thread + 32; s < splits; s += 32) maximum = fmaxf(maximum, base[static_cast<size_t>(s) * stride + head_width]);
    maximum = warp_max(maximum);
    float denominator = 0.0f, acc[DIMS] = {};
    for (int first = 0; first < splits; first += 32) {
        float weight = 0.0f;
        if (first > 0 && first + thread < splits) state = *reinterpret_cast<const float2 *>(base + static_cast<size_t>(first + thread) * stride + head_width);
        if (first + thread < splits) weight = expf(state.x - maximum);
        const int count = min(32, splits - first);
        for (int s = 0; s < count; s += BATCH) {
            if (first + s > 0) fetch(first + s);
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                if (s + i >= count) break;
                const float w = __shfl_sync(0xffffffffu, weight, s + i);
                denominator = fmaf(__shfl_sync(0xffffffffu, state.y, s + i), w, denominator);
#pragma unroll
                for (int d = 0; d < DIMS; d++)
                    if (thread + 32 * d < head_width) acc[d] = fmaf(part[i][d], w, acc[d]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < DIMS; i++)
        if (thread + 32 * i < head_width)
            out[static_cast<size_t>(pair) * head_width + thread + 32 * i] = static_cast<uint16_t>(f32_to_bf16_bits(denominator == 0.0f ? 0.0f : acc[i] / denominator));
}

template <int HD, int GROUP, int QL>
cudaError_t launch_f32(const AttentionArgs &a, cudaStream_t stream) {
    auto kernel = attention_f32_kernel<HD, GROUP, QL>;
    constexpr size_t smem = sizeof(typename AttentionF32<HD, GROUP, QL>::Shared);
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (status != cudaSuccess) return status;
    const int groups = a.blocks != nullptr ? a.row_blocks : a.lanes / a.lanes_per_stream * ((a.lanes_per_stream + QL - 1) / QL);
    const dim3 grid(a.kv.kv_heads, a.max_splits, groups);
    status = launch_dependent(kernel, grid, dim3(128), smem, 1, stream, a.q, a.kv, a.meta, a.lanes, a.lanes_per_stream, a.q_heads, a.scale, a.split_tokens,
                              a.max_splits, a.scratch, a.blocks);
    if (status != cudaSuccess) return status;
    return launch_dependent(attention_f32_merge_kernel, dim3((a.lanes * a.q_heads + 3) / 4), dim3(128), 0, 1, stream, a.scratch, a.out, a.kv, a.meta, a.lanes,
                            a.q_heads, a.kv.head_width, a.split_tokens, a.max_splits);
}

template <int HD>
cudaError_t launch_f32_of_width(const AttentionArgs &args, cudaStream_t stream) {
    switch (args.group) {
    case 1: return launch_f32<HD, 1, 4>(args, stream);
    case 2: return launch_f32<HD, 2, 4>(args, stream);
    case 4: return launch_f32<HD, 4, 4>(args, stream);
    default: return launch_f32<HD, 8, 2>(args, stream);
    }
}

// Heads of at most 32 (tiny models, short contexts: latency, not bandwidth): one warp per (lane, q head), scalar f32; its
// threads take every 32nd token with a softmax of their own and merge in the end.  HD: the head width where rows are whole
// 16-byte words, else 0.  The rows of a token are requested together, and the merge halves the dims a thread holds with
// every exchange.  (Element by element and five exchanges per dim: 7.6 us for a 50-token context; this 2.5.)
template <int HD>
__global__ void attention_small_kernel(const uint16_t *__restrict__ q, uint16_t *__restrict__ out, KvLayer kv,
                                       LaneTable lanes_meta, int lanes, int q_heads, float scale) {
    constexpr int WIDTH = HD > 0 ? HD : 32;
    grid_launch_dependents();
    grid_dependency_wait();
    const int index = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), thread = threadIdx.x & 31;
    if (index >= lanes * q_heads) return;
    const int lane = index / q_heads, head = index % q_heads;
    const int slot = lanes_meta.slot[lane];
    if (slot < 0) return;
    const int hd = HD > 0 ? HD : kv.head_width;
    const int kv_head = head / (q_heads / kv.kv_heads);
    const uint32_t tick = lanes_meta.position[lane];
    const uint32_t capacity = kv.capacity;
    const uint32_t tokens = tick + 1u < capacity ? tick + 1u : capacity;
    const uint32_t first_tick = tick + 1u - tokens;
    auto read_row = [&](const uint16_t *row, float (&values)[WIDTH]) {
        if (HD > 0) {
            uint4 words[WIDTH / 8];
#pragma unroll
            for (int i = 0; i < WIDTH / 8; i++) words[i] = reinterpret_cast<const uint4 *>(row)[i];
#pragma unroll
            for (int i = 0; i < WIDTH / 8; i++) {
                const uint32_t four[4] = {words[i].x, words[i].y, words[i].z, words[i].w};
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    values[8 * i + 2 * w] = bf16_lo(four[w]);
                    values[8 * i + 2 * w + 1] = bf16_hi(four[w]);
                }
            }
        } else {
#pragma unroll
            for (int d = 0; d < WIDTH; d++) values[d] = d < hd ? bf16_bits_to_f32(row[d]) : 0.0f;
        }
    };
    float query[WIDTH], acc[WIDTH];
    read_row(q + (static_cast<size_t>(lane) * q_heads + head) * hd, query);
#pragma unroll
    for (int d = 0; d < WIDTH; d++) acc[d] = 0.0f;
    float maximum = LOWEST, denominator = 0.0f;
    for (uint32_t i = thread; i < tokens; i += 32) {
        uint32_t ring = first_tick + i;
        if (ring >= capacity) ring %= capacity;
        const uint16_t *row = kv.pool + kv_token_offset(kv, slot, ring, kv_head, false);
        float key[WIDTH], value[WIDTH];
        read_row(row, key);
        read_row(row + static_cast<size_t>(kv.kv_heads) * kv.page_tokens * hd, value);
        float dot = 0.0f;
#pragma unroll
        for (int d = 0; d < WIDTH; d++) dot = fmaf(query[d], key[d], dot);
        const float score = dot * scale, next_max = fmaxf(maximum, score);
        const float alpha = expf(maximum - next_max), beta = expf(score - next_max);
        denominator = denominator * alpha + beta;
        maximum = next_max;
#pragma unroll
        for (int d = 0; d < WIDTH; d++) acc[d] = acc[d] * alpha + beta * value[d];
    }
    const float whole_max = warp_max(maximum), weight = expf(maximum - whole_max);
    denominator = warp_sum(denominator * weight);
#pragma unroll
    for (int d = 0; d < WIDTH; d++) acc[d] *= weight;
    // the dims' sums over the warp: every exchange (distance 16, 8, ..) adds the partner's share of half of them
    int dim = 0;
#pragma unroll
    for (int step = 0; step < 5; step++) {
        const int distance = 16 >> step, live = WIDTH >> step;
        if (live > 1) {
            const bool upper = (thread & distance) != 0;
#pragma unroll
            for (int i = 0; i < live / 2; i++) {
                const float keep = upper ? acc[live / 2 + i] : acc[i], send = upper ? acc[i] : acc[live / 2 + i];
                acc[i] = keep + __shfl_xor_sync(0xffffffffu, send, distance);
            }
            if (upper) dim += live / 2;
        } else {
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], distance);  // fewer dims than threads: several end up with the same one
        }
    }
    constexpr int SHARERS = 32 / WIDTH;
    if (thread % SHARERS == 0 && dim < hd)
        out[(static_cast<size_t>(lane) * q_heads + head) * hd + dim] =
            static_cast<uint16_t>(f32_to_bf16_bits(denominator == 0.0f ? 0.0f : acc[0] / denominator));
}

// Log-sum-exp merge of the split partials; one warp per (lane, q head).
__global__ void attention_merge_kernel(const float *__restrict__ scratch, uint16_t *__restrict__ out, KvLayer kv,
                                       LaneTable lanes_meta, int lanes, int q_heads, int head_width, int split_tokens,
                                       int max_splits) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int pair = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), thread = threadIdx.x & 31;
    if (pair >= lanes * q_heads) return;
    const int lane = pair / q_heads;
    if (lanes_meta.slot[lane] < 0) return;
    const uint32_t tick = lanes_meta.position[lane];
    const uint32_t tokens = tick + 1u < kv.capacity ? tick + 1u : kv.capacity;
    const int splits = min(static_cast<int>((tokens + split_tokens - 1) / split_tokens), max_splits), stride = head_width + 2;
    const float *base = scratch + static_cast<size_t>(pair) * max_splits * stride;
    // the first splits' states and rows are requested together: one trip to memory for contexts of a few splits
    constexpr int BATCH = 8;
    float2 part[BATCH][2];  // two dimensions per thread and 64 of the head
    auto fetch = [&](int first) {
#pragma unroll
        for (int i = 0; i < BATCH; i++)
#pragma unroll
            for (int d = 0; d < 2; d++)
                if (first + i < splits && 2 * thread + 64 * d < head_width)
                    part[i][d] = reinterpret_cast<const float2 *>(base + static_cast<size_t>(first + i) * stride)[thread + 32 * d];
    };
    float2 state = make_float2(LOWEST, 0.0f);
    if (thread < splits) state = *reinterpret_cast<const float2 *>(base + static_cast<size_t>(thread) * stride + head_width);
    fetch(0);
    float maximum = state.x;
    for (int s = thread + 32; s < splits; s += 32) maximum = fmaxf(maximum, base[static_cast<size_t>(s) * stride + head_width]);
    maximum = warp_max(maximum);
    float denominator = 0.0f;
    float2 acc[2] = {};
    for (int first = 0; first < splits; first += 32) {
        float weight = 0.0f;
        if (first + thread < splits) {
            if (first > 0) state = *reinterpret_cast<const float2 *>(base + static_cast<size_t>(first + thread) * stride + head_width);
            weight = expf(state.x - maximum);
            denominator = fmaf(state.y, weight, denominator);
        }
        const int count = min(32, splits - first);
        for (int s = 0; s < count; s += BATCH) {
            if (first + s > 0) fetch(first + s);
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                if (s + i >= count) break;
                const float w = __shfl_sync(0xffffffffu, weight, s + i);
#pragma unroll
                for (int d = 0; d < 2; d++)
                    if (2 * thread + 64 * d < head_width) {
                        acc[d].x = fmaf(part[i][d].x, w, acc[d].x);
                        acc[d].y = fmaf(part[i][d].y, w, acc[d].y);
                    }
            }
        }
    }
    denominator = warp_sum(denominator);
    const float inverse = denominator == 0.0f ? 0.0f : 1.0f / denominator;
#pragma unroll
    for (int i = 0; i < 2; i++)
        if (2 * thread + 64 * i < head_width)
            *reinterpret_cast<uint32_t *>(out + static_cast<size_t>(pair) * head_width + 2 * thread + 64 * i) = pack_bf16(acc[i].x * inverse, acc[i].y * inverse);
}

template <int HD, int ROW_WARPS, int TOKEN_WARPS>
cudaError_t launch_tiles(const AttentionArgs &args, dim3 grid, cudaStream_t stream) {
    auto kernel = attention_tile_kernel<HD, ROW_WARPS, TOKEN_WARPS>;
    constexpr size_t smem = attention_smem<HD, ROW_WARPS, TOKEN_WARPS>();
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
    if (status != cudaSuccess) return status;
    return launch_dependent(kernel, grid, dim3(ROW_WARPS * TOKEN_WARPS * 32), smem, 1, stream, args);
}

template <int HD>
cudaError_t launch_tiles_of_width(AttentionArgs args, int streams, cudaStream_t stream) {
    const int rows = args.lanes_per_stream * args.group;
    auto grid = [&](int block_rows) {
        if (args.blocks == nullptr) args.row_blocks = (rows + block_rows - 1) / block_rows;
        return dim3(static_cast<unsigned int>(args.blocks != nullptr ? args.row_blocks : streams * args.row_blocks), static_cast<unsigned int>(args.kv.kv_heads), static_cast<unsigned int>(args.max_splits));
    };
    if (attention_is_prefill(args.lanes_per_stream, args.q_heads, args.kv.kv_heads)) {
        const dim3 blocks = grid(128);
        return launch_tiles<HD, 8, 1>(args, blocks, stream);
    }
    if (rows <= 16) {
        const dim3 blocks = grid(16);
        return launch_tiles<HD, 1, 4>(args, blocks, stream);
    }
    const dim3 blocks = grid(32);
    return launch_tiles<HD, 2, 4>(args, blocks, stream);
}

}  // namespace

// Up to 96 rows (lanes x query heads per kv head) of a stream run the small-batch form: three blocks of 32 rows read the
// context three times at most, and from there on the 128-row form wastes less than it saves.
bool attention_is_prefill(int lanes_per_stream, int q_heads, int kv_heads) { return lanes_per_stream * (q_heads / kv_heads) > 96; }

int attention_block_lanes(int lanes_per_stream, int q_heads, int kv_heads, int head_width, bool scalar_f32) {
    const int group = q_heads / kv_heads;
    if ((head_width != 64 && head_width != 128) || (group != 1 && group != 2 && group != 4 && group != 8)) return 1;
    if (scalar_f32) return group == 8 ? 2 : 4;
    const int rows = lanes_per_stream * group;
    return (attention_is_prefill(lanes_per_stream, q_heads, kv_heads) ? 128 : rows <= 16 ? 16 : 32) / group;
}

cudaError_t launch_attention(const uint16_t *q, uint16_t *out, const KvLayer &kv, const LaneTable &lanes_meta,
                             int lanes, int lanes_per_stream, int q_heads, float scale, int split_tokens, int max_splits,
                             float *scratch, bool scalar_f32, cudaStream_t stream, const AttentionBlock *blocks, int block_count) {
    if (lanes <= 0) return cudaSuccess;
    if (lanes_per_stream <= 0 || (blocks == nullptr && lanes % lanes_per_stream != 0)) return cudaErrorInvalidValue;
    const int group = q_heads / kv.kv_heads;
    const bool wide = kv.head_width == 64 || kv.head_width == 128;
    if (!wide || (group != 1 && group != 2 && group != 4 && group != 8)) {
        if (kv.head_width > 32) return cudaErrorInvalidValue;
        auto kernel = kv.head_width == 32 ? attention_small_kernel<32> : kv.head_width == 16 ? attention_small_kernel<16>
                    : kv.head_width == 8 ? attention_small_kernel<8> : attention_small_kernel<0>;
        return launch_dependent(kernel, dim3((lanes * q_heads + 3) / 4), dim3(128), 0, 1, stream, q, out, kv, lanes_meta, lanes, q_heads, scale);
    }
    AttentionArgs args = {};
    args.q = q;
    args.out = out;
    args.kv = kv;
    args.meta = lanes_meta;
    args.lanes = lanes;
    args.lanes_per_stream = lanes_per_stream;
    args.q_heads = q_heads;
    args.group = group;
    args.scale = scale;
    args.split_tokens = split_tokens;
    args.max_splits = max_splits;
    args.scratch = scratch;
    args.blocks = blocks;
    args.row_blocks = block_count;
    if (scalar_f32) return kv.head_width == 128 ? launch_f32_of_width<128>(args, stream) : launch_f32_of_width<64>(args, stream);
    const int streams = lanes / lanes_per_stream;
    cudaError_t status = kv.head_width == 128 ? launch_tiles_of_width<128>(args, streams, stream) : launch_tiles_of_width<64>(args, streams, stream);
    if (status != cudaSuccess || max_splits == 1) return status;
    return launch_dependent(attention_merge_kernel, dim3((lanes * q_heads + 3) / 4), dim3(128), 0, 1, stream, scratch, out, kv, lanes_meta, lanes, q_heads,
                            kv.head_width, split_tokens, max_splits);
}

// ---- rotary embedding of q and k and the KV append in one launch -------------------------------------------------
// rotary_bf16.comp.template:99-109 (five bf16 roundings per element; cos/sin from the table the mounter fills with the
// same f32 pow/cos/sin sequence), parallel_head_norm_rope_2way_bf16.comp.template:166-209 where norm weights are given
// (per-head RMSNorm rounded to bf16 first), then the append of append_gqa_attention_bf16.comp.template:189-215.  One
// warp per (lane, head): query heads go to q_out, key heads and values straight into the lane's KV slot.
namespace {

constexpr int ROPE_WARPS = 8;
__global__ void __launch_bounds__(ROPE_WARPS * 32) rope_append_kernel(const __grid_constant__ RopeAppend r, const KvLayer kv, const LaneTable meta) {
    extern __shared__ float rows[];  // [warp][head width]
    grid_launch_dependents();
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5, thread = threadIdx.x & 31, lane = blockIdx.x, head = blockIdx.y * ROPE_WARPS + warp;
    const int width = kv.head_width;
    if (head >= r.q_heads + 2 * kv.kv_heads) return;
    const int part = head < r.q_heads ? 0 : (head < r.q_heads + kv.kv_heads ? 1 : 2);  // q, k, v
    const int own_head = part == 0 ? head : head - r.q_heads - (part == 2 ? kv.kv_heads : 0);
    const int heads = part == 0 ? r.q_heads : kv.kv_heads;
    const uint16_t *in = (part == 0 ? r.q : part == 1 ? r.k : r.v) + (static_cast<size_t>(lane) * heads + own_head) * width;
    uint16_t *out;
    if (part == 0) {
        out = r.q_out + (static_cast<size_t>(lane) * heads + own_head) * width;
    } else {
        const int slot = meta.slot[lane];
        if (slot < 0 || kv.capacity == 0) return;
        out = kv.pool + kv_token_offset(kv, slot, meta.position[lane] % kv.capacity, own_head, part == 2);
    }
    if (part == 2) {
        for (int word = thread; word < width / 2; word += 32) reinterpret_cast<uint32_t *>(out)[word] = reinterpret_cast<const uint32_t *>(in)[word];
        return;
    }
    float *values = rows + warp * width;
    for (int word = thread; word < width / 2; word += 32) {
        const uint32_t packed = reinterpret_cast<const uint32_t *>(in)[word];
        values[2 * word] = bf16_lo(packed);
        values[2 * word + 1] = bf16_hi(packed);
    }
    const uint16_t *norm = part == 0 ? r.q_norm : r.k_norm;
    if (norm != nullptr) {
        __syncwarp();
        // the squares are added as rope_kernel's CTA of `lanes_of` threads adds them: per thread, per warp, over the warps
        const int lanes_of = min((width / 2 + 31) / 32 * 32, 256);
        float total = 0.0f;
        for (int first = 0; first < lanes_of; first += 32) {
            float sum = 0.0f;
            for (int d = first + thread; d < width; d += lanes_of) sum = fmaf(values[d], values[d], sum);
            total += warp_sum(sum);
        }
        const float inv_rms = 1.0f / sqrtf(total / static_cast<float>(width) + r.eps);
        for (int d = thread; d < width; d += 32) values[d] = round_bf16(values[d] * inv_rms * (bf16_bits_to_f32(norm[d]) + r.norm_offset));
    }
    __syncwarp();
    const RopeForm &form = part == 0 ? r.q_form : r.k_form;
    const int half = form.rotary / 2;
    const uint32_t *table = form.cos_sin + static_cast<size_t>(meta.position[lane] % form.positions) * half;
    auto rotated = [&](int d) {
        if (d >= form.rotary) return values[d];
        const uint32_t packed = table[form.interleaved ? d / 2 : d % half];
        float other;
        if (form.interleaved) other = (d & 1) == 0 ? -values[d + 1] : values[d - 1];
        else other = d < half ? -values[d + half] : values[d - half];
        return round_bf16(values[d] * bf16_lo(packed)) + round_bf16(other * bf16_hi(packed));
    };
    for (int word = thread; word < width / 2; word += 32) reinterpret_cast<uint32_t *>(out)[word] = pack_bf16(rotated(2 * word), rotated(2 * word + 1));
}

// Heads of 128 that are rotated whole, halves against one another, without norms (most dense models): a thread holds dims
// 2 t, 2 t + 1 and their partners 64 further on, so a head needs no shared memory, and a warp has the rows of HEADS heads in
// flight under one set of factors.  512 lanes x 48 heads: 12.8 -> 9.0 us.
template <int HEADS>
__global__ void __launch_bounds__(ROPE_WARPS * 32) rope_append_whole_kernel(const __grid_constant__ RopeAppend r, const KvLayer kv, const LaneTable meta) {
    constexpr int WIDTH = 128;
    grid_launch_dependents();
    grid_dependency_wait();
    const int warp = threadIdx.x >> 5, thread = threadIdx.x & 31, lane = blockIdx.x, first = (blockIdx.y * ROPE_WARPS + warp) * HEADS;
    const int heads = r.q_heads + 2 * kv.kv_heads;
    if (first >= heads) return;
    const int slot = meta.slot[lane];
    const uint32_t position = meta.position[lane];
    const bool stored = slot >= 0 && kv.capacity != 0;  // keys and values
    const size_t row = stored ? kv_token_offset(kv, slot, position % kv.capacity, 0, false) : 0;
    const uint2 q_factors = r.q_heads > 0 ? reinterpret_cast<const uint2 *>(r.q_form.cos_sin + static_cast<size_t>(position % r.q_form.positions) * (WIDTH / 2))[thread] : make_uint2(0, 0);
    const uint2 k_factors = reinterpret_cast<const uint2 *>(r.k_form.cos_sin + static_cast<size_t>(position % r.k_form.positions) * (WIDTH / 2))[thread];
    uint32_t low[HEADS], high[HEADS];
#pragma unroll
    for (int h = 0; h < HEADS; h++) {
        const int head = first + h;
        if (head >= heads) break;
        const uint32_t *in = reinterpret_cast<const uint32_t *>(
            head < r.q_heads ? r.q + (static_cast<size_t>(lane) * r.q_heads + head) * WIDTH
            : head < r.q_heads + kv.kv_heads ? r.k + (static_cast<size_t>(lane) * kv.kv_heads + head - r.q_heads) * WIDTH
                                             : r.v + (static_cast<size_t>(lane) * kv.kv_heads + head - r.q_heads - kv.kv_heads) * WIDTH);
        low[h] = in[thread];
        high[h] = in[thread + 32];
    }
#pragma unroll
    for (int h = 0; h < HEADS; h++) {
        const int head = first + h;
        if (head >= heads) break;
        const bool query = head < r.q_heads, value = head >= r.q_heads + kv.kv_heads;
        if (!query && !stored) continue;
        if (!value) {
            const uint2 factors = query ? q_factors : k_factors;
            const float c0 = bf16_lo(factors.x), s0 = bf16_hi(factors.x), c1 = bf16_lo(factors.y), s1 = bf16_hi(factors.y);
            const float x0 = bf16_lo(low[h]), x1 = bf16_hi(low[h]), y0 = bf16_lo(high[h]), y1 = bf16_hi(high[h]);
            low[h] = pack_bf16(round_bf16(x0 * c0) + round_bf16(-y0 * s0), round_bf16(x1 * c1) + round_bf16(-y1 * s1));
            high[h] = pack_bf16(round_bf16(y0 * c0) + round_bf16(x0 * s0), round_bf16(y1 * c1) + round_bf16(x1 * s1));
        }
        const size_t kv_half = value ? static_cast<size_t>(kv.kv_heads) * kv.page_tokens * WIDTH : 0;
        const int own = head - r.q_heads - (value ? kv.kv_heads : 0);
        uint32_t *out = reinterpret_cast<uint32_t *>(query ? r.q_out + (static_cast<size_t>(lane) * r.q_heads + head) * WIDTH
                                                           : kv.pool + row + kv_half + static_cast<size_t>(own) * kv.page_tokens * WIDTH);
        out[thread] = low[h];
        out[thread + 32] = high[h];
    }
}

}  // namespace

cudaError_t launch_rope_append(const RopeAppend &rope, const KvLayer &kv, const LaneTable &lanes_meta, int lanes, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    const int heads = rope.q_heads + 2 * kv.kv_heads;
    auto whole = [&](const RopeForm &form) { return form.rotary == 128 && !form.interleaved; };
    if (kv.head_width == 128 && (rope.q_heads == 0 || whole(rope.q_form)) && whole(rope.k_form) && rope.q_norm == nullptr && rope.k_norm == nullptr) {
        // a head per warp while the lanes do not fill the chip
        constexpr int MANY = 6;
        if (lanes >= multiprocessors()) return launch_dependent(rope_append_whole_kernel<MANY>, dim3(lanes, (heads + ROPE_WARPS * MANY - 1) / (ROPE_WARPS * MANY)), dim3(ROPE_WARPS * 32), 0, 1, stream, rope, kv, lanes_meta);
        return launch_dependent(rope_append_whole_kernel<1>, dim3(lanes, (heads + ROPE_WARPS - 1) / ROPE_WARPS), dim3(ROPE_WARPS * 32), 0, 1, stream, rope, kv, lanes_meta);
    }
    return launch_dependent(rope_append_kernel, dim3(lanes, (heads + ROPE_WARPS - 1) / ROPE_WARPS), dim3(ROPE_WARPS * 32),
                            static_cast<size_t>(ROPE_WARPS) * kv.head_width * sizeof(float), 1, stream, rope, kv, lanes_meta);
}

// greedy_sampler_f32.comp.template:31-34,52-109: arg-max with ties -> lowest id.  Two stages so that a
// 128k-entry vocabulary is scanned by many CTAs: stage 1 reduces ARGMAX_CHUNKS slices per lane, stage 2 the
// partial winners (chunks are ordered by token id, so "lower id wins a tie" carries over).
constexpr int ARGMAX_CHUNKS = 64;

__device__ __forceinline__ void argmax_combine(float &best, uint32_t &token, float other, uint32_t other_token) {
    if (other_token != 0xffffffffu && (token == 0xffffffffu || other > best || (other == best && other_token < token))) {
        best = other;
        token = other_token;
    }
}

__device__ __forceinline__ void argmax_block_reduce(float &best, uint32_t &token, float *shared_logit, uint32_t *shared_token) {
    for (int offset = 16; offset > 0; offset >>= 1) {
        float other = __shfl_xor_sync(0xffffffffu, best, offset);
        uint32_t other_token = __shfl_xor_sync(0xffffffffu, token, offset);
        argmax_combine(best, token, other, other_token);
    }
    if ((threadIdx.x & 31) == 0) {
        shared_logit[threadIdx.x >> 5] = best;
        shared_token[threadIdx.x >> 5] = token;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        int warps = blockDim.x >> 5;
        best = static_cast<int>(threadIdx.x) < warps ? shared_logit[threadIdx.x] : 0.0f;
        token = static_cast<int>(threadIdx.x) < warps ? shared_token[threadIdx.x] : 0xffffffffu;
        for (int offset = 16; offset > 0; offset >>= 1) {
            float other = __shfl_xor_sync(0xffffffffu, best, offset);
            uint32_t other_token = __shfl_xor_sync(0xffffffffu, token, offset);
            argmax_combine(best, token, other, other_token);
        }
    }
}

__global__ void argmax_partial_kernel(const float *__restrict__ logits, float *__restrict__ partial_logit,
                                      uint32_t *__restrict__ partial_token, int vocab) {
    grid_launch_dependents();
    grid_dependency_wait();
    __shared__ float shared_logit[32];
    __shared__ uint32_t shared_token[32];
    const int lane = blockIdx.y, chunk = blockIdx.x;
    const int per_chunk = (vocab + ARGMAX_CHUNKS - 1) / ARGMAX_CHUNKS;
    const int begin = chunk * per_chunk, end = min(vocab, begin + per_chunk);
    const float *row = logits + static_cast<size_t>(lane) * vocab;
    float best = 0.0f;
    uint32_t token = 0xffffffffu;
#pragma unroll 4
    for (int index = begin + threadIdx.x; index < end; index += blockDim.x) {
        float candidate = row[index];
        if (token == 0xffffffffu || candidate > best) {  // strictly greater keeps the lowest id within a thread
            best = candidate;
            token = static_cast<uint32_t>(index);
        }
    }
    argmax_block_reduce(best, token, shared_logit, shared_token);
    if (threadIdx.x == 0) {
        partial_logit[lane * ARGMAX_CHUNKS + chunk] = best;
        partial_token[lane * ARGMAX_CHUNKS + chunk] = token;
    }
}

__global__ void argmax_final_kernel(const float *__restrict__ partial_logit, const uint32_t *__restrict__ partial_token,
                                    uint32_t *__restrict__ records) {
    grid_launch_dependents();
    grid_dependency_wait();
    __shared__ float shared_logit[32];
    __shared__ uint32_t shared_token[32];
    const int lane = blockIdx.x;
    float best = partial_logit[lane * ARGMAX_CHUNKS + threadIdx.x];
    uint32_t token = partial_token[lane * ARGMAX_CHUNKS + threadIdx.x];
    argmax_block_reduce(best, token, shared_logit, shared_token);
    if (threadIdx.x == 0) {
        uint32_t *record = records + static_cast<size_t>(lane) * 4;
        record[0] = token == 0xffffffffu ? 0u : token;
        record[1] = __float_as_uint(best);
        record[2] = 0u;
        record[3] = 0u;
    }
}

size_t argmax_scratch_bytes(int lanes) { return static_cast<size_t>(lanes) * ARGMAX_CHUNKS * 8; }

cudaError_t launch_argmax(const float *logits, uint32_t *records, int lanes, int vocab, void *scratch, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    float *partial_logit = static_cast<float *>(scratch);
    uint32_t *partial_token = reinterpret_cast<uint32_t *>(partial_logit + static_cast<size_t>(lanes) * ARGMAX_CHUNKS);
    dim3 grid(ARGMAX_CHUNKS, lanes);
    cudaError_t status = launch_dependent(argmax_partial_kernel, grid, dim3(256), 0, 1, stream, logits, partial_logit, partial_token, vocab);
    if (status != cudaSuccess) return status;
    return launch_dependent(argmax_final_kernel, dim3(lanes), dim3(ARGMAX_CHUNKS), 0, 1, stream, partial_logit, partial_token, records);
}

// ---- greedy arg-max without a caller-provided scratch buffer -------------------------------------------------
// Same two kernels as launch_argmax, with the per-chunk partial winners kept in a fixed device array that is part
// of the library image (32 KB, enough for STATIC_ARGMAX_MAX_LANES lanes).  Nothing is allocated, by this function
// or on its behalf: the array's device address is looked up once per device (cudaGetSymbolAddress; the array's
// name on the host side is not a device pointer) with that device current, and cached.
// Every partial slot the second kernel reads is written by the first kernel of the same call, so nothing needs
// clearing between calls; the array does keep the previous call's partials and is shared by all callers in the
// process, so two calls that overlap in time on one device (different streams or threads) race on it.
constexpr int STATIC_ARGMAX_MAX_LANES = 64;
constexpr int STATIC_ARGMAX_MAX_DEVICES = 64;
static __device__ __align__(256) unsigned char static_argmax_scratch[STATIC_ARGMAX_MAX_LANES * ARGMAX_CHUNKS * 8];

int argmax_static_max_lanes() { return STATIC_ARGMAX_MAX_LANES; }

cudaError_t launch_argmax_static(const float *logits, uint32_t *records, int lanes, int vocab, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (lanes > STATIC_ARGMAX_MAX_LANES) return cudaErrorInvalidValue;
    static std::atomic<void *> device_address[STATIC_ARGMAX_MAX_DEVICES];  // zero-initialised; every thread that looks it up stores the same value
    int device = 0;
    cudaError_t status = cudaGetDevice(&device);
    if (status != cudaSuccess) return status;
    if (device < 0 || device >= STATIC_ARGMAX_MAX_DEVICES) return cudaErrorInvalidDevice;
    void *address = device_address[device].load(std::memory_order_acquire);
    if (address == nullptr) {
        status = cudaGetSymbolAddress(&address, static_argmax_scratch);
        if (status != cudaSuccess) return status;
        device_address[device].store(address, std::memory_order_release);
    }
    return launch_argmax(logits, records, lanes, vocab, address, stream);
}

}  // namespace nerve
