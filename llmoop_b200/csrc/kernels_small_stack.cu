// A whole forward of a small dense bf16 model in one launch, a CTA per stream: the embedding and the draft adapter, all layers,
// the final norm, the logits and their arg-max.
//
// A model whose layers are some tens of KB of weights is latency only: as separate kernels a layer is seven dependent
// launches of 1.2 to 2.5 us each for less than a microsecond of work, and a forward has ten more around the layers.  Here a
// stream's lanes stay in one CTA's shared memory from the first step to the last; a layer's weights arrive by bulk copies
// while the layer before it is computed (the first two layers' before the previous kernel has ended), and the steps are
// separated by block barriers.  Streams share nothing but the weights, so a stream's values do not depend on its company.
// The matrices are multiplied on mma.sync (16 rows a warp, eight lanes a tile; tcgen05's 128 rows would be padding): scalar
// f32 took 0.6 us per pass of 64 rows, 8.5 us a layer of hidden 64 and FFN 128 for two lanes.  Sums of 16 columns start
// from zero and join in f32 with Kahan's correction: the tensor core cuts the low bits of what it aligns, and uncorrected
// sums of 32 columns lay 20 to 40 % further from 64-bit sums than scalar f32 (RMS of N(0, 1) times N(0, 0.02), 64 to 512
// columns: 4.7e-8 to 8.7e-8 of the sum's, scalar 3.9e-8 to 6.2e-8; as here 3.8e-8 to 4.1e-8; 32 columns: 3.5e-8 to scalar
// 3.0e-8, which is why fewer than 64 are left to the scalar kernels).
//
// The operations and their rounding points are those of the kernels this replaces: embedding_lookup_bf16.comp.template:31-46,
// rms_norm_bf16.comp.template:49-72, bf16 linears with f32 sums, rotary_bf16.comp.template:99-109,
// append_gqa_attention_bf16.comp.template:189-339, silu_multiply_bf16.comp.template:30-52, add_bf16.comp.template:17-24.
#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

namespace {

constexpr int THREADS = 512, WARPS = THREADS / 32;
constexpr int SHARED_LIMIT = 220 * 1024;  // the rest is the kernel's own arrays
constexpr unsigned int SPIN_LIMIT = 1u << 18;
constexpr int PAGES_HELD = 512;  // pages of a stream's block table row kept in shared memory
constexpr float LOWEST = -3.4028234663852886e38f;

constexpr int PAD = 8;  // bf16 values behind a row of activations: rows 16 bytes apart in the banks

struct Sizes {  // of a lane's row and of a layer's weights
    int q_width, kv_width, floats, halves, inner, weights;
};
__host__ __device__ inline Sizes sizes_of(const SmallStackShape &s) {
    Sizes z;
    z.q_width = s.q_heads * s.head_width;
    z.kv_width = s.kv_heads * s.head_width;
    z.floats = s.hidden + z.q_width + 2 * z.kv_width;         // the hidden row; q | k | v
    z.inner = z.q_width > s.ffn ? z.q_width : s.ffn;          // the attention output or the SiLU products
    z.halves = 2 * s.hidden + PAD + z.inner + PAD;            // the norms of the hidden row (and of the embedding); inner
    z.weights = 2 * (s.hidden * (2 * z.q_width + 2 * z.kv_width) + 3 * s.hidden * s.ffn + 2 * s.hidden);  // the norms' behind the matrices
    return z;
}

__device__ __forceinline__ uint32_t shared_address(const void *object) { return static_cast<uint32_t>(__cvta_generic_to_shared(object)); }
__device__ __forceinline__ void mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// sum + part, with what the addition rounds away kept for the next one
__device__ __forceinline__ void join(float &sum, float &lost, float part) {
    const float corrected = __fsub_rn(part, lost), next = __fadd_rn(sum, corrected);
    lost = __fsub_rn(__fsub_rn(next, sum), corrected);
    sum = next;
}

// rows x k bf16 weights times the lanes' bf16 inputs (shared memory, `pitch` apart); finish(row, lane, sums) for every output.
// With two matrices (gate and up) both sums of a row end in one thread.  The columns of a unit of 32 go to the MMAs' k slots
// as a thread's 16 bytes hold them, alike on both sides.  Lanes beyond the last read what lies there: `finish` drops them.
template <int MATRICES, class Finish>
__device__ __forceinline__ void multiply(const uint16_t *first, const uint16_t *second, int rows, int k, const uint16_t *x, int pitch, int lanes, const Finish &finish) {
    const int warp = threadIdx.x >> 5, g = (threadIdx.x & 31) >> 2, j = threadIdx.x & 3;
    for (int tile = warp; tile < rows >> 4; tile += WARPS) {
        for (int lane0 = 0; lane0 < lanes; lane0 += 8) {
            float sums[MATRICES][4], lost[MATRICES][4];
#pragma unroll
            for (int a = 0; a < MATRICES; a++)
#pragma unroll
                for (int e = 0; e < 4; e++) sums[a][e] = lost[a][e] = 0.0f;
            const uint16_t *in = x + (lane0 + g) * pitch + j * 8;
#pragma unroll 2
            for (int unit = 0; unit < k >> 5; unit++) {
                const uint4 b = *reinterpret_cast<const uint4 *>(in + unit * 32);
#pragma unroll
                for (int a = 0; a < MATRICES; a++) {
                    const uint16_t *row = (a == 0 ? first : second) + (tile * 16 + g) * k + unit * 32 + j * 8;
                    const uint4 upper = *reinterpret_cast<const uint4 *>(row), lower = *reinterpret_cast<const uint4 *>(row + 8 * k);
                    float even[4] = {0.0f, 0.0f, 0.0f, 0.0f}, odd[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                    mma(even, upper.x, lower.x, upper.y, lower.y, b.x, b.y);
                    mma(odd, upper.z, lower.z, upper.w, lower.w, b.z, b.w);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        join(sums[a][e], lost[a][e], even[e]);
                        join(sums[a][e], lost[a][e], odd[e]);
                    }
                }
            }
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int lane = lane0 + 2 * j + (e & 1);
                float mine[MATRICES];
#pragma unroll
                for (int a = 0; a < MATRICES; a++) mine[a] = sums[a][e];
                finish(tile * 16 + g + 8 * (e >> 1), lane, mine);
            }
        }
    }
}

// One warp per lane; `read(lane, column)` gives the row.
template <class Read>
__device__ __forceinline__ void normalise(const Read &read, const uint16_t *weight, uint16_t *y, int pitch, int width, int lanes, float eps, float offset) {
    const int thread = threadIdx.x & 31;
    for (int m = threadIdx.x >> 5; m < lanes; m += WARPS) {
        float sum = 0.0f;
        for (int i = thread; i < width; i += 32) sum = fmaf(read(m, i), read(m, i), sum);
        sum = warp_sum(sum);
        const float inverse = 1.0f / sqrtf(sum * (1.0f / static_cast<float>(width)) + eps);
        for (int i = thread; i < width; i += 32)
            y[m * pitch + i] = static_cast<uint16_t>(f32_to_bf16_bits(read(m, i) * inverse * (bf16_bits_to_f32(weight[i]) + offset)));
    }
}

// One warp per (lane, q head) as in attention_small_kernel, the query and the output in shared memory; the rows of up to four
// tokens per thread are requested together.  `pages`: the stream's row of the block table.
template <int HD>
__device__ __forceinline__ void attend(const float *query_row, uint16_t *out, const KvLayer &kv, const int32_t *pages, uint32_t tick, int kv_head, float scale) {
    constexpr int WORDS = HD / 8, BATCH = HD <= 16 ? 4 : 2;
    const int thread = threadIdx.x & 31;
    const uint32_t capacity = kv.capacity, tokens = tick + 1u < capacity ? tick + 1u : capacity, first_tick = tick + 1u - tokens;
    float query[HD], acc[HD];
#pragma unroll
    for (int d = 0; d < HD; d++) query[d] = query_row[d], acc[d] = 0.0f;
    float maximum = LOWEST, denominator = 0.0f;
    const int half = kv.kv_heads * kv.page_tokens * HD;
    for (uint32_t first = thread; first < tokens; first += 32 * BATCH) {
        uint4 key[BATCH][WORDS], value[BATCH][WORDS];
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            const uint32_t i = first + 32 * b;
            if (i >= tokens) break;
            uint32_t ring = first_tick + i;
            if (ring >= capacity) ring %= capacity;
            const int page = static_cast<int>(ring / kv.page_tokens), within = static_cast<int>(ring - page * kv.page_tokens);
            const uint16_t *row = kv.pool + static_cast<size_t>(pages[page]) * 2 * half + (kv_head * kv.page_tokens + within) * HD;
#pragma unroll
            for (int w = 0; w < WORDS; w++) {
                key[b][w] = __ldcg(reinterpret_cast<const uint4 *>(row) + w);
                value[b][w] = __ldcg(reinterpret_cast<const uint4 *>(row + half) + w);
            }
        }
#pragma unroll
        for (int b = 0; b < BATCH; b++) {
            if (first + 32 * b >= tokens) break;
            float dot = 0.0f;
#pragma unroll
            for (int w = 0; w < WORDS; w++) {
                const uint32_t words[4] = {key[b][w].x, key[b][w].y, key[b][w].z, key[b][w].w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    dot = fmaf(query[8 * w + 2 * e], bf16_lo(words[e]), dot);
                    dot = fmaf(query[8 * w + 2 * e + 1], bf16_hi(words[e]), dot);
                }
            }
            const float score = dot * scale, next = fmaxf(maximum, score), alpha = expf(maximum - next), beta = expf(score - next);
            denominator = denominator * alpha + beta;
            maximum = next;
#pragma unroll
            for (int w = 0; w < WORDS; w++) {
                const uint32_t words[4] = {value[b][w].x, value[b][w].y, value[b][w].z, value[b][w].w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    acc[8 * w + 2 * e] = acc[8 * w + 2 * e] * alpha + beta * bf16_lo(words[e]);
                    acc[8 * w + 2 * e + 1] = acc[8 * w + 2 * e + 1] * alpha + beta * bf16_hi(words[e]);
                }
            }
        }
    }
    const float whole = warp_max(maximum), weight = expf(maximum - whole);
    denominator = warp_sum(denominator * weight);
    // the dims' sums over the warp: every exchange adds the partner's share of half of them
    int dim = 0;
#pragma unroll
    for (int d = 0; d < HD; d++) acc[d] *= weight;
#pragma unroll
    for (int step = 0; step < 5; step++) {
        const int distance = 16 >> step, live = HD >> step;
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
    if (thread % (32 / HD) == 0) out[dim] = static_cast<uint16_t>(f32_to_bf16_bits(denominator == 0.0f ? 0.0f : acc[0] / denominator));
}

template <int HD>
__global__ void __launch_bounds__(THREADS, 1) small_stack_kernel(const SmallStackLayer *__restrict__ layers, int layer_count, const SmallStackShape shape,
                                                                 const __grid_constant__ SmallForward forward, const LaneTable meta, int lanes, int *error_flag) {
    extern __shared__ __align__(128) uint8_t smem[];
    // what every layer needs again: the descriptions of two layers, the lanes' positions, slots and rotary factors, the
    // stream's pages (a global load in front of a dependent one would cost as much as a matrix)
    __shared__ SmallStackLayer described[2];
    __shared__ uint32_t ticks[SMALL_STACK_MAX_LANES];
    __shared__ int32_t slots[SMALL_STACK_MAX_LANES];
    __shared__ uint32_t rotations[SMALL_STACK_MAX_LANES * (HD / 2)];
    __shared__ int32_t page_row[PAGES_HELD];
    __shared__ unsigned long long best[SMALL_STACK_MAX_LANES];  // arg-max keys
    const Sizes z = sizes_of(shape);
    uint64_t *arrived = reinterpret_cast<uint64_t *>(smem);  // [2]
    uint8_t *weights = smem + 128;                           // [2][z.weights]
    float *x = reinterpret_cast<float *>(weights + 2 * static_cast<size_t>(z.weights)), *qkv = x + shape.hidden;
    const int stride = z.floats, pitch = z.halves, padded_lanes = (lanes + 7) & ~7, first_lane = blockIdx.x * lanes, thread = threadIdx.x;
    uint16_t *normed = reinterpret_cast<uint16_t *>(x + lanes * stride), *inner = normed + 2 * shape.hidden + PAD;
    const int matrix_bytes[4] = {2 * shape.hidden * (z.q_width + 2 * z.kv_width), 2 * shape.hidden * z.q_width, 4 * shape.hidden * shape.ffn, 2 * shape.hidden * shape.ffn};
    grid_launch_dependents();
    auto request = [&](int layer) {  // q, k, v, o, gate, up and down, one behind the other
        const SmallStackLayer &spec = layers[layer];
        const uint32_t barrier = shared_address(arrived + (layer & 1));
        uint32_t to = shared_address(weights + static_cast<size_t>(layer & 1) * z.weights);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barrier), "r"(z.weights) : "memory");
        const int bytes[9] = {2 * shape.hidden * z.q_width, 2 * shape.hidden * z.kv_width, 2 * shape.hidden * z.kv_width, 2 * shape.hidden * z.q_width,
                              2 * shape.hidden * shape.ffn, 2 * shape.hidden * shape.ffn, 2 * shape.hidden * shape.ffn, 2 * shape.hidden, 2 * shape.hidden};
#pragma unroll
        for (int i = 0; i < 9; i++) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to),
                         "l"(__cvta_generic_to_global(spec.weights[i])), "r"(bytes[i]), "r"(barrier)
                         : "memory");
            to += bytes[i];
        }
    };
    if (thread == 0) {
        for (int i = 0; i < 2; i++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(shared_address(arrived + i)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
        request(0);
        if (layer_count > 1) request(1);
    }
    constexpr int LAYER_WORDS = static_cast<int>(sizeof(SmallStackLayer) / sizeof(uint32_t));
    auto describe = [&](int layer) {  // by the second warp
        if (thread >= 32 && thread < 32 + LAYER_WORDS && layer < layer_count)
            reinterpret_cast<uint32_t *>(&described[layer & 1])[thread - 32] = reinterpret_cast<const uint32_t *>(layers + layer)[thread - 32];
    };
    describe(0);
    describe(1);
    grid_dependency_wait();  // (the weights are nobody's output)
    if (thread < lanes) {
        ticks[thread] = meta.position[first_lane + thread];
        slots[thread] = meta.slot[first_lane + thread];
    }
    if (thread < padded_lanes) best[thread] = 0ull;
    for (int i = thread; i < lanes * shape.hidden; i += THREADS) {
        const int m = i / shape.hidden, column = i - m * shape.hidden;
        const uint32_t token = __ldcg(forward.tokens + first_lane + m);
        x[m * stride + column] =
            round_bf16(token < static_cast<uint32_t>(forward.vocab) ? bf16_bits_to_f32(__ldg(forward.embedding + static_cast<size_t>(token) * shape.hidden + column)) * forward.embedding_scale : 0.0f);
    }
    __syncthreads();
    if (forward.adapter != nullptr) {  // the draft's input: a linear of the norms of the token's embedding and of the hidden state handed on
        const uint16_t *given = forward.hidden_in + static_cast<size_t>(first_lane) * shape.hidden;
        normalise([&](int m, int i) { return x[m * stride + i]; }, forward.adapter_norms[0], normed + (forward.embedding_first ? 0 : shape.hidden), pitch, shape.hidden, lanes,
                  forward.adapter_eps, forward.adapter_offset);
        normalise([&](int m, int i) { return bf16_bits_to_f32(__ldcg(given + m * shape.hidden + i)); }, forward.adapter_norms[1],
                  normed + (forward.embedding_first ? shape.hidden : 0), pitch, shape.hidden, lanes, forward.adapter_eps, forward.adapter_offset);
        __syncthreads();
        multiply<1>(forward.adapter, nullptr, shape.hidden, 2 * shape.hidden, normed, pitch, lanes, [&](int row, int m, const float *sum) {
            if (m < lanes) x[m * stride + row] = round_bf16(sum[0]);
        });
        __syncthreads();
    }
    for (int i = thread; i < lanes * (HD / 2); i += THREADS)
        rotations[i] = __ldg(shape.rope_table + static_cast<size_t>(ticks[i / (HD / 2)] % shape.rope_positions) * (HD / 2) + i % (HD / 2));
    const int slot = slots[0];  // the lanes are one stream's
    const int32_t *pages = described[0].kv.block_table + static_cast<size_t>(slot < 0 ? 0 : slot) * described[0].kv.pages_per_slot;
    if (described[0].kv.pages_per_slot <= PAGES_HELD) {
        for (int i = thread; i < described[0].kv.pages_per_slot; i += THREADS) page_row[i] = __ldcg(pages + i);
        pages = page_row;
    }
    for (int layer = 0; layer < layer_count; layer++) {
        const SmallStackLayer &spec = described[layer & 1];
        const KvLayer &kv = spec.kv;
        const uint16_t *matrix = reinterpret_cast<const uint16_t *>(weights + static_cast<size_t>(layer & 1) * z.weights);
        {
            unsigned int spins = 0;
            uint32_t done = 0;
            while (true) {
                asm volatile(
                    "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\nselp.u32 %0, 1, 0, p;\n}\n"
                    : "=r"(done)
                    : "r"(shared_address(arrived + (layer & 1))), "r"(static_cast<uint32_t>(layer >> 1) & 1u), "r"(20000u)
                    : "memory");
                if (done) break;
                if (++spins > SPIN_LIMIT) {
                    atomicExch(error_flag, 3);
                    break;
                }
            }
        }
        const uint16_t *norms = matrix + z.weights / 2 - 2 * shape.hidden;
        normalise([&](int m, int i) { return x[m * stride + i]; }, norms, normed, pitch, shape.hidden, lanes, shape.eps, shape.norm_offset);
        __syncthreads();
        const int qkv_rows = z.q_width + 2 * z.kv_width;
        multiply<1>(matrix, nullptr, qkv_rows, shape.hidden, normed, pitch, lanes, [&](int row, int m, const float *sum) {
            if (m < lanes) qkv[m * stride + row] = round_bf16(sum[0]);
        });
        matrix += matrix_bytes[0] / 2;
        __syncthreads();
        // rotation of q (in place) and of k on its way into its page, v beside it; two dims of a head per thread
        const int heads = shape.q_heads + 2 * shape.kv_heads, pairs = HD / 2;
        for (int i = thread; i < lanes * heads * pairs; i += THREADS) {
            const int m = i / (heads * pairs), head = (i / pairs) % heads, f = i % pairs;
            float *row = qkv + m * stride + head * HD;
            float low = row[f], high = row[f + pairs];
            if (head < shape.q_heads + shape.kv_heads) {
                const uint32_t rotation = rotations[m * pairs + f];
                const float cosine = bf16_lo(rotation), sine = bf16_hi(rotation);
                const float turned_low = round_bf16(round_bf16(low * cosine) + round_bf16(-high * sine)), turned_high = round_bf16(round_bf16(high * cosine) + round_bf16(low * sine));
                low = turned_low;
                high = turned_high;
            }
            if (head < shape.q_heads) {
                row[f] = low;
                row[f + pairs] = high;
            } else if (slot >= 0) {
                const bool value = head >= shape.q_heads + shape.kv_heads;
                const int kv_head = head - shape.q_heads - (value ? shape.kv_heads : 0);
                const uint32_t ring = ticks[m] % kv.capacity;
                uint16_t *to = kv.pool + (static_cast<size_t>(pages[ring / kv.page_tokens]) * 2 + (value ? 1 : 0)) * kv.kv_heads * kv.page_tokens * HD +
                               (static_cast<size_t>(kv_head) * kv.page_tokens + ring % kv.page_tokens) * HD;
                to[f] = static_cast<uint16_t>(f32_to_bf16_bits(low));
                to[f + pairs] = static_cast<uint16_t>(f32_to_bf16_bits(high));
            }
        }
        __syncthreads();
        const int group = shape.q_heads / shape.kv_heads;
        for (int index = thread >> 5; index < lanes * shape.q_heads; index += WARPS) {
            const int m = index / shape.q_heads, head = index - m * shape.q_heads;
            uint16_t *out = inner + m * pitch + head * HD;
            if (slot >= 0) attend<HD>(qkv + m * stride + head * HD, out, kv, pages, ticks[m], head / group, shape.attention_scale);
            else if ((thread & 31) < HD) out[thread & 31] = 0;
        }
        __syncthreads();
        auto add_residual = [&](int row, int m, const float *sum) {
            if (m < lanes) x[m * stride + row] = round_bf16(round_bf16(sum[0]) + x[m * stride + row]);
        };
        multiply<1>(matrix, nullptr, shape.hidden, z.q_width, inner, pitch, lanes, add_residual);
        matrix += matrix_bytes[1] / 2;
        __syncthreads();
        normalise([&](int m, int i) { return x[m * stride + i]; }, norms + shape.hidden, normed, pitch, shape.hidden, lanes, shape.eps, shape.norm_offset);
        __syncthreads();
        multiply<2>(matrix, matrix + matrix_bytes[2] / 4, shape.ffn, shape.hidden, normed, pitch, lanes, [&](int row, int m, const float *sum) {
            if (m < lanes) inner[m * pitch + row] = static_cast<uint16_t>(f32_to_bf16_bits(rounded_silu(round_bf16(sum[0])) * round_bf16(sum[1])));
        });
        matrix += matrix_bytes[2] / 2;
        __syncthreads();
        multiply<1>(matrix, nullptr, shape.hidden, shape.ffn, inner, pitch, lanes, add_residual);
        __syncthreads();
        describe(layer + 2);
        if (thread == 0 && layer + 2 < layer_count) {
            asm volatile("fence.proxy.async;" ::: "memory");  // the buffer has been read by every thread
            request(layer + 2);
        }
    }
    if (forward.normalized == nullptr) return;
    normalise([&](int m, int i) { return x[m * stride + i]; }, forward.final_norm, normed, pitch, shape.hidden, lanes, forward.final_eps, forward.final_offset);
    __syncthreads();
    for (int i = thread; i < lanes * shape.hidden; i += THREADS) {
        const int m = i / shape.hidden, column = i - m * shape.hidden;
        forward.normalized[static_cast<size_t>(first_lane) * shape.hidden + i] = normed[m * pitch + column];
    }
    if (forward.logits == nullptr) return;
    // the logits, and the greatest of a lane's (the lowest token of equals): the larger key, an order of f32 as whole numbers
    // in front of the token's complement
    multiply<1>(forward.table, nullptr, forward.vocab, shape.hidden, normed, pitch, lanes, [&](int row, int m, const float *sum) {
        const float logit = sum[0] * forward.logits_scale;
        if (m < lanes) forward.logits[static_cast<size_t>(first_lane + m) * forward.vocab + row] = logit;
        const uint32_t bits = __float_as_uint(logit + 0.0f), order = logit != logit ? 1u : ((bits & 0x80000000u) ? ~bits : bits | 0x80000000u);
        unsigned long long key = (static_cast<unsigned long long>(order) << 32) | static_cast<uint32_t>(~row);
#pragma unroll
        for (int distance = 4; distance < 32; distance *= 2) {  // the rows of a tile sit eight threads apart
            const unsigned long long other = __shfl_xor_sync(0xffffffffu, key, distance);
            key = other > key ? other : key;
        }
        if ((threadIdx.x & 31) < 4) atomicMax(best + m, key);
    });
    if (forward.records == nullptr) return;
    __syncthreads();
    if (thread < lanes) {
        const uint32_t token = ~static_cast<uint32_t>(best[thread]), order = static_cast<uint32_t>(best[thread] >> 32);
        uint32_t *record = forward.records + static_cast<size_t>(first_lane + thread) * 4;
        record[0] = token;
        record[1] = (order & 0x80000000u) ? order & 0x7fffffffu : ~order;
        record[2] = 0u;
        record[3] = 0u;
    }
}

size_t shared_bytes(const SmallStackShape &shape, int lanes) {
    const Sizes z = sizes_of(shape);
    return 128 + 2 * static_cast<size_t>(z.weights) + static_cast<size_t>(lanes) * z.floats * sizeof(float) + static_cast<size_t>((lanes + 7) & ~7) * z.halves * sizeof(uint16_t);
}

}  // namespace

// Two layers' weights and a stream's lanes have to fit a CTA's shared memory, and the logits of one CTA may not cost what the
// launches did.  A verify pass of 2 lanes (kernels of the single operations in brackets): hidden 64, FFN 128, 2 layers,
// vocabulary 256, 20.6 us (34.5), 8 lanes 26 (50), 16 streams 21 (62), 1900 tokens of context 71 (101); hidden 96 with the
// largest layers that fit and vocabulary 1024 27.8 us (36.4), 1900 tokens 87 (104), but vocabulary 4096 46.5 (37.2).
//
// The context counts, too: a warp walks the whole window of a (lane, q head), where the other route spreads it over the chip.
// A layer takes 10, 15 or 62 ns a token (heads of 8, 16, 32) for every sixteen of them, the other route 13 to 19 however many
// they are, but some 15 us more to begin with (whole calls with the host, hidden 64, 2 layers, 4 heads of 16: 8 lanes 80 us and
// 111 at 16 tokens, 199 and 180 at 1900, 2029 and 1239 at 32000; 2 lanes 76 and 133, 127 and 164, 965 and 1247; 32 lanes 133 and
// 130, 592 and 195 at 1900; 3 layers of 8 heads of 8, 8 lanes: 96 and 134, 159 and 153 at 512; a layer of 2 heads of 32, 8 lanes:
// 78 and 104, 106 and 100 at 512).  So what a whole window takes on top may not exceed those 15 us.  The window is the
// mount's capacity, not the context, and up to eight lanes the rule is that of eight: what else is in a batch may not
// change the route of a stream.
bool small_stack_supported(const SmallStackShape &shape, int vocab, uint32_t capacity, int lanes) {
    if (shape.head_width != 8 && shape.head_width != 16 && shape.head_width != 32) return false;
    if (shape.kv_heads < 1 || shape.q_heads < 1 || shape.q_heads % shape.kv_heads != 0) return false;
    const Sizes z = sizes_of(shape);
    if (shape.hidden < 64 || shape.ffn < 64 || z.q_width < 64) return false;
    if (shape.hidden % 32 != 0 || shape.ffn % 32 != 0 || z.q_width % 32 != 0 || (z.q_width + 2 * z.kv_width) % 16 != 0 || z.kv_width % 8 != 0) return false;
    if (vocab % 16 != 0 || vocab > SMALL_STACK_MAX_VOCAB || lanes < 1 || lanes > SMALL_STACK_MAX_LANES) return false;
    const int decided = lanes < 8 ? 8 : lanes, rounds = (decided * shape.q_heads + WARPS - 1) / WARPS;
    const long long nanoseconds = rounds * (shape.head_width == 8 ? 10 : shape.head_width == 16 ? 15 : 62) - 16;
    return shared_bytes(shape, decided) <= SHARED_LIMIT && nanoseconds * capacity <= 15000;
}

cudaError_t launch_small_stack(const SmallStackLayer *layers_device, int layer_count, const SmallStackShape &shape, const SmallForward &forward, const LaneTable &lanes_meta,
                               uint32_t capacity, int streams, int lanes_per_stream, int *error_flag, cudaStream_t stream) {
    if (streams < 1 || layer_count < 1 || !small_stack_supported(shape, forward.vocab, capacity, lanes_per_stream)) return cudaErrorInvalidValue;
    auto kernel = shape.head_width == 32 ? small_stack_kernel<32> : shape.head_width == 16 ? small_stack_kernel<16> : small_stack_kernel<8>;
    // (never lowered: a captured launch keeps its own size)
    const cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SHARED_LIMIT);
    if (status != cudaSuccess) return status;
    return launch_dependent(kernel, dim3(streams), dim3(THREADS), shared_bytes(shape, lanes_per_stream), 1, stream, layers_device, layer_count, shape, forward, lanes_meta,
                            lanes_per_stream, error_flag);
}

}  // namespace nerve
