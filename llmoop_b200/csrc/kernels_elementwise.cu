// Element-wise and per-lane kernels: embedding gather, RMSNorm, residual add,
// SiLU*up, concatenate, RoPE (optionally with per-head RMSNorm), FP8 activation
// quantisation, MoE routing and reduce.  All are HBM/L2-trivial (KBs per lane);
// they exist to keep the reference's bf16 rounding points, and are sized so a
// verify batch (<= 160 lanes) fills the SMs with one CTA per lane (x head).
#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

// Bound by the pages' bytes (32 pages of 64 KB in 33 layers: 140 MB moved); four CTAs share a page so that a single
// stream's page still spreads over the chip.
constexpr int PAGE_COPY_PARTS = 4;
__global__ void __launch_bounds__(256) copy_pages_kernel(const PagePool *__restrict__ pools, const PageCopy *__restrict__ pages) {
    grid_launch_dependents();
    grid_dependency_wait();
    const PagePool pool = pools[blockIdx.y];
    const PageCopy page = pages[blockIdx.x];
    const uint8_t *from = pool.base + static_cast<size_t>(page.from) * pool.page_bytes;
    uint8_t *to = pool.base + static_cast<size_t>(page.to) * pool.page_bytes;
    const size_t first = blockIdx.z * blockDim.x + threadIdx.x, stride = static_cast<size_t>(PAGE_COPY_PARTS) * blockDim.x;
    if (pool.page_bytes % 16 == 0) {
#pragma unroll 4
        for (size_t i = first; i < pool.page_bytes / 16; i += stride) reinterpret_cast<uint4 *>(to)[i] = reinterpret_cast<const uint4 *>(from)[i];
    } else {
        for (size_t i = first; i < pool.page_bytes / 4; i += stride) reinterpret_cast<uint32_t *>(to)[i] = reinterpret_cast<const uint32_t *>(from)[i];
    }
}

cudaError_t launch_copy_pages(const PagePool *pools, int layers, const PageCopy *pages, int count, cudaStream_t stream) {
    if (layers <= 0 || count <= 0) return cudaSuccess;
    return launch_dependent(copy_pages_kernel, dim3(count, layers, PAGE_COPY_PARTS), dim3(256), 0, 1, stream, pools, pages);
}

// embedding_lookup_bf16.comp.template:31-46: out = bf16(bf16(row) * scale); a
// token id >= vocab leaves the frame untouched.
__global__ void embedding_kernel(const uint32_t *__restrict__ table, const uint32_t *__restrict__ tokens,
                                 uint32_t *__restrict__ out, int width_words, int vocab, float scale) {
    grid_launch_dependents();
    grid_dependency_wait();
    int lane = blockIdx.y;
    uint32_t token = tokens[lane];
    if (token >= static_cast<uint32_t>(vocab)) return;
    for (int word = blockIdx.x * blockDim.x + threadIdx.x; word < width_words; word += gridDim.x * blockDim.x) {
        uint32_t packed = table[static_cast<size_t>(token) * width_words + word];
        out[static_cast<size_t>(lane) * width_words + word] = pack_bf16(bf16_lo(packed) * scale, bf16_hi(packed) * scale);
    }
}

cudaError_t launch_embedding(const uint16_t *table, const uint32_t *tokens, uint16_t *out, int lanes, int width,
                             int vocab, float scale, cudaStream_t stream) {
    int words = width / 2;
    dim3 grid((words + 255) / 256, lanes);
    return launch_dependent(embedding_kernel, grid, dim3(256), 0, 1, stream, reinterpret_cast<const uint32_t *>(table), tokens, reinterpret_cast<uint32_t *>(out), words, vocab, scale);
}

// rms_norm_bf16.comp.template:49-72: y = bf16(x * rsqrt(mean(x^2) + eps) * (w + offset)), f32 math.  A row is one CTA's:
// latency, not bandwidth.  A thread's words (WORDS of them, blockDim apart, or more than that in a loop) and their weights
// are requested together and stay in registers between the two passes (one lane of 4096: 4.1 -> 1.7 us).
template <int WORDS>
__global__ void rms_norm_kernel(const uint32_t *__restrict__ x, const uint32_t *__restrict__ weight,
                                uint32_t *__restrict__ y, int width_words, float inv_width, float eps, float offset) {
    __shared__ float partial[32];
    const uint32_t *row = x + static_cast<size_t>(blockIdx.x) * width_words;
    uint32_t *out = y + static_cast<size_t>(blockIdx.x) * width_words;
    const int step = blockDim.x;
    constexpr int HELD = WORDS > 0 ? WORDS : 1;
    uint32_t values[HELD], weights[HELD];
    grid_launch_dependents();
    if (WORDS > 0) {  // (the weights are nobody's output)
#pragma unroll
        for (int i = 0; i < WORDS; i++)
            if (static_cast<int>(threadIdx.x) + i * step < width_words) weights[i] = __ldg(weight + threadIdx.x + i * step);
    }
    grid_dependency_wait();
    float sum = 0.0f;
    auto square = [&](uint32_t packed) {
        const float lo = bf16_lo(packed), hi = bf16_hi(packed);
        sum = fmaf(lo, lo, sum);
        sum = fmaf(hi, hi, sum);
    };
    if (WORDS > 0) {
#pragma unroll
        for (int i = 0; i < WORDS; i++)
            if (static_cast<int>(threadIdx.x) + i * step < width_words) values[i] = row[threadIdx.x + i * step];
#pragma unroll
        for (int i = 0; i < WORDS; i++)
            if (static_cast<int>(threadIdx.x) + i * step < width_words) square(values[i]);
    } else {
        for (int word = threadIdx.x; word < width_words; word += step) square(row[word]);
    }
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = sum;
    __syncthreads();
    float total = 0.0f;
    for (int warp = 0; warp < (step >> 5); warp++) total += partial[warp];
    // IEEE sqrt and divide (nvcc's default -prec-sqrt/-prec-div), as a CPU evaluates 1/sqrt(v)
    const float inv_rms = 1.0f / sqrtf(total * inv_width + eps);
    auto norm = [&](uint32_t packed, uint32_t w) { return pack_bf16(bf16_lo(packed) * inv_rms * (bf16_lo(w) + offset), bf16_hi(packed) * inv_rms * (bf16_hi(w) + offset)); };
    if (WORDS > 0) {
#pragma unroll
        for (int i = 0; i < WORDS; i++)
            if (static_cast<int>(threadIdx.x) + i * step < width_words) out[threadIdx.x + i * step] = norm(values[i], weights[i]);
    } else {
        for (int word = threadIdx.x; word < width_words; word += step) out[word] = norm(row[word], weight[word]);
    }
}

cudaError_t launch_rms_norm(const uint16_t *x, const uint16_t *weight, uint16_t *y, int lanes, int width, float eps,
                            float weight_offset, cudaStream_t stream) {
    int words = width / 2;
    int threads = words >= 1024 ? 512 : (words >= 256 ? 256 : (words >= 64 ? 64 : 32));
    const int held = (words + threads - 1) / threads;
    auto kernel = held <= 2 ? rms_norm_kernel<2> : held <= 4 ? rms_norm_kernel<4> : held <= 8 ? rms_norm_kernel<8> : rms_norm_kernel<0>;
    return launch_dependent(kernel, dim3(lanes), dim3(threads), 0, 1, stream, reinterpret_cast<const uint32_t *>(x), reinterpret_cast<const uint32_t *>(weight), reinterpret_cast<uint32_t *>(y), words, 1.0f / static_cast<float>(width), eps, weight_offset);
}

// add_bf16.comp.template:17-24
__global__ void add_kernel(const uint32_t *__restrict__ a, const uint32_t *__restrict__ b, uint32_t *__restrict__ y,
                           size_t words) {
    grid_launch_dependents();
    grid_dependency_wait();
    for (size_t word = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; word < words;
         word += static_cast<size_t>(gridDim.x) * blockDim.x) {
        uint32_t left = a[word], right = b[word];
        y[word] = pack_bf16(bf16_lo(left) + bf16_lo(right), bf16_hi(left) + bf16_hi(right));
    }
}

cudaError_t launch_add(const uint16_t *a, const uint16_t *b, uint16_t *y, size_t count, cudaStream_t stream) {
    size_t words = count / 2;
    int blocks = static_cast<int>((words + 255) / 256);
    blocks = std::min(blocks, multiprocessors() * 8);
    if (blocks < 1) blocks = 1;
    return launch_dependent(add_kernel, dim3(blocks), dim3(256), 0, 1, stream, reinterpret_cast<const uint32_t *>(a), reinterpret_cast<const uint32_t *>(b), reinterpret_cast<uint32_t *>(y), words);
}

// After the tensor-parallel all-reduce of a row-parallel linear: the reference's linear rounds its f32 sum to bf16
// and its residual_add rounds again (add_bf16.comp.template:17-24).
__global__ void round_add_kernel(const float *__restrict__ sums, const uint16_t *__restrict__ residual, uint16_t *__restrict__ out,
                                 size_t count) {
    grid_launch_dependents();
    grid_dependency_wait();
    for (size_t index = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; index < count;
         index += static_cast<size_t>(gridDim.x) * blockDim.x) {
        float value = round_bf16(sums[index]);
        if (residual != nullptr) value += bf16_bits_to_f32(residual[index]);
        out[index] = static_cast<uint16_t>(f32_to_bf16_bits(value));
    }
}

cudaError_t launch_round_add(const float *sums, const uint16_t *residual, uint16_t *out, size_t count, cudaStream_t stream) {
    int blocks = static_cast<int>((count + 255) / 256);
    blocks = std::min(blocks, multiprocessors() * 8);
    if (blocks < 1) blocks = 1;
    return launch_dependent(round_add_kernel, dim3(blocks), dim3(256), 0, 1, stream, sums, residual, out, count);
}

// silu_multiply_bf16.comp.template:30-52: bf16(bf16(silu(gate)) * up)
__global__ void silu_multiply_kernel(const uint32_t *__restrict__ gate, const uint32_t *__restrict__ up,
                                     uint32_t *__restrict__ y, size_t words) {
    grid_launch_dependents();
    grid_dependency_wait();
    for (size_t word = blockIdx.x * static_cast<size_t>(blockDim.x) + threadIdx.x; word < words;
         word += static_cast<size_t>(gridDim.x) * blockDim.x) {
        uint32_t g = gate[word], u = up[word];
        y[word] = pack_bf16(rounded_silu(bf16_lo(g)) * bf16_lo(u), rounded_silu(bf16_hi(g)) * bf16_hi(u));
    }
}

cudaError_t launch_silu_multiply(const uint16_t *gate, const uint16_t *up, uint16_t *y, size_t count,
                                 cudaStream_t stream) {
    size_t words = count / 2;
    int blocks = static_cast<int>((words + 255) / 256);
    blocks = std::min(blocks, multiprocessors() * 8);
    if (blocks < 1) blocks = 1;
    return launch_dependent(silu_multiply_kernel, dim3(blocks), dim3(256), 0, 1, stream, reinterpret_cast<const uint32_t *>(gate), reinterpret_cast<const uint32_t *>(up), reinterpret_cast<uint32_t *>(y), words);
}

// concatenate_bf16.comp.template:20-30 (per lane: [a | b])
template <typename Word>
__global__ void concat_kernel(const Word *__restrict__ a, const Word *__restrict__ b, Word *__restrict__ y,
                              int words_a, int words_b) {
    grid_launch_dependents();
    grid_dependency_wait();
    int lane = blockIdx.x;
    int total = words_a + words_b;
    for (int word = blockIdx.y * blockDim.x + threadIdx.x; word < total; word += gridDim.y * blockDim.x)
        y[static_cast<size_t>(lane) * total + word] =
            word < words_a ? a[static_cast<size_t>(lane) * words_a + word] : b[static_cast<size_t>(lane) * words_b + word - words_a];
}

cudaError_t launch_concat(const uint16_t *a, const uint16_t *b, uint16_t *y, int lanes, int width_a, int width_b,
                          cudaStream_t stream) {
    if (width_a % 8 == 0 && width_b % 8 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(y)) & 15) == 0)
        return launch_dependent(concat_kernel<uint4>, dim3(lanes, ((width_a + width_b) / 8 + 255) / 256), dim3(256), 0, 1, stream, reinterpret_cast<const uint4 *>(a),
                                reinterpret_cast<const uint4 *>(b), reinterpret_cast<uint4 *>(y), width_a / 8, width_b / 8);
    return launch_dependent(concat_kernel<uint32_t>, dim3(lanes), dim3(256), 0, 1, stream, reinterpret_cast<const uint32_t *>(a), reinterpret_cast<const uint32_t *>(b), reinterpret_cast<uint32_t *>(y), width_a / 2, width_b / 2);
}

// rotary_bf16.comp.template:99-109 (five bf16 roundings per element) with
// cos/sin taken from a table the mounter fills with the same f32 pow/cos/sin
// sequence; parallel_head_norm_rope_2way_bf16.comp.template:166-209 when
// norm_weight is given (per-head RMSNorm rounded to bf16 first).
// One CTA per (head, lane); blockDim = head_width/2 rounded up to a warp.
__global__ void rope_kernel(const uint16_t *__restrict__ x, uint16_t *__restrict__ y, const uint32_t *__restrict__ cos_sin,
                            uint32_t table_positions, const uint32_t *__restrict__ positions, int heads, int head_width,
                            int rotary, int interleaved, const uint16_t *__restrict__ norm_weight, float eps, float offset) {
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ float values[];  // head_width normalised (or raw) inputs as f32
    __shared__ float partial[32];
    int head = blockIdx.x, lane = blockIdx.y;
    const uint16_t *in = x + (static_cast<size_t>(lane) * heads + head) * head_width;
    uint16_t *out = y + (static_cast<size_t>(lane) * heads + head) * head_width;
    float sum = 0.0f;
    for (int d = threadIdx.x; d < head_width; d += blockDim.x) {
        float value = bf16_bits_to_f32(in[d]);
        values[d] = value;
        sum = fmaf(value, value, sum);
    }
    if (norm_weight != nullptr) {
        sum = warp_sum(sum);
        if ((threadIdx.x & 31) == 0) partial[threadIdx.x >> 5] = sum;
        __syncthreads();
        float total = 0.0f;
        for (int warp = 0; warp < (blockDim.x >> 5); warp++) total += partial[warp];
        float inv_rms = 1.0f / sqrtf(total / static_cast<float>(head_width) + eps);
        for (int d = threadIdx.x; d < head_width; d += blockDim.x)
            values[d] = round_bf16(values[d] * inv_rms * (bf16_bits_to_f32(norm_weight[d]) + offset));
    }
    __syncthreads();
    uint32_t position = positions[lane] % table_positions;
    int half = rotary / 2;
    for (int d = threadIdx.x; d < head_width; d += blockDim.x) {
        float result;
        if (d >= rotary) {
            result = values[d];
        } else {
            int frequency = interleaved ? d / 2 : d % half;
            uint32_t packed = cos_sin[static_cast<size_t>(position) * half + frequency];
            float cosine = bf16_lo(packed), sine = bf16_hi(packed);
            float other;
            if (interleaved) other = (d & 1) == 0 ? -values[d + 1] : values[d - 1];
            else other = d < half ? -values[d + half] : values[d - half];
            float direct = round_bf16(values[d] * cosine);
            float rotated = round_bf16(other * sine);
            result = direct + rotated;
        }
        out[d] = static_cast<uint16_t>(f32_to_bf16_bits(result));
    }
}

cudaError_t launch_rope(const uint16_t *x, uint16_t *y, const uint32_t *cos_sin, uint32_t table_positions,
                        const uint32_t *positions, int lanes, int heads, int head_width, int rotary, int interleaved,
                        const uint16_t *norm_weight, float eps, float weight_offset, cudaStream_t stream) {
    int threads = ((head_width / 2 + 31) / 32) * 32;
    if (threads > 256) threads = 256;
    dim3 grid(heads, lanes);
    return launch_dependent(rope_kernel, grid, dim3(threads), head_width * sizeof(float), 1, stream, x, y, cos_sin, table_positions, positions, heads, head_width, rotary, interleaved, norm_weight, eps, weight_offset);
}

// quantize_fp8_e4m3.comp.template:41-60: per 128-column block scale = absmax/448
// (1 when the block is all zero), q = e4m3(x / scale).  One warp per block.
__global__ void quantize_fp8_kernel(const uint32_t *__restrict__ x, uint32_t *__restrict__ q, float *__restrict__ scales,
                                    int blocks_total) {
    grid_launch_dependents();
    grid_dependency_wait();
    int block = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (block >= blocks_total) return;
    int lane = threadIdx.x & 31;
    // 128 columns = 64 words; each thread takes 2 words = 4 values
    const uint32_t *src = x + static_cast<size_t>(block) * 64 + lane * 2;
    uint32_t w0 = src[0], w1 = src[1];
    float v0 = bf16_lo(w0), v1 = bf16_hi(w0), v2 = bf16_lo(w1), v3 = bf16_hi(w1);
    float lane_max = fmaxf(fmaxf(fabsf(v0), fabsf(v1)), fmaxf(fabsf(v2), fabsf(v3)));
    float block_max = warp_max(lane_max);
    float scale = block_max > 0.0f ? block_max / 448.0f : 1.0f;
    if (lane == 0) scales[block] = scale;
    uint32_t packed = static_cast<uint32_t>(f32_to_e4m3(v0 / scale)) | (static_cast<uint32_t>(f32_to_e4m3(v1 / scale)) << 8) |
                      (static_cast<uint32_t>(f32_to_e4m3(v2 / scale)) << 16) |
                      (static_cast<uint32_t>(f32_to_e4m3(v3 / scale)) << 24);
    q[static_cast<size_t>(block) * 32 + lane] = packed;
}

cudaError_t launch_quantize_fp8(const uint16_t *x, uint8_t *q, float *scales, int lanes, int k, cudaStream_t stream) {
    int blocks_total = lanes * (k / 128);
    int warps_per_cta = 8;
    return launch_dependent(quantize_fp8_kernel, dim3((blocks_total + warps_per_cta - 1) / warps_per_cta), dim3(warps_per_cta * 32), 0, 1, stream, reinterpret_cast<const uint32_t *>(x), reinterpret_cast<uint32_t *>(q), scales, blocks_total);
}

// moe_topk_bf16.comp.template:42-84.  One warp per lane: top_k rounds of
// arg-max (first max wins: lowest expert id among equals), softmax over the
// selected logits accumulated in score order, routes sorted by expert id,
// word = bf16(weight) << 16 | expert.
// One warp per token.  A score and its expert make one key (bf16 bits in an order of unsigned numbers, then the smaller
// expert first), so that a choice is one warp-wide maximum: bound by that chain of top_k steps (128 experts, top 8: 9.7 us
// with five exchanges of two values per step and one thread for the weights, now 3.6).
__global__ void moe_topk_kernel(const uint16_t *__restrict__ router_logits, uint32_t *__restrict__ routes, int experts,
                                int top_k) {
    extern __shared__ uint16_t scores[];  // [experts] in an order of unsigned numbers; 0: chosen, or never to be chosen (-inf, NaN)
    __shared__ int selected[64];
    __shared__ float terms[64];
    grid_launch_dependents();
    grid_dependency_wait();
    const int token = blockIdx.x, lane = threadIdx.x;
    const uint16_t *logits = router_logits + static_cast<size_t>(token) * experts;
    auto key_of = [&](int e) { return scores[e] == 0 ? 0u : (static_cast<uint32_t>(scores[e]) << 16) | (0xffffu - static_cast<uint32_t>(e)); };
    uint32_t mine = 0;  // the largest of this thread's keys
    for (int e = lane; e < experts; e += 32) {
        uint32_t bits = logits[e], magnitude = bits & 0x7fffu;
        if (magnitude == 0) bits = 0;  // -0 ties with 0
        const bool never = magnitude > 0x7f80u || bits == 0xff80u;
        scores[e] = static_cast<uint16_t>(never ? 0u : (bits & 0x8000u) ? 0xffffu - bits : bits | 0x8000u);
        mine = max(mine, key_of(e));
    }
    for (int route = 0; route < top_k; route++) {
        const uint32_t best = __reduce_max_sync(0xffffffffu, mine);
        const int expert = best == 0 ? 0 : static_cast<int>(0xffffu - (best & 0xffffu));  // every remaining score is -inf or NaN: the shader keeps expert 0
        if (lane == 0) selected[route] = expert;
        if (best != 0 && mine == best) {
            scores[expert] = 0;
            mine = 0;
            for (int e = lane; e < experts; e += 32) mine = max(mine, key_of(e));
        }
    }
    __syncwarp();
    const float maximum = bf16_bits_to_f32(logits[selected[0]]);
    for (int route = lane; route < top_k; route += 32) terms[route] = expf(bf16_bits_to_f32(logits[selected[route]]) - maximum);
    __syncwarp();
    float denominator = 0.0f;
    for (int route = 0; route < top_k; route++) denominator += terms[route];  // in the order of choice
    for (int route = lane; route < top_k; route += 32) {  // written in the order of the experts
        const int expert = selected[route];
        int place = 0;
        for (int other = 0; other < top_k; other++) place += selected[other] < expert || (selected[other] == expert && other < route);
        routes[static_cast<size_t>(token) * top_k + place] = (static_cast<uint32_t>(f32_to_bf16_bits(terms[route] / denominator)) << 16) | static_cast<uint32_t>(expert);
    }
}

cudaError_t launch_moe_topk(const uint16_t *router_logits, uint32_t *routes, int lanes, int experts, int top_k,
                            cudaStream_t stream) {
    if (top_k > 64 || experts > 65536) return cudaErrorInvalidValue;  // (a route holds sixteen bits of expert)
    const size_t smem = static_cast<size_t>(experts) * sizeof(uint16_t);
    if (smem > 48 * 1024) {
        const cudaError_t status = cudaFuncSetAttribute(moe_topk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (status != cudaSuccess) return status;
    }
    return launch_dependent(moe_topk_kernel, dim3(lanes), dim3(32), smem, 1, stream, router_logits, routes, experts, top_k);
}

// moe_reduce_bf16.comp.template:28-45: bf16-rounded running sum over the routes
// in route (expert-id) order, then * routed scale.
// A thread adds one word up; its contributions are requested eight at a time (one after the other, four words a thread: 5.8 us
// for 24 tokens of 2048, now 1.6).
__global__ void moe_reduce_kernel(const uint32_t *__restrict__ outputs, uint32_t *__restrict__ y, int hidden_words,
                                  int top_k, float routed_scale) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int token = blockIdx.x, word = blockIdx.y * blockDim.x + threadIdx.x;
    if (word >= hidden_words) return;
    const uint32_t *source = outputs + static_cast<size_t>(token) * top_k * hidden_words + word;
    float lo = 0.0f, hi = 0.0f;
    constexpr int BATCH = 8;
    for (int first = 0; first < top_k; first += BATCH) {
        uint32_t contribution[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; i++)
            if (first + i < top_k) contribution[i] = source[static_cast<size_t>(first + i) * hidden_words];
#pragma unroll
        for (int i = 0; i < BATCH; i++) {
            if (first + i >= top_k) break;
            lo = round_bf16(lo + bf16_lo(contribution[i]));
            hi = round_bf16(hi + bf16_hi(contribution[i]));
        }
    }
    y[static_cast<size_t>(token) * hidden_words + word] = pack_bf16(lo * routed_scale, hi * routed_scale);
}

cudaError_t launch_moe_reduce(const uint16_t *outputs, uint16_t *y, int lanes, int hidden_size, int top_k,
                              float routed_scale, cudaStream_t stream) {
    const int words = hidden_size / 2;
    return launch_dependent(moe_reduce_kernel, dim3(lanes, (words + 255) / 256), dim3(256), 0, 1, stream, reinterpret_cast<const uint32_t *>(outputs),
                            reinterpret_cast<uint32_t *>(y), words, top_k, routed_scale);
}

}  // namespace nerve
