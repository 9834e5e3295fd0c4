// Launches of the persistent decode stack kernel as a C function: layers with given weights, lanes of one or several streams.
#include <vector>

#include "../llmoop_b200/csrc/kernels.cuh"

// What goes in, as device pointers; q, k, v, o, gate, up and down: packed words and scales.
struct StackLayers {
    const void *words[7], *scales[7], *input_norm, *post_norm, *rope;
    void *hidden, *pool, *attention_out;
    const void *table, *positions, *slots;
    int lanes, lanes_per_stream, hidden_width, q_heads, kv_heads, head_width, ffn, page_tokens, pages_per_slot, attended, layers, launches;
    float eps, norm_offset, attention_scale, milliseconds;
};

// 0, a CUDA error, -1: not a shape of this kernel, -2 - n: the kernel's error word
extern "C" __attribute__((visibility("default"))) int stack_layers(StackLayers *t) {
    using namespace nerve;
    StackShape shape{};
    shape.hidden = t->hidden_width;
    shape.q_heads = t->q_heads;
    shape.kv_heads = t->kv_heads;
    shape.head_width = t->head_width;
    shape.ffn = t->ffn;
    shape.eps = t->eps;
    shape.norm_offset = t->norm_offset;
    shape.attention_scale = t->attention_scale;
    shape.rope_table = static_cast<const uint32_t *>(t->rope);
    shape.rope_positions = 1;
    int device = 0;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&shape.grid, cudaDevAttrMultiProcessorCount, device);
    size_t shared = 0;
    if (!decode_stack_supported(shape, t->lanes, &shared)) return -1;

    std::vector<void *> owned;
    cudaError_t status = cudaSuccess;
    auto allocate = [&](size_t bytes) -> void * {
        void *p = nullptr;
        if (status == cudaSuccess) status = cudaMalloc(&p, bytes < 16 ? 16 : bytes);
        if (status == cudaSuccess) status = cudaMemset(p, 0, bytes < 16 ? 16 : bytes);
        owned.push_back(p);
        return p;
    };
    const int q_width = t->q_heads * t->head_width, kv_width = t->kv_heads * t->head_width, splits = (t->attended + 63) / 64;
    auto segment = [&](int i, int rows, int rope) {
        return RelayoutSegment{static_cast<const uint32_t *>(t->words[i]), static_cast<const uint16_t *>(t->scales[i]), rows, rope};
    };
    auto stream = [&](std::vector<RelayoutSegment> segments, bool pair, int k) {
        int rows = 0;
        for (const RelayoutSegment &s : segments) rows += s.rows;
        if (pair) rows /= 2;
        uint8_t *out = static_cast<uint8_t *>(allocate(int4_cta_stream_bytes(rows, k, pair, shape.grid)));
        if (status == cudaSuccess) status = launch_int4_cta_streams(segments.data(), static_cast<int>(segments.size()), pair, k, shape.grid, out, nullptr);
        return out;
    };
    std::vector<StackLayer> layers(t->layers);
    for (StackLayer &layer : layers) {
        layer.qkv = stream({segment(0, q_width, t->head_width), segment(1, kv_width, t->head_width), segment(2, kv_width, 0)}, false, t->hidden_width);
        layer.o = stream({segment(3, t->hidden_width, 0)}, false, q_width);
        layer.gate_up = stream({segment(4, t->ffn, 0), segment(5, t->ffn, 0)}, true, t->hidden_width);
        layer.down = stream({segment(6, t->hidden_width, 0)}, false, t->ffn);
        layer.input_norm = static_cast<const uint16_t *>(t->input_norm);
        layer.post_norm = static_cast<const uint16_t *>(t->post_norm);
        layer.kv = KvLayer{static_cast<uint16_t *>(t->pool), static_cast<const int32_t *>(t->table), t->pages_per_slot, t->page_tokens, t->kv_heads, t->head_width,
                           static_cast<uint32_t>(t->pages_per_slot * t->page_tokens)};
    }
    StackLayer *on_device = static_cast<StackLayer *>(allocate(layers.size() * sizeof(StackLayer)));
    if (status == cudaSuccess) status = cudaMemcpy(on_device, layers.data(), layers.size() * sizeof(StackLayer), cudaMemcpyHostToDevice);
    StackBuffers buffers{};
    buffers.hidden = static_cast<uint16_t *>(t->hidden);
    buffers.q = static_cast<uint16_t *>(allocate(8 * static_cast<size_t>(q_width) * 2));
    buffers.attention_scratch = static_cast<float *>(allocate(static_cast<size_t>(t->lanes) * t->q_heads * (splits + (splits + 31) / 32) * (t->head_width + 2) * 4));
    buffers.attention_out = static_cast<uint16_t *>(t->attention_out);
    buffers.activation = static_cast<uint8_t *>(allocate(stack_activation_bytes(t->ffn)));
    buffers.residual = static_cast<uint8_t *>(allocate(stack_residual_bytes(t->ffn, t->hidden_width > q_width ? t->hidden_width : q_width)));
    buffers.barrier = static_cast<unsigned int *>(allocate(STACK_BARRIER_WORDS * 4));
    buffers.error_flag = static_cast<int *>(allocate(4));
    const LaneTable meta{static_cast<const uint32_t *>(t->positions), static_cast<const int32_t *>(t->slots)};
    cudaEvent_t begin, end;
    cudaEventCreate(&begin);
    cudaEventCreate(&end);
    cudaEventRecord(begin);
    for (int i = 0; i < t->launches && status == cudaSuccess; i++)
        status = launch_decode_stack(on_device, t->layers, shape, buffers, meta, t->lanes, t->lanes_per_stream, 64, splits, nullptr);
    cudaEventRecord(end);
    const cudaError_t finished = cudaDeviceSynchronize();
    if (status == cudaSuccess) status = finished;
    cudaEventElapsedTime(&t->milliseconds, begin, end);
    int error = 0;
    if (status == cudaSuccess) status = cudaMemcpy(&error, buffers.error_flag, 4, cudaMemcpyDeviceToHost);
    for (void *p : owned) cudaFree(p);
    cudaEventDestroy(begin);
    cudaEventDestroy(end);
    if (status != cudaSuccess) return static_cast<int>(status);
    return error != 0 ? -2 - error : 0;
}

extern "C" __attribute__((visibility("default"))) size_t stream_bytes(int rows, int k, int pair) { return nerve::int4_cta_stream_bytes(rows, k, pair != 0, 148); }
