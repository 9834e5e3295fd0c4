// The attention launches of the kernel-per-operator path as a C function, so that a test can read the f32 partials the engine
// keeps to itself.  A ragged batch is given as the lanes of each stream.
#include <vector>

#include "../llmoop_b200/csrc/kernels_attention.cu"

extern "C" __attribute__((visibility("default"))) int attention_partials(const void *q, void *out, void *pool, const void *table, const void *positions, const void *slots,
                                                                          int lanes, int lanes_per_stream, int q_heads, int kv_heads, int head_width, int page_tokens,
                                                                          int pages_per_slot, float scale, int split_tokens, int max_splits, void *scratch, int scalar_f32,
                                                                          const int *ragged_lanes, int ragged_streams) {
    using namespace nerve;
    KvLayer kv{};
    kv.pool = static_cast<uint16_t *>(pool);
    kv.block_table = static_cast<const int32_t *>(table);
    kv.pages_per_slot = pages_per_slot;
    kv.page_tokens = page_tokens;
    kv.kv_heads = kv_heads;
    kv.head_width = head_width;
    kv.capacity = static_cast<uint32_t>(pages_per_slot * page_tokens);
    const LaneTable meta{static_cast<const uint32_t *>(positions), static_cast<const int32_t *>(slots)};
    AttentionBlock *blocks = nullptr;
    int count = 0;
    if (ragged_streams > 0) {
        const int block_lanes = attention_block_lanes(lanes_per_stream, q_heads, kv_heads, head_width, scalar_f32 != 0);
        std::vector<AttentionBlock> host;
        int first = 0;
        for (int s = 0; s < ragged_streams; s++) {
            for (int index = 0; index * block_lanes < ragged_lanes[s]; index++) host.push_back(AttentionBlock{first, ragged_lanes[s], index});
            first += ragged_lanes[s];
        }
        count = static_cast<int>(host.size());
        if (cudaMalloc(&blocks, host.size() * sizeof(AttentionBlock)) != cudaSuccess) return -1;
        if (cudaMemcpy(blocks, host.data(), host.size() * sizeof(AttentionBlock), cudaMemcpyHostToDevice) != cudaSuccess) return -1;
    }
    const cudaError_t status = launch_attention(static_cast<const uint16_t *>(q), static_cast<uint16_t *>(out), kv, meta, lanes, lanes_per_stream, q_heads, scale, split_tokens,
                                                max_splits, static_cast<float *>(scratch), scalar_f32 != 0, nullptr, blocks, count);
    const cudaError_t finished = cudaDeviceSynchronize();
    if (blocks != nullptr) cudaFree(blocks);
    return static_cast<int>(status != cudaSuccess ? status : finished);
}
