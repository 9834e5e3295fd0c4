// Launchers for the sm_100a kernels of the MTP decode path.  Activations are
// bf16 row-major [lane][width]; `lanes` is the batch of (stream, tick) pairs
// processed in one launch (verify candidates, prefill chunk, or multi-stream
// decode).  All functions enqueue on `stream` and return the launch status.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace nerve {

// Per-launch description of the lanes that touch transient state.
struct LaneTable {
    const uint32_t *position;  // [lanes] stream tick (low 32 bits) of each lane
    const int32_t *slot;       // [lanes] stream slot of each lane (row of block_table)
};

// Paged KV state of one attention layer.  Page p holds `page_tokens` tokens:
//   K at kv + p*page_elems + (head*page_tokens + t)*head_width
//   V at the same offset + page_elems/2
// A stream's logical token index i lives in page block_table[slot][ (i / page_tokens) % pages_per_slot ].
struct KvLayer {
    uint16_t *pool;
    const int32_t *block_table;  // [slots][pages_per_slot]
    int pages_per_slot;
    int page_tokens;
    int kv_heads;
    int head_width;
    uint32_t capacity;  // pages_per_slot * page_tokens (ring length in tokens)
};

// Copies of KV pages within their pools: pages[i].from -> pages[i].to in every layer's pool.
struct PagePool {
    uint8_t *base;
    size_t page_bytes;  // a multiple of 4
};
struct PageCopy {
    int32_t from, to;
};
constexpr int MAX_PAGE_COPIES = 1024;  // of one launch
cudaError_t launch_copy_pages(const PagePool *pools, int layers, const PageCopy *pages, int count, cudaStream_t stream);

cudaError_t launch_embedding(const uint16_t *table, const uint32_t *tokens, uint16_t *out, int lanes, int width,
                             int vocab, float scale, cudaStream_t stream);

cudaError_t launch_rms_norm(const uint16_t *x, const uint16_t *weight, uint16_t *y, int lanes, int width, float eps,
                            float weight_offset, cudaStream_t stream);

cudaError_t launch_add(const uint16_t *a, const uint16_t *b, uint16_t *y, size_t count, cudaStream_t stream);
cudaError_t launch_silu_multiply(const uint16_t *gate, const uint16_t *up, uint16_t *y, size_t count, cudaStream_t stream);
cudaError_t launch_concat(const uint16_t *a, const uint16_t *b, uint16_t *y, int lanes, int width_a, int width_b,
                          cudaStream_t stream);

// RoPE from a host-built table: cos_sin[(position % table_positions) * rotary/2 + f] = {bf16 cos, bf16 sin} packed
// in one u32 (cos low).  Optional per-head RMSNorm first (norm_weight != nullptr).
cudaError_t launch_rope(const uint16_t *x, uint16_t *y, const uint32_t *cos_sin, uint32_t table_positions,
                        const uint32_t *positions, int lanes, int heads, int head_width, int rotary, int interleaved,
                        const uint16_t *norm_weight, float eps, float weight_offset, cudaStream_t stream);

enum LinearEpilogue {
    EPILOGUE_BF16 = 0,            // y = bf16(sum)
    EPILOGUE_RESIDUAL_ROUNDED = 1,  // y = bf16(bf16(sum) + residual)        (BF16 / INT4 packages)
    EPILOGUE_RESIDUAL_F32 = 2,    // y = bf16(sum + residual)                (FP8 packages)
    EPILOGUE_F32_SCALED = 3,      // y_f32 = sum * scale                     (logits; tensor-parallel partial sums)
};

// y[m][n] = sum_k x[m][k] * W[n][k], bf16 weights.  The form fixes the order of additions: by the number of lanes, or the
// caller's choice (tensor cores where K allows).
enum LinearForm { LINEAR_AUTO, LINEAR_SCALAR, LINEAR_TENSOR };
bool linear_bf16_is_scalar(int lanes, int n, int k, LinearForm form);
// Up to three matrices that share their input (q, k, v) in one launch.
struct LinearBranches {
    int count = 0;
    const void *w[3] = {};
    const uint16_t *scale[3] = {};  // FP8: block scales
    void *y[3] = {};
    int n[3] = {};
    void add(const void *weights, const uint16_t *scales, void *out, int rows) {
        w[count] = weights;
        scale[count] = scales;
        y[count] = out;
        n[count++] = rows;
    }
};
// bf16, eight lanes or fewer at a time in scalar f32 (the form launch_linear_bf16 takes for LINEAR_SCALAR or up to eight lanes).
cudaError_t launch_linear_bf16_scalar(const uint16_t *x, const LinearBranches &branches, const uint16_t *residual, int lanes, int k, int epilogue, float scale,
                                      cudaStream_t stream);
cudaError_t launch_linear_fp8_multi(const uint8_t *xq, const float *xscale, const LinearBranches &branches, const uint16_t *residual, int lanes, int k,
                                    int epilogue, cudaStream_t stream);
cudaError_t launch_linear_bf16(const uint16_t *x, const uint16_t *w, void *y, const uint16_t *residual, int lanes,
                               int n, int k, int epilogue, float scale, cudaStream_t stream, int *error_flag = nullptr, LinearForm form = LINEAR_AUTO);
// y = bf16( silu_bf16(bf16(x.Wg)) * bf16(x.Wu) )
cudaError_t launch_linear_silu_multiply_bf16(const uint16_t *x, const uint16_t *wg, const uint16_t *wu, uint16_t *y,
                                             int lanes, int n, int k, cudaStream_t stream);

// INT4 compressed-tensors weight-only linear: qweight [n][k/8] u32, scales bf16 [n][k/group].
// Batches of more than 8 lanes run the tensor-core GEMM, which reads the activations from `prepared`
// (launch_prepare_activations of the same x); smaller ones read x.
// error_flag (optional device word): set to 3 by the GEMM if one of its bounded waits expires.
cudaError_t launch_linear_int4(const uint16_t *x, const void *prepared, const uint32_t *qweight, const uint16_t *scales, uint16_t *y,
                               const uint16_t *residual, int lanes, int n, int k, int group, int epilogue,
                               cudaStream_t stream, int *error_flag = nullptr);

// FP8 W8A8: xq e4m3 [lanes][k], xscale f32 [lanes][k/128]; w e4m3 [n][k]; wscale bf16 [ceil(n/128)][k/128].
cudaError_t launch_quantize_fp8(const uint16_t *x, uint8_t *q, float *scales, int lanes, int k, cudaStream_t stream);
cudaError_t launch_linear_fp8(const uint8_t *xq, const float *xscale, const uint8_t *w, const uint16_t *wscale,
                              uint16_t *y, const uint16_t *residual, int lanes, int n, int k, int epilogue,
                              cudaStream_t stream);
cudaError_t launch_linear_silu_multiply_fp8(const uint8_t *xq, const float *xscale, const uint8_t *wg,
                                            const uint16_t *wg_scale, const uint8_t *wu, const uint16_t *wu_scale,
                                            uint16_t *y, int lanes, int n, int k, cudaStream_t stream);

// MoE (softmax over the selected experts, routes sorted by expert id).
cudaError_t launch_moe_topk(const uint16_t *router_logits, uint32_t *routes, int lanes, int experts, int top_k,
                            cudaStream_t stream);
// The (token, route) pairs of a batch grouped by expert, up to eight of one expert to a tile.
struct MoeGroups {
    int4 *tiles;      // {expert, first place in order, count, 0}
    int *order;       // pair = token * top_k + route
    int *tile_count;
};
size_t moe_group_bytes(int lanes, int top_k, int experts);
MoeGroups moe_groups(void *scratch, int lanes, int top_k, int experts);  // carves moe_group_bytes bytes
cudaError_t launch_moe_group(const uint32_t *routes, const MoeGroups &groups, int lanes, int top_k, int experts, cudaStream_t stream);
// xq / xscale: the hidden frames [lanes], or the intermediates [lanes * top_k], as launch_quantize_fp8 writes them.
cudaError_t launch_moe_gate_up_fp8(const uint8_t *xq, const float *xscale, const MoeGroups &groups, const uint8_t *w,
                                   const uint16_t *wscale, uint16_t *intermediates, int lanes, int hidden_size,
                                   int inter, int experts, int top_k, cudaStream_t stream);
cudaError_t launch_moe_down_fp8(const uint8_t *xq, const float *xscale, const MoeGroups &groups, const uint32_t *routes, const uint8_t *w,
                                const uint16_t *wscale, uint16_t *outputs, int lanes, int hidden_size, int inter,
                                int experts, int top_k, cudaStream_t stream);
cudaError_t launch_moe_reduce(const uint16_t *outputs, uint16_t *y, int lanes, int hidden_size, int top_k,
                              float routed_scale, cudaStream_t stream);

// Rotary embedding of q and k (with a per-head RMSNorm in front where norm weights are given) and the append of K and V
// at every lane's position, in one launch.
struct RopeForm {
    const uint32_t *cos_sin;  // [position][rotary / 2] packed (sin << 16 | cos) bf16
    uint32_t positions;
    int rotary, interleaved;  // rotary 0: the values as they are
};
struct RopeAppend {
    const uint16_t *q, *k, *v;
    uint16_t *q_out;
    const uint16_t *q_norm, *k_norm;  // nullptr = no norm
    float eps, norm_offset;
    int q_heads;                      // 0: k and v only
    RopeForm q_form, k_form;
};
cudaError_t launch_rope_append(const RopeAppend &rope, const KvLayer &kv, const LaneTable &lanes_meta, int lanes, cudaStream_t stream);
// Causal GQA attention over the stream's pages, split over the context: split s covers split_tokens tokens, partials are
// merged by a second kernel (max_splits 1: none).  scratch holds [lanes][q_heads][max_splits][head_width + 2] f32.
// Lanes are stream-major: every stream of the batch contributes `lanes_per_stream` consecutive lanes - or, in a ragged
// batch, up to as many, described by a device array of blocks of attention_block_lanes lanes of one stream each.
// scalar_f32: the form for layers whose attention output is quantised to FP8.
struct AttentionBlock {
    int first_lane, lanes;  // of the stream
    int index;              // of the block in the stream
};
int attention_block_lanes(int lanes_per_stream, int q_heads, int kv_heads, int head_width, bool scalar_f32);
bool attention_is_prefill(int lanes_per_stream, int q_heads, int kv_heads);  // the form with 128 query rows per CTA
cudaError_t launch_attention(const uint16_t *q, uint16_t *out, const KvLayer &kv, const LaneTable &lanes_meta,
                             int lanes, int lanes_per_stream, int q_heads, float scale, int split_tokens, int max_splits,
                             float *scratch, bool scalar_f32, cudaStream_t stream, const AttentionBlock *blocks = nullptr, int block_count = 0);

// INT4 multi-branch forms (one launch for q/k/v; gate/up with the SiLU*up epilogue).
cudaError_t launch_linear_int4_multi(const uint16_t *x, const void *prepared, int branches, const uint32_t *const *qweights,
                                     const uint16_t *const *scales, uint16_t *const *ys, const int *ns,
                                     const uint16_t *residual, int lanes, int k, int epilogue, cudaStream_t stream,
                                     int *error_flag = nullptr);
cudaError_t launch_linear_int4_silu_pair(const uint16_t *x, const void *prepared, const uint32_t *gate_q, const uint16_t *gate_s,
                                         const uint32_t *up_q, const uint16_t *up_s, uint16_t *y, int lanes, int n,
                                         int k, cudaStream_t stream, int *error_flag = nullptr);

// ---- streaming output projection for at most 8 lanes (kernels_projection.cu) ----
// logits[lane][row] = scale * x[lane] . table[first_row + row], f32, rows of a slice that starts at a multiple of 16.
// `streamed_table` is the copy launch_projection_table makes of the whole bf16 table (projection_table_bytes bytes).
// With `rounded` set the kernel is a plain bf16 linear instead: rounded[lane][row] = bf16(sum), `logits` and `scale` unused.
size_t projection_table_bytes(int rows, int k);
cudaError_t launch_projection_table(const uint16_t *table, void *out, int rows, int k, cudaStream_t stream);
bool output_projection_supported(int lanes, int k);
cudaError_t launch_output_projection(const uint16_t *x, const void *streamed_table, int first_row, float *logits, int lanes, int rows, int k, float scale,
                                     int grid, int *error_flag, cudaStream_t stream, uint16_t *rounded = nullptr);

// ---- INT4 g128 GEMM on the tcgen05 tensor cores for more than 8 lanes (kernels_int4_gemm.cu) ----
// `prepared` holds the activations in the GEMM's operand form (int4_activation_bytes bytes, 16-byte aligned), written
// by launch_prepare_activations from bf16 [lanes][k].  y and the epilogues as for launch_linear_int4
// (EPILOGUE_F32_SCALED writes f32 * scale); with `silu` the two matrices are a gate/up pair and ys[0] takes
// bf16(silu_bf16(bf16 gate) * bf16 up).  error_flag (optional device word) is set to 3 if a bounded wait expires.
bool linear_int4_gemm_supported(int lanes, int n, int k);
size_t int4_activation_bytes(int lanes, int k);
cudaError_t launch_prepare_activations(const uint16_t *x, void *prepared, int lanes, int k, cudaStream_t stream);
// ... of the RMSNorm of x (the values launch_rms_norm writes, up to the order in which the squares are added), without writing
// them
cudaError_t launch_rms_norm_prepared(const uint16_t *x, const uint16_t *weight, void *prepared, int lanes, int width, float eps, float weight_offset,
                                     cudaStream_t stream);
cudaError_t launch_linear_int4_gemm(const void *prepared, int branches, const uint32_t *const *qweights, const uint16_t *const *scales, void *const *ys,
                                    const int *ns, const uint16_t *residual, int lanes, int k, int epilogue, float scale, bool silu, int *error_flag,
                                    cudaStream_t stream);
// bf16 weights, batches of more than 8 lanes (tcgen05): called by launch_linear_bf16.
bool linear_bf16_gemm_supported(int lanes, int n, int k);
cudaError_t launch_linear_bf16_gemm(const uint16_t *x, const uint16_t *w, void *y, const uint16_t *residual, int lanes, int n, int k, int epilogue,
                                    float scale, int *error_flag, cudaStream_t stream);

// ---- persistent decode stack (kernels_stack.cu) ----
// One cooperative launch runs a whole stack of dense INT4 g128 Llama-style layers for a batch of at most 8 lanes:
// every CTA (one per SM) streams its share of each weight matrix while grid-wide barriers separate the steps of a
// layer.  Weights are read from per-CTA byte streams written at mount (launch_int4_cta_streams).

// How the CTAs of a grid share one matrix of `tiles` 16-row tiles over K = groups * 128 columns.  CTA c owns tiles c,
// c + grid, ...  The rows of a gate/up pair alternate tile by tile (gate, up, gate, ..) and go to the CTAs in runs of
// sixteen, so that the 128 columns of a run, a quantisation group of the down projection, end in one CTA.  A CTA works on
// `slots` of its tiles at a time (one pass): 16 warps as slots / 2 pairs of tiles times `width` groups of K, the warp at
// place i of a pair taking groups i, i + width, ... (no more of them than there are groups: a short K leaves warps without a
// tile rather than have its stream padded).  Step s of a pass is one stage of the CTA's stream: for every present
// tile the 16x128 blocks of groups s * width .. s * width + width - 1 (1 KB of nibbles each, zero beyond `groups`), followed
// by the same blocks' 32-byte scale-pair rows.
struct MatrixSchedule {
    int tiles, groups, run, slots, width, steps, grid;
};
__host__ __device__ inline MatrixSchedule stack_schedule(int tiles, int groups, bool pair, int grid) {
    MatrixSchedule s;
    s.run = pair ? 16 : 1;
    s.tiles = pair ? 2 * tiles : tiles;
    s.groups = groups;
    s.grid = grid;
    const int most = (s.tiles / s.run + grid - 1) / grid * s.run;
    int pairs = 1;
    while (2 * pairs < most && pairs < 8) pairs *= 2;
    s.slots = 2 * pairs;
    s.width = 16 / pairs;
    while (s.width / 2 >= groups) s.width /= 2;
    s.steps = (groups + s.width - 1) / s.width;
    return s;
}
__host__ __device__ inline int stack_cta_tiles(const MatrixSchedule &s, int cta) {
    const int runs = s.tiles / s.run;
    return (runs / s.grid + (cta < runs % s.grid ? 1 : 0)) * s.run;
}
__host__ __device__ inline int stack_cta_tile(const MatrixSchedule &s, int cta, int i) { return (cta + i / s.run * s.grid) * s.run + i % s.run; }
// Bytes of the stream in front of CTA `cta`'s share (every tile costs width * steps units of 1056 bytes).
__host__ __device__ inline size_t stack_cta_offset(const MatrixSchedule &s, int cta) {
    const int runs = s.tiles / s.run, extra = runs % s.grid;
    const size_t tiles_before = (static_cast<size_t>(cta) * (runs / s.grid) + (cta < extra ? cta : extra)) * s.run;
    return tiles_before * s.width * s.steps * 1056;
}
__host__ __device__ inline size_t stack_stream_bytes(const MatrixSchedule &s) { return static_cast<size_t>(s.tiles) * s.width * s.steps * 1056; }

struct StackLayer {
    const uint8_t *qkv, *o, *gate_up, *down;  // per-CTA streams of the four matrix steps
    const uint16_t *input_norm, *post_norm;
    KvLayer kv;
};
struct StackShape {
    int hidden, q_heads, kv_heads, head_width, ffn;
    float eps, norm_offset, attention_scale;
    const uint32_t *rope_table;  // [position][head_width / 2] packed (sin << 16 | cos) bf16
    uint32_t rope_positions;
    int grid;                    // CTAs the streams were written for (the device's SM count at mount)
};
struct StackBuffers {
    uint16_t *hidden;            // [lanes][hidden] residual stream, updated in place
    uint16_t *q;                 // [lanes][q_heads * head_width]
    float *attention_scratch;    // split partials
    uint16_t *attention_out;     // [lanes][q_heads * head_width]
    uint8_t *activation;         // [lanes][ffn] in operand form: stack_activation_bytes(ffn) bytes (see kernels_stack.cu)
    uint8_t *residual;           // what the operand form loses where a group's values lie far apart: stack_residual_bytes(..) bytes
    unsigned int *barrier;       // STACK_BARRIER_WORDS words, zero before the first launch
    int *error_flag;             // set when a bounded wait expires (2: grid barrier or peer, 3: weight pipeline)
    unsigned long long *timing;  // optional [layers][32] nanosecond stamps of CTA 0 (step boundaries), or nullptr
    unsigned int barrier_handicap;  // test hook: arrivals the grid barriers wait for on top of the grid's own (0 in service);
                                    // they can never come, so the first barrier gives up after a short bounded wait
};
constexpr int STACK_BARRIER_WORDS = 1024;  // two barrier words, then the attention arrival counters (kv heads x lane groups)
// Tensor-parallel exchange of the persistent kernel: every rank holds the same residual stream and its shard of
// each layer.  The o and down projections push their f32 partial sums into every peer's inbox - value and exchange
// number in one 8-byte store over NVLink - and the thread that owns an output element waits for the peers' words
// in its own rank's inbox, then adds all shares in rank order.
// Inbox of a rank: [2 parities][STACK_TP_MAX_RANKS sources][8 lanes][hidden] 8-byte words.
constexpr int STACK_TP_MAX_RANKS = 8;
constexpr int STACK_TP_WORD_CONSUMED = 2;                // control word: exchanges done by earlier launches
constexpr unsigned int STACK_TP_SPIN_LIMIT = 1u << 25;   // polls of one inbox word: ranks start their launches a host jitter apart
struct StackTp {
    int rank = 0, size = 1;                            // size 1: no exchange
    float *exchange[STACK_TP_MAX_RANKS] = {};          // every rank's inbox as seen from this GPU (own entry: local memory)
    unsigned long long *counter[STACK_TP_MAX_RANKS] = {};  // every rank's 16 control words
};
constexpr int STACK_TP_WORD_VOTES = 3;                   // control word: arg-max votes taken so far (tensor_parallel_argmax)
constexpr int STACK_TP_VOTE_LANES = 64;                  // lanes one vote can carry
// Behind the 16 control words: the vote area [2 parities][STACK_TP_MAX_RANKS][STACK_TP_VOTE_LANES][2] 8-byte words.
constexpr size_t STACK_TP_CONTROL_BYTES = 16 * sizeof(unsigned long long) + 2 * STACK_TP_MAX_RANKS * STACK_TP_VOTE_LANES * 2 * sizeof(unsigned long long);
inline size_t stack_tp_exchange_floats(int hidden) { return static_cast<size_t>(2) * STACK_TP_MAX_RANKS * 8 * hidden * 2; }

// One source matrix of a stream copy.  rope_head_width > 0 orders the rows of every head so that MMA rows
// r and r + 8 of a tile are the rotary partners (d, d + head_width / 2).
struct RelayoutSegment {
    const uint32_t *qweight;
    const uint16_t *scales;
    int rows;
    int rope_head_width;
};
// Segments share K; their tiles follow one another, or - with `pair` - those of segment 0 and 1 alternate (gate, up).  Every segment's row count must be a multiple of 16.  `rows` of int4_cta_stream_bytes is the sum of
// the segments' rows (one segment's for a pair).
size_t int4_cta_stream_bytes(int rows, int k, bool pair, int grid);
cudaError_t launch_int4_cta_streams(const RelayoutSegment *segments, int count, bool pair, int k, int grid, uint8_t *out,
                                    cudaStream_t stream);
size_t stack_activation_bytes(int ffn);  // of StackBuffers::activation, for any batch
size_t stack_residual_bytes(int ffn, int widest);  // of StackBuffers::residual; `widest`: of the hidden and the query rows
// Whether the stack kernel is built for this shape and batch; *smem_bytes receives its dynamic shared memory.
bool decode_stack_supported(const StackShape &shape, int lanes, size_t *smem_bytes);
cudaError_t launch_decode_stack(const StackLayer *layers_device, int layer_count, const StackShape &shape,
                                const StackBuffers &buffers, const LaneTable &lanes_meta, int lanes, int lanes_per_stream,
                                int split_tokens, int max_splits, cudaStream_t stream, const StackTp *tp_device = nullptr, int tp_size = 1);

// ---- small dense bf16 models (kernels_small_stack.cu) ----
// A whole forward in one launch, a CTA per stream, for layers whose weights fit a CTA's shared memory twice.
struct SmallStackLayer {
    const uint16_t *weights[9];  // q, k, v, o, gate, up, down (bf16 row-major), the weights of the two norms: 16-byte aligned
    KvLayer kv;
};
struct SmallStackShape {
    int hidden, q_heads, kv_heads, head_width, ffn;
    float eps, norm_offset, attention_scale;
    const uint32_t *rope_table;  // [position][head_width / 2] packed (sin << 16 | cos) bf16, halves rotated against one another
    uint32_t rope_positions;
};
struct SmallForward {
    const uint16_t *embedding;  // [vocab][hidden]
    const uint32_t *tokens;     // [lanes]
    float embedding_scale;
    int vocab;
    // a draft's input adapter (nullptr: none): [hidden][2 hidden], the norms of the embedding and of hidden_in
    const uint16_t *adapter, *adapter_norms[2], *hidden_in;
    float adapter_eps, adapter_offset;
    int embedding_first;  // the embedding's norm takes the first columns
    // the final norm's rows [lanes][hidden] (nullptr: ends behind the layers), the logits [lanes][vocab] (nullptr: none), the
    // arg-max records (nullptr: none)
    const uint16_t *final_norm;
    float final_eps, final_offset;
    uint16_t *normalized;
    const uint16_t *table;
    float logits_scale;
    float *logits;
    uint32_t *records;
};
constexpr int SMALL_STACK_MAX_LANES = 32;  // per stream
constexpr int SMALL_STACK_MAX_VOCAB = 1024;
bool small_stack_supported(const SmallStackShape &shape, int vocab, uint32_t capacity, int lanes_per_stream);
cudaError_t launch_small_stack(const SmallStackLayer *layers_device, int layer_count, const SmallStackShape &shape, const SmallForward &forward, const LaneTable &lanes_meta,
                               uint32_t capacity, int streams, int lanes_per_stream, int *error_flag, cudaStream_t stream);

// Tensor-parallel row-parallel linears: out = bf16(bf16(sum) + residual) (or bf16(sum) without residual) from the
// all-reduced f32 sums [count].
cudaError_t launch_round_add(const float *sums, const uint16_t *residual, uint16_t *out, size_t count, cudaStream_t stream);

// ---- glue of the speculative cycle (all tiny) ----
// dst[i] = src[index[i]] for rows of `width` bf16.
// Times (nanoseconds, device clock) and the status of a speculative cycle.
enum CycleMark { CYCLE_BEGIN, CYCLE_DRAFTED, CYCLE_VERIFIED, CYCLE_END, CYCLE_STATUS, CYCLE_MARKS };
cudaError_t launch_begin_cycle(const uint32_t *host_state, uint32_t *state, int state_words, const uint16_t *pending, const int32_t *host_slots, uint16_t *gathered, int rows,
                               uint16_t *backup, int max_streams, int hidden, unsigned long long *marks, cudaStream_t stream);
cudaError_t launch_finish_cycle(const uint32_t *results, int words, unsigned long long *marks, const int *error_word, uint32_t *host_results, cudaStream_t stream);
cudaError_t launch_gather_rows(const uint16_t *src, const int32_t *index, uint16_t *dst, int rows, int width,
                               cudaStream_t stream);
// Hidden inputs of the draft catch-up: lane (s, 0) takes pending[slot[s]], lane (s, i>0) takes normalized (s, i-1).
cudaError_t launch_shift_hidden(const uint16_t *pending, const int32_t *slots, const uint16_t *normalized,
                                uint16_t *dst, int streams, int lanes_per_stream, int hidden, unsigned long long *marks, cudaStream_t stream);
// The same for lanes of any number per stream (neighbouring lanes of one slot are one stream's), and the way back: the
// normalised frame of every stream's last lane becomes its pending hidden state.
cudaError_t launch_shift_hidden_lanes(const uint16_t *pending, const int32_t *slots, const uint16_t *normalized, uint16_t *dst, int lanes, int hidden,
                                      cudaStream_t stream);
cudaError_t launch_commit_hidden(const uint16_t *normalized, const int32_t *slots, uint16_t *pending, int lanes, int hidden, cudaStream_t stream);
// After draft step `step`: token = forced[s][step] unless it is 0xffffffff, else the sampled record; written to
// next_tokens[s] and verify_tokens[s][step + 1].
cudaError_t launch_draft_select(const uint32_t *records, const uint32_t *forced, int step, int streams, int drafts,
                                uint32_t *next_tokens, uint32_t *verify_tokens, unsigned long long *marks, cudaStream_t stream);
// Longest-matching-prefix acceptance + stop truncation (speculative_decode.rs:54-105) per stream, then
// pending[slot[s]] = normalized lane (s, committed-1).  out row = {accepted, committed, emitted_count, 0,
// emitted[drafts+1], targets[drafts+1]}.  own_drafts[s] <= drafts: how many of the drafts count for the stream.
cudaError_t launch_accept(const uint32_t *verify_tokens, const uint32_t *target_records, const uint32_t *stop_tokens,
                          const int32_t *stop_counts, const int32_t *own_drafts, int max_stop, int streams, int drafts, uint32_t *out,
                          const uint16_t *normalized, uint16_t *pending, const int32_t *slots, int hidden,
                          cudaStream_t stream);

// Vocabulary-parallel greedy sampling under tensor parallelism: every rank has taken the arg-max of its own slice of
// the vocabulary (records_local: {token within the slice, logit bits, ..} per lane, as launch_argmax writes them);
// the ranks push (logit, global token), tagged with the vote number, into each other's vote areas over NVLink, wait
// (bounded) for all of them and all pick the same winner - highest logit, ties to the lowest token id.  One block.
// The vote number lives on the device (control word STACK_TP_WORD_VOTES), so the launch can be replayed from a graph.
cudaError_t launch_tensor_parallel_argmax(const uint32_t *records_local, uint32_t first_token, uint32_t *records, int lanes, const StackTp *tp_device,
                                          int *error_flag, cudaStream_t stream);

// Greedy arg-max (ties -> lowest id); record = {token, logit bits, 0, 0} per lane.
// `scratch` holds argmax_scratch_bytes(lanes) bytes of per-chunk partial winners.
size_t argmax_scratch_bytes(int lanes);
cudaError_t launch_argmax(const float *logits, uint32_t *records, int lanes, int vocab, void *scratch, cudaStream_t stream);
// The same with the partial winners in a fixed device array of the library (no allocation anywhere); at most
// argmax_static_max_lanes() lanes, one call at a time per device.
int argmax_static_max_lanes();
cudaError_t launch_argmax_static(const float *logits, uint32_t *records, int lanes, int vocab, cudaStream_t stream);

// ---- seeded temperature / top-k / top-p / min-p sampler (kernels_sampler.cu) ----
constexpr int SAMPLER_MAX_TOP_K = 64;
struct SamplerParams {   // one per stream slot
    uint32_t method;     // 0 greedy (arg-max, record flags 0), 1 temperature_top_k_top_p
    uint32_t top_k;      // 1..SAMPLER_MAX_TOP_K
    uint32_t seed;
    float temperature, top_p, min_p;
};
size_t sampler_scratch_bytes(int lanes);
// One record {token, logit bits, sampled flag, 0} per lane; lane l uses table[slots[l]] (slot 0 when slots is
// NULL) and the uniform of stream tick ticks[l].
cudaError_t launch_sample(const float *logits, uint32_t *records, int lanes, int vocab, const SamplerParams *table, const int32_t *slots,
                          const uint32_t *ticks, void *scratch, cudaStream_t stream);

}  // namespace nerve
