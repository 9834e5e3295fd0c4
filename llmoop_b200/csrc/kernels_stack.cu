// Persistent decode stack: one cooperative launch runs every layer of a dense INT4 g128 Llama-style stack
// (rms_norm, q/k/v, RoPE, KV append, attention, o + residual, rms_norm, gate/up + SiLU, down + residual:
// the kernel list of one reference layer component, runtime-rs/shaders/*.comp.template) for a batch of at most
// 8 lanes - the verify batch and the draft / single-tick steps of the speculative decode cycle.
//
// Why one launch: at these batch sizes a layer is ~112 MB of weights (~17 us of HBM time) cut into a dozen
// dependent steps; as separate kernels every step pays a launch, a pipeline fill and a drain.  Here one CTA per
// SM stays resident and the weight stream never stops for a step boundary:
//
//  * weights: at mount every matrix is rewritten as one contiguous byte stream per CTA, in exactly the order the
//    CTA consumes it (see stack_schedule in kernels.cuh).  A stream is a sequence of stages; a stage is up to two
//    16x128 blocks of packed nibbles (1 KB each) and their 32 bytes of scales for each of 16 warps.
//  * a producer thread (warp 16) walks the CTA's stages of all matrices of all layers and brings them into a ring
//    in shared memory with one bulk asynchronous copy per stage (mbarrier transaction counts; no cluster forms),
//    as far ahead as the ring allows - through the grid barriers, the attention step and the epilogues.
//  * 16 consumer warps: a warp multiplies two tiles of 16 rows with every width-th group (128 columns) of K, so a
//    matrix costs one cross-warp reduction and one epilogue pass per CTA instead of one per tile.  The products are
//    integers: weights as signed bytes, activations as four signed bytes each, mma.sync m16n8k32 with exact 32-bit
//    sums (see "matrix blocks"); the group scale multiplies the group's sum in f32 as in
//    linear_int4_ct.comp.template:80-150.
//  * activations: the inputs of q/k/v and gate/up (rms_norm_bf16.comp.template:49-72) and of o are brought into
//    operand form in shared memory by every CTA; the inputs of down leave the SiLU epilogue in operand form (the
//    eight tiles of a gate/up pass are one quantisation group of down's columns) and ride a ring of their own, one
//    slice per step, once the grid barrier in front of the step has opened.
//  * attention: a team of four warps per (kv head, 64-token split, lane group) on the tensor cores (query rows in
//    shared memory, K and V rows in registers, all loads of an item requested before its arithmetic); the team that
//    completes a kv head's last split queues the merge, and after its items the CTA's sixteen warps merge one
//    (lane, q head) row each - no grid barrier between the splits and their merge.  Lane groups of more than 32
//    splits are merged in two levels (ranges of 32 splits spread over every warp of the grid, then the ranges of a
//    row by one warp), with a grid barrier before each level.
//  * registers: everything that outlives a step is kept in shared memory (StackShared), the steps are inlined into one
//    loop, and the consumers take the registers that the producers hand back.  Half the time of an earlier form of this
//    kernel was spills: with 227 KB of an SM's memory given to the ring the first-level cache holds about fifty bytes per
//    thread, and what a function saved around a call came back from L2.
//  * tensor parallelism (the EXCHANGE instances): o and down push their f32 partial sums, tagged with the exchange
//    number in the same 8-byte store, into every peer's inbox over NVLink; the owner of an output element waits
//    for the peers' words in its own memory and adds them in rank order.  No barrier crosses the link.
//
// Every wait is bounded: when a bound expires the kernel sets the error word and leaves.
#include <cstddef>
#include <cstdlib>

#include "common.cuh"
#include "kernels.cuh"

namespace nerve {

namespace {

constexpr int CONSUMER_WARPS = 16;
constexpr int CONSUMER_THREADS = CONSUMER_WARPS * 32;
constexpr int STACK_THREADS = CONSUMER_THREADS + 128;  // + the producer warps (registers are allotted four warps at a time)
// Registers: a launch gives 96 to each of the 640 threads; the producers hand 64 of theirs back, the consumers take 16 more.
constexpr int PRODUCER_REGISTERS = 32, CONSUMER_REGISTERS = 112;
static_assert(CONSUMER_THREADS * CONSUMER_REGISTERS + 128 * PRODUCER_REGISTERS <= STACK_THREADS * 96, "the consumers' registers come out of the producers'");
constexpr int UNIT_BYTES = 1024;                      // packed nibbles of a 16x128 block
constexpr int UNIT_SCALE_BYTES = 32;                  // its eight scale pairs
constexpr int UNIT_TOTAL = UNIT_BYTES + UNIT_SCALE_BYTES;
constexpr int STAGE_BYTES = 2 * CONSUMER_WARPS * UNIT_TOTAL;  // a step of a pass: two blocks per consumer warp (33 792 bytes)
constexpr int MAX_STAGES = 16;
constexpr uint32_t EMPTY = 8 * MAX_STAGES, SLICE_FULL = 16 * MAX_STAGES, SLICE_EMPTY = 24 * MAX_STAGES;  // barrier arrays, from a slot's `full`
// Activations in operand form (see stage_rows): two halves and eight factors per group of 128 columns.
__host__ __device__ constexpr uint32_t operand_half_bytes(int lanes) { return static_cast<uint32_t>(lanes) * 256u; }
__host__ __device__ constexpr uint32_t operand_group_bytes(int lanes) { return 2u * operand_half_bytes(lanes) + 32u; }
constexpr uint32_t PRODUCT_BYTES = 8 * 128 * sizeof(float);  // a group of SiLU products of every lane, before it takes operand form
constexpr unsigned int BARRIER_SPIN_LIMIT = 1u << 20;
constexpr unsigned int PIPE_SPIN_LIMIT = 1u << 18;  // attempts of about 20 us each at most
constexpr unsigned int OPEN_SPIN_LIMIT = 1u << 28;  // polls of the barrier count by the slice producer: it has to outlast the consumers' own waits
constexpr int BARRIERS_PER_LAYER = 5;  // after q/k/v, attention, o, gate/up, down
constexpr int ARRIVAL_WORDS_OFFSET = 16;  // attention arrival counters sit behind the two barrier words

// ------------------------------------------------------------------------------------------ per-CTA streams

struct RelayoutArgs {
    RelayoutSegment segment[3];
    int first_tile[4];
    int count;
    int pair;
    int k;
    MatrixSchedule schedule;
};

// Block (step, cta) writes one step of one CTA's stream: the present tiles' blocks, then their scale pairs.
__global__ void int4_cta_stream_kernel(const RelayoutArgs args, uint8_t *__restrict__ out) {
    const MatrixSchedule &s = args.schedule;
    const int cta = blockIdx.y;
    const int here = stack_cta_tiles(s, cta);
    const int pass = blockIdx.x / s.steps, step = blockIdx.x % s.steps;
    int present = here - pass * s.slots;
    if (present <= 0) return;
    if (present > s.slots) present = s.slots;
    const int groups = args.k >> 7;
    uint8_t *base = out + stack_cta_offset(s, cta) + static_cast<size_t>(pass) * s.slots * s.width * s.steps * UNIT_TOTAL +
                    static_cast<size_t>(step) * present * s.width * UNIT_TOTAL;
    uint4 *weights_out = reinterpret_cast<uint4 *>(base);
    uint32_t *scales_out = reinterpret_cast<uint32_t *>(base + static_cast<size_t>(present) * s.width * UNIT_BYTES);
    auto locate = [&](int unit_in_step, int &group, int &which, int &local_tile) {
        const int slot = unit_in_step / s.width;
        group = step * s.width + unit_in_step % s.width;
        if (group >= s.groups) return false;  // padding of a ragged last step: zeros under zero scales
        const int tile = stack_cta_tile(s, cta, pass * s.slots + slot);
        which = 0;
        local_tile = tile;
        if (args.pair) {  // gate and up rows alternate
            which = tile & 1;
            local_tile = tile >> 1;
        } else {
            while (which + 1 < args.count && tile >= args.first_tile[which + 1]) which++;
            local_tile = tile - args.first_tile[which];
        }
        return true;
    };
    auto source_row = [&](const RelayoutSegment &segment, int local_tile, int mma_row) {
        if (segment.rope_head_width > 0) {
            const int tiles_per_head = segment.rope_head_width / 16;
            const int head = local_tile / tiles_per_head, th = local_tile % tiles_per_head;
            const int d = mma_row < 8 ? 8 * th + mma_row : segment.rope_head_width / 2 + 8 * th + (mma_row - 8);
            return head * segment.rope_head_width + d;
        }
        return local_tile * 16 + mma_row;
    };
    const int units = present * s.width;
    for (int index = threadIdx.x; index < units * 64; index += blockDim.x) {
        const int unit_in_step = index >> 6, half = (index >> 5) & 1, lane = index & 31;
        const int g = lane >> 2, j = lane & 3;
        int group = 0, which = 0, local_tile = 0;
        uint4 value = make_uint4(0, 0, 0, 0);
        if (locate(unit_in_step, group, which, local_tile)) {
            const RelayoutSegment &segment = args.segment[which];
            const int row = source_row(segment, local_tile, g + 8 * half);
            value = *reinterpret_cast<const uint4 *>(segment.qweight + static_cast<size_t>(row) * (args.k >> 3) + group * 16 + j * 4);
            value.x ^= 0x88888888u, value.y ^= 0x88888888u, value.z ^= 0x88888888u, value.w ^= 0x88888888u;  // q -> q - 8 in two's complement
        }
        weights_out[index] = value;
    }
    for (int index = threadIdx.x; index < units * 8; index += blockDim.x) {
        const int unit_in_step = index >> 3, g = index & 7;
        int group = 0, which = 0, local_tile = 0;
        uint32_t value = 0;
        if (locate(unit_in_step, group, which, local_tile)) {
            const RelayoutSegment &segment = args.segment[which];
            const uint32_t low = segment.scales[static_cast<size_t>(source_row(segment, local_tile, g)) * groups + group];
            const uint32_t high = segment.scales[static_cast<size_t>(source_row(segment, local_tile, g + 8)) * groups + group];
            value = low | (high << 16);
        }
        scales_out[index] = value;
    }
}

// ------------------------------------------------------------------------------------------ small helpers

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// 16x32 signed bytes times 32x8 signed bytes, exact sums.  D and C are different operands: C starts a chain.
__device__ __forceinline__ void mma_s8_16832(int32_t (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int32_t c0,
                                             int32_t c1, int32_t c2, int32_t c3) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};\n"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}

// Pairs of f32 in one register pair (two IEEE operations per instruction).
__device__ __forceinline__ unsigned long long pair_of(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ unsigned long long pair_add(unsigned long long a, unsigned long long b) {
    unsigned long long v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ unsigned long long pair_multiply(unsigned long long a, unsigned long long b) {
    unsigned long long v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ unsigned long long pair_fma(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}

__device__ __forceinline__ uint32_t load_acquire(const unsigned int *address) {
    uint32_t value;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(value) : "l"(address) : "memory");
    return value;
}

__device__ __forceinline__ void cta_sync() { asm volatile("bar.sync 1, 512;" ::: "memory"); }  // of the consumers
__device__ __forceinline__ void team_barrier(int barrier_id) { asm volatile("bar.sync %0, 128;" ::"r"(barrier_id) : "memory"); }

// ---- mbarrier / bulk copy (shared-space addresses)
__device__ __forceinline__ void mbarrier_init(uint32_t address, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(address), "r"(count) : "memory");
}
__device__ __forceinline__ void mbarrier_arrive(uint32_t address) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(address) : "memory");
}
__device__ __forceinline__ void mbarrier_arrive_expect(uint32_t address, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(address), "r"(bytes) : "memory");
}
// One attempt at waiting for the phase of the given parity: the thread is suspended by the hardware until the
// phase completes or about `MBARRIER_SUSPEND_NS` have passed, so a waiting warp issues almost nothing.
constexpr uint32_t MBARRIER_SUSPEND_NS = 20000;
__device__ __forceinline__ bool mbarrier_test(uint32_t address, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(done)
        : "r"(address), "r"(parity), "r"(MBARRIER_SUSPEND_NS)
        : "memory");
    return done != 0;
}
// global -> this CTA's shared memory, completion counted in bytes on `barrier`
__device__ __forceinline__ void bulk_load(uint32_t destination, const void *source, uint32_t bytes, uint32_t barrier) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(destination),
                 "l"(__cvta_generic_to_global(source)), "r"(bytes), "r"(barrier)
                 : "memory");
}
__device__ __forceinline__ uint32_t shared_load_acquire(uint32_t address) {
    uint32_t value;
    asm volatile("ld.acquire.cta.shared::cta.u32 %0, [%1];" : "=r"(value) : "r"(address) : "memory");
    return value;
}
__device__ __forceinline__ void shared_store_release(uint32_t address, uint32_t value) {
    asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(address), "r"(value) : "memory");
}
// Shared-memory loads by shared-space address (kept in program order behind the waits that make their data valid).
template <int OFFSET>
__device__ __forceinline__ uint4 shared_load16(uint32_t address) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4+%5];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(address), "n"(OFFSET) : "memory");
    return v;
}
// ------------------------------------------------------------------------------------------ the CTA's view of a matrix

struct PhaseInfo {
    int tiles_here;       // 16-row tiles of this CTA, see stack_cta_tile
    int passes;           // rounds of `slots` tiles
    int slots, width, steps, groups;
    int width_log2;       // width is a power of two
    int window;           // steps whose activations are staged at a time
    uint32_t cta_offset;  // bytes from the matrix's stream to this CTA's share
};

struct StackArgs {
    const StackLayer *layers;
    int layer_count;
    StackShape shape;
    StackBuffers buffers;
    LaneTable lanes_meta;
    int lanes, lanes_per_stream, max_splits;
    int stages;
    int slice_slots, slice_bytes;        // ring of activation slices (down, one step each) inside the scratch area
    uint32_t scratch_bytes;
    const StackTp *tp;  // device copy of the exchange description, or nullptr (single GPU)
    int tp_size;
};

// Merges a CTA can be left with in a layer: at most one per work item, of at most (1024 - 16) arrival counters x 32 splits
// on 148 CTAs.
constexpr int ATTENTION_MERGE_LIST = 256;
struct AttentionItem {
    int16_t kv_head, split;     // the kv head, the context split
    int16_t lane0, lanes;       // the query lanes
    int32_t slot, arrival;      // the stream's slot; kv_head * group_slots + lane group, the split counter
    int32_t count, splits;      // tokens of the split (0: nothing to do); splits of the whole context
    uint32_t first_tick, ring_base;  // of its first token
};
// What a warp does in a pass of a matrix: two tiles of 16 rows, every width-th group of K.
struct WarpBlocks {
    uint32_t unit, scales;      // its first block inside a stage, and on to that block's scales
    uint32_t next_tile;         // on to the second tile's block (its scales are 1 / 32 of that further)
    uint32_t x;                 // its group of the first step: from the staged rows, inside the slice of a step
    uint32_t x_step;            // on to the group of the next step; slices: to the next slot
    int steps;                  // steps that hold a group of the warp (0 if it has no tile)
    int tiles;                  // 1 or 2
};
struct OperandPlace {  // where a thread's B fragments are inside a group: in the first half, and the same with the neighbour's term
    uint32_t first, second, half, factor;
};

// What the CTA's threads share, at the start of its shared memory; the scratch area (staged rows and SiLU products /
// attention teams / slices of down) and the ring follow.  All state that outlives a step is kept
// here, not in registers: a value that is live across the steps' functions is spilled, and with 227 KB of the SM's memory
// given to the ring the spills miss the first-level cache (a version with 0.5 KB of them took twice the time).
struct StackShared {
    uint64_t full[MAX_STAGES], empty[MAX_STAGES], slice_full[MAX_STAGES], slice_empty[MAX_STAGES];
    StackArgs a;
    PhaseInfo info[4];
    StackLayer layer[2];        // the current layer's description (layer & 1) and the next one's, copied ahead of their use
    uint32_t scratch, ring;     // offsets from the start
    uint32_t products;          // where the SiLU products of a pass of gate/up go, f32 [lane][128]: an offset
    uint32_t place;             // where the consumers stand in the two rings (pack_place)
    uint32_t open_word;         // counted grid barriers passed (read by the producer of slices)
    uint32_t barrier_target;    // arrivals expected at the grid barriers so far
    uint32_t barrier_limit;     // polls
    WarpBlocks blocks[4][CONSUMER_WARPS];  // of the first pass of each matrix step
    OperandPlace operand_place[32];     // by lane of the warp
    uint32_t output[CONSUMER_THREADS];     // o and down: the thread's first output in the residual stream (see matrix_step)
    uint32_t exchanges;         // tensor-parallel exchanges of earlier launches
    // lanes
    uint32_t tick[8];
    int32_t slot[8];
    uint64_t kv_row[8];         // element offset of the lane's K row (kv head 0) in a layer's pool, ~0 if it has none
    uint32_t rope[8 * 64];      // [lane][HD / 2] rotary factors of the lanes' positions
    // attention: for each team the KV rows of its first work item (the block table is shared by all layers, so the rows
    // of a (split, lane group) are the same in every layer's pool)
    int32_t group_slots;        // lane groups of all streams
    AttentionItem item[4];
    AttentionItem later_item[2][4];  // taken in turn: an item without tokens has no barrier behind the reading of its count
    int32_t merge_count;        // (kv head, lane group) pairs whose last split this CTA's teams completed in this layer ...
    uint16_t merge_list[ATTENTION_MERGE_LIST];  // ... and which: kv_head * group_slots + group_slot
    uint32_t row_base[4][64];   // offset (in rows of HD elements) of token t's K row of kv head 0 in a layer's pool
    float norm_partial[4 * CONSUMER_WARPS];
    alignas(16) float reduce[CONSUMER_WARPS][2][128];  // the warps' partial sums: [warp][tile of its pair][row][lane]
};
extern __shared__ __align__(128) uint8_t smem_raw[];
__device__ __forceinline__ StackShared &shared() { return *reinterpret_cast<StackShared *>(smem_raw); }
__device__ __forceinline__ uint32_t shared_address(const void *object) { return static_cast<uint32_t>(__cvta_generic_to_shared(object)); }
__device__ __forceinline__ uint4 smem16(uint32_t offset) { return *reinterpret_cast<const uint4 *>(smem_raw + offset); }
__device__ __forceinline__ uint32_t smem4(uint32_t offset) { return *reinterpret_cast<const uint32_t *>(smem_raw + offset); }
// The thread's number, read anew: what is derived from it is not kept across the steps of a layer.
__device__ __forceinline__ int thread_now() {
    int thread;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(thread));
    return thread;
}

// All CTAs of the (cooperative, co-resident) grid meet here; only the consumer warps take part.  A wait that does not
// complete within the spin limit sets the error flag and lets the CTA go on (its results are then garbage, the host sees
// the flag); once the flag is up nobody waits any more.  Counted barriers are those the producer of slices waits for.
__device__ __forceinline__ void grid_meet(bool counted) {
    cta_sync();
    if (threadIdx.x == 0) {
        StackShared &sh = shared();
        unsigned int *counter = sh.a.buffers.barrier;
        int *error_flag = sh.a.buffers.error_flag;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");  // covers the CTA's writes before the barrier above
        const unsigned int target = sh.barrier_target + gridDim.x, limit = sh.barrier_limit;
        sh.barrier_target = target;
        unsigned int spins = 0;
        while (load_acquire(counter) < target) {
            if (++spins > limit) {
                atomicExch(error_flag, 2);
                break;
            }
            if ((spins & 63u) == 0 && *reinterpret_cast<volatile int *>(error_flag) != 0) break;
        }
        if (counted) shared_store_release(shared_address(&sh.open_word), sh.open_word + 1u);
    }
    cta_sync();
}
__device__ __forceinline__ void stamp(int layer, int index) {  // step times of CTA 0, for tests and profiles
    unsigned long long *timing = shared().a.buffers.timing;
    if (timing != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        timing[layer * 32 + index] = now;
    }
}

__device__ __forceinline__ const uint8_t *layer_stream(const StackLayer &layer, int phase) {
    return phase == 0 ? layer.qkv : (phase == 1 ? layer.o : (phase == 2 ? layer.gate_up : layer.down));
}

__device__ __forceinline__ int stage_present(const PhaseInfo &pi, int pass) {
    const int left = pi.tiles_here - pass * pi.slots;
    return left < pi.slots ? left : pi.slots;
}

// ------------------------------------------------------------------------------------------ producers
// Two single threads (lane 0 of warps 16 and 17) walk the CTA's sequence - for every layer the four matrices, for
// every matrix its passes and steps - each on its own: one requests the weights, a step of a pass as one
// stage, the other the activation slice of every step of down (once the grid barrier in front of it has
// opened).  A slot is free when the consumer warps have released its previous use (the `empty` barrier); its
// `full` barrier completes with the producer's arrival plus the bytes of the copy.

struct RingPosition {
    uint32_t slot, parity;  // parity of the `empty` phase that frees the slot for the next use
};
__device__ __forceinline__ void ring_advance(RingPosition &position, uint32_t stages) {
    if (++position.slot == stages) {
        position.slot = 0;
        position.parity ^= 1u;
    }
}
// false: gave up (the error flag is set, or was set by somebody else)
__device__ __forceinline__ bool wait_slot_free(uint32_t empty_address, const RingPosition &position, int *error_flag) {
    unsigned int spins = 0;
    while (!mbarrier_test(empty_address + position.slot * 8, position.parity)) {
        if (++spins > PIPE_SPIN_LIMIT) {
            atomicExch(error_flag, 3);
            return false;
        }
        if ((spins & 255u) == 0 && *reinterpret_cast<volatile int *>(error_flag) != 0) return false;
    }
    return true;
}
// After giving up: let the copies that are still in flight land before the CTA's shared memory goes away.
__device__ __forceinline__ void linger() {
    for (int i = 0; i < 64; i++) __nanosleep(1000);
}

__device__ __forceinline__ void produce_weights() {
    const StackShared &sh = shared();
    int *error_flag = sh.a.buffers.error_flag;
    const uint32_t stages = static_cast<uint32_t>(sh.a.stages), ring = shared_address(smem_raw + sh.ring), empty = shared_address(sh.empty), full = shared_address(sh.full);
    RingPosition position{0u, 1u};
    for (int layer = 0; layer < sh.a.layer_count; layer++) {
        const StackLayer *spec = sh.a.layers + layer;
        for (int phase = 0; phase < 4; phase++) {
            const PhaseInfo pi = sh.info[phase];
            if (pi.passes == 0) continue;
            const uint8_t *source = layer_stream(*spec, phase) + pi.cta_offset;
            for (int pass = 0; pass < pi.passes; pass++) {
                const uint32_t bytes = static_cast<uint32_t>(stage_present(pi, pass) * pi.width * UNIT_TOTAL);
                for (int step = 0; step < pi.steps; step++) {
                    if (!wait_slot_free(empty, position, error_flag)) return linger();
                    mbarrier_arrive_expect(full + position.slot * 8, bytes);
                    bulk_load(ring + position.slot * static_cast<uint32_t>(STAGE_BYTES), source, bytes, full + position.slot * 8);
                    source += bytes;
                    ring_advance(position, stages);
                }
            }
        }
    }
}

__device__ __forceinline__ void produce_activations() {
    const StackShared &sh = shared();
    int *error_flag = sh.a.buffers.error_flag;
    const uint32_t slots = static_cast<uint32_t>(sh.a.slice_slots), slices = shared_address(smem_raw + sh.scratch), empty = shared_address(sh.slice_empty),
                   full = shared_address(sh.slice_full), slice_bytes = static_cast<uint32_t>(sh.a.slice_bytes), group_bytes = operand_group_bytes(sh.a.lanes);
    RingPosition position{0u, 1u};
    const PhaseInfo pi = sh.info[3];
    if (pi.passes == 0) return;
    for (int layer = 0; layer < sh.a.layer_count; layer++) {
        // the slices were written by other CTAs with ordinary stores before the grid barrier counted here; the
        // scratch area they land in is free once this CTA's consumers have passed that barrier, too
        const uint32_t needed = static_cast<uint32_t>(layer * BARRIERS_PER_LAYER + 4);
        unsigned int spins = 0;
        while (shared_load_acquire(shared_address(&sh.open_word)) < needed) {
            if (++spins > OPEN_SPIN_LIMIT) {
                atomicExch(error_flag, 3);
                return linger();
            }
            if ((spins & 255u) == 0 && *reinterpret_cast<volatile int *>(error_flag) != 0) return linger();
            __nanosleep(20);
        }
        asm volatile("fence.proxy.async;" ::: "memory");  // ... and the copy engine reads them
        for (int pass = 0; pass < pi.passes; pass++) {
            const uint8_t *source = sh.a.buffers.activation;
            for (int first_group = 0; first_group < pi.groups; first_group += pi.width) {
                if (!wait_slot_free(empty, position, error_flag)) return linger();
                const int groups = pi.groups - first_group < pi.width ? pi.groups - first_group : pi.width;
                const uint32_t bytes = static_cast<uint32_t>(groups) * group_bytes;
                mbarrier_arrive_expect(full + position.slot * 8, bytes);
                bulk_load(slices + position.slot * slice_bytes, source, bytes, full + position.slot * 8);
                source += bytes;
                ring_advance(position, slots);
            }
        }
    }
}

// Waits (bounded) until a barrier's phase of the given parity is complete.
__device__ __forceinline__ void wait_barrier(uint32_t barrier, uint32_t parity) {
    unsigned int spins = 0;
    while (!mbarrier_test(barrier, parity)) {
        int *error_flag = shared().a.buffers.error_flag;
        if (++spins > PIPE_SPIN_LIMIT) {
            atomicExch(error_flag, 3);
            break;
        }
        if ((spins & 255u) == 0 && *reinterpret_cast<volatile int *>(error_flag) != 0) break;
    }
}
// ------------------------------------------------------------------------------------------ activation staging

// The operand form of activations.  A group (128 columns) of a lane is held as whole numbers X of 31 bits over one
// power of two - x = X 2^(e - 29), e the exponent of the largest magnitude of the group (of the warp's two groups where
// rows are staged) - and X as four signed bytes, X = t0 2^24 + t1 2^16 + t2 2^8 + t3: the group's products with the four-bit
// weights then add up exactly in 32-bit integers, whatever their order, and what f32 rounds is the group's sum, as in
// linear_int4_ct.comp.template:80-150.  A bf16 value down to 2^-22 of that largest is carried exactly, a smaller one to
// 2^(e - 30), which is no further off than an fp16 number (2^-25) while the largest is below 64.  A group with a larger
// one that has values it cannot hold keeps what they lost, X' 2^(e - 59), in the same form in global memory
// (StackBuffers::residual); its factor and its digits are negative, and add_residuals multiplies the rest.  (With three
// bytes the rows without a weight on a large column were off by 1e-2 of a group's sum where it was 10000 beside N(0, 1)
// products times 0.05.  The fourth byte is free up to four lanes - the MMA's columns were there - and costs a fourth column
// tile from five on.)
//
// A group that holds a NaN has a NaN for its factor, so that all its sums are.  One with infinities has zeros, a factor of -0 and
// +-1 for them in the residual, whose factor is an infinity then: a row whose weight there is not 0 gets an infinity, any
// other a NaN, as from the products (of several infinities in one group the sum of the weights decides).
//
// A group takes operand_group_bytes(lanes) bytes: [half h][lane][term t][j] pieces of 16 bytes (the B fragments of
// MMAs 2h and 2h + 1 for thread column j: the digits of the eight columns of word 4j + 2h, even columns first, then
// those of word 4j + 2h + 1; where lane + h is odd the terms are in the order 1, 0, 3, 2, so that a term of two neighbours falls
// into different banks), then one f32 factor per lane, what a unit of t3 times a weight of one is worth.
__device__ __forceinline__ uint32_t operand_word_offset(int word, int m, int lanes) {  // of the lane's terms
    return static_cast<uint32_t>((word >> 1) & 1) * operand_half_bytes(lanes) + static_cast<uint32_t>(m) * 256u + static_cast<uint32_t>(word >> 2) * 16u +
           static_cast<uint32_t>(word & 1) * 8u;
}
__host__ __device__ constexpr uint32_t term_offset(int term, int lane_and_half) { return static_cast<uint32_t>(term ^ (lane_and_half & 1)) * 64u; }
// From the exponent field of a group's largest magnitude: the factor onto X / 2^8, and the group's factor (2^-4 of a unit since
// the MMA sees sixteen times the weights); of finite groups.
__device__ __forceinline__ float operand_scale(uint32_t exponent) { return __uint_as_float((275u - (exponent < 40u ? 40u : exponent)) << 23); }
__device__ __forceinline__ float operand_factor(uint32_t exponent) { return __uint_as_float(((exponent < 40u ? 40u : exponent) - 33u) << 23); }
__device__ __forceinline__ bool operand_may_lose(uint32_t exponent) { return exponent >= 133u; }  // (133: 64; 255: not finite)
constexpr float RESIDUAL_SCALE = 4194304.0f, RESIDUAL_UNIT = 0x1p-30f;  // what is left in units of t3, onto X' / 2^8; the factors' ratio
__device__ __forceinline__ float special_factor(bool nan, bool infinite) { return __uint_as_float(nan ? 0x7fc00000u : (infinite ? 0x80000000u : 0u)); }
__device__ __forceinline__ float residual_factor(float factor) {
    const uint32_t bits = __float_as_uint(factor);
    return bits >> 31 == 0 ? 0.0f : (bits == 0x80000000u ? INFINITY : -factor * RESIDUAL_UNIT);  // (NaN is positive)
}
// A pair of values as X + 0x00808080: 2^7 in front of the lower digits makes their bytes unsigned, so that no digit borrows from
// the next.  f32 rounds to whole numbers where it is 1.5 * 2^23 + X; it does so for X / 2^8, then for the 2^8 of what is left.
// (Additions of integers are multiply-adds by an opaque one: they leave the half-rate integer pipe to the permutes.)
struct DigitConstants {  // made where they are used: the compiler would keep them in registers through the whole layer
    uint32_t one, byte, digits;
    unsigned long long bias, minus, byte_pair;  // pairs
};
__device__ __forceinline__ DigitConstants digit_constants() {
    DigitConstants c;
    asm volatile("mov.b32 %0, 1;" : "=r"(c.one));
    asm volatile("mov.b32 %0, 256;" : "=r"(c.byte));
    asm volatile("mov.b32 %0, 0x75408080;" : "=r"(c.digits));  // 0x00808080 - 2^8 0x4B400000 - 0x4B400000
    asm volatile("mov.b64 %0, 0x4B4000004B400000;" : "=l"(c.bias));
    asm volatile("mov.b64 %0, 0xBF800000BF800000;" : "=l"(c.minus));
    asm volatile("mov.b64 %0, 0x4380000043800000;" : "=l"(c.byte_pair));
    return c;
}
// `left`: what X leaves of the values, in units of X.
__device__ __forceinline__ void operand_wholes(unsigned long long x, unsigned long long scales, const DigitConstants &c, uint32_t &first, uint32_t &second, unsigned long long &left) {
    const unsigned long long high = pair_fma(x, scales, c.bias), rest = pair_fma(x, scales, pair_fma(high, c.minus, c.bias)), low = pair_fma(rest, c.byte_pair, c.bias);
    left = pair_fma(rest, c.byte_pair, pair_fma(low, c.minus, c.bias));
    first = static_cast<uint32_t>(high) * c.byte + (static_cast<uint32_t>(low) * c.one + c.digits);
    second = static_cast<uint32_t>(high >> 32) * c.byte + (static_cast<uint32_t>(low >> 32) * c.one + c.digits);
}
// The digits of four whole numbers as four words (term 0 first).
__device__ __forceinline__ void operand_digits(uint32_t y0, uint32_t y1, uint32_t y2, uint32_t y3, uint32_t (&terms)[4]) {
    const uint32_t low01 = __byte_perm(y0, y1, 0x5140), low23 = __byte_perm(y2, y3, 0x5140), high01 = __byte_perm(y0, y1, 0x7362), high23 = __byte_perm(y2, y3, 0x7362);
    terms[0] = __byte_perm(high01, high23, 0x7632);
    terms[1] = __byte_perm(high01, high23, 0x5410) ^ 0x80808080u;
    terms[2] = __byte_perm(low01, low23, 0x7632) ^ 0x80808080u;
    terms[3] = __byte_perm(low01, low23, 0x5410) ^ 0x80808080u;
}
__device__ __forceinline__ uint32_t operand_negative(uint32_t y) { return 0x01010100u - y; }
constexpr uint32_t OPERAND_ZERO = 0x00808080u;
__device__ __forceinline__ uint32_t operand_of_infinity(uint32_t bits) {  // of an f32: +-1 if it is infinite
    return (bits & 0x7fffffffu) != 0x7f800000u ? OPERAND_ZERO : (bits >> 31 ? OPERAND_ZERO - 1u : OPERAND_ZERO + 1u);
}
__device__ __forceinline__ uint32_t larger_halves(uint32_t a, uint32_t b) {
    uint32_t v;
    asm("max.u16x2 %0, %1, %2;" : "=r"(v) : "r"(a), "r"(b));
    return v;
}

// What the four bytes cannot hold of a thread's eight columns (see the operand form); by the sixteen threads of a group together.
// `place`: its pieces in shared memory, already written; `residual`: those in the residual's group.
__device__ __noinline__ void keep_residual(uint4 raw, uint32_t exponent, int lane_and_half, uint8_t *place, uint8_t *residual, float *factor) {
    const DigitConstants c = digit_constants();
    const float scale = operand_scale(exponent);
    const uint32_t words[4] = {raw.x, raw.y, raw.z, raw.w}, half_warp = 0xffffu << (thread_now() & 16);
    uint32_t whole[4][2], rest[4][2], terms[2][4];
    float marked = -operand_factor(exponent);
    if (exponent == 255u) {  // (of the warp's two groups; a finite one beside it counts nothing: no sum of the row is)
        bool nan = false, infinite = false;
#pragma unroll
        for (int w = 0; w < 4; w++)
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const uint32_t bits = i == 0 ? words[w] << 16 : words[w] & 0xffff0000u;
                nan |= (bits & 0x7fffffffu) > 0x7f800000u;
                infinite |= (bits & 0x7fffffffu) == 0x7f800000u;
                whole[w][i] = OPERAND_ZERO;
                rest[w][i] = operand_of_infinity(bits);
            }
        nan = __any_sync(half_warp, nan);
        infinite = __any_sync(half_warp, infinite);
        marked = special_factor(nan, infinite);
    } else {
        unsigned long long left[4];
        bool lost = false;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            operand_wholes(pair_of(bf16_lo(words[w]), bf16_hi(words[w])), pair_of(scale, scale), c, whole[w][0], whole[w][1], left[w]);
            lost |= ((left[w] | (left[w] >> 32)) & 0x7fffffffu) != 0;
        }
        if (!__any_sync(half_warp, lost)) return;
#pragma unroll
        for (int w = 0; w < 4; w++) {
            whole[w][0] = operand_negative(whole[w][0]), whole[w][1] = operand_negative(whole[w][1]);
            operand_wholes(left[w], pair_of(RESIDUAL_SCALE, RESIDUAL_SCALE), c, rest[w][0], rest[w][1], left[w]);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++) operand_digits(whole[0][i], whole[1][i], whole[2][i], whole[3][i], terms[i]);
#pragma unroll
    for (int t = 0; t < 4; t++) *reinterpret_cast<uint2 *>(place + term_offset(t, lane_and_half)) = make_uint2(terms[0][t], terms[1][t]);
    if (factor != nullptr) *factor = marked;
#pragma unroll
    for (int i = 0; i < 2; i++) operand_digits(rest[0][i], rest[1][i], rest[2][i], rest[3][i], terms[i]);
#pragma unroll
    for (int t = 0; t < 4; t++) *reinterpret_cast<uint2 *>(residual + term_offset(t, lane_and_half)) = make_uint2(terms[0][t], terms[1][t]);  // (every CTA writes the same)
}

// Rows into operand form, groups [first_group, first_group + groups) of them: with `weight` their rms_norm
// (rms_norm_bf16.comp.template:49-72), without it the bf16 values as they are.  Each CTA repeats it: 8 KB per lane
// from L2.  A thread owns chunk t (and t + 512 when CHUNKS = 2) of each lane, four lanes at a time: one pass over
// registers for the sums of squares, one block-wide exchange, then normalise, round, find the exponent and cut the digits.
// With FROM_GROUP (no weight) the threads own chunks from the first group on, whose operand form goes `destination` bytes into
// the scratch area.
template <int CHUNKS, int LANES, bool FROM_GROUP = false>  // chunks per thread and lane: columns <= CHUNKS * 8 * CONSUMER_THREADS; lanes at a time (1, 2 or 4)
__device__ __forceinline__ void stage_rows(const uint16_t *x, const uint16_t *weight, int width, int first_group, int groups, uint32_t destination = 0) {
    const StackShared &sh = shared();
    uint8_t *operands = smem_raw + sh.scratch + destination;
    float *partial = shared().norm_partial;
    const int lanes = sh.a.lanes, per_lane = width >> 3, thread = thread_now(), warp = thread >> 5, lane = thread & 31, first_chunk = thread + (FROM_GROUP ? first_group * 16 : 0);
    const float eps = sh.a.shape.eps, offset = sh.a.shape.norm_offset;
    const uint4 *source = reinterpret_cast<const uint4 *>(x);
    uint4 scale_words[CHUNKS];
#pragma unroll
    for (int c = 0; c < CHUNKS; c++) {
        const int chunk = first_chunk + c * CONSUMER_THREADS;
        scale_words[c] = weight != nullptr && chunk < per_lane ? __ldg(reinterpret_cast<const uint4 *>(weight) + chunk) : make_uint4(0, 0, 0, 0);
    }
#pragma unroll 1
    for (int m0 = 0; m0 < lanes; m0 += LANES) {
        uint4 raw[LANES][CHUNKS];
#pragma unroll
        for (int mm = 0; mm < LANES; mm++)
#pragma unroll
            for (int c = 0; c < CHUNKS; c++) {
                const int chunk = first_chunk + c * CONSUMER_THREADS;
                // lanes beyond the batch read the last lane again (their results are not stored)
                const int m = m0 + mm < lanes ? m0 + mm : lanes - 1;
                raw[mm][c] = __ldcg(source + static_cast<size_t>(m) * per_lane + (chunk < per_lane ? chunk : 0));
            }
        float my_inverse = 1.0f;
        if (weight != nullptr) {
            float sums[LANES];
#pragma unroll
            for (int mm = 0; mm < LANES; mm++) {
                float sum = 0.0f;
#pragma unroll
                for (int c = 0; c < CHUNKS; c++) {
                    if (CHUNKS > 1 && thread + c * CONSUMER_THREADS >= per_lane) continue;
                    const uint32_t words[4] = {raw[mm][c].x, raw[mm][c].y, raw[mm][c].z, raw[mm][c].w};
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        const float lo = bf16_lo(words[w]), hi = bf16_hi(words[w]);
                        sum = fmaf(lo, lo, sum);
                        sum = fmaf(hi, hi, sum);
                    }
                }
                sums[mm] = (CHUNKS > 1 || thread < per_lane) ? sum : 0.0f;
            }
            float total;
            if (LANES == 4) {
                // the four sums cross the warp together: after two exchanges a thread holds the sum of lane 2 * bit0 + bit1
                const bool odd = lane & 1;
                const float keep0 = odd ? sums[LANES / 2] : sums[0], keep1 = odd ? sums[LANES - 1] : sums[LANES / 4];
                const float send0 = odd ? sums[0] : sums[LANES / 2], send1 = odd ? sums[LANES / 4] : sums[LANES - 1];
                const float a0 = keep0 + __shfl_xor_sync(0xffffffffu, send0, 1), a1 = keep1 + __shfl_xor_sync(0xffffffffu, send1, 1);
                const bool upper = lane & 2;
                float sum = (upper ? a1 : a0) + __shfl_xor_sync(0xffffffffu, upper ? a0 : a1, 2);
                sum += __shfl_xor_sync(0xffffffffu, sum, 4);
                sum += __shfl_xor_sync(0xffffffffu, sum, 8);
                sum += __shfl_xor_sync(0xffffffffu, sum, 16);
                if (lane < 4) partial[(2 * (lane & 1) + (lane >> 1)) * CONSUMER_WARPS + warp] = sum;
            } else {
#pragma unroll
                for (int mm = 0; mm < LANES; mm++) {
#pragma unroll
                    for (int step = 1; step < 32; step *= 2) sums[mm] += __shfl_xor_sync(0xffffffffu, sums[mm], step);
                    if (lane == 0) partial[mm * CONSUMER_WARPS + warp] = sums[mm];
                }
            }
            cta_sync();
            // every warp adds up the 16 partials of the lanes: lanes 8k .. 8k+7 of the warp take lane m0 + k
            const int k = (lane >> 3) < LANES ? lane >> 3 : 0;
            total = partial[k * CONSUMER_WARPS + (lane & 7) * 2] + partial[k * CONSUMER_WARPS + (lane & 7) * 2 + 1];
            total += __shfl_xor_sync(0xffffffffu, total, 1);
            total += __shfl_xor_sync(0xffffffffu, total, 2);
            total += __shfl_xor_sync(0xffffffffu, total, 4);
            // IEEE sqrt and divide, as a CPU evaluates 1/sqrt(v)
            my_inverse = 1.0f / sqrtf(total * (1.0f / static_cast<float>(width)) + eps);
        }
#pragma unroll
        for (int c = 0; c < CHUNKS; c++) {
            const int chunk = first_chunk + c * CONSUMER_THREADS, group = (chunk >> 4) - first_group;
            unsigned long long norm[4];
            if (weight != nullptr) {
                const uint32_t sc[4] = {scale_words[c].x, scale_words[c].y, scale_words[c].z, scale_words[c].w};
#pragma unroll
                for (int w = 0; w < 4; w++) norm[w] = pair_of(bf16_lo(sc[w]) + offset, bf16_hi(sc[w]) + offset);
            }
            uint32_t largest[LANES];
#pragma unroll
            for (int mm = 0; mm < LANES; mm++) {
                uint32_t words[4] = {raw[mm][c].x, raw[mm][c].y, raw[mm][c].z, raw[mm][c].w};
                if (weight != nullptr) {
                    const float inv_rms = __shfl_sync(0xffffffffu, my_inverse, mm * 8);
                    const unsigned long long inverse = pair_of(inv_rms, inv_rms);
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        // rounded to nearest even, as the shaders' f32_to_bf16 for every finite value
                        const unsigned long long v = pair_multiply(pair_multiply(pair_of(bf16_lo(words[w]), bf16_hi(words[w])), inverse), norm[w]);
                        asm("{\n.reg .f32 lo, hi;\nmov.b64 {lo, hi}, %1;\ncvt.rn.bf16x2.f32 %0, hi, lo;\n}" : "=r"(words[w]) : "l"(v));
                    }
                    raw[mm][c] = make_uint4(words[0], words[1], words[2], words[3]);
                }
                if (chunk >= per_lane) words[0] = words[1] = words[2] = words[3] = 0;  // beyond the row: no part of the warp's exponent
                const uint32_t most =
                    larger_halves(larger_halves(words[0] & 0x7fff7fffu, words[1] & 0x7fff7fffu), larger_halves(words[2] & 0x7fff7fffu, words[3] & 0x7fff7fffu));
                largest[mm] = larger_halves(most, most >> 16) & 0x7f80u;
            }
#pragma unroll
            for (int mm = 0; mm < LANES; mm++) largest[mm] = __reduce_max_sync(0xffffffffu, largest[mm]) >> 7;
            if (chunk < per_lane && group >= 0 && group < groups) {
                const int word = chunk & 15;
                uint8_t *block = operands + static_cast<uint32_t>(group) * operand_group_bytes(lanes), *place = block + operand_word_offset(word, m0, lanes);
                const uint32_t flip = (word & 2) * 32;
                uint8_t *const pieces[2] = {place + flip, place - flip};  // even and odd ones
                const DigitConstants constants = digit_constants();
#pragma unroll
                for (int mm = 0; mm < LANES; mm++) {
                    if (m0 + mm >= lanes) break;
                    const float scale = operand_scale(largest[mm]);
                    const unsigned long long scales = pair_of(scale, scale);
                    const uint32_t words[4] = {raw[mm][c].x, raw[mm][c].y, raw[mm][c].z, raw[mm][c].w};
                    uint32_t whole[4][2], even[4], odd[4];
#pragma unroll
                    for (int w = 0; w < 4; w++) {
                        unsigned long long left;
                        operand_wholes(pair_of(bf16_lo(words[w]), bf16_hi(words[w])), scales, constants, whole[w][0], whole[w][1], left);
                    }
                    operand_digits(whole[0][0], whole[1][0], whole[2][0], whole[3][0], even);
                    operand_digits(whole[0][1], whole[1][1], whole[2][1], whole[3][1], odd);
#pragma unroll
                    for (int t = 0; t < 4; t++) *reinterpret_cast<uint2 *>(pieces[(t + mm) & 1] + 256 * mm + term_offset(t, mm)) = make_uint2(even[t], odd[t]);  // (m0 is even)
                    if (word == 0) *reinterpret_cast<float *>(block + 2 * operand_half_bytes(lanes) + 4 * (m0 + mm)) = operand_factor(largest[mm]);
                }
                uint32_t most = largest[0];
#pragma unroll
                for (int mm = 1; mm < LANES; mm++) most = max(most, largest[mm]);
                if (operand_may_lose(most)) {  // (rare, and apart from the loop: a call in it would cost it registers)
#pragma unroll
                    for (int mm = 0; mm < LANES; mm++)
                        if (m0 + mm < lanes && operand_may_lose(largest[mm]))
                            keep_residual(raw[mm][c], largest[mm], mm + (word >> 1), place + 256 * mm,
                                          sh.a.buffers.residual + static_cast<size_t>((sh.a.shape.ffn >> 7) + (chunk >> 4)) * operand_group_bytes(lanes) +
                                              operand_word_offset(word, m0 + mm, lanes),
                                          word == 0 ? reinterpret_cast<float *>(block + 2 * operand_half_bytes(lanes) + 4 * (m0 + mm)) : nullptr);
                }
            }
        }
        if (m0 + LANES < lanes) cta_sync();  // `partial` is rewritten for the next four lanes
    }
    cta_sync();
}

// Rows too wide for a thread's two chunks (o's inputs: no norm looks at whole ones), 8192 columns at a time.
__device__ __noinline__ void stage_wide_rows(const uint16_t *x, int width, int first_group, int groups) {
    const int end = first_group + groups < width >> 7 ? first_group + groups : width >> 7, at_a_time = 2 * CONSUMER_THREADS / 16;
    for (int group = first_group; group < end; group += at_a_time)
        stage_rows<2, 2, true>(x, nullptr, width, group, end - group < at_a_time ? end - group : at_a_time, static_cast<uint32_t>(group - first_group) * operand_group_bytes(shared().a.lanes));
}
template <int TILES>
__device__ __forceinline__ void stage_any(const uint16_t *x, const uint16_t *weight, int width, int first_group, int groups) {
    if (width > 2 * 8 * CONSUMER_THREADS) return stage_wide_rows(x, width, first_group, groups);
    const bool narrow = width <= 8 * CONSUMER_THREADS;
    if (TILES == 1 && shared().a.lanes == 1) return narrow ? stage_rows<1, 1>(x, weight, width, first_group, groups) : stage_rows<2, 1>(x, weight, width, first_group, groups);
    constexpr int LANES = TILES == 1 ? 2 : 4;
    return narrow ? stage_rows<1, LANES>(x, weight, width, first_group, groups) : stage_rows<2, 2>(x, weight, width, first_group, groups);
}

// A group's 128 columns of one lane (bf16 values as f32 in shared memory) into operand form in global memory, by one warp.
__device__ __forceinline__ void store_operand_group(uint8_t *block, uint8_t *residual, const float *columns, int m, int lanes) {
    const int lane = thread_now() & 31, word = lane >> 1, odd = lane & 1;
    const DigitConstants c = digit_constants();
    float v[4];
#pragma unroll
    for (int i = 0; i < 4; i++) v[i] = columns[word * 8 + odd + 2 * i];
    const uint32_t exponent = __reduce_max_sync(0xffffffffu, max(max(__float_as_uint(v[0]) & 0x7fffffffu, __float_as_uint(v[1]) & 0x7fffffffu),
                                                                 max(__float_as_uint(v[2]) & 0x7fffffffu, __float_as_uint(v[3]) & 0x7fffffffu))) >> 23;
    const float scale = operand_scale(exponent);
    float factor = operand_factor(exponent);
    uint32_t terms[4], whole[4];
    unsigned long long left[2];
#pragma unroll
    for (int i = 0; i < 2; i++) operand_wholes(pair_of(v[2 * i], v[2 * i + 1]), pair_of(scale, scale), c, whole[2 * i], whole[2 * i + 1], left[i]);
    const uint32_t at = operand_word_offset(word, m, lanes) + 4 * odd;
    const unsigned long long any = (left[0] | left[1]) & 0x7fffffff7fffffffull;
    if (operand_may_lose(exponent) && (exponent == 255u || __any_sync(0xffffffffu, any != 0))) {
        uint32_t rest[4];
        if (exponent == 255u) {
            bool nan = false, infinite = false;
#pragma unroll
            for (int i = 0; i < 4; i++) {
                nan |= v[i] != v[i];
                infinite |= fabsf(v[i]) == INFINITY;
                whole[i] = OPERAND_ZERO;
                rest[i] = operand_of_infinity(__float_as_uint(v[i]));
            }
            nan = __any_sync(0xffffffffu, nan);
            infinite = __any_sync(0xffffffffu, infinite);
            factor = special_factor(nan, infinite);
        } else {
            factor = -factor;
#pragma unroll
            for (int i = 0; i < 4; i++) whole[i] = operand_negative(whole[i]);
#pragma unroll
            for (int i = 0; i < 2; i++) operand_wholes(left[i], pair_of(RESIDUAL_SCALE, RESIDUAL_SCALE), c, rest[2 * i], rest[2 * i + 1], left[i]);
        }
        operand_digits(rest[0], rest[1], rest[2], rest[3], terms);
#pragma unroll
        for (int t = 0; t < 4; t++) *reinterpret_cast<uint32_t *>(residual + at + term_offset(t, m + (word >> 1))) = terms[t];
    }
    operand_digits(whole[0], whole[1], whole[2], whole[3], terms);
#pragma unroll
    for (int t = 0; t < 4; t++) *reinterpret_cast<uint32_t *>(block + at + term_offset(t, m + (word >> 1))) = terms[t];
    if (lane == 0) *reinterpret_cast<float *>(block + 2 * operand_half_bytes(lanes) + 4 * m) = factor;
}

// ------------------------------------------------------------------------------------------ attention
// A team of four warps serves one context split (64 tokens) of one kv head for the Q = QL * GROUP <= 16 query
// vectors of QL consecutive lanes of a stream (append_gqa_attention_bf16.comp.template:217-339: f32 scores of
// bf16 q.k, f32 softmax, f32 p.v).  Warp w of the team scores tokens 16w .. 16w + 15: q rows are the A operand of
// S = Q K^T, K rows the B operand (both read with 16-byte loads; the head dimension is permuted identically on both
// sides).  The warps agree on the split's row maxima, hand their probabilities on as A fragments - split into a bf16
// high and low part, p = hi + lo to 2^-17 - and warp w then sums dims [w HD / 4, (w + 1) HD / 4) of O = P V over all 64
// tokens, V as the B operand, its token pairs assembled with byte permutes; the products of 16 tokens add up in the
// tensor core, the four parts in f32.  (Each warp summing all dims over its own tokens needed the parts added through
// 17 KB of shared memory per team, in two rounds.)  The team writes one partial (unnormalised output, maximum, sum) per
// query to the scratch.  The team that completes a kv head's last split queues the merge of all of them.

constexpr int Q_PITCH_PAD = 64;  // bytes: 16-byte reads of a quarter warp fall into distinct banks
template <int HD>
__host__ __device__ constexpr size_t attention_team_bytes() {
    // query rows, later the probabilities' fragments (high and low), then maxima and sums [warp][row] and the rows of 64 tokens
    constexpr size_t rows = 16 * (HD * 2 + Q_PITCH_PAD), fragments = 2 * 4 * 32 * 16;
    return (rows > fragments ? rows : fragments) + (2 * 4 * 16 + 64) * 4;
}

// The scratch of a layer's attention step: every (lane, q head, split) partial is HD floats of unnormalised output in
// `values` [lane][q head][split][HD] (16-byte aligned rows) and (maximum, sum) in `stats` [lane][q head][split][2]
// behind all the values - together the (HD + 2) floats per partial the scratch is sized for.
__device__ __forceinline__ float *attention_stats(float *scratch, int lanes, int q_heads, int max_splits, int head_width) {
    return scratch + static_cast<size_t>(lanes) * q_heads * max_splits * head_width;
}

// Log-sum-exp merge of up to 32 partials of one (lane, q head) row by one warp: lane s of the warp weighs partial s,
// every lane owns HD / 32 consecutive output dims, and the weighted rows are summed in order, the loads of eight or
// sixteen partials in flight at a time.  `values` points at the lane's dims of the first partial (rows of HD floats),
// `stats` at its (maximum, sum).  Leaves the block's maximum, its sum and the lane's unnormalised dims.
constexpr int MERGE_BLOCK = 32;
template <int HD>
__device__ __forceinline__ void attention_merge_block(const float *__restrict__ values, const float2 *__restrict__ stats, int count, float &maximum,
                                                      float &denominator, float (&acc)[HD / 32]) {
    constexpr int VEC = HD / 32;
    static_assert(VEC == 1 || VEC == 2 || VEC == 4, "a lane owns one, two or four output dims");
    constexpr int CHUNK = VEC == 4 ? 8 : 16;  // rows in flight at a time; a divisor of the block, whose weights sit in the warp's lanes
    static_assert(MERGE_BLOCK % CHUNK == 0, "rounds of the merge must not straddle a block");
    const int lane_id = thread_now() & 31;
    const int last = count - 1;
    // Rows beyond the last partial are read as the last one again and weigh nothing, so no load is predicated.
    float part[CHUNK][VEC];
    auto fetch = [&](int first) {
#pragma unroll
        for (int u = 0; u < CHUNK; u++) {
            const float *source = values + static_cast<size_t>(first + u < last ? first + u : last) * HD;
            if (VEC == 4) {
                const float4 raw = __ldcg(reinterpret_cast<const float4 *>(source));
                part[u][0] = raw.x, part[u][VEC > 1 ? 1 : 0] = raw.y, part[u][VEC > 2 ? 2 : 0] = raw.z, part[u][VEC > 3 ? 3 : 0] = raw.w;
            } else if (VEC == 2) {
                const float2 raw = __ldcg(reinterpret_cast<const float2 *>(source));
                part[u][0] = raw.x, part[u][VEC > 1 ? 1 : 0] = raw.y;
            } else {
                part[u][0] = __ldcg(source);
            }
        }
    };
#pragma unroll
    for (int v = 0; v < VEC; v++) acc[v] = 0.0f;
    // the statistics and the first rows are requested together
    const float2 pair = __ldcg(stats + (lane_id < last ? lane_id : last));
    fetch(0);
    maximum = warp_max(lane_id < count ? pair.x : -3.4028234663852886e38f);
    const float weight = lane_id < count ? expf(pair.x - maximum) : 0.0f;
    denominator = warp_sum(lane_id < count ? pair.y * weight : 0.0f);
#pragma unroll 1
    for (int s = 0; s < count; s += CHUNK) {
        if (s != 0) fetch(s);
#pragma unroll
        for (int u = 0; u < CHUNK; u++) {
            const float w = __shfl_sync(0xffffffffu, weight, s + u);  // 0 in the lanes beyond the last partial
#pragma unroll
            for (int v = 0; v < VEC; v++) acc[v] += part[u][v] * w;
        }
    }
}

// How many 64-token splits the partials of a query lane's rows cover: those of the newest lane of its group of QL
// lanes (a team writes every row of its group for every split of the group; rows of older lanes are masked there).
__device__ __forceinline__ int attention_own_splits(uint32_t capacity, uint32_t tick);
__device__ __forceinline__ int attention_group_splits(uint32_t capacity, int query_lane, int ql) {
    const StackShared &sh = shared();
    const int per_stream = sh.a.lanes_per_stream, stream = query_lane / per_stream, first = ((query_lane % per_stream) / ql) * ql;
    uint32_t tick = 0;
    for (int i = first; i < first + ql && i < per_stream; i++) {
        const uint32_t other = sh.tick[stream * per_stream + i];
        if (other > tick) tick = other;
    }
    return attention_own_splits(capacity, tick);
}

// The splits of one lane's own attended window.
__device__ __forceinline__ int attention_own_splits(uint32_t capacity, uint32_t tick) {
    const uint32_t tokens = tick + 1u < capacity ? tick + 1u : capacity;
    const int splits = static_cast<int>((tokens + 63u) / 64u), most = shared().a.max_splits;
    return splits < most ? splits : most;
}

// The scratch behind the split partials: per row and range of MERGE_BLOCK splits one merged partial, laid out like
// the split partials (values, then statistics).  Used by rows of more than MERGE_BLOCK splits.
__device__ __forceinline__ float *attention_range_values(const StackArgs &a, int head_width) {
    return a.buffers.attention_scratch + static_cast<size_t>(a.lanes) * a.shape.q_heads * a.max_splits * (head_width + 2);
}
__device__ __forceinline__ int attention_ranges(int max_splits) { return (max_splits + MERGE_BLOCK - 1) / MERGE_BLOCK; }

// The merged output of a row, rounded to bf16 (the warp's lanes own consecutive dims).
template <int HD>
__device__ __forceinline__ void attention_write_row(int query_lane, int head, float denominator, const float (&acc)[HD / 32]) {
    constexpr int VEC = HD / 32;
    const StackArgs &a = shared().a;
    uint16_t *out = a.buffers.attention_out + (static_cast<size_t>(query_lane) * a.shape.q_heads + head) * HD + (thread_now() & 31) * VEC;
    uint32_t bits[VEC];
#pragma unroll
    for (int v = 0; v < VEC; v++) bits[v] = f32_to_bf16_bits(denominator == 0.0f ? 0.0f : acc[v] / denominator);
    if (VEC == 4) *reinterpret_cast<uint2 *>(out) = make_uint2(bits[0] | (bits[VEC > 1 ? 1 : 0] << 16), bits[VEC > 2 ? 2 : 0] | (bits[VEC > 3 ? 3 : 0] << 16));
    else if (VEC == 2) *reinterpret_cast<uint32_t *>(out) = bits[0] | (bits[VEC > 1 ? 1 : 0] << 16);
    else *out = static_cast<uint16_t>(bits[0]);
}

// A row of at most MERGE_BLOCK splits: merged and written out by one warp.
template <int HD>
__device__ __forceinline__ void attention_merge_row(int splits, int query_lane, int head) {
    constexpr int VEC = HD / 32;
    const StackArgs &a = shared().a;
    const int lane_id = thread_now() & 31;
    const size_t row = (static_cast<size_t>(query_lane) * a.shape.q_heads + head) * a.max_splits;
    float maximum, denominator, acc[VEC];
    attention_merge_block<HD>(a.buffers.attention_scratch + row * HD + lane_id * VEC,
                              reinterpret_cast<const float2 *>(attention_stats(a.buffers.attention_scratch, a.lanes, a.shape.q_heads, a.max_splits, HD)) + row, splits, maximum,
                              denominator, acc);
    attention_write_row<HD>(query_lane, head, denominator, acc);
}

// Longer rows, first level: one range of MERGE_BLOCK splits of a row into one partial.
template <int HD>
__device__ __forceinline__ void attention_merge_range(int splits, int query_lane, int head, int range) {
    constexpr int VEC = HD / 32;
    const StackArgs &a = shared().a;
    const int lane_id = thread_now() & 31;
    const size_t row = static_cast<size_t>(query_lane) * a.shape.q_heads + head;
    const size_t first = row * a.max_splits + static_cast<size_t>(range) * MERGE_BLOCK;
    const int count = splits - range * MERGE_BLOCK < MERGE_BLOCK ? splits - range * MERGE_BLOCK : MERGE_BLOCK;
    float maximum, denominator, acc[VEC];
    attention_merge_block<HD>(a.buffers.attention_scratch + first * HD + lane_id * VEC,
                              reinterpret_cast<const float2 *>(attention_stats(a.buffers.attention_scratch, a.lanes, a.shape.q_heads, a.max_splits, HD)) + first, count, maximum,
                              denominator, acc);
    const int ranges = attention_ranges(a.max_splits);
    float *values = attention_range_values(a, HD);
    float *out = values + (row * ranges + range) * HD + lane_id * VEC;
#pragma unroll
    for (int v = 0; v < VEC; v++) out[v] = acc[v];
    if (lane_id == 0) {
        float2 *statistics = reinterpret_cast<float2 *>(values + static_cast<size_t>(a.lanes) * a.shape.q_heads * ranges * HD) + row * ranges + range;
        *statistics = make_float2(maximum, denominator);
    }
}

// Second level: the row's range partials merged and written out.
template <int HD>
__device__ __forceinline__ void attention_merge_ranges(int splits, int query_lane, int head) {
    constexpr int VEC = HD / 32;
    const StackArgs &a = shared().a;
    const int lane_id = thread_now() & 31;
    const size_t row = static_cast<size_t>(query_lane) * a.shape.q_heads + head;
    const int ranges = attention_ranges(a.max_splits), count = (splits + MERGE_BLOCK - 1) / MERGE_BLOCK;
    const float *values = attention_range_values(a, HD);
    float maximum, denominator, acc[VEC];
    attention_merge_block<HD>(values + row * ranges * HD + lane_id * VEC,
                              reinterpret_cast<const float2 *>(values + static_cast<size_t>(a.lanes) * a.shape.q_heads * ranges * HD) + row * ranges, count, maximum,
                              denominator, acc);
    attention_write_row<HD>(query_lane, head, denominator, acc);
}

// Loads through L2 that stay where they are written (the compiler may not sink them towards their use).
__device__ __forceinline__ uint4 load16_now(const void *address) {
    uint4 v;
    asm volatile("ld.global.cg.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(address) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t load4_now(const void *address) {
    uint32_t v;
    asm volatile("ld.global.cg.u32 %0, [%1];" : "=r"(v) : "l"(address) : "memory");
    return v;
}
__device__ __forceinline__ uint32_t load2_now(const void *address) {
    uint16_t v;
    asm volatile("ld.global.cg.u16 %0, [%1];" : "=h"(v) : "l"(address) : "memory");
    return v;
}
__device__ __forceinline__ uint2 load8_now(const void *address) {
    uint2 v;
    asm volatile("ld.global.cg.v2.u32 {%0,%1}, [%2];" : "=r"(v.x), "=r"(v.y) : "l"(address) : "memory");
    return v;
}

template <int HD>
__device__ __forceinline__ size_t attention_row_base(const KvLayer &kv, int slot, uint32_t ring_base, int token) {
    uint32_t ring = ring_base + static_cast<uint32_t>(token);
    if (ring >= kv.capacity) ring -= kv.capacity;
    const int page = static_cast<int>(ring / kv.page_tokens), within = static_cast<int>(ring % kv.page_tokens);
    const int physical = kv.block_table[static_cast<size_t>(slot) * kv.pages_per_slot + page];
    return static_cast<size_t>(physical) * 2 * kv.kv_heads * kv.page_tokens * HD + static_cast<size_t>(within) * HD;
}

// What work item `item` of the launch's attention steps is.
template <int QL>
__device__ __forceinline__ AttentionItem attention_item(const KvLayer &kv, int item) {
    const StackShared &sh = shared();
    const int per_stream = sh.a.lanes_per_stream, groups_per_stream = (per_stream + QL - 1) / QL, max_splits = sh.a.max_splits;
    AttentionItem it;
    const int rest = item / kv.kv_heads, group_slot = rest / max_splits, stream = group_slot / groups_per_stream, first = (group_slot - stream * groups_per_stream) * QL;
    it.kv_head = static_cast<int16_t>(item - rest * kv.kv_heads);
    it.split = static_cast<int16_t>(rest - group_slot * max_splits);
    it.lane0 = static_cast<int16_t>(stream * per_stream + first);
    const int left = per_stream - first;
    it.lanes = static_cast<int16_t>(left < QL ? left : QL);
    it.slot = sh.slot[it.lane0];
    it.arrival = it.kv_head * sh.group_slots + group_slot;
    it.count = 0;
    if (it.slot < 0) return it;
    uint32_t newest = 0;
    for (int i = 0; i < it.lanes; i++) newest = sh.tick[it.lane0 + i] > newest ? sh.tick[it.lane0 + i] : newest;
    const uint32_t tokens = newest + 1u < kv.capacity ? newest + 1u : kv.capacity;  // attended window of the newest lane
    const uint32_t begin = static_cast<uint32_t>(it.split) * 64u;
    if (begin >= tokens) return it;
    it.first_tick = newest + 1u - tokens + begin;
    it.ring_base = it.first_tick % kv.capacity;
    it.count = static_cast<int32_t>(tokens - begin < 64u ? tokens - begin : 64u);
    const int splits = static_cast<int>((tokens + 63u) / 64u);
    it.splits = splits < max_splits ? splits : max_splits;
    return it;
}

template <int HD, int GROUP, int QL>
__device__ __forceinline__ void attention_team_item(int layer, const AttentionItem &it, bool rows_cached) {
    constexpr int Q = QL * GROUP;
    constexpr int QW = HD / 32;         // 16-byte pieces of a q / k row per thread
    constexpr int DIMS = HD / 4;        // head dims of the output per warp
    constexpr int DPT = DIMS / 8;       // of which one thread column owns this many: 4, 2 or 1
    static_assert(Q <= 16 && HD % 32 == 0 && DPT <= 4, "attention team shape");
    StackShared &sh = shared();
    const int thread = thread_now(), team = thread >> 7, team_thread = thread & 127, team_warp = team_thread >> 5, lane = thread & 31, g = lane >> 2, j = lane & 3;
    const int barrier_id = 2 + team;
    uint8_t *team_smem = smem_raw + sh.scratch + static_cast<uint32_t>(team) * static_cast<uint32_t>(attention_team_bytes<HD>());
    float *team_max = reinterpret_cast<float *>(team_smem + attention_team_bytes<HD>() - (2 * 4 * 16 + 64) * 4);  // [4][16]
    float *team_sum = team_max + 4 * 16;                                                                          // [4][16]
    uint32_t *team_rows = reinterpret_cast<uint32_t *>(team_sum + 4 * 16);                                        // [64]
    const KvLayer &kv = sh.layer[layer & 1].kv;
    const int count = it.count, lane0 = it.lane0, kv_head = it.kv_head, q_heads = sh.a.shape.q_heads;
    stamp(layer, 20);
    // row numbers (units of HD elements, kv head 0) of the split's K rows: cached for the team's first item, else looked
    // up through the block table, a token per thread
    const uint32_t *rows = sh.row_base[team];
    if (!rows_cached) {
        if (team_thread < 64) team_rows[team_thread] = team_thread < count ? static_cast<uint32_t>(attention_row_base<HD>(kv, it.slot, it.ring_base, team_thread) / HD) : 0u;
        team_barrier(barrier_id);
        rows = team_rows;
    }
    // ---- the query rows, as asynchronous copies (they would hold 32 registers per thread)
    constexpr uint32_t Q_PITCH = HD * 2 + Q_PITCH_PAD;
    const uint32_t q_shared = shared_address(team_smem);
#pragma unroll
    for (int piece = team_thread; piece < 16 * QW * 4; piece += 128) {
        const int row = piece / (QW * 4), part = piece % (QW * 4);
        const uint32_t destination = q_shared + static_cast<uint32_t>(row) * Q_PITCH + static_cast<uint32_t>(part) * 16u;
        if (row / GROUP < it.lanes && row < Q) {
            const uint16_t *source = sh.a.buffers.q + (static_cast<size_t>(lane0 + row / GROUP) * q_heads + kv_head * GROUP + row % GROUP) * HD + part * 8;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(destination), "l"(source) : "memory");
        } else {
            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};" ::"r"(destination), "r"(0u) : "memory");
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    // ---- K rows of tokens g and g + 8 of the warp's sixteen, requested before the arithmetic
    const size_t head_offset = static_cast<size_t>(kv_head) * kv.page_tokens * HD;
    const uint16_t *keys = kv.pool + head_offset + j * 8, *values = kv.pool + head_offset + static_cast<size_t>(kv.kv_heads) * kv.page_tokens * HD + team_warp * DIMS + g * DPT;
    const int token0 = 16 * team_warp;
    uint4 kf[2][QW];
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
        const int token = token0 + nt * 8 + g;
        const uint16_t *krow = keys + static_cast<size_t>(rows[token]) * HD;
#pragma unroll
        for (int w = 0; w < QW; w++) kf[nt][w] = token < count ? load16_now(krow + w * 32) : make_uint4(0, 0, 0, 0);
    }
    uint32_t tick_row[2];
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int query = (g + 8 * r) / GROUP;
        tick_row[r] = g + 8 * r < Q && query < it.lanes ? sh.tick[lane0 + query] : 0xffffffffu;
    }
    const uint32_t capacity = kv.capacity, first_tick = it.first_tick;
    const float scale = sh.a.shape.attention_scale;
    asm volatile("cp.async.wait_all;" ::: "memory");
    team_barrier(barrier_id);  // the query rows are in shared memory
    float s[2][4];
    {
        float part[2][2][4];  // two chains per tile of eight tokens
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int c = 0; c < 4; c++) part[nt][0][c] = part[nt][1][c] = 0.0f;
#pragma unroll
        for (int w = 0; w < QW; w++) {
            const uint32_t at = q_shared + static_cast<uint32_t>(g) * Q_PITCH + static_cast<uint32_t>(w) * 64u + static_cast<uint32_t>(j) * 16u;
            const uint4 q0 = shared_load16<0>(at), q1 = shared_load16<8 * Q_PITCH>(at);
#pragma unroll
            for (int nt = 0; nt < 2; nt++) {
                mma_bf16_16816(part[nt][0], q0.x, q1.x, q0.y, q1.y, kf[nt][w].x, kf[nt][w].y);
                mma_bf16_16816(part[nt][1], q0.z, q1.z, q0.w, q1.w, kf[nt][w].z, kf[nt][w].w);
            }
        }
#pragma unroll
        for (int nt = 0; nt < 2; nt++)
#pragma unroll
            for (int c = 0; c < 4; c++) s[nt][c] = part[nt][0][c] + part[nt][1][c];
    }
    // the V rows (the warp's dims) of tokens 2j, 2j + 1, 2j + 8, 2j + 9 of every sixteen, in the K rows' registers: they
    // arrive during the softmax
    constexpr int VW = DPT > 2 ? 2 : 1;
    uint32_t v[4][4][VW];
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int t = 0; t < 4; t++) {
            const int token = 16 * k + 2 * j + (t & 1) + 8 * (t >> 1);
            const uint16_t *vrow = values + static_cast<size_t>(rows[token]) * HD;
            v[k][t][0] = v[k][t][VW - 1] = 0u;
            if (token < count) {
                if (DPT == 4) {
                    const uint2 raw = load8_now(vrow);
                    v[k][t][0] = raw.x;
                    v[k][t][VW - 1] = raw.y;
                } else {
                    v[k][t][0] = DPT == 2 ? load4_now(vrow) : load2_now(vrow);
                }
            }
        }
    stamp(layer, 21);

    // ---- causal / ring mask, scale; the team's row maxima; probabilities
    float row_max[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            const int token = token0 + nt * 8 + 2 * j + (c & 1);
            const uint32_t tick = tick_row[c >> 1], token_tick = first_tick + token;
            const bool visible = token < count && tick != 0xffffffffu && token_tick <= tick && token_tick + capacity > tick;
            s[nt][c] = visible ? s[nt][c] * scale : -INFINITY;
            row_max[c >> 1] = fmaxf(row_max[c >> 1], s[nt][c]);
        }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        row_max[r] = fmaxf(row_max[r], __shfl_xor_sync(0xffffffffu, row_max[r], 1));
        row_max[r] = fmaxf(row_max[r], __shfl_xor_sync(0xffffffffu, row_max[r], 2));
        if (j == 0) team_max[team_warp * 16 + g + 8 * r] = row_max[r];
    }
    team_barrier(barrier_id);
    float row_sum[2] = {0.0f, 0.0f};
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int row = g + 8 * r;
        row_max[r] = fmaxf(fmaxf(team_max[row], team_max[16 + row]), fmaxf(team_max[32 + row], team_max[48 + row]));
        row_max[r] = fmaxf(row_max[r], -3.4028234663852886e38f);
    }
#pragma unroll
    for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int c = 0; c < 4; c++) {
            s[nt][c] = s[nt][c] == -INFINITY ? 0.0f : expf(s[nt][c] - row_max[c >> 1]);
            row_sum[c >> 1] += s[nt][c];
        }
#pragma unroll
    for (int r = 0; r < 2; r++) {
        row_sum[r] += __shfl_xor_sync(0xffffffffu, row_sum[r], 1);
        row_sum[r] += __shfl_xor_sync(0xffffffffu, row_sum[r], 2);
        if (j == 0) team_sum[team_warp * 16 + g + 8 * r] = row_sum[r];
    }
    // the probabilities as the A fragment of the warp's 16 tokens, high and low bf16 parts, for every warp of the team (the
    // query rows are read: the maxima's barrier lies behind the products)
    uint4 *fragments = reinterpret_cast<uint4 *>(team_smem);  // [high, low][16 tokens][lane]
    {
        uint32_t ph[4], pl[4];
#pragma unroll
        for (int f = 0; f < 4; f++) {
            const float first = s[f >> 1][2 * (f & 1)], second = s[f >> 1][2 * (f & 1) + 1];
            ph[f] = pack_bf16(first, second);
            pl[f] = pack_bf16(first - bf16_lo(ph[f]), second - bf16_hi(ph[f]));
        }
        fragments[team_warp * 32 + lane] = make_uint4(ph[0], ph[1], ph[2], ph[3]);
        fragments[128 + team_warp * 32 + lane] = make_uint4(pl[0], pl[1], pl[2], pl[3]);
    }
    stamp(layer, 22);
    team_barrier(barrier_id);

    // ---- O = P V: the warp's dims over the split's tokens; thread column g owns dims DPT g .. DPT g + DPT - 1 of them
    float o[DPT][4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint4 high = fragments[k * 32 + lane], low = fragments[128 + k * 32 + lane];
#pragma unroll
        for (int i = 0; i < DPT; i++) {
            const uint32_t selector = (i & 1) ? 0x7632u : 0x5410u;
            const uint32_t b0 = __byte_perm(v[k][0][i >> 1], v[k][1][i >> 1], selector), b1 = __byte_perm(v[k][2][i >> 1], v[k][3][i >> 1], selector);
            float part[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            mma_bf16_16816(part, high.x, high.y, high.z, high.w, b0, b1);
            mma_bf16_16816(part, low.x, low.y, low.z, low.w, b0, b1);
#pragma unroll
            for (int c = 0; c < 4; c++) o[i][c] = k == 0 ? part[c] : o[i][c] + part[c];
        }
    }
    // accumulator column 2j (+1) of tile i is dim DPT * (2j (+1)) + i
    float *scratch = sh.a.buffers.attention_scratch;
    const int max_splits = sh.a.max_splits;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        const int row = g + 8 * r;
        if (tick_row[r] == 0xffffffffu) continue;  // padding
        const size_t partial = (static_cast<size_t>(lane0 + row / GROUP) * q_heads + kv_head * GROUP + row % GROUP) * max_splits + it.split;
        float *out = scratch + partial * HD + team_warp * DIMS + 2 * j * DPT;
        float sums[2][DPT];
#pragma unroll
        for (int half = 0; half < 2; half++)
#pragma unroll
            for (int i = 0; i < DPT; i++) sums[half][i] = o[i][2 * r + half];
        if (DPT == 4) {
            *reinterpret_cast<float4 *>(out) = make_float4(sums[0][0], sums[0][DPT > 1 ? 1 : 0], sums[0][DPT > 2 ? 2 : 0], sums[0][DPT - 1]);
            *reinterpret_cast<float4 *>(out + 4) = make_float4(sums[1][0], sums[1][DPT > 1 ? 1 : 0], sums[1][DPT > 2 ? 2 : 0], sums[1][DPT - 1]);
        } else if (DPT == 2) {
            *reinterpret_cast<float4 *>(out) = make_float4(sums[0][0], sums[0][DPT - 1], sums[1][0], sums[1][DPT - 1]);
        } else {
            *reinterpret_cast<float2 *>(out) = make_float2(sums[0][0], sums[1][0]);
        }
        if (team_warp == 0 && j == 0)
            *reinterpret_cast<float2 *>(attention_stats(scratch, sh.a.lanes, q_heads, max_splits, HD) + partial * 2) =
                make_float2(row_max[r], team_sum[row] + team_sum[16 + row] + team_sum[32 + row] + team_sum[48 + row]);
    }
    // ---- the team that completes the kv head's last split notes the merge of its queries for the CTA; groups of more than
    // MERGE_BLOCK splits are merged in two levels by the whole grid after the items
    stamp(layer, 23);
    team_barrier(barrier_id);  // the team's partials are written, and its shared arrays free for its next item
    if (it.splits <= MERGE_BLOCK && team_thread == 0) {
        unsigned int *arrival = sh.a.buffers.barrier + ARRIVAL_WORDS_OFFSET + it.arrival;
        unsigned int before;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(before) : "l"(arrival) : "memory");  // covers the team's writes before the barrier
        if (before == static_cast<unsigned int>(it.splits - 1)) {
            *arrival = 0u;  // for the next layer (several grid barriers away)
            sh.merge_list[atomicAdd(&sh.merge_count, 1)] = static_cast<uint16_t>(it.arrival);
        }
    }
    stamp(layer, 24);
}

template <int GROUP>
struct AttentionTeam {
    static constexpr int QL = GROUP >= 8 ? 2 : (GROUP >= 4 ? 4 : (16 / GROUP > 8 ? 8 : 16 / GROUP));
};

// ------------------------------------------------------------------------------------------ matrix blocks
// A 16x128 block times the lanes of a batch, as signed bytes: the packed weights are q - 8 in two's complement, so a
// nibble in the upper half of its byte is sixteen times the weight (one AND for eight weights, a shift in front for
// the other eight), and an activation is four bytes (see the operand form).  Up to two lanes have their terms in
// the eight columns of one MMA, up to four in two, up to eight in four:
//   TILES 1: column 4 lane + term;  TILES 2: tile 0 column 2 lane + term (0, 1), tile 1 column 2 lane + term - 2;
//   TILES 4: tile `term`, column `lane`.
// Why integers: with exact fp16 operands (q - 8) and per-group f32 sums a block cost 72 instructions of dequantisation
// (nine for eight nibbles, most at half rate) and eight MMAs; here 24 and 4 TILES, mma.sync taking 32 bytes of K at the
// rate of 16 fp16.  The accumulators start at 1.5 * 2^23 as an integer, which is the f32 of 1.5 * 2^23 + the sum.
constexpr float SUM_BIAS_F32 = 12582912.0f;

// f32 sums of a thread over its groups: rows g and g + 8 of one lane (TILES 1: of lane j / 2 in the even thread columns,
// TILES 2: of lane j), or of lanes 2j and 2j + 1 as a pair (TILES 4).
template <int TILES>
struct Accumulators {
    float row[2];
};
template <>
struct Accumulators<4> {
    unsigned long long row[2];
};
template <int TILES>
struct ActivationOperands {
    uint4 b[TILES][2];
    float factor[2];
};
// `load16(offset)`: of the group's pieces.
template <int TILES, class Load>
__device__ __forceinline__ void load_pieces(ActivationOperands<TILES> &x, const OperandPlace &place, const Load &load16) {
#pragma unroll
    for (int h = 0; h < 2; h++) {
        const uint32_t first = (h == 0 ? place.first : place.second) + h * place.half, second = (h == 0 ? place.second : place.first) + h * place.half;
        x.b[0][h] = load16(first);
        if (TILES == 2) x.b[TILES - 1][h] = load16(first + 128);
        if (TILES == 4) x.b[TILES > 1 ? 1 : 0][h] = load16(second), x.b[TILES > 2 ? 2 : 0][h] = load16(first + 128), x.b[TILES - 1][h] = load16(second + 128);
    }
}
template <int TILES>
__device__ __forceinline__ void load_activations(ActivationOperands<TILES> &x, uint32_t group, const OperandPlace &place) {
    load_pieces<TILES>(x, place, [&](uint32_t offset) { return smem16(group + offset); });
    if (TILES == 4) {
        const float2 both = *reinterpret_cast<const float2 *>(smem_raw + group + place.factor);
        x.factor[0] = both.x, x.factor[1] = both.y;
    } else {
        x.factor[0] = x.factor[1] = *reinterpret_cast<const float *>(smem_raw + group + place.factor);
    }
}
// Constants of the products, made where a pass begins: the compiler would keep them in registers through the whole layer.
struct ProductConstants {
    int32_t bias;
    uint32_t sixteen;  // a multiplication goes to the FMA pipe: AND and shift share a pipe of half the rate
    unsigned long long unbias, term0, term1, term2;  // pairs
};
__device__ __forceinline__ ProductConstants product_constants() {
    ProductConstants c;
    asm volatile("mov.b32 %0, 0x4B400000;" : "=r"(c.bias));
    asm volatile("mov.b32 %0, 16;" : "=r"(c.sixteen));
    asm volatile("mov.b64 %0, 0xCB400000CB400000;" : "=l"(c.unbias));
    asm volatile("mov.b64 %0, 0x4B8000004B800000;" : "=l"(c.term0));
    asm volatile("mov.b64 %0, 0x4780000047800000;" : "=l"(c.term1));
    asm volatile("mov.b64 %0, 0x4380000043800000;" : "=l"(c.term2));
    return c;
}
// BLOCKS blocks (of different tiles) against the same activations, their chains of MMAs side by side.
template <int TILES, int BLOCKS>
__device__ __forceinline__ void block_products(uint4 (*rows)[2], const uint32_t *scales, const ActivationOperands<TILES> &x, const ProductConstants &c,
                                               Accumulators<TILES> *acc) {
    int32_t sums[BLOCKS][TILES][4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
#pragma unroll
        for (int b = 0; b < BLOCKS; b++) {
            const uint4 &upper = rows[b][0], &lower = rows[b][1];
            const uint32_t wa = i == 0 ? upper.x : (i == 1 ? upper.y : (i == 2 ? upper.z : upper.w)), wb = i == 0 ? lower.x : (i == 1 ? lower.y : (i == 2 ? lower.z : lower.w));
            const uint32_t a0 = (wa * c.sixteen) & 0xf0f0f0f0u, a1 = (wb * c.sixteen) & 0xf0f0f0f0u, a2 = wa & 0xf0f0f0f0u, a3 = wb & 0xf0f0f0f0u;
#pragma unroll
            for (int t = 0; t < TILES; t++) {
                const uint4 &columns = x.b[t][i >> 1];
                const uint32_t b0 = (i & 1) ? columns.z : columns.x, b1 = (i & 1) ? columns.w : columns.y;
                int32_t(&sum)[4] = sums[b][t];
                if (i == 0) mma_s8_16832(sum, a0, a1, a2, a3, b0, b1, c.bias, c.bias, c.bias, c.bias);
                else mma_s8_16832(sum, a0, a1, a2, a3, b0, b1, sum[0], sum[1], sum[2], sum[3]);
            }
        }
    }
    // the group's sum t0 2^24 + t1 2^16 + t2 2^8 + t3, rounded to f32 (the lower terms' roundings are below that of what they
    // join, unless it is zero), times the scale
#pragma unroll
    for (int b = 0; b < BLOCKS; b++) {
        const float scale[2] = {__uint_as_float(scales[b] << 16), __uint_as_float(scales[b] & 0xffff0000u)};
        if constexpr (TILES == 4) {
            const unsigned long long factors = pair_of(x.factor[0], x.factor[1]);
#pragma unroll
            for (int r = 0; r < 2; r++) {
                unsigned long long term[4];
#pragma unroll
                for (int t = 0; t < 4; t++) term[t] = pair_add(pair_of(__int_as_float(sums[b][t][2 * r]), __int_as_float(sums[b][t][2 * r + 1])), c.unbias);
                const unsigned long long sum = pair_fma(term[0], c.term0, pair_fma(term[1], c.term1, pair_fma(term[2], c.term2, term[3])));
                acc[b].row[r] = pair_fma(pair_multiply(factors, pair_of(scale[r], scale[r])), sum, acc[b].row[r]);
            }
        } else {
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const float first = __int_as_float(sums[b][0][2 * r]) - SUM_BIAS_F32, second = __int_as_float(sums[b][0][2 * r + 1]) - SUM_BIAS_F32;
                float low;  // of terms 2 and 3, which TILES 1 has one thread column further
                if constexpr (TILES == 1) low = __shfl_down_sync(0xffffffffu, fmaf(first, 256.0f, second), 1);
                else low = fmaf(__int_as_float(sums[b][TILES - 1][2 * r]) - SUM_BIAS_F32, 256.0f, __int_as_float(sums[b][TILES - 1][2 * r + 1]) - SUM_BIAS_F32);
                acc[b].row[r] = fmaf(scale[r] * x.factor[0], fmaf(first, 16777216.0f, fmaf(second, 65536.0f, low)), acc[b].row[r]);
            }
        }
    }
}
// A tile's sums of the warp, to sums[row][lane].
template <int TILES>
__device__ __forceinline__ void store_sums(float *sums, const Accumulators<TILES> &acc) {
    const int lane = thread_now() & 31, g = lane >> 2, j = lane & 3;
#pragma unroll
    for (int r = 0; r < 2; r++) {
        float *row = sums + (g + 8 * r) * 8;
        if constexpr (TILES == 4) *reinterpret_cast<unsigned long long *>(row + 2 * j) = acc.row[r];
        else if (TILES == 2) row[j] = acc.row[r];
        else if ((j & 1) == 0) row[j >> 1] = acc.row[r];
    }
}

// Where the warps stand in the two rings, in one word: slot, slice slot, and the parities of both.
struct RingPlace {
    uint32_t slot, parity, slice_slot, slice_parity;
};
__device__ __forceinline__ RingPlace unpack_place(uint32_t packed) { return {packed & 255u, (packed >> 16) & 1u, (packed >> 8) & 255u, (packed >> 17) & 1u}; }
__device__ __forceinline__ uint32_t pack_place(const RingPlace &at) { return at.slot | (at.slice_slot << 8) | (at.parity << 16) | (at.slice_parity << 17); }

__device__ __forceinline__ WarpBlocks warp_blocks(int phase, int pass, int warp) {
    const StackShared &sh = shared();
    const PhaseInfo &pi = sh.info[phase];
    const int width = pi.width, pair = warp >> pi.width_log2, group = warp & (width - 1), present = stage_present(pi, pass), tiles = present - 2 * pair;
    const uint32_t group_bytes = operand_group_bytes(sh.a.lanes), first = static_cast<uint32_t>(2 * pair * width + group);
    WarpBlocks b;
    b.unit = sh.ring + first * UNIT_BYTES;
    b.scales = static_cast<uint32_t>(present * width) * UNIT_BYTES + first * UNIT_SCALE_BYTES - first * UNIT_BYTES;
    b.next_tile = static_cast<uint32_t>(width) * UNIT_BYTES;
    b.x = sh.scratch + static_cast<uint32_t>(group) * group_bytes;
    b.x_step = phase == 3 ? static_cast<uint32_t>(sh.a.slice_bytes) : static_cast<uint32_t>(width) * group_bytes;
    b.steps = tiles <= 0 || group >= pi.groups ? 0 : (pi.groups - group + width - 1) >> pi.width_log2;
    b.tiles = tiles > 1 ? 2 : 1;
    return b;
}

template <int TILES>
__device__ __forceinline__ Accumulators<TILES> *carried_sums(int warp, int lane) {  // inside the warp's own part of `reduce`
    static_assert(2 * 32 * sizeof(Accumulators<TILES>) <= sizeof(shared().reduce[0]), "a warp's carried sums fit its part");
    return reinterpret_cast<Accumulators<TILES> *>(&shared().reduce[warp][0][0]) + 2 * lane;
}
// The sign bit of a thread's factors: a group of its lanes has a residual.  `second`: the mask of the second lane's (TILES 4).
__device__ __forceinline__ uint32_t second_lane_mask() { return 2 * (thread_now() & 3) + 1 < shared().a.lanes ? 0x80000000u : 0u; }
template <int TILES>
__device__ __forceinline__ uint32_t factor_signs(const float (&factor)[2], uint32_t second) {
    return TILES == 4 ? __float_as_uint(factor[0]) | (__float_as_uint(factor[1]) & second) : __float_as_uint(factor[0]);
}

// The residuals of the warp's groups (see the operand form) times their weights, read again from the stream in global memory,
// onto the sums of a pass (or of a window of it).  A lane's value does not depend on which other lanes have one.
template <int TILES>
__device__ __noinline__ void add_residuals(int phase, int layer, int pass, int first_step, bool carry) {
    StackShared &sh = shared();
    const int thread = thread_now(), warp = thread >> 5, lane = thread & 31;
    const PhaseInfo &pi = sh.info[phase];
    const WarpBlocks blocks = warp_blocks(phase, pass, warp);
    const OperandPlace place = sh.operand_place[lane];
    const uint32_t group_bytes = operand_group_bytes(sh.a.lanes), stage = static_cast<uint32_t>(stage_present(pi, pass) * pi.width * UNIT_TOTAL);
    const uint8_t *stream = layer_stream(sh.layer[layer & 1], phase) + pi.cta_offset + static_cast<size_t>(pass) * pi.slots * pi.width * pi.steps * UNIT_TOTAL + (blocks.unit - sh.ring);
    const uint8_t *residuals = sh.a.buffers.residual + (phase == 3 ? 0 : static_cast<size_t>(sh.a.shape.ffn >> 7) * group_bytes);
    const int last = first_step + pi.window < blocks.steps ? first_step + pi.window : blocks.steps;
    const ProductConstants constants = product_constants();
    const uint32_t second = second_lane_mask();
    Accumulators<TILES> acc[2];
    acc[0].row[0] = acc[0].row[1] = acc[1].row[0] = acc[1].row[1] = 0;
    for (int step = first_step; step < last; step++) {
        const size_t group = static_cast<size_t>(step * pi.width + (warp & (pi.width - 1))) * group_bytes;
        ActivationOperands<TILES> x;
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const uint32_t at = place.factor + (TILES == 4 ? 4u * i : 0u);
            x.factor[i] = phase == 3 ? __ldcg(reinterpret_cast<const float *>(sh.a.buffers.activation + group + at))
                                     : *reinterpret_cast<const float *>(smem_raw + blocks.x + static_cast<uint32_t>(step - first_step) * blocks.x_step + at);
        }
        if (!__any_sync(0xffffffffu, factor_signs<TILES>(x.factor, second) >> 31)) continue;
#pragma unroll
        for (int i = 0; i < 2; i++) x.factor[i] = residual_factor(x.factor[i]);
        load_pieces<TILES>(x, place, [&](uint32_t offset) { return __ldcg(reinterpret_cast<const uint4 *>(residuals + group + offset)); });
        for (int t = 0; t < blocks.tiles; t++) {
            const uint8_t *unit = stream + static_cast<size_t>(step) * stage + t * blocks.next_tile;
            uint4 rows[1][2] = {{__ldg(reinterpret_cast<const uint4 *>(unit) + lane), __ldg(reinterpret_cast<const uint4 *>(unit) + 32 + lane)}};
            const uint32_t scales[1] = {__ldg(reinterpret_cast<const uint32_t *>(stream + static_cast<size_t>(step) * stage + blocks.scales + t * (blocks.next_tile / 32u)) + (lane >> 2))};
            block_products<TILES, 1>(rows, scales, x, constants, acc + t);
        }
    }
    for (int t = 0; t < 2; t++) {
        if (carry) {
            Accumulators<TILES> &sums = carried_sums<TILES>(warp, lane)[t];
            for (int r = 0; r < 2; r++) {
                if constexpr (TILES == 4) sums.row[r] = pair_add(sums.row[r], acc[t].row[r]);
                else sums.row[r] += acc[t].row[r];
            }
            continue;
        }
        const int g = lane >> 2, j = lane & 3;  // as store_sums
        for (int r = 0; r < 2; r++) {
            float *row = sh.reduce[warp][t] + (g + 8 * r) * 8;
            if constexpr (TILES == 4) {
                unsigned long long *both = reinterpret_cast<unsigned long long *>(row + 2 * j);
                *both = pair_add(*both, acc[t].row[r]);
            } else if (TILES == 2) {
                row[j] += acc[t].row[r];
            } else if ((j & 1) == 0) {
                row[j >> 1] += acc[t].row[r];
            }
        }
    }
}

// Every stage holds, for this warp, the blocks of two tiles and one group of K, multiplied by the same activations: tiles
// 2 pair and 2 pair + 1 of the pass, group step * width + place.  Leaves the sums in `reduce` - of a window that is not
// the pass's last, the thread's own sums, which its next window starts from.
template <int TILES, bool X_IN_SLICE>
__device__ __forceinline__ uint32_t consume_pass(int phase, int layer, int pass, int first_step) {
    StackShared &sh = shared();
    const int thread = thread_now(), warp = thread >> 5, lane = thread & 31;
    const int left = sh.info[phase].steps - first_step, window = sh.info[phase].window, steps = left < window ? left : window;
    const WarpBlocks blocks = pass == 0 ? sh.blocks[phase][warp] : warp_blocks(phase, pass, warp);
    const OperandPlace place = sh.operand_place[lane];
    const int active = blocks.steps - first_step < steps ? blocks.steps - first_step : steps, tiles = blocks.tiles;
    const uint32_t scales_from_unit = blocks.scales - static_cast<uint32_t>(lane) * 16u + static_cast<uint32_t>(lane >> 2) * 4u, next_tile = blocks.next_tile,
                   x_step = blocks.x_step;
    static_assert(offsetof(StackShared, empty) == offsetof(StackShared, full) + EMPTY && offsetof(StackShared, slice_full) == offsetof(StackShared, full) + SLICE_FULL &&
                      offsetof(StackShared, slice_empty) == offsetof(StackShared, full) + SLICE_EMPTY,
                  "a slot's barriers are found from its first one");
    RingPlace at = unpack_place(sh.place);
    const uint32_t full = shared_address(sh.full), last_barrier = full + 8u * (static_cast<uint32_t>(sh.a.stages) - 1), ring_bytes = (static_cast<uint32_t>(sh.a.stages) - 1) * STAGE_BYTES;
    const uint32_t last_slice_barrier = full + 8u * static_cast<uint32_t>(sh.a.slice_slots - 1), slices_bytes = static_cast<uint32_t>(sh.a.slice_slots - 1) * x_step;
    uint32_t barrier = full + at.slot * 8u, slice_barrier = full + at.slice_slot * 8u;
    uint32_t unit = blocks.unit + static_cast<uint32_t>(lane) * 16u + at.slot * static_cast<uint32_t>(STAGE_BYTES);
    uint32_t x = blocks.x + (X_IN_SLICE ? at.slice_slot * x_step : 0u);
    const ProductConstants constants = product_constants();
    uint32_t signs = 0;
    const uint32_t second = TILES == 4 ? second_lane_mask() : 0u;
    Accumulators<TILES> acc[2];
#pragma unroll
    for (int t = 0; t < 2; t++) {
        acc[t].row[0] = acc[t].row[1] = 0;
        if (first_step > 0) acc[t] = carried_sums<TILES>(warp, lane)[t];
    }
#pragma unroll 1
    for (int step = 0; step < steps; step++) {
        wait_barrier(barrier, at.parity);
        if (X_IN_SLICE) wait_barrier(slice_barrier + SLICE_FULL, at.slice_parity);
        if (step < active) {
            ActivationOperands<TILES> operands;
            uint4 rows[2][2];
            uint32_t row_scales[2];
            rows[0][0] = smem16(unit);
            rows[0][1] = smem16(unit + 512);
            row_scales[0] = smem4(unit + scales_from_unit);
            load_activations<TILES>(operands, x, place);
            signs |= factor_signs<TILES>(operands.factor, second);
            if (tiles > 1) {
                rows[1][0] = smem16(unit + next_tile);
                rows[1][1] = smem16(unit + next_tile + 512);
                row_scales[1] = smem4(unit + scales_from_unit + next_tile / 32u);
                if constexpr (TILES == 4) {  // (four chains each; the sums of both would not fit the registers)
                    block_products<TILES, 1>(rows, row_scales, operands, constants, acc);
                    block_products<TILES, 1>(rows + 1, row_scales + 1, operands, constants, acc + 1);
                } else {
                    block_products<TILES, 2>(rows, row_scales, operands, constants, acc);
                }
            } else {
                block_products<TILES, 1>(rows, row_scales, operands, constants, acc);
            }
        }
        __syncwarp();
        if (lane == 0) {
            mbarrier_arrive(barrier + EMPTY);
            if (X_IN_SLICE) mbarrier_arrive(slice_barrier + SLICE_EMPTY);
        }
        if (barrier == last_barrier) {
            barrier = full;
            unit -= ring_bytes;
            at.parity ^= 1u;
        } else {
            barrier += 8u;
            unit += STAGE_BYTES;
        }
        if (X_IN_SLICE) {
            if (slice_barrier == last_slice_barrier) {
                slice_barrier = full;
                x -= slices_bytes;
                at.slice_parity ^= 1u;
            } else {
                slice_barrier += 8u;
                x += x_step;
            }
        } else {
            x += x_step;
        }
    }
    at.slot = (barrier - full) >> 3;
    at.slice_slot = (slice_barrier - full) >> 3;
#pragma unroll
    for (int t = 0; t < 2; t++) {
        if (steps < left) carried_sums<TILES>(warp, lane)[t] = acc[t];
        else store_sums<TILES>(sh.reduce[warp][t], acc[t]);
    }
    if (__any_sync(0xffffffffu, signs >> 31)) add_residuals<TILES>(phase, layer, pass, first_step, steps < left);
    return pack_place(at);
}

// ------------------------------------------------------------------------------------------ the kernel

// One matrix step of a layer: stage the activations, stream the CTA's weights, finish the outputs.  Phase 0: q | k | v,
// 1: o, 2: gate and up, 3: down.  EXCHANGE: the tensor-parallel form (o and down leave partial sums that are exchanged
// between the ranks).
template <int HD, bool EXCHANGE, int TILES>
__device__ __forceinline__ void matrix_step(int phase, int layer) {
    StackShared &sh = shared();
    stamp(layer, 4 * phase);
    int pass = 0, first_step = 0;
#pragma unroll 1
    while (pass < sh.info[phase].passes) {
        // ---- activations of q/k/v and gate/up: normalised rows, of o: the attention outputs, staged by every CTA - in
        // windows of a pass's steps where whole rows are too large; those of down arrive in slices
        const int window = sh.info[phase].window;
        if (phase != 3 && (pass == 0 || first_step > 0 || window < sh.info[phase].steps || (phase == 2 && sh.products == sh.scratch))) {  // (products over the rows)
            const StackLayer &spec = sh.layer[layer & 1];
            stage_any<TILES>(phase == 1 ? sh.a.buffers.attention_out : sh.a.buffers.hidden, phase == 0 ? spec.input_norm : (phase == 2 ? spec.post_norm : nullptr),
                             phase == 1 ? sh.a.shape.q_heads * HD : sh.a.shape.hidden, first_step * sh.info[phase].width, window * sh.info[phase].width);
        }
        if (pass == 0 && first_step == 0) stamp(layer, 4 * phase + 1);
        // Epilogue roles: thread t finishes output (high = t & 1, lane m = (t >> 1) & 7, row = ((t >> 4) & 7) + 8 * high)
        // of tile (t >> 7) + 4 * round of the pass - of gate/up the pair of tiles -, so the rotary partner rows r and r + 8
        // of a lane sit in neighbouring threads.  The first round's residual value is requested before the arithmetic.
        uint32_t residual = 0;
        if (phase & 1) {
            const int thread = thread_now();
            if (((thread >> 1) & 7) < sh.a.lanes && (thread >> 7) < stage_present(sh.info[phase], pass))
                residual = __ldcg(sh.a.buffers.hidden + sh.output[thread] + pass * sh.info[phase].slots * static_cast<int>(gridDim.x) * 16);
        }
        const uint32_t place = phase == 3 ? consume_pass<TILES, true>(phase, layer, pass, first_step) : consume_pass<TILES, false>(phase, layer, pass, first_step);
        stamp(layer, 26 + phase);
        cta_sync();
        if (thread_now() == 0) sh.place = place;  // read again behind the next meeting
        first_step += window;
        if (first_step < sh.info[phase].steps) {
            cta_sync();  // every warp is through with the window, its place noted
            continue;
        }
        first_step = 0;
        const int thread = thread_now(), m = (thread >> 1) & 7, row = ((thread >> 4) & 7) + 8 * (thread & 1);
        const bool lane_present = m < sh.a.lanes;
        const int tiles = phase == 2 ? stage_present(sh.info[phase], pass) >> 1 : stage_present(sh.info[phase], pass), width = sh.info[phase].width;
#pragma unroll 1
        for (int slot = thread >> 7; slot < tiles; slot += 4) {  // uniform over the warp
            float first = 0.0f, second = 0.0f;
            const float *src = &sh.reduce[(phase == 2 ? slot : slot >> 1) * width][phase == 2 ? 0 : slot & 1][row * 8 + m];
            for (int w = 0; w < width; w++) {
                first += src[w * 256];
                if (phase == 2) second += src[w * 256 + 128];
            }
            if (phase == 0) {
                // q / k: rotary_bf16.comp.template:99-109 (non-interleaved, rotary width = head width, five bf16
                // roundings); k and v go into the lane's KV page (append_gqa_attention_bf16.comp.template:189-215)
                const int tile = static_cast<int>(blockIdx.x) + (pass * sh.info[phase].slots + slot) * static_cast<int>(gridDim.x);
                const int q_tiles = (sh.a.shape.q_heads * HD) >> 4, k_tiles = (sh.a.shape.kv_heads * HD) >> 4;
                const float mine_value = round_bf16(first);
                const float partner = __shfl_xor_sync(0xffffffffu, mine_value, 1);  // the row 8 further (or 8 back)
                if (lane_present) {
                    const KvLayer &kv = sh.layer[layer & 1].kv;
                    const size_t kv_token = sh.kv_row[m];
                    const bool kv_writable = kv_token != ~0ull;
                    const size_t head_stride = static_cast<size_t>(kv.page_tokens) * HD;
                    if (tile < q_tiles + k_tiles) {
                        const bool is_q = tile < q_tiles, high = row >= 8;
                        const int local = is_q ? tile : tile - q_tiles;
                        const int head = local / (HD >> 4), d = 8 * (local % (HD >> 4)) + (row & 7) + (high ? HD / 2 : 0);
                        const uint32_t rotation = sh.rope[m * (HD >> 1) + 8 * (local % (HD >> 4)) + (row & 7)];
                        const float cosine = bf16_lo(rotation), sine = bf16_hi(rotation);
                        // d < half: x cos + (-x[d + half]) sin;  d >= half: x cos + x[d - half] sin
                        const float other = high ? partner : -partner;
                        const uint16_t value = static_cast<uint16_t>(f32_to_bf16_bits(round_bf16(mine_value * cosine) + round_bf16(other * sine)));
                        if (is_q) sh.a.buffers.q[(static_cast<size_t>(m) * sh.a.shape.q_heads + head) * HD + d] = value;
                        else if (kv_writable) kv.pool[kv_token + static_cast<size_t>(head) * head_stride + d] = value;
                    } else if (kv_writable) {
                        const int index = (tile - q_tiles - k_tiles) * 16 + row;
                        kv.pool[kv_token + static_cast<size_t>(kv.kv_heads + index / HD) * head_stride + index % HD] = static_cast<uint16_t>(f32_to_bf16_bits(first));
                    }
                }
            } else if (phase == 2) {
                // silu_multiply_bf16.comp.template:30-52: bf16(silu_bf16(bf16 gate) * bf16 up)
                if (lane_present)
                    *reinterpret_cast<float *>(smem_raw + sh.products + (m * 128 + slot * 16 + row) * 4) = round_bf16(rounded_silu(round_bf16(first)) * round_bf16(second));
            } else if (lane_present) {
                float total = first;
                uint16_t *out = sh.a.buffers.hidden + sh.output[thread] + (pass * sh.info[phase].slots + slot - (thread >> 7)) * static_cast<int>(gridDim.x) * 16;
                if constexpr (EXCHANGE) {
                    // this rank's share of the sum over K goes to every peer's inbox, value and exchange number in
                    // one 8-byte store; the peers' shares arrive in this rank's inbox the same way
                    const StackTp &tp = *sh.a.tp;
                    int *error_flag = sh.a.buffers.error_flag;
                    const uint32_t number = sh.exchanges + static_cast<uint32_t>(2 * layer + (phase == 1 ? 1 : 2));
                    const size_t element = static_cast<size_t>(number & 1u) * STACK_TP_MAX_RANKS * 8 * sh.a.shape.hidden + (out - sh.a.buffers.hidden);
                    const unsigned long long word = (static_cast<unsigned long long>(number) << 32) | __float_as_uint(first);
                    for (int r = 0; r < tp.size; r++)
                        if (r != tp.rank)
                            asm volatile("st.relaxed.sys.global.u64 [%0], %1;" ::"l"(reinterpret_cast<unsigned long long *>(tp.exchange[r]) + element +
                                                                                  static_cast<size_t>(tp.rank) * 8 * sh.a.shape.hidden),
                                         "l"(word)
                                         : "memory");
                    total = 0.0f;
                    unsigned int spins = 0;
                    bool gave_up = false;
                    for (int r = 0; r < tp.size; r++) {  // rank order on every rank: the replicas stay bit-identical
                        float part = first;
                        if (r != tp.rank) {
                            const unsigned long long *source =
                                reinterpret_cast<const unsigned long long *>(tp.exchange[tp.rank]) + element + static_cast<size_t>(r) * 8 * sh.a.shape.hidden;
                            unsigned long long got = 0;
                            while (!gave_up) {
                                asm volatile("ld.relaxed.sys.global.u64 %0, [%1];" : "=l"(got) : "l"(source) : "memory");
                                if (static_cast<uint32_t>(got >> 32) == number) break;
                                if (++spins > STACK_TP_SPIN_LIMIT) {
                                    atomicExch(error_flag, 2);
                                    gave_up = true;
                                } else if ((spins & 255u) == 0 && *reinterpret_cast<volatile int *>(error_flag) != 0) {
                                    gave_up = true;
                                }
                            }
                            part = __uint_as_float(static_cast<uint32_t>(got));
                        }
                        total += part;
                    }
                }
                // linear + residual_add (add_bf16.comp.template:17-24): bf16(bf16(product) + residual), in place
                const uint32_t before = slot < 4 ? residual : __ldcg(out);
                *out = static_cast<uint16_t>(f32_to_bf16_bits(round_bf16(total) + bf16_bits_to_f32(before)));
            }
        }
        if (phase == 2) {
            // the pass's eight tiles of gate and of up are one group of down's columns: into operand form, one warp per lane
            cta_sync();
            const int warp = thread_now() >> 5, lanes = sh.a.lanes;
            if (warp < lanes)
                store_operand_group(sh.a.buffers.activation + static_cast<size_t>(blockIdx.x + pass * gridDim.x) * operand_group_bytes(lanes),
                                    sh.a.buffers.residual + static_cast<size_t>(blockIdx.x + pass * gridDim.x) * operand_group_bytes(lanes),
                                    reinterpret_cast<const float *>(smem_raw + sh.products) + warp * 128, warp, lanes);
        }
        pass++;
        if (pass < sh.info[phase].passes) cta_sync();  // the partial sums are rewritten by the next pass
    }
    stamp(layer, 4 * phase + 2);
}

// Attention of a layer: (kv head, split, stream x lane group) items, one team of four warps each, spread over the SMs
// first; the teams' shared arrays reuse the scratch area (nothing is staged right now).
template <int HD, int GROUP>
__device__ __forceinline__ void attention_step(int layer) {
    constexpr int QL = AttentionTeam<GROUP>::QL;
    StackShared &sh = shared();
    const int total = sh.a.shape.kv_heads * sh.a.max_splits * sh.group_slots;
    {
        const int team = thread_now() >> 7;
        int round = 0;
#pragma unroll 1
        for (int item = blockIdx.x + gridDim.x * team; item < total; item += gridDim.x * 4, round++) {
            AttentionItem &later = sh.later_item[round & 1][team];
            if (round > 0) {
                // (last read two rounds ago: every warp of the team has arrived at the barrier between since)
                if ((thread_now() & 127) == 0) later = attention_item<QL>(sh.layer[layer & 1].kv, item);
                team_barrier(2 + team);
            }
            const AttentionItem &it = round == 0 ? sh.item[team] : later;
            if (it.count > 0) attention_team_item<HD, GROUP, QL>(layer, it, round == 0);
        }
    }
    cta_sync();
    stamp(layer, 17);
    {
        // merge the heads whose last split was completed here: one (lane, q head) row per warp and round
        const int requests = sh.merge_count;
        if (requests > 0) {  // (the partials are visible: the counting thread acquired them in front of the meeting above)
            const int group_slots = sh.group_slots, per_stream = sh.a.lanes_per_stream, groups_per_stream = (per_stream + QL - 1) / QL;
            for (int index = thread_now() >> 5; index < requests * QL * GROUP; index += CONSUMER_WARPS) {
                const int request = sh.merge_list[index / (QL * GROUP)], row = index % (QL * GROUP);
                const int kv_head = request / group_slots, group_slot = request % group_slots;
                const int group_index = group_slot % groups_per_stream;
                const int query_lane = (group_slot / groups_per_stream) * per_stream + group_index * QL + row / GROUP;
                if (query_lane < sh.a.lanes && group_index * QL + row / GROUP < per_stream && sh.slot[query_lane] >= 0)
                    attention_merge_row<HD>(attention_own_splits(sh.layer[layer & 1].kv.capacity, sh.tick[query_lane]), query_lane, kv_head * GROUP + row % GROUP);
            }
        }
    }
    if (sh.a.max_splits > MERGE_BLOCK) {
        // ---- groups of more than MERGE_BLOCK splits: every warp of the grid merges ranges of MERGE_BLOCK splits into one
        // partial each, then one warp per row merges the row's range partials
        const int ranges = attention_ranges(sh.a.max_splits), q_heads = sh.a.shape.q_heads, rows = sh.a.lanes * q_heads;
        const uint32_t capacity = sh.layer[layer & 1].kv.capacity;
        grid_meet(false);
        for (int task = blockIdx.x + gridDim.x * (thread_now() >> 5); task < rows * ranges; task += gridDim.x * CONSUMER_WARPS) {
            const int row = task / ranges, range = task % ranges, query_lane = row / q_heads;
            if (sh.slot[query_lane] < 0) continue;
            const int splits = attention_group_splits(capacity, query_lane, QL);
            if (splits > MERGE_BLOCK && range * MERGE_BLOCK < splits) attention_merge_range<HD>(splits, query_lane, row % q_heads, range);
        }
        grid_meet(false);
        for (int row = blockIdx.x + gridDim.x * (thread_now() >> 5); row < rows; row += gridDim.x * CONSUMER_WARPS) {
            const int query_lane = row / q_heads;
            if (sh.slot[query_lane] < 0) continue;
            const int splits = attention_group_splits(capacity, query_lane, QL);
            if (splits > MERGE_BLOCK) attention_merge_ranges<HD>(splits, query_lane, row % q_heads);
        }
    }
}

constexpr int LAYER_WORDS = static_cast<int>(sizeof(StackLayer) / sizeof(uint32_t));
static_assert(sizeof(StackLayer) % sizeof(uint32_t) == 0 && sizeof(StackArgs) % sizeof(uint32_t) == 0, "descriptions are copied word by word");

// At the top of a layer: the next layer's description into the other copy (last read before the previous layer's final
// barrier; stages of the next layer are requested behind this layer's first meeting at the earliest), and the K and V rows this CTA's teams will read in this layer's attention step on their way into L2.
template <int HD>
__device__ __forceinline__ void begin_layer(int layer) {
    StackShared &sh = shared();
    const int thread = thread_now();
    if (thread >= 32 && thread < 32 + LAYER_WORDS && layer + 1 < sh.a.layer_count)
        reinterpret_cast<uint32_t *>(&sh.layer[(layer + 1) & 1])[thread - 32] = reinterpret_cast<const uint32_t *>(sh.a.layers + layer + 1)[thread - 32];
    const KvLayer &kv = sh.layer[layer & 1].kv;
    const int team = thread >> 7, team_thread = thread & 127;
    if (team_thread < sh.item[team].count) {
        const size_t half_page = static_cast<size_t>(kv.kv_heads) * kv.page_tokens * HD;
        const uint16_t *row = kv.pool + static_cast<size_t>(sh.row_base[team][team_thread]) * HD + static_cast<size_t>(sh.item[team].kv_head) * kv.page_tokens * HD;
#pragma unroll
        for (int line = 0; line < (HD * 2 + 127) / 128; line++) {
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t *>(row) + line * 128));
            asm volatile("prefetch.global.L2 [%0];" ::"l"(reinterpret_cast<const uint8_t *>(row + half_page) + line * 128));
        }
    }
}

// What the consumers look up once per launch: the lanes' positions, pages and rotary factors, the KV rows of each team's
// first attention item.
template <int HD, int GROUP>
__device__ __forceinline__ void prepare_launch() {
    constexpr int QL = AttentionTeam<GROUP>::QL;
    StackShared &sh = shared();
    const int thread = threadIdx.x, lanes = sh.a.lanes;
    if (thread < 4 * CONSUMER_WARPS) sh.blocks[thread >> 4][thread & 15] = warp_blocks(thread >> 4, 0, thread & 15);
    if (thread < 8) {
        const uint32_t tick = thread < lanes ? sh.a.lanes_meta.position[thread] : 0u;
        const int slot = thread < lanes ? sh.a.lanes_meta.slot[thread] : -1;
        sh.tick[thread] = tick;
        sh.slot[thread] = slot;
        const KvLayer &kv = sh.layer[0].kv;
        uint64_t row = ~0ull;
        if (slot >= 0 && kv.capacity != 0) {
            const uint32_t ring_token = tick % kv.capacity;
            const int physical = kv.block_table[static_cast<size_t>(slot) * kv.pages_per_slot + ring_token / kv.page_tokens];
            row = static_cast<uint64_t>(physical) * 2 * kv.kv_heads * kv.page_tokens * HD + static_cast<uint64_t>(ring_token % kv.page_tokens) * HD;
        }
        sh.kv_row[thread] = row;
    }
    for (int index = thread; index < lanes * (HD >> 1); index += CONSUMER_THREADS) {
        const int m = index / (HD >> 1);
        sh.rope[index] = __ldg(sh.a.shape.rope_table + static_cast<size_t>(sh.a.lanes_meta.position[m] % sh.a.shape.rope_positions) * (HD >> 1) + (index - m * (HD >> 1)));
    }
    cta_sync();
    const int per_stream = sh.a.lanes_per_stream, groups_per_stream = (per_stream + QL - 1) / QL, group_slots = lanes / per_stream * groups_per_stream;
    const int total = sh.a.shape.kv_heads * sh.a.max_splits * group_slots;
    const int team = thread >> 7, team_thread = thread & 127;
    const int item = static_cast<int>(blockIdx.x) + static_cast<int>(gridDim.x) * team;
    if (thread == 0) {
        sh.merge_count = 0;
        sh.group_slots = group_slots;
    }
    cta_sync();
    const KvLayer &kv = sh.layer[0].kv;
    if (team_thread == 0) {
        sh.item[team].count = 0;
        if (item < total && kv.capacity != 0) sh.item[team] = attention_item<QL>(kv, item);
    }
    cta_sync();
    if (team_thread < 64)
        sh.row_base[team][team_thread] =
            team_thread < sh.item[team].count ? static_cast<uint32_t>(attention_row_base<HD>(kv, sh.item[team].slot, sh.item[team].ring_base, team_thread) / HD) : 0u;
    sh.output[thread] = static_cast<uint32_t>(((thread >> 1) & 7) * sh.a.shape.hidden + (static_cast<int>(blockIdx.x) + (thread >> 7) * static_cast<int>(gridDim.x)) * 16 +
                                              ((thread >> 4) & 7) + 8 * (thread & 1));
    cta_sync();
}

// The matrices' schedules and the rings' barriers.
template <int TILES>
__device__ __forceinline__ void prepare_rings(int q_width, int kv_width) {
    StackShared &sh = shared();
    const int thread = threadIdx.x, lanes = sh.a.lanes;
    if (thread < 4) {
        const StackShape &shape = sh.a.shape;
        const int grid = static_cast<int>(gridDim.x), cta = static_cast<int>(blockIdx.x);
        const MatrixSchedule s = thread == 0   ? stack_schedule((q_width + 2 * kv_width) >> 4, shape.hidden >> 7, false, grid)
                                 : thread == 1 ? stack_schedule(shape.hidden >> 4, q_width >> 7, false, grid)
                                 : thread == 2 ? stack_schedule(shape.ffn >> 4, shape.hidden >> 7, true, grid)
                                               : stack_schedule(shape.hidden >> 4, shape.ffn >> 7, false, grid);
        PhaseInfo &pi = sh.info[thread];
        pi.tiles_here = stack_cta_tiles(s, cta);
        pi.passes = (pi.tiles_here + s.slots - 1) / s.slots;
        pi.slots = s.slots;
        pi.width = s.width;
        pi.width_log2 = 31 - __clz(s.width);
        pi.steps = s.steps;
        pi.groups = s.groups;
        pi.window = pi.steps;
        if (thread != 3 && static_cast<uint32_t>(pi.groups) * operand_group_bytes(lanes) > sh.a.scratch_bytes)
            pi.window = static_cast<int>((sh.a.scratch_bytes) / operand_group_bytes(lanes)) / pi.width;
        pi.cta_offset = static_cast<uint32_t>(stack_cta_offset(s, cta));
    }
    if (thread < MAX_STAGES) {
        mbarrier_init(shared_address(&sh.full[thread]), 1);               // the producer's arrival with the byte count
        mbarrier_init(shared_address(&sh.empty[thread]), CONSUMER_WARPS);  // one arrival per consumer warp
        mbarrier_init(shared_address(&sh.slice_full[thread]), 1);
        mbarrier_init(shared_address(&sh.slice_empty[thread]), CONSUMER_WARPS);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async;" ::: "memory");
    }
    if (thread >= 32 && thread < 64) {
        // columns without a lane repeat lane 0's, their results are dropped
        const int g = (thread & 31) >> 2, j = thread & 3;
        const int column = TILES == 1 ? g >> 2 : (TILES == 2 ? g >> 1 : g), m = column < lanes ? column : 0, term = TILES == 1 ? g & 3 : (TILES == 2 ? g & 1 : 0);
        const int summed = TILES == 1 ? j >> 1 : (TILES == 2 ? j : 2 * j);  // the lane (the first of two) of the thread's sums
        const uint32_t row = static_cast<uint32_t>(m) * 256u + static_cast<uint32_t>(j) * 16u;
        OperandPlace place;
        place.half = operand_half_bytes(lanes);
        place.first = row + term_offset(term, m);
        place.second = row + term_offset(term, m + 1);
        place.factor = 2 * place.half + static_cast<uint32_t>(summed < lanes ? summed : 0) * 4u;
        sh.operand_place[thread & 31] = place;
    }
    if (thread == 64) {
        sh.scratch = (static_cast<uint32_t>(sizeof(StackShared)) + 127u) & ~127u;
        sh.ring = sh.scratch + sh.a.scratch_bytes;
        const uint32_t staged = static_cast<uint32_t>(sh.a.shape.hidden >> 7) * operand_group_bytes(lanes);
        sh.products = staged + PRODUCT_BYTES <= sh.a.scratch_bytes ? sh.scratch + staged : sh.scratch;
        sh.place = 0u;
        sh.barrier_target = sh.a.buffers.barrier_handicap;
        sh.barrier_limit = sh.a.buffers.barrier_handicap != 0 ? (1u << 12) : BARRIER_SPIN_LIMIT;
        sh.open_word = 0u;
        sh.exchanges = sh.a.tp != nullptr ? static_cast<uint32_t>(sh.a.tp->counter[sh.a.tp->rank][STACK_TP_WORD_CONSUMED]) : 0u;
    }
    __syncthreads();
}

// TILES: MMA columns in eights (stack_tiles).
template <int HD, int GROUP, bool EXCHANGE, int TILES>
__global__ void __launch_bounds__(STACK_THREADS, 1) decode_stack_kernel(const __grid_constant__ StackArgs args) {
    StackShared &sh = shared();
    for (int word = threadIdx.x; word < static_cast<int>(sizeof(StackArgs) / sizeof(uint32_t)); word += STACK_THREADS)
        reinterpret_cast<uint32_t *>(&sh.a)[word] = reinterpret_cast<const uint32_t *>(&args)[word];
    if (threadIdx.x >= 256 && threadIdx.x < 256 + LAYER_WORDS)
        reinterpret_cast<uint32_t *>(&sh.layer[0])[threadIdx.x - 256] = reinterpret_cast<const uint32_t *>(args.layers)[threadIdx.x - 256];
    if (args.layer_count > 1 && threadIdx.x >= 384 && threadIdx.x < 384 + LAYER_WORDS)
        reinterpret_cast<uint32_t *>(&sh.layer[1])[threadIdx.x - 384] = reinterpret_cast<const uint32_t *>(args.layers + 1)[threadIdx.x - 384];
    if (args.buffers.timing != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        args.buffers.timing[16] = now;
    }
    __syncthreads();
    prepare_rings<TILES>(sh.a.shape.q_heads * HD, sh.a.shape.kv_heads * HD);
    if (threadIdx.x >= CONSUMER_THREADS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(PRODUCER_REGISTERS));
        if (threadIdx.x == CONSUMER_THREADS) produce_weights();
        else if (threadIdx.x == CONSUMER_THREADS + 32) produce_activations();
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(CONSUMER_REGISTERS));
    prepare_launch<HD, GROUP>();
#pragma unroll 1
    for (int layer = 0; layer < sh.a.layer_count; layer++) {
        begin_layer<HD>(layer);
#pragma unroll 1
        for (int phase = 0; phase < 4; phase++) {
            matrix_step<HD, EXCHANGE, TILES>(phase, layer);
#pragma unroll 1
            for (bool attended = phase != 0;; attended = true) {
                if (phase < 3 || layer + 1 < sh.a.layer_count) grid_meet(true);
                if (phase != 0 || !attended) stamp(layer, 4 * phase + 3);
                if (attended) break;
                attention_step<HD, GROUP>(layer);
            }
            if (phase == 0) {
                if (threadIdx.x == 0) sh.merge_count = 0;  // read again after the next layer's q/k/v barrier at the earliest
                stamp(layer, 18);
            }
        }
    }

    if (args.buffers.timing != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long now;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
        args.buffers.timing[30] = now;
    }
    // The last CTA to leave rearms the barrier words for the next launch (every CTA has passed its last barrier
    // before it counts itself out).
    if (threadIdx.x == 0) {
        unsigned int *counter = args.buffers.barrier;
        const unsigned int gone = atomicAdd(counter + 1, 1u);
        if (gone == gridDim.x - 1) {
            counter[0] = 0u;
            counter[1] = 0u;
            // the next launch counts on from here
            if constexpr (EXCHANGE) args.tp->counter[args.tp->rank][STACK_TP_WORD_CONSUMED] = sh.exchanges + static_cast<uint32_t>(2 * args.layer_count);
            __threadfence();
        }
    }
}

struct StackPlanSmem {
    size_t scratch, total;
    int stages, slice_slots, slice_bytes;
};

template <int HD>
bool plan_smem_for(const StackShape &shape, int lanes, int grid, StackPlanSmem *plan) {
    const int q_width = shape.q_heads * shape.head_width, widest = q_width > shape.hidden ? q_width : shape.hidden;
    const MatrixSchedule qkv = stack_schedule((q_width + 2 * shape.kv_heads * shape.head_width) >> 4, shape.hidden >> 7, false, grid);
    const MatrixSchedule o = stack_schedule(shape.hidden >> 4, q_width >> 7, false, grid);
    const MatrixSchedule down = stack_schedule(shape.hidden >> 4, shape.ffn >> 7, false, grid);
    const size_t group = operand_group_bytes(lanes), limit = 227 * 1024;
    const size_t stage = STAGE_BYTES;
    const size_t fixed = (sizeof(StackShared) + 127) & ~static_cast<size_t>(127);
    // what the scratch has to hold: the attention teams, two slices of down, a step's groups of the staged rows
    const size_t slice = static_cast<size_t>(down.width < down.groups ? down.width : down.groups) * group;
    size_t least = 4 * attention_team_bytes<HD>();
    if (2 * slice > least) least = 2 * slice;
    const size_t window = static_cast<size_t>(qkv.width > o.width ? qkv.width : o.width) * group;
    if (window > least) least = window;
    if (PRODUCT_BYTES > least) least = PRODUCT_BYTES;
    // ... and whole rows, unless the ring would be left with less than two stages
    size_t scratch = static_cast<size_t>(widest >> 7) * group;
    if (shape.ffn >> 7 > grid) scratch += PRODUCT_BYTES;  // several passes of gate/up: the products beside the rows
    if (scratch < least) scratch = least;
    if (fixed + 128 + scratch + 2 * stage > limit) scratch = fixed + 128 + least + 2 * stage > limit ? least : limit - fixed - 128 - 2 * stage;
    scratch = (scratch + 127) & ~static_cast<size_t>(127);
    if (fixed + scratch + 2 * stage > limit) return false;
    int slice_slots = static_cast<int>(scratch / slice);
    if (slice_slots > MAX_STAGES) slice_slots = MAX_STAGES;
    int stages = static_cast<int>((limit - fixed - scratch) / stage);
    if (stages > MAX_STAGES) stages = MAX_STAGES;
    plan->scratch = scratch;
    plan->stages = stages;
    plan->slice_slots = slice_slots;
    plan->slice_bytes = static_cast<int>(slice);
    plan->total = fixed + scratch + static_cast<size_t>(stages) * stage;
    return true;
}

bool plan_smem(const StackShape &shape, int lanes, int grid, StackPlanSmem *plan) {
    const int group = shape.kv_heads > 0 ? shape.q_heads / shape.kv_heads : 0;
    if (shape.head_width == 128 && (group == 4 || group == 8)) return plan_smem_for<128>(shape, lanes, grid, plan);
    if (shape.head_width == 64 && group == 4) return plan_smem_for<64>(shape, lanes, grid, plan);
    if (shape.head_width == 32 && group == 2) return plan_smem_for<32>(shape, lanes, grid, plan);
    return false;
}

template <int HD, int GROUP, bool EXCHANGE, int TILES>
cudaError_t launch_instance_of(const StackArgs &args, size_t smem, int grid, cudaStream_t stream) {
    // the attribute is per device and per kernel instance: set it on every launch (a cheap host-side call)
    cudaError_t status = cudaFuncSetAttribute(decode_stack_kernel<HD, GROUP, EXCHANGE, TILES>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (status != cudaSuccess) return status;
    // the consumers would wait forever for registers that the launch did not bring
    cudaFuncAttributes attributes;
    status = cudaFuncGetAttributes(&attributes, decode_stack_kernel<HD, GROUP, EXCHANGE, TILES>);
    if (status != cudaSuccess) return status;
    if (attributes.numRegs * STACK_THREADS < CONSUMER_THREADS * CONSUMER_REGISTERS + (STACK_THREADS - CONSUMER_THREADS) * PRODUCER_REGISTERS)
        return cudaErrorInvalidDeviceFunction;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(grid);
    config.blockDim = dim3(STACK_THREADS);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeCooperative;  // all CTAs co-resident: they wait on one another
    attribute[0].val.cooperative = 1;
    config.attrs = attribute;
    config.numAttrs = 1;
    return cudaLaunchKernelEx(&config, decode_stack_kernel<HD, GROUP, EXCHANGE, TILES>, args);
}

// MMA columns of a batch in eights: four terms per lane.
constexpr int stack_tiles(int lanes) { return lanes <= 2 ? 1 : (lanes <= 4 ? 2 : 4); }

template <int HD, int GROUP, bool EXCHANGE>
cudaError_t launch_instance_of(const StackArgs &args, size_t smem, int grid, cudaStream_t stream) {
    switch (stack_tiles(args.lanes)) {
        case 1: return launch_instance_of<HD, GROUP, EXCHANGE, 1>(args, smem, grid, stream);
        case 2: return launch_instance_of<HD, GROUP, EXCHANGE, 2>(args, smem, grid, stream);
        default: return launch_instance_of<HD, GROUP, EXCHANGE, 4>(args, smem, grid, stream);
    }
}
template <int HD, int GROUP>
cudaError_t launch_instance(const StackArgs &args, size_t smem, int grid, cudaStream_t stream) {
    return args.tp_size > 1 ? launch_instance_of<HD, GROUP, true>(args, smem, grid, stream) : launch_instance_of<HD, GROUP, false>(args, smem, grid, stream);
}

}  // namespace

size_t stack_activation_bytes(int ffn) { return static_cast<size_t>(ffn >> 7) * operand_group_bytes(8); }

size_t stack_residual_bytes(int ffn, int widest) { return static_cast<size_t>((ffn >> 7) + (widest >> 7)) * operand_group_bytes(8); }

size_t int4_cta_stream_bytes(int rows, int k, bool pair, int grid) {
    return stack_stream_bytes(stack_schedule(rows / 16, k / 128, pair, grid));
}

cudaError_t launch_int4_cta_streams(const RelayoutSegment *segments, int count, bool pair, int k, int grid, uint8_t *out, cudaStream_t stream) {
    if (count < 1 || count > 3 || (pair && count != 2) || k % 128 != 0 || grid < 1) return cudaErrorInvalidValue;
    RelayoutArgs args = {};
    args.count = count;
    args.pair = pair ? 1 : 0;
    args.k = k;
    int tiles = 0;
    for (int i = 0; i < count; i++) {
        if (segments[i].rows % 16 != 0) return cudaErrorInvalidValue;
        if (segments[i].rope_head_width > 0 && (segments[i].rope_head_width % 16 != 0 || segments[i].rows % segments[i].rope_head_width != 0))
            return cudaErrorInvalidValue;
        args.segment[i] = segments[i];
        args.first_tile[i] = tiles;
        if (!pair || i == 0) tiles += segments[i].rows / 16;
    }
    if (pair && (segments[0].rows != segments[1].rows || segments[0].rows % 128 != 0)) return cudaErrorInvalidValue;
    args.first_tile[count] = tiles;
    args.schedule = stack_schedule(tiles, k / 128, pair, grid);
    const int passes = (stack_cta_tiles(args.schedule, 0) + args.schedule.slots - 1) / args.schedule.slots;
    if (tiles == 0) return cudaSuccess;
    int4_cta_stream_kernel<<<dim3(passes * args.schedule.steps, grid), 256, 0, stream>>>(args, out);
    return cudaGetLastError();
}

bool decode_stack_supported(const StackShape &shape, int lanes, size_t *smem_bytes) {
    if (lanes < 1 || lanes > 8 || shape.grid < 1) return false;
    if (shape.hidden > 2 * 8 * CONSUMER_THREADS || shape.hidden % 128 != 0 || shape.ffn % 128 != 0 || (shape.q_heads * shape.head_width) % 128 != 0) return false;
    if (((shape.q_heads + 2 * shape.kv_heads) * shape.head_width) % 16 != 0 || shape.kv_heads * 8 > STACK_BARRIER_WORDS - ARRIVAL_WORDS_OFFSET) return false;
    StackPlanSmem plan;
    if (!plan_smem(shape, lanes, shape.grid, &plan)) return false;
    if (smem_bytes) *smem_bytes = plan.total;
    return true;
}

cudaError_t launch_decode_stack(const StackLayer *layers_device, int layer_count, const StackShape &shape,
                                const StackBuffers &buffers, const LaneTable &lanes_meta, int lanes, int lanes_per_stream,
                                int split_tokens, int max_splits, cudaStream_t stream, const StackTp *tp_device, int tp_size) {
    StackPlanSmem plan;
    if (lanes < 1 || lanes > 8 || !plan_smem(shape, lanes, shape.grid, &plan) || lanes_per_stream <= 0 || lanes % lanes_per_stream != 0 ||
        layer_count < 1 || split_tokens != 64 || max_splits > MERGE_BLOCK * MERGE_BLOCK)
        return cudaErrorInvalidValue;
    StackArgs args;
    args.layers = layers_device;
    args.layer_count = layer_count;
    args.shape = shape;
    args.buffers = buffers;
    args.lanes_meta = lanes_meta;
    args.lanes = lanes;
    args.lanes_per_stream = lanes_per_stream;
    args.max_splits = max_splits;
    if (tp_size < 1 || tp_size > STACK_TP_MAX_RANKS || (tp_size > 1 && tp_device == nullptr)) return cudaErrorInvalidValue;
    args.tp = tp_size > 1 ? tp_device : nullptr;
    args.tp_size = tp_size;
    args.stages = plan.stages;
    args.slice_slots = plan.slice_slots;
    args.slice_bytes = plan.slice_bytes;
    args.scratch_bytes = static_cast<uint32_t>(plan.scratch);
    const int group = shape.q_heads / shape.kv_heads;
    if (shape.head_width == 128 && group == 4) return launch_instance<128, 4>(args, plan.total, shape.grid, stream);
    if (shape.head_width == 128 && group == 8) return launch_instance<128, 8>(args, plan.total, shape.grid, stream);
    if (shape.head_width == 64 && group == 4) return launch_instance<64, 4>(args, plan.total, shape.grid, stream);
    return launch_instance<32, 2>(args, plan.total, shape.grid, stream);
}

}  // namespace nerve
