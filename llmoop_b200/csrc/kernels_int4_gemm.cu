// INT4 g128 weight-only linear for batches of more than eight lanes (prefill chunks, many-stream verify and draft
// batches) on the fifth-generation tensor cores: y[m][n] = sum_k x[m][k] * (q[n][k] - 8) * scale[n][k / 128], the
// arithmetic of linear_int4_ct.comp.template:80-150 (tile structure of the reference's prefill kernel:
// linear_batch_cooperative_int4.comp.template:78-212).
//
// Operands.  (q - 8) has at most three significant bits and a bf16 scale eight, so their product fits the eleven of
// fp16 exactly: the weights enter the tensor core as fp16 (q - 8) * scale * 2^p with p chosen per row so that the
// row's largest scale lies in [2^11, 2^12) - exact for every scale down to 2^-29 of the largest, and below that the
// loss is 2^-40 of the row's largest weight.  The activations are bf16 times a power of two chosen per lane so that
// the lane's largest value lies in [2^14, 2^15), as fp16: exact down to 2^-29 of the largest value.  Both powers of
// two come off again in the epilogue.  (Rows whose scales are close together take a cheaper form, dequantise_word_raw, in
// another range of exponents.)  No group scale is left to apply to partial sums, so the f32 accumulator stays
// in tensor memory over the whole of K (one that is read back, scaled and added up in registers for every group of
// 128 columns ran at 140-175 TFLOP/s: the tensor pipe was idle 87 % of the time).  The tensor core truncates its running
// sum, so the longest chain decides the error against 64 bits: before the output's rounding 3e-7 of the output for 16
// lanes of 4096 x 4096, at most 9e-6 (512 lanes of 4096 x 14336), where per-group sums had 1e-7 to 3e-7; of the bf16
// outputs, which their rounding puts 1.66e-3 off, it changes the sixth digit.
//
// Roles.  A CTA computes ROW_TILES x 128 weight rows (M side) by up to 256 / ROW_TILES lanes (N side):
//   8 x ROW_TILES warps bring their rows' packed nibbles into shared memory with cp.async several groups ahead (32 rows x 64
//              bytes per warp and group, private to the warp), turn them into fp16 and write them into tensor memory
//              (tcgen05.st): the A operand never touches shared memory, whose bandwidth the B operand needs;
//   the next warp: one thread issues the MMAs (A from tensor memory, B from shared memory) and commits;
//   the last warp: one thread copies the activations, which prepare_activations_kernel left in global memory in the
//              order of the 128-byte-swizzled shared-memory tiles: two bulk copies per group of 128 columns.
// With ROW_TILES = 2 every activation byte read from L2 feeds two MMAs; stages of half a group make room for 160 lanes there.  K may be split over a cluster of CTAs whose
// partial sums meet through distributed shared memory (shapes with too few tiles to fill the chip).
// Waits are bounded; a wait that expires sets the error word, and the CTA still frees its tensor memory.  No bounded wait
// counts the time of the kernel in front: every role passes the (unbounded) dependency wait before its first wait that
// hangs on the activations, which only then are copied.
#include <cuda_fp16.h>

#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

namespace {

template <int ROW_TILES>
constexpr int gemm_threads() { return ROW_TILES * 256 + 64; }
constexpr unsigned int GEMM_SPIN_LIMIT = 1u << 22;  // tries of 1.5 us
constexpr int GEMM_MAX_B_STAGES = 8, GEMM_MAX_A_STAGES = 4;  // of 64 or 128 columns of K each
constexpr size_t GEMM_SMEM_ONE = 225 * 1024, GEMM_SMEM_TWO = 111 * 1024;  // one or two CTAs per SM
constexpr size_t GEMM_BARRIER_BYTES = 256, GEMM_TAIL_BYTES = GEMM_BARRIER_BYTES + 256 * sizeof(float);  // barriers, lane factors

// Shared-memory matrix descriptor, K-major, 128-byte swizzle: start address / 16 in bits 0-13, 1024 bytes between
// 8-row atoms / 16 in bits 32-45, descriptor version 1 in bits 46-47, swizzle mode 2 (128 bytes) in bits 61-63.
__device__ __forceinline__ uint64_t swizzled_descriptor(uint32_t shared_address) {
    return static_cast<uint64_t>((shared_address & 0x3FFFFu) >> 4) | (1ull << 16) | (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}

__device__ __forceinline__ bool wait_barrier(uint32_t barrier, uint32_t parity, int *error_flag) {
    unsigned int spins = 0;
    while (true) {
        uint32_t done;
        asm volatile(
            "{\n"
            ".reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n"
            "}\n"
            : "=r"(done)
            : "r"(barrier), "r"(parity)
            : "memory");
        if (done) return true;
        if (++spins > GEMM_SPIN_LIMIT) {
            if (error_flag != nullptr) *static_cast<volatile int *>(error_flag) = 3;  // (may be mapped host memory)
            return false;
        }
    }
}
__device__ __forceinline__ void commit_to(uint32_t barrier) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(barrier) : "memory");
}
// One lane of a converged warp.  The issuing warps run their loops as a whole, on values the compiler can keep in uniform
// registers, and only the instructions themselves under this predicate: with the loop inside a one-thread branch every
// MMA operand was moved to a uniform register first, and a group of eight MMAs took 890 cycles to issue instead of 325.
__device__ __forceinline__ bool elect_one() {
    uint32_t elected;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(elected));
    return elected != 0;
}
__device__ __forceinline__ uint32_t shared_address(const void *pointer) { return static_cast<uint32_t>(__cvta_generic_to_shared(pointer)); }

// Half-precision pair arithmetic on 32-bit words.
__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
    uint32_t out;
    asm("mul.rn.f16x2 %0, %1, %2;" : "=r"(out) : "r"(a), "r"(b));
    return out;
}
// The nibbles of `word` as fp16 (q - 8) * scale, pairs (0,4) (1,5) (2,6) (3,7): a nibble in the low mantissa bits of
// 1024 is 1024 + q, one in the next four is 1024 + 16 q; the offset comes off exactly and the product is exact.
__device__ __forceinline__ void dequantise_word(uint32_t word, uint32_t scale2, uint32_t (&out)[4]) {
    const uint32_t shifted = word >> 8;
    uint32_t a, b, c, d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(a) : "r"(word), "n"(0x000F000F), "n"(0x64006400));
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(b) : "r"(word), "n"(0x00F000F0), "n"(0x64006400));
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(c) : "r"(shifted), "n"(0x000F000F), "n"(0x64006400));
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(shifted), "n"(0x00F000F0), "n"(0x64006400));
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(a) : "r"(a), "r"(0x64086408u));                      // - 1032
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(b) : "r"(b), "r"(0x2C002C00u), "r"(0xD480D480u));  // / 16 - 72
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(c) : "r"(c), "r"(0x64086408u));
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(d) : "r"(d), "r"(0x2C002C00u), "r"(0xD480D480u));
    out[0] = mul2(a, scale2);
    out[1] = mul2(b, scale2);
    out[2] = mul2(c, scale2);
    out[3] = mul2(d, scale2);
}

// The same values x 2^-24 in four operations less, from the nibbles where they stand: as fp16 bit patterns they are q x 2^-24
// (x 16 in the next four bits), subnormal and exact, and one fused multiply-add with 2^24 s and -8 s makes (q - 8) s of
// them - exact as long as s keeps its eight bits above 2^-24, that is for rows whose scales lie within a factor of 64.
// (28672 x 8192, rows of either kind: 43.0 and 31.2 us for 16 lanes, 46.5 and 34.5 for 32, 80.5 and 68.0 for 160.)
__device__ __forceinline__ uint32_t fma2(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t out;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(out) : "r"(a), "r"(b), "r"(c));
    return out;
}
__device__ __forceinline__ void dequantise_word_raw(uint32_t word, uint32_t scale2, uint32_t scale2_16th, uint32_t offset2, uint32_t (&out)[4]) {
    const uint32_t shifted = word >> 8;
    out[0] = fma2(word & 0x000F000Fu, scale2, offset2);
    out[1] = fma2(word & 0x00F000F0u, scale2_16th, offset2);
    out[2] = fma2(shifted & 0x000F000Fu, scale2, offset2);
    out[3] = fma2(shifted & 0x00F000F0u, scale2_16th, offset2);
}

// A power of two as f32 from its biased exponent.
__device__ __forceinline__ float power_of_two(int biased_exponent) { return __uint_as_float(static_cast<uint32_t>(biased_exponent) << 23); }

struct GemmArgs {
    const uint8_t *x;          // prepared activations: [k / 64][lane block of 8] atoms of 1024 bytes
    const float *x_factor;     // [lanes] power of two that undoes the lane's scaling
    const uint32_t *qweights[3];  // up to three matrices that share the activations (q, k, v; gate, up) in one launch:
    const uint16_t *scale_rows[3];
    void *ys[3];
    int ns[3];
    int first_tile[4];         // ... matrix b owns the 128-row tiles first_tile[b] .. first_tile[b + 1] - 1
    const uint16_t *residual;
    int lanes, lane_blocks, tile_lanes, k, epilogue, silu, paired;
    float scale;
    int *error_flag;
    int a_stages, b_stages, raw_stages;
    uint32_t tmem_columns, barrier_offset;
};

// Which 32 rows a quarter of a row tile holds: the matrix and the first row.  A SiLU pair (matrix 0 gate, 1 up, equal
// shapes) takes the same rows of both: as two row tiles, or as the two halves of one.
template <int ROW_TILES>
__device__ __forceinline__ void locate_rows(const GemmArgs &a, int block_tile, int row_tile, int quarter, int &matrix, int &row) {
    if (a.silu) {
        if (ROW_TILES == 2) {
            matrix = row_tile;
            row = block_tile * 128 + quarter * 32;
        } else {
            matrix = quarter >> 1;
            row = block_tile * 64 + (quarter & 1) * 32;
        }
        return;
    }
    const int tile = block_tile * ROW_TILES + row_tile;
    matrix = 0;
    row = 1 << 30;
    if (tile >= a.first_tile[3]) return;  // the odd tile out: repeats the last row, nothing of it is stored
    while (matrix < 2 && tile >= a.first_tile[matrix + 1]) matrix++;
    row = (tile - a.first_tile[matrix]) * 128 + quarter * 32;
}

// PARTS: stages of both operands to a group of 128 columns (1 or 2).  Half groups leave tensor memory for two row tiles of
// 129 to 160 lanes: 28672 x 8192 with 160 lanes is one wave then instead of two (82 -> 72 us), 28672 x 4096 with 2048 lanes
// seven instead of eleven waves of 256 lanes (490 -> 407 us).
template <int ROW_TILES, int PARTS>
__global__ void __launch_bounds__(gemm_threads<ROW_TILES>(), ROW_TILES == 1 ? 2 : 1) linear_int4_gemm_kernel(const __grid_constant__ GemmArgs a) {
    constexpr int ROWS = 128 * ROW_TILES, WARPS = 8 * ROW_TILES;  // warps that prepare the A operand: two sets, one for every other group
    constexpr uint32_t SLOT = WARPS * 2048;                         // one raw stage: 32 rows x 64 bytes of every such warp
    extern __shared__ __align__(1024) uint8_t smem[];
    // [B stages][raw nibbles of eight warps][row scales][barriers]; the f32 partial sums take the front in the end
    const int splits = gridDim.z, split = blockIdx.z;
    const int groups = a.k >> 7, first_group = groups * split / splits, own_groups = groups * (split + 1) / splits - first_group;
    const int m0 = blockIdx.x * a.tile_lanes;
    const int n_lanes = min(a.tile_lanes, a.lane_blocks * 8 - m0);  // multiple of 16
    constexpr uint32_t A_COLUMNS = 64 / PARTS;  // of tensor memory, per stage and row tile
    const uint32_t b_stage_bytes = static_cast<uint32_t>(a.tile_lanes) * (256 / PARTS);
    uint8_t *const raw = smem + static_cast<size_t>(a.b_stages) * b_stage_bytes;
    uint16_t *const scales = reinterpret_cast<uint16_t *>(raw + a.raw_stages * SLOT);
    const uint32_t a_full = shared_address(smem) + a.barrier_offset, a_empty = a_full + 8 * GEMM_MAX_A_STAGES, b_full = a_empty + 8 * GEMM_MAX_A_STAGES,
                   b_empty = b_full + 8 * GEMM_MAX_B_STAGES, all_done = b_empty + 8 * GEMM_MAX_B_STAGES, tmem_slot = all_done + 8;
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp: uniform
    grid_launch_dependents();

    if (threadIdx.x == 0) {
        for (int s = 0; s < GEMM_MAX_A_STAGES; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(a_full + s * 8), "r"(4 * ROW_TILES) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a_empty + s * 8) : "memory");
        }
        for (int s = 0; s < GEMM_MAX_B_STAGES; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_full + s * 8) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(b_empty + s * 8) : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(all_done) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(a.tmem_columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
    tmem = __reduce_or_sync(0xffffffffu, tmem);  // a uniform register
    const uint32_t d_stride = (static_cast<uint32_t>(a.tile_lanes) + 31u) & ~31u, tmem_a = tmem + ROW_TILES * d_stride;

    bool alive = true;
    float row_factor = 1.0f;  // operand warps: the power of two that undoes the row's scaling
    const int quarter = warp & 3, row_tile = (warp >> 2) % ROW_TILES, set = warp / (4 * ROW_TILES);
    if (warp < WARPS) {
        int matrix, row0;
        locate_rows<ROW_TILES>(a, blockIdx.y, row_tile, quarter, matrix, row0);
        const int n = a.ns[matrix];
        const int items = (own_groups - set + 1) / 2;  // groups set, set + 2, ...
        // cp.async: four neighbouring threads bring the 64 bytes of one row; the chunk's place is swizzled with the row
        const uint8_t *source[4];
        uint32_t destination[4];
        const uint32_t warp_raw = shared_address(raw) + static_cast<uint32_t>(warp) * 2048;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int r = (lane >> 2) + 8 * i, global_row = min(row0 + r, n - 1);
            source[i] = reinterpret_cast<const uint8_t *>(a.qweights[matrix]) + static_cast<size_t>(global_row) * (a.k >> 1) +
                        static_cast<size_t>(first_group) * 64 + (lane & 3) * 16;
            destination[i] = warp_raw + static_cast<uint32_t>(r * 64 + (((lane & 3) ^ ((r >> 1) & 3)) * 16));
        }
        int requested = 0;            // items asked for so far
        uint32_t request_slot = 0;    // ... and the slot of the next one, in bytes
        const uint32_t slots_end = static_cast<uint32_t>(a.raw_stages) * SLOT;
        auto request = [&]() {
            if (requested < items) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(destination[i] + request_slot), "l"(source[i]) : "memory");
                    source[i] += 128;
                }
                requested++;
                request_slot = request_slot + SLOT == slots_end ? 0 : request_slot + SLOT;
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
#pragma unroll
        for (int i = 0; i < 4; i++) source[i] += set * 64;
        for (int item = 0; item < a.raw_stages - 1; item++) request();
        // the row's scales into shared memory ([group][row], read by this thread alone) and their largest exponent
        float factor;
        bool raw_operands;  // of all the warp's rows: their largest scale enters as [2^14, 2^15) x 2^-24
        {
            const uint16_t *row_scales = a.scale_rows[matrix] + static_cast<size_t>(min(row0 + lane, n - 1)) * groups + first_group;
            uint16_t *const own = scales + row_tile * 128 + quarter * 32 + lane;
            uint32_t largest = 16u << 7, smallest = 0x7FFFu;  // of the magnitudes that are not zero
            auto note = [&](uint32_t bits) {
                const uint32_t magnitude = bits & 0x7FFFu;
                largest = max(largest, magnitude);
                smallest = min(smallest, magnitude == 0 ? 0x7FFFu : magnitude);
            };
            if (groups % 8 == 0 && own_groups % 8 == 0 && (reinterpret_cast<uintptr_t>(row_scales) & 15) == 0) {
                constexpr int BATCH = 4;  // 16-byte loads in flight
                for (int g = 0; g < own_groups; g += 8 * BATCH) {
                    uint4 eight[BATCH];
#pragma unroll
                    for (int i = 0; i < BATCH; i++)
                        if (g + 8 * i < own_groups) eight[i] = __ldg(reinterpret_cast<const uint4 *>(row_scales + g + 8 * i));
#pragma unroll
                    for (int i = 0; i < BATCH; i++) {
                        if (g + 8 * i >= own_groups) break;
                        const uint32_t words[4] = {eight[i].x, eight[i].y, eight[i].z, eight[i].w};
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const uint32_t bits = (words[j >> 1] >> (16 * (j & 1))) & 0xFFFFu;
                            note(bits);
                            own[(g + 8 * i + j) * ROWS] = static_cast<uint16_t>(bits);
                        }
                    }
                }
            } else {
#pragma unroll 8
                for (int g = 0; g < own_groups; g++) {
                    const uint16_t bits = __ldg(row_scales + g);
                    note(bits);
                    own[g * ROWS] = bits;
                }
            }
            const int exponent = static_cast<int>(largest >> 7);
            raw_operands = __all_sync(0xffffffffu, static_cast<int>(smallest >> 7) + 6 >= exponent && exponent <= 244);
            factor = power_of_two(raw_operands ? 268 - exponent : min(265 - exponent, 254));
            row_factor = power_of_two(raw_operands ? exponent + 10 : max(exponent - 11, 1));
        }
        const uint32_t read_base = warp_raw + static_cast<uint32_t>(lane * 64);
        const uint32_t read_swizzle = static_cast<uint32_t>((lane >> 1) & 3);
        const uint32_t tmem_rows = tmem_a + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(row_tile) * A_COLUMNS;
        const uint16_t *scale = scales + set * ROWS + row_tile * 128 + quarter * 32 + lane;
        uint32_t read_slot = 0;
        // ring position of the item's group among the A stages, and the parity of its last release (the first round waits for none)
        int stage = set * PARTS;
        uint32_t parity = 1;
        bool first_round = true;
        auto advance = [&](int by) {
            stage += by;
            if (stage >= a.a_stages) {
                stage -= a.a_stages;
                parity ^= 1;
                if (first_round) grid_dependency_wait();  // from here on the MMAs release the stages
                first_round = false;
            }
        };
        auto prepare = [&](auto raw) {
            for (int item = 0; item < items; item++) {
                request();
                switch (a.raw_stages) {  // the item's own copies have landed
                case 3: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
                case 4: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
                case 5: asm volatile("cp.async.wait_group 4;" ::: "memory"); break;
                default: asm volatile("cp.async.wait_group 5;" ::: "memory"); break;
                }
                __syncwarp();
                uint32_t scale2 = __half_as_ushort(__float2half_rn(bf16_bits_to_f32(*scale) * factor));
                scale2 |= scale2 << 16;
                scale += 2 * ROWS;
                uint4 words[4];
#pragma unroll
                for (int c = 0; c < 4; c++) {
                    const uint32_t address = read_base + read_slot + ((static_cast<uint32_t>(c) ^ read_swizzle) * 16);
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(words[c].x), "=r"(words[c].y), "=r"(words[c].z), "=r"(words[c].w) : "r"(address));
                }
                read_slot = read_slot + SLOT == slots_end ? 0 : read_slot + SLOT;
                const uint32_t scale2_16th = mul2(scale2, 0x2C002C00u), offset2 = mul2(scale2, 0x80088008u);  // s / 16; -2^-21 s
#pragma unroll
                for (int part = 0; part < PARTS; part++) {
                    if (alive && !wait_barrier(a_empty + stage * 8, parity, a.error_flag)) alive = false;
                    if (!alive) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t target = tmem_rows + static_cast<uint32_t>(stage) * (A_COLUMNS * ROW_TILES);
#pragma unroll
                    for (int c = 0; c < 4 / PARTS; c++) {
                        const uint4 packed = words[part * (4 / PARTS) + c];
                        uint32_t v[4][4];
                        const uint32_t four[4] = {packed.x, packed.y, packed.z, packed.w};
#pragma unroll
                        for (int w = 0; w < 4; w++) {
                            if (raw) dequantise_word_raw(four[w], scale2, scale2_16th, offset2, v[w]);
                            else dequantise_word(four[w], scale2, v[w]);
                        }
                        asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(target + c * 16),
                                     "r"(v[0][0]), "r"(v[0][1]), "r"(v[0][2]), "r"(v[0][3]), "r"(v[1][0]), "r"(v[1][1]), "r"(v[1][2]), "r"(v[1][3]), "r"(v[2][0]),
                                     "r"(v[2][1]), "r"(v[2][2]), "r"(v[2][3]), "r"(v[3][0]), "r"(v[3][1]), "r"(v[3][2]), "r"(v[3][3])
                                     : "memory");
                    }
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(a_full + stage * 8) : "memory");
                    advance(part + 1 < PARTS ? 1 : PARTS + 1);  // over the other set's group
                }
                if (!alive) break;
            }
        };
        if (raw_operands) prepare(std::true_type{});
        else prepare(std::false_type{});
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp == WARPS) {
        // instruction descriptor: f32 accumulator, A and B fp16, both K-major, N / 8 in bits 17-22, M / 16 in bits 24-28
        const uint32_t instruction = (1u << 4) | (static_cast<uint32_t>(n_lanes / 8) << 17) | (8u << 24);
        const uint64_t b_first = swizzled_descriptor(shared_address(smem)), b_half = static_cast<uint64_t>(n_lanes) * 8;  // descriptors count 16 bytes
        int stage_a = 0, stage_b = 0;
        uint32_t parity_a = 0, parity_b = 0;
        grid_dependency_wait();
        for (int part = 0; part < own_groups * PARTS; part++) {
            if (!wait_barrier(b_full + stage_b * 8, parity_b, a.error_flag) || !wait_barrier(a_full + stage_a * 8, parity_a, a.error_flag)) {
                alive = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            if (elect_one()) {
                const uint64_t b_stage = b_first + static_cast<uint64_t>(stage_b) * (b_stage_bytes >> 4);
#pragma unroll
                for (int t = 0; t < ROW_TILES; t++) {
                    const uint32_t d_address = tmem + t * d_stride, a_address = tmem_a + static_cast<uint32_t>(stage_a * ROW_TILES + t) * A_COLUMNS;
#pragma unroll
                    for (int step = 0; step < 8 / PARTS; step++) {  // K = 16 per instruction; four steps to a 128-byte row of the swizzled tile
                        const uint64_t b_descriptor = b_stage + (step >> 2) * b_half + (step & 3) * 2;
                        const uint32_t accumulate = (part > 0 || step > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n"
                            ".reg .pred p;\n"
                            "setp.ne.b32 p, %4, 0;\n"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
                            "}\n" ::"r"(d_address),
                            "r"(a_address + step * 8), "l"(b_descriptor), "r"(instruction), "r"(accumulate)
                            : "memory");
                    }
                }
                commit_to(a_empty + stage_a * 8);
                commit_to(b_empty + stage_b * 8);
            }
            __syncwarp();
            if (++stage_a == a.a_stages) {
                stage_a = 0;
                parity_a ^= 1;
            }
            if (++stage_b == a.b_stages) {
                stage_b = 0;
                parity_b ^= 1;
            }
        }
        if (elect_one()) commit_to(all_done);
        __syncwarp();
    } else {
        grid_dependency_wait();
        const uint8_t *source = a.x + static_cast<size_t>(2 * first_group) * a.lane_blocks * 1024 + static_cast<size_t>(m0 >> 3) * 1024;
        const size_t part_bytes = static_cast<size_t>(a.lane_blocks) * 1024;
        const uint32_t bytes = static_cast<uint32_t>(n_lanes) * 128;
        int stage = 0;
        uint32_t parity = 1;  // the first round waits for no release
        for (int item = 0; item < own_groups * PARTS; item++) {
            if (!wait_barrier(b_empty + stage * 8, parity, a.error_flag)) {
                for (int g = item > a.b_stages ? item - a.b_stages : 0; g < item; g++)  // the copies in flight land before the CTA gives its memory up
                    wait_barrier(b_full + (g % a.b_stages) * 8, static_cast<uint32_t>((g / a.b_stages) & 1), a.error_flag);
                break;
            }
            if (elect_one()) {
                const uint32_t target = shared_address(smem) + static_cast<uint32_t>(stage) * b_stage_bytes, full = b_full + stage * 8;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full), "r"(2 / PARTS * bytes) : "memory");
#pragma unroll
                for (int part = 0; part < 2 / PARTS; part++)
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(target + part * bytes),
                                 "l"(source + static_cast<size_t>(part) * part_bytes), "r"(bytes), "r"(full)
                                 : "memory");
            }
            __syncwarp();
            source += 2 / PARTS * part_bytes;
            if (++stage == a.b_stages) {
                stage = 0;
                parity ^= 1;
            }
        }
    }
    __syncwarp();
    grid_dependency_wait();  // outputs may be inputs of the kernel in front

    // ---- accumulators -> f32 [lane][row] in shared memory (every copy and MMA that used it is done by then)
    float *const sums = reinterpret_cast<float *>(smem);
    float *const factors = reinterpret_cast<float *>(smem + a.barrier_offset + GEMM_BARRIER_BYTES);
    if (threadIdx.x < n_lanes && m0 + static_cast<int>(threadIdx.x) < a.lanes) factors[threadIdx.x] = a.x_factor[m0 + threadIdx.x];
    if (warp < WARPS) {
        if (!wait_barrier(all_done, 0u, a.error_flag)) alive = false;
    }
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp < WARPS && alive) {  // the two sets share the lanes; both know the row's factor
        const int local_row = row_tile * 128 + quarter * 32 + lane;
        for (int column = set * 16; column < n_lanes; column += 32) {
            uint32_t d[16];
            asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                         : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]),
                           "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
                         : "r"(tmem + (static_cast<uint32_t>(quarter * 32) << 16) + row_tile * d_stride + static_cast<uint32_t>(column))
                         : "memory");
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int i = 0; i < 16; i++) sums[(column + i) * ROWS + local_row] = __uint_as_float(d[i]) * row_factor;
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(a.tmem_columns) : "memory");
    const bool good = __syncthreads_and(alive ? 1 : 0) != 0;
    if (splits > 1) {
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }

    // ---- outputs: this CTA's share of the tile's lanes; a thread keeps two neighbouring rows and walks the lanes
    const int lane_begin = n_lanes * split / splits, lane_end = min(n_lanes * (split + 1) / splits, a.lanes - m0);
    const int pairs = a.silu ? ROWS / 4 : ROWS / 2, r = (threadIdx.x & (pairs - 1)) * 2;  // pairs is a power of two
    int matrix, row;
    locate_rows<ROW_TILES>(a, blockIdx.y, r >> 7, (r >> 5) & 3, matrix, row);
    row += r & 31;
    const int n = a.ns[matrix];
    if (good && threadIdx.x < WARPS * 32 && row < n) {
        auto pair_sum = [&](int m, int at) {
            if (splits == 1) return *reinterpret_cast<const float2 *>(sums + m * ROWS + at);
            // every split's share is asked for before the first one is added: one round trip to the peers instead of one each
            float2 part[8];
            const uint32_t local = shared_address(sums + m * ROWS + at);
#pragma unroll
            for (int s = 0; s < 8; s++) {
                if (s >= splits) break;
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(s));
                asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(part[s].x), "=f"(part[s].y) : "r"(remote));
            }
            float2 sum = part[0];
#pragma unroll
            for (int s = 1; s < 8; s++) {
                if (s >= splits) break;
                sum.x += part[s].x;
                sum.y += part[s].y;
            }
            return sum;
        };
        const bool whole = a.paired && (n & 1) == 0;  // both rows exist and their outputs share an aligned word
        const bool second_row = row + 1 < n;
        const int step = WARPS * 32 / pairs;
        constexpr int BATCH = 8;
        for (int m = lane_begin + static_cast<int>(threadIdx.x) / pairs; m < lane_end; m += step * BATCH) {
            float2 sum[BATCH], other[BATCH];  // other: the up rows of a SiLU pair, or the residual
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int mi = m + i * step;
                if (mi >= lane_end) break;
                sum[i] = pair_sum(mi, r);
                other[i] = make_float2(0.0f, 0.0f);
                if (a.silu) {
                    other[i] = pair_sum(mi, r + ROWS / 2);
                } else if (a.residual != nullptr) {
                    const uint16_t *residual = a.residual + static_cast<size_t>(m0 + mi) * n + row;
                    if (whole) {
                        const uint32_t both = *reinterpret_cast<const uint32_t *>(residual);
                        other[i] = make_float2(bf16_lo(both), bf16_hi(both));
                    } else {
                        other[i].x = bf16_bits_to_f32(residual[0]);
                        if (second_row) other[i].y = bf16_bits_to_f32(residual[1]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < BATCH; i++) {
                const int mi = m + i * step;
                if (mi >= lane_end) break;
                const float factor = factors[mi];
                const size_t out = static_cast<size_t>(m0 + mi) * n + row;
                float first = sum[i].x * factor, second = sum[i].y * factor;
                if (a.epilogue == EPILOGUE_F32_SCALED) {
                    float *y = static_cast<float *>(a.ys[matrix]) + out;
                    y[0] = first * a.scale;
                    if (second_row) y[1] = second * a.scale;
                    continue;
                }
                if (a.silu) {
                    first = rounded_silu(round_bf16(first)) * round_bf16(other[i].x * factor);
                    second = rounded_silu(round_bf16(second)) * round_bf16(other[i].y * factor);
                } else if (a.residual != nullptr) {
                    first = (a.epilogue == EPILOGUE_RESIDUAL_ROUNDED ? round_bf16(first) : first) + other[i].x;
                    second = (a.epilogue == EPILOGUE_RESIDUAL_ROUNDED ? round_bf16(second) : second) + other[i].y;
                }
                uint16_t *y = static_cast<uint16_t *>(a.ys[matrix]) + out;
                if (whole) {
                    *reinterpret_cast<uint32_t *>(y) = pack_bf16(first, second);
                } else {
                    y[0] = static_cast<uint16_t>(f32_to_bf16_bits(first));
                    if (second_row) y[1] = static_cast<uint16_t>(f32_to_bf16_bits(second));
                }
            }
        }
    }
    if (splits > 1) {  // nobody leaves while a peer may still read its sums
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

// bf16 [lanes][k] -> fp16 x 2^e in the GEMM's tile order, one CTA per lane (lanes beyond the batch are zero): largest
// magnitude of the row, then the conversion; a 16-byte piece of eight columns holds them in the order (0,4)(1,5)(2,6)
// (3,7) the nibble pairs come out in, at its swizzled place in the 8-lane x 64-column atom.  With NORM the row is the
// RMSNorm of x (rms_norm_bf16.comp.template:49-72), kept in shared memory between its two passes.
// HELD: 16-byte pieces of the row per thread, kept in registers (0: any number, kept in shared memory or read again); the
// norm's weights are nobody's output and are on their way while the kernel in front still runs (32 x 4096: 4.1 -> 2.7 us).
constexpr int PREPARE_THREADS = 512;
template <bool NORM, int HELD>
__global__ void __launch_bounds__(PREPARE_THREADS) prepare_activations_kernel(const uint16_t *__restrict__ x, const uint16_t *__restrict__ weight, float eps,
                                                                             float weight_offset, uint8_t *__restrict__ out, float *__restrict__ factors, int lanes,
                                                                             int lane_blocks, int k) {
    constexpr int WARPS = PREPARE_THREADS / 32, REGISTERS = HELD > 0 ? HELD : 1;
    extern __shared__ __align__(16) uint4 normalised[];
    __shared__ float warp_sums[WARPS];
    __shared__ uint32_t warp_largest[WARPS];
    const int m = blockIdx.x, pieces = k >> 3;
    uint4 held[REGISTERS], weights[REGISTERS];
    auto each_piece = [&](auto body) {  // body(register, piece)
        if (HELD > 0) {
#pragma unroll
            for (int i = 0; i < REGISTERS; i++)
                if (static_cast<int>(threadIdx.x) + i * PREPARE_THREADS < pieces) body(i, static_cast<int>(threadIdx.x) + i * PREPARE_THREADS);
        } else {
            for (int p = threadIdx.x; p < pieces; p += PREPARE_THREADS) body(0, p);
        }
    };
    grid_launch_dependents();
    if (NORM && HELD > 0) each_piece([&](int i, int p) { weights[i] = __ldg(reinterpret_cast<const uint4 *>(weight) + p); });
    grid_dependency_wait();
    const uint4 *row = reinterpret_cast<const uint4 *>(x + static_cast<size_t>(m) * k);
    uint32_t largest = 0;
    auto note = [&](const uint4 &v) {
        const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int i = 0; i < 4; i++) largest = max(largest, max((words[i] & 0x7FFFu), (words[i] >> 16) & 0x7FFFu));
    };
    if (m < lanes) {
        if (HELD > 0) each_piece([&](int i, int p) { held[i] = row[p]; });
        if (NORM) {
            float sum = 0.0f;
            each_piece([&](int i, int p) {
                const uint4 v = HELD > 0 ? held[i] : row[p];
                if (HELD == 0) normalised[p] = v;
                const uint32_t words[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    sum = fmaf(bf16_lo(words[w]), bf16_lo(words[w]), sum);
                    sum = fmaf(bf16_hi(words[w]), bf16_hi(words[w]), sum);
                }
            });
            sum = warp_sum(sum);
            if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = sum;
            __syncthreads();
            float total = 0.0f;
#pragma unroll
            for (int w = 0; w < WARPS; w++) total += warp_sums[w];
            const float inv_rms = 1.0f / sqrtf(total * (1.0f / static_cast<float>(k)) + eps);
            each_piece([&](int i, int p) {
                const uint4 v = HELD > 0 ? held[i] : normalised[p], w = HELD > 0 ? weights[i] : reinterpret_cast<const uint4 *>(weight)[p];
                auto norm = [&](uint32_t value, uint32_t factor) {
                    return pack_bf16(bf16_lo(value) * inv_rms * (bf16_lo(factor) + weight_offset), bf16_hi(value) * inv_rms * (bf16_hi(factor) + weight_offset));
                };
                const uint4 y = make_uint4(norm(v.x, w.x), norm(v.y, w.y), norm(v.z, w.z), norm(v.w, w.w));
                if (HELD > 0) held[i] = y;
                else normalised[p] = y;
                note(y);
            });
        } else {
            each_piece([&](int i, int p) { note(HELD > 0 ? held[i] : row[p]); });
        }
        largest = __reduce_max_sync(0xffffffffu, largest);
        if ((threadIdx.x & 31) == 0) warp_largest[threadIdx.x >> 5] = largest;
        __syncthreads();
#pragma unroll
        for (int w = 0; w < WARPS; w++) largest = max(largest, warp_largest[w]);
    }
    const int exponent = max(static_cast<int>(largest >> 7), 16);
    const float factor = power_of_two(min(268 - exponent, 254));
    if (m < lanes && threadIdx.x == 0) factors[m] = power_of_two(max(exponent - 14, 1));
    each_piece([&](int i, int p) {
        uint4 packed = make_uint4(0, 0, 0, 0);
        if (m < lanes) {
            const uint4 v = HELD > 0 ? held[i] : NORM ? normalised[p] : row[p];
            auto both = [&](uint32_t lo, uint32_t hi) {
                const __half2 h = __floats2half2_rn(__uint_as_float(lo) * factor, __uint_as_float(hi) * factor);
                return *reinterpret_cast<const uint32_t *>(&h);
            };
            packed.x = both(v.x << 16, v.z << 16);
            packed.y = both(v.x & 0xffff0000u, v.z & 0xffff0000u);
            packed.z = both(v.y << 16, v.w << 16);
            packed.w = both(v.y & 0xffff0000u, v.w & 0xffff0000u);
        }
        *reinterpret_cast<uint4 *>(out + (static_cast<size_t>(p >> 3) * lane_blocks + (m >> 3)) * 1024 + (m & 7) * 128 + (((p & 7) ^ (m & 7)) * 16)) = packed;
    });
}
template <bool NORM>
auto prepare_kernel(int k) {
    const int pieces = k / 8;
    return pieces <= PREPARE_THREADS ? prepare_activations_kernel<NORM, 1> : pieces <= 2 * PREPARE_THREADS ? prepare_activations_kernel<NORM, 2>
           : pieces <= 4 * PREPARE_THREADS ? prepare_activations_kernel<NORM, 4> : prepare_activations_kernel<NORM, 0>;
}

struct GemmPlan {
    int row_tiles = 1, parts = 1, lane_tiles = 1, tile_lanes = 16, splits = 1, a_stages = 2, b_stages = 2, raw_stages = 3;
    uint32_t tmem_columns = 512;
    size_t smem = 0;
};

// Tile shape and K split by an estimate of the launch's time in SM cycles, fitted to the times of every plan at 84 points
// (16 .. 2048 lanes of six matrices from 4096 x 4096 to 28672 x 8192; the plan it takes is 2 % slower than the best one on
// average, an estimate without the dequantisation's latency took 7 %).  Per group of 128 columns a CTA needs 5.6 cycles per
// lane and row tile on the tensor cores (4 at the pipe's nominal rate) or the time of its operand warps, which wait more
// than they work: two CTAs of an SM do not slow one another down.  A wave that is not full costs as much as a full one, and
// every CTA pays for filling its pipeline and for its epilogue, split ones for meeting their peers.  The number of splits goes
// with the lanes of the launch, and with it the order of a lane's sums: from nine lanes on a lane's last bits depend on what
// shares its batch.  (Splits by the matrix alone would cost 6 % of an 8B layer's GEMM time at 512 lanes and 14 % at 32, by
// this estimate.)
GemmPlan plan_gemm(int matrix_tiles, int lanes, int groups, bool silu) {
    const int sms = multiprocessors();
    const int padded = (lanes + 15) / 16 * 16;
    GemmPlan best;
    double best_cycles = 1e30;
    for (int form = 0; form < 3; form++) {
        const int row_tiles = form == 0 ? 1 : 2, parts = form == 2 ? 2 : 1;
        const int most = form == 0 ? 256 : form == 1 ? 128 : 160;
        const int fewest_tiles = (padded + most - 1) / most;
        // (a SiLU pair covers 64 rows of both matrices per row tile)
        const int blocks = silu ? (row_tiles == 2 ? matrix_tiles / 2 : matrix_tiles) : (matrix_tiles + row_tiles - 1) / row_tiles;
        for (int lane_tiles = fewest_tiles; lane_tiles <= fewest_tiles + 2; lane_tiles++) {
            const int tile_lanes = ((padded + lane_tiles - 1) / lane_tiles + 15) / 16 * 16;
            if (tile_lanes > most || (form == 2 && tile_lanes <= 128) || (lane_tiles > 1 && tile_lanes * (lane_tiles - 1) >= padded)) continue;
            for (int splits = 1; splits <= 8 && (splits == 1 || splits * 2 <= groups); splits *= 2) {
                const int own = (groups + splits - 1) / splits;
                GemmPlan plan;
                plan.row_tiles = row_tiles;
                plan.parts = parts;
                plan.lane_tiles = lane_tiles;
                plan.tile_lanes = tile_lanes;
                plan.splits = splits;
                const size_t scales = static_cast<size_t>(own) * 256 * row_tiles, b_stage = static_cast<size_t>(tile_lanes) * (256 / parts);
                const size_t sums = static_cast<size_t>(tile_lanes) * 512 * row_tiles;
                int per_sm = 0;
                for (int share = row_tiles == 1 && tile_lanes <= 64 ? 2 : 1; share >= 1 && per_sm == 0; share--) {
                    const size_t limit = share == 2 ? GEMM_SMEM_TWO : GEMM_SMEM_ONE;
                    // stages: the pair that looks furthest ahead, counted in stages of B, on its shorter side (a raw slot holds
                    // two groups, and the one being read does not count)
                    int best_ahead = 0;
                    for (int raw = 3; raw <= 6; raw++)
                        for (int b = 2; b <= GEMM_MAX_B_STAGES; b++) {
                            const size_t bytes = std::max(static_cast<size_t>(b) * b_stage + static_cast<size_t>(raw) * 16384 * row_tiles + scales, sums);
                            const int ahead = std::min(2 * parts * (raw - 1), b);
                            if (bytes > limit || ahead <= best_ahead) continue;
                            best_ahead = ahead;
                            plan.b_stages = b;
                            plan.raw_stages = raw;
                            plan.smem = bytes;
                            per_sm = share;
                        }
                }
                if (per_sm == 0) continue;
                const int d_columns = (tile_lanes + 31) / 32 * 32 * row_tiles;
                plan.tmem_columns = per_sm == 2 ? 256 : 512;
                plan.a_stages = std::min(GEMM_MAX_A_STAGES, (static_cast<int>(plan.tmem_columns) - d_columns) / (64 / parts * row_tiles));
                if (plan.a_stages < parts + 1) continue;
                const int ctas = blocks * lane_tiles * splits, together = ctas > sms ? per_sm : 1;
                const double dequantise = row_tiles == 2 ? 430.0 : together == 2 ? 350.0 : 680.0;
                const double per_group = 200.0 + row_tiles * std::max(5.6 * tile_lanes, dequantise);
                const int waves = (ctas + sms * per_sm - 1) / (sms * per_sm);
                const double cycles = waves * (own * per_group * together + 7700.0 + 25.0 * row_tiles * tile_lanes) +
                                      (splits > 1 ? 650.0 * splits + 25.0 * row_tiles * tile_lanes : 0.0);
                if (cycles < best_cycles) {
                    best_cycles = cycles;
                    best = plan;
                }
            }
        }
    }
    return best;
}

}  // namespace

bool linear_int4_gemm_supported(int lanes, int n, int k) { return lanes > 8 && k % 128 == 0 && k >= 128 && n >= 1; }

size_t int4_activation_bytes(int lanes, int k) {
    const size_t padded = static_cast<size_t>(lanes + 15) / 16 * 16;
    return padded * k * 2 + padded * sizeof(float);
}

static float *activation_factors(void *prepared, int lanes, int k) {
    const size_t padded = static_cast<size_t>(lanes + 15) / 16 * 16;
    return reinterpret_cast<float *>(static_cast<uint8_t *>(prepared) + padded * k * 2);
}

cudaError_t launch_prepare_activations(const uint16_t *x, void *prepared, int lanes, int k, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    const int padded = (lanes + 15) / 16 * 16;
    return launch_dependent(prepare_kernel<false>(k), dim3(padded), dim3(PREPARE_THREADS), 0, 1, stream, x, static_cast<const uint16_t *>(nullptr), 0.0f,
                            0.0f, static_cast<uint8_t *>(prepared), activation_factors(prepared, lanes, k), lanes, padded / 8, k);
}

cudaError_t launch_rms_norm_prepared(const uint16_t *x, const uint16_t *weight, void *prepared, int lanes, int width, float eps, float weight_offset,
                                     cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    const int padded = (lanes + 15) / 16 * 16;
    auto kernel = prepare_kernel<true>(width);
    const size_t smem = width / 8 <= 4 * PREPARE_THREADS ? 0 : static_cast<size_t>(width) * 2;
    if (smem > 48 * 1024) {
        cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (status != cudaSuccess) return status;
    }
    return launch_dependent(kernel, dim3(padded), dim3(PREPARE_THREADS), smem, 1, stream, x, weight, eps, weight_offset,
                            static_cast<uint8_t *>(prepared), activation_factors(prepared, lanes, width), lanes, padded / 8, width);
}

cudaError_t launch_linear_int4_gemm(const void *prepared, int branches, const uint32_t *const *qweights, const uint16_t *const *scales, void *const *ys,
                                    const int *ns, const uint16_t *residual, int lanes, int k, int epilogue, float scale, bool silu, int *error_flag,
                                    cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (branches < 1 || branches > 3 || (residual != nullptr && branches != 1) || (silu && (branches != 2 || ns[0] != ns[1]))) return cudaErrorInvalidValue;
    GemmArgs args = {};
    int tiles = 0;
    for (int b = 0; b < 3; b++) {
        const int source = b < branches ? b : branches - 1;
        if (b < branches && !linear_int4_gemm_supported(lanes, ns[b], k)) return cudaErrorInvalidValue;
        args.qweights[b] = qweights[source];
        args.scale_rows[b] = scales[source];
        args.ys[b] = ys[source];
        args.ns[b] = ns[source];
        args.first_tile[b] = tiles;
        if (b < branches) tiles += (ns[b] + 127) / 128;
    }
    args.first_tile[3] = tiles;
    for (int b = branches; b < 3; b++) args.first_tile[b] = tiles;  // no tile belongs to an absent matrix ...
    const GemmPlan plan = plan_gemm(tiles, lanes, k >> 7, silu);
    if (plan.smem == 0) return cudaErrorInvalidValue;
    args.x = static_cast<const uint8_t *>(prepared);
    args.x_factor = activation_factors(const_cast<void *>(prepared), lanes, k);
    args.residual = residual;
    args.lanes = lanes;
    args.lane_blocks = (lanes + 15) / 16 * 2;
    args.tile_lanes = plan.tile_lanes;
    args.k = k;
    args.epilogue = epilogue;
    args.silu = silu ? 1 : 0;
    uintptr_t addresses = reinterpret_cast<uintptr_t>(residual);
    for (int b = 0; b < branches; b++) addresses |= reinterpret_cast<uintptr_t>(ys[b]);
    args.paired = addresses % 4 == 0 ? 1 : 0;
    args.scale = scale;
    args.error_flag = error_flag;
    args.a_stages = plan.a_stages;
    args.b_stages = plan.b_stages;
    args.raw_stages = plan.raw_stages;
    args.tmem_columns = plan.tmem_columns;
    args.barrier_offset = static_cast<uint32_t>(plan.smem);
    int blocks = (tiles + plan.row_tiles - 1) / plan.row_tiles;
    if (silu) blocks = (ns[0] + 64 * plan.row_tiles - 1) / (64 * plan.row_tiles);
    const dim3 grid(plan.lane_tiles, blocks, plan.splits);
    auto kernel = plan.row_tiles == 1 ? linear_int4_gemm_kernel<1, 1> : plan.parts == 1 ? linear_int4_gemm_kernel<2, 1> : linear_int4_gemm_kernel<2, 2>;
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(GEMM_SMEM_ONE + GEMM_TAIL_BYTES));
    if (status != cudaSuccess) return status;
    return launch_dependent(kernel, grid, dim3(plan.row_tiles == 2 ? gemm_threads<2>() : gemm_threads<1>()), plan.smem + GEMM_TAIL_BYTES, plan.splits, stream, args);
}

}  // namespace nerve
