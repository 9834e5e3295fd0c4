// bf16 linear for batches of more than eight lanes (the draft adapter's linear over a prefill chunk, the output
// projection of a many-stream verify batch, routers) on the fifth-generation tensor cores: y[m][n] = sum_k x[m][k] *
// w[n][k], the arithmetic of linear_bf16.comp.template / tied_output_projection_batch_bf16.comp.template:52-142 (bf16
// operands, f32 accumulation over the whole of K, one rounding or the logit scale at the end).
//
// Persistent: one CTA per SM walks output tiles of 128 weight rows (MMA M) x up to 256 lanes (MMA N).  One warp copies
// both operands with TMA (128-byte-swizzled tiles of 64 columns) into a ring as deep as shared memory allows, straight
// on into the next tile; one warp issues the MMAs into one of two accumulators in tensor memory; four warps write the
// finished accumulator out while the other one fills.  The weight bytes are the bound up to 64 lanes (a 128256 x 4096 table of
// 1.05 GB: 160-167 us, the copy rate), the stores of the outputs show from there on (160 lanes: 200 us), and from 200 lanes
// on the tensor pipe is it.  (The form this replaced - 64 lanes to a tile, operands copied by all threads between two
// barriers per block - read that table for 32 lanes in 640 us.)
// Waits are bounded; a wait that expires sets the error word, and the CTA still frees its tensor memory.  The unbounded wait
// for the kernel in front comes before them in every role, so none of them counts that kernel's time.
#include <cuda.h>

#include <algorithm>

#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

namespace {

constexpr int ROWS = 128, BLOCK_K = 128;                 // weight rows per tile; columns per stage (two swizzled halves of 64)
constexpr int THREADS = 256, MAX_STAGES = 6;
constexpr uint32_t A_BYTES = ROWS * BLOCK_K * 2;
constexpr size_t SMEM_LIMIT = 226 * 1024, CONTROL_BYTES = 256;
constexpr unsigned int SPIN_LIMIT = 1u << 22;  // tries of 1.5 us

__device__ __forceinline__ uint64_t swizzled_descriptor(uint32_t shared_address) {  // K-major, 128-byte swizzle, 1024 bytes between 8-row atoms
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
        if (++spins > SPIN_LIMIT) {
            if (error_flag != nullptr) *static_cast<volatile int *>(error_flag) = 3;  // (may be mapped host memory)
            return false;
        }
    }
}
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
__device__ __forceinline__ void commit_to(uint32_t barrier) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(barrier) : "memory");
}
__device__ __forceinline__ void copy_tile(uint32_t target, const CUtensorMap *map, int column, int row, uint32_t barrier) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(target), "l"(map), "r"(column), "r"(row),
                 "r"(barrier)
                 : "memory");
}

struct BgemmArgs {
    CUtensorMap weights, activations;  // boxes of 64 columns x 128 rows, and x tile_lanes lanes
    void *y;
    const uint16_t *residual;
    int lanes, n, k, epilogue;
    float scale;
    int *error_flag;
    int tile_lanes, lane_tiles, tiles, stages;
};

__global__ void __launch_bounds__(THREADS, 1) linear_bf16_gemm_kernel(const __grid_constant__ BgemmArgs a) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;  // warp: uniform
    const uint32_t b_bytes = static_cast<uint32_t>(a.tile_lanes) * BLOCK_K * 2, stage_bytes = A_BYTES + b_bytes;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    const uint32_t full = base + static_cast<uint32_t>(a.stages) * stage_bytes, empty = full + 8 * MAX_STAGES, acc_full = empty + 8 * MAX_STAGES, acc_empty = acc_full + 16,
                   tmem_slot = acc_empty + 16;
    const int blocks = a.k / BLOCK_K;
    grid_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < MAX_STAGES; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + s * 8) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty + s * 8) : "memory");
        }
        for (int s = 0; s < 2; s++) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(acc_full + s * 8) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(acc_empty + s * 8) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const uint32_t acc_columns = (static_cast<uint32_t>(a.tile_lanes) + 31u) & ~31u;
    uint32_t columns = 32;
    while (columns < 2 * acc_columns) columns *= 2;
    if (warp == 2) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tmem_slot), "r"(columns) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    uint32_t tmem;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(tmem) : "r"(tmem_slot) : "memory");
    tmem = __reduce_or_sync(0xffffffffu, tmem);  // a uniform register

    if (warp == 0) {  // ---- copies
        int stage = 0, issued = 0;
        uint32_t parity = 1;  // the first round waits for no release
        // the weights of the first stages do not wait for the kernel in front
        const int first_tile = blockIdx.x, ahead = first_tile < a.tiles ? min(a.stages, blocks) : 0;
        if (elect_one())
            for (int block = 0; block < ahead; block++) {
                const uint32_t target = base + static_cast<uint32_t>(block) * stage_bytes;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full + block * 8), "r"(stage_bytes) : "memory");
                for (int half = 0; half < 2; half++)
                    copy_tile(target + half * (A_BYTES / 2), &a.weights, block * BLOCK_K + half * 64, first_tile / a.lane_tiles * ROWS, full + block * 8);
            }
        __syncwarp();
        grid_dependency_wait();
        bool alive = true;
        for (int tile = first_tile; tile < a.tiles && alive; tile += gridDim.x) {
            const int row0 = tile / a.lane_tiles * ROWS, m0 = tile % a.lane_tiles * a.tile_lanes;
            for (int block = 0; block < blocks; block++) {
                if (!wait_barrier(empty + stage * 8, parity, a.error_flag)) {
                    for (int s = 0; s < a.stages && s < issued; s++) {  // the copies in flight land before the CTA gives its memory up
                        const int which = (issued - 1 - s) % a.stages;
                        wait_barrier(full + which * 8, static_cast<uint32_t>(((issued - 1 - s) / a.stages) & 1), a.error_flag);
                    }
                    alive = false;
                    break;
                }
                if (elect_one()) {
                    const uint32_t target = base + static_cast<uint32_t>(stage) * stage_bytes, barrier = full + stage * 8;
                    if (issued >= ahead) {
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(barrier), "r"(stage_bytes) : "memory");
                        for (int half = 0; half < 2; half++) copy_tile(target + half * (A_BYTES / 2), &a.weights, block * BLOCK_K + half * 64, row0, barrier);
                    }
                    for (int half = 0; half < 2; half++) copy_tile(target + A_BYTES + half * (b_bytes / 2), &a.activations, block * BLOCK_K + half * 64, m0, barrier);
                }
                __syncwarp();
                issued++;
                if (++stage == a.stages) {
                    stage = 0;
                    parity ^= 1;
                }
            }
        }
    } else if (warp == 1) {  // ---- MMAs
        // instruction descriptor: f32 accumulator, A and B bf16, both K-major, N / 8 in bits 17-22, M / 16 in bits 24-28
        const uint32_t instruction = (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(a.tile_lanes / 8) << 17) | (8u << 24);
        const uint64_t first = swizzled_descriptor(base), b_half = b_bytes / 2 >> 4;
        int stage = 0, round = 0;
        uint32_t parity = 0;
        bool alive = true;
        grid_dependency_wait();
        for (int tile = blockIdx.x; tile < a.tiles && alive; tile += gridDim.x, round++) {
            const uint32_t accumulator = tmem + (round & 1) * acc_columns;
            if (!wait_barrier(acc_empty + (round & 1) * 8, static_cast<uint32_t>((round / 2 + 1) & 1), a.error_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int block = 0; block < blocks; block++) {
                if (!wait_barrier(full + stage * 8, parity, a.error_flag)) {
                    alive = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (elect_one()) {
                    const uint64_t a_stage = first + static_cast<uint64_t>(stage) * (stage_bytes >> 4), b_stage = a_stage + (A_BYTES >> 4);
#pragma unroll
                    for (int step = 0; step < 8; step++) {  // K = 16 per instruction; four steps to a 128-byte row of a swizzled half
                        const uint64_t a_descriptor = a_stage + (step >> 2) * (A_BYTES / 2 >> 4) + (step & 3) * 2, b_descriptor = b_stage + (step >> 2) * b_half + (step & 3) * 2;
                        const uint32_t accumulate = (block > 0 || step > 0) ? 1u : 0u;
                        asm volatile(
                            "{\n"
                            ".reg .pred p;\n"
                            "setp.ne.b32 p, %4, 0;\n"
                            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n"
                            "}\n" ::"r"(accumulator),
                            "l"(a_descriptor), "l"(b_descriptor), "r"(instruction), "r"(accumulate)
                            : "memory");
                    }
                    commit_to(empty + stage * 8);
                    if (block == blocks - 1) commit_to(acc_full + (round & 1) * 8);
                }
                __syncwarp();
                if (++stage == a.stages) {
                    stage = 0;
                    parity ^= 1;
                }
            }
        }
    } else if (warp >= 4) {  // ---- outputs: thread = weight row
        grid_dependency_wait();
        const int quarter = warp & 3;
        int round = 0;
        for (int tile = blockIdx.x; tile < a.tiles; tile += gridDim.x, round++) {
            const int row = tile / a.lane_tiles * ROWS + quarter * 32 + lane, m0 = tile % a.lane_tiles * a.tile_lanes, count = min(a.tile_lanes, a.lanes - m0);
            if (!wait_barrier(acc_full + (round & 1) * 8, static_cast<uint32_t>((round / 2) & 1), a.error_flag)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t accumulator = tmem + (static_cast<uint32_t>(quarter * 32) << 16) + (round & 1) * acc_columns;
            for (int column = 0; column < count; column += 16) {
                uint32_t d[16];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                             : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]),
                               "=r"(d[10]), "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
                             : "r"(accumulator + static_cast<uint32_t>(column))
                             : "memory");
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (row >= a.n) continue;
                float residual[16];
                if (a.residual != nullptr)
#pragma unroll
                    for (int i = 0; i < 16; i++)
                        if (column + i < count) residual[i] = bf16_bits_to_f32(a.residual[static_cast<size_t>(m0 + column + i) * a.n + row]);
#pragma unroll
                for (int i = 0; i < 16; i++) {
                    if (column + i >= count) break;
                    const size_t index = static_cast<size_t>(m0 + column + i) * a.n + row;
                    float sum = __uint_as_float(d[i]);
                    if (a.epilogue == EPILOGUE_F32_SCALED) {
                        reinterpret_cast<float *>(a.y)[index] = sum * a.scale;
                    } else {
                        if (a.epilogue == EPILOGUE_RESIDUAL_ROUNDED) sum = round_bf16(sum) + residual[i];
                        else if (a.epilogue == EPILOGUE_RESIDUAL_F32) sum = sum + residual[i];
                        reinterpret_cast<uint16_t *>(a.y)[index] = static_cast<uint16_t>(f32_to_bf16_bits(sum));
                    }
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(acc_empty + (round & 1) * 8) : "memory");
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 2) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns) : "memory");
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *, const cuuint32_t *, const cuuint32_t *,
                                 CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {  // the driver's entry point, found through the runtime (the library does not link libcuda)
    static const EncodeTiled found = [] {
        void *pointer = nullptr;
        cudaDriverEntryPointQueryResult result;
        const cudaError_t status = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &pointer, cudaEnableDefault, &result);
        return status == cudaSuccess && result == cudaDriverEntryPointSuccess ? reinterpret_cast<EncodeTiled>(pointer) : nullptr;
    }();
    return found;
}
bool encode(CUtensorMap *map, const uint16_t *matrix, int rows, int k, int box_rows) {
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(k), static_cast<cuuint64_t>(rows)}, strides[1] = {static_cast<cuuint64_t>(k) * 2};
    const cuuint32_t box[2] = {64, static_cast<cuuint32_t>(box_rows)}, steps[2] = {1, 1};
    const EncodeTiled function = encode_tiled();
    return function != nullptr && function(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<uint16_t *>(matrix), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                           CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

}  // namespace

bool linear_bf16_gemm_supported(int lanes, int n, int k) { return lanes > 8 && k % 128 == 0 && k >= 128 && n >= 1; }

cudaError_t launch_linear_bf16_gemm(const uint16_t *x, const uint16_t *w, void *y, const uint16_t *residual, int lanes, int n, int k, int epilogue,
                                    float scale, int *error_flag, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (!linear_bf16_gemm_supported(lanes > 8 ? lanes : 9, n, k)) return cudaErrorInvalidValue;
    BgemmArgs args = {};
    // as few lane tiles as 256 lanes allow, of equal size: every tile reads its weight rows again (from L2)
    const int padded = (lanes + 15) / 16 * 16;
    args.lane_tiles = (padded + 255) / 256;
    args.tile_lanes = ((padded + args.lane_tiles - 1) / args.lane_tiles + 15) / 16 * 16;
    args.lane_tiles = (padded + args.tile_lanes - 1) / args.tile_lanes;
    args.tiles = (n + ROWS - 1) / ROWS * args.lane_tiles;
    args.stages = std::min<int>(MAX_STAGES, static_cast<int>(SMEM_LIMIT / (A_BYTES + static_cast<size_t>(args.tile_lanes) * BLOCK_K * 2)));
    if (!encode(&args.weights, w, n, k, ROWS) || !encode(&args.activations, x, lanes, k, args.tile_lanes)) return cudaErrorInvalidValue;
    args.y = y;
    args.residual = residual;
    args.lanes = lanes;
    args.n = n;
    args.k = k;
    args.epilogue = epilogue;
    args.scale = scale;
    args.error_flag = error_flag;
    cudaError_t status = cudaFuncSetAttribute(linear_bf16_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(SMEM_LIMIT + CONTROL_BYTES));
    if (status != cudaSuccess) return status;
    const size_t smem = static_cast<size_t>(args.stages) * (A_BYTES + static_cast<size_t>(args.tile_lanes) * BLOCK_K * 2) + CONTROL_BYTES;
    return launch_dependent(linear_bf16_gemm_kernel, dim3(std::min(args.tiles, multiprocessors())), dim3(THREADS), smem, 1, stream, args);
}

}  // namespace nerve
