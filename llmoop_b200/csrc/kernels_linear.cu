// Weight-streaming linears for small lane counts (verify M = k+1, draft M = 1,
// multi-stream batches): y[m][n] = sum_k x[m][k] * W[n][k].
//
// All of these are HBM-bound: every weight byte is read once per launch, the
// activations (KBs) stay in L1/L2.  Algorithmic bytes per output row:
//   INT4 g128: k/2 packed + 2*k/128 scale bytes;  BF16: 2*k;  FP8: k + block scales.
//
// INT4 path (linear_int4_ct.comp.template:80-150 semantics): at 4 lanes a
// scalar-FMA kernel needs ~6 ALU ops per nibble (unpack, offset, 4 FMAs), i.e.
// ~280 thread-ops/clk/SM to keep up with HBM, above the 128/clk an SM issues,
// so the dot products run on the tensor cores even at M <= 8:
// mma.sync.m16n8k16 with A = 16 weight rows dequantised in registers to bf16
// (exact: 128+q built with one lop3, minus 136), B = up to 8 activation lanes,
// f32 accumulators; the group scale is applied to the f32 partial after every
// 128-column group, so rounding happens only once at the bf16 store.
// The K permutation inside an mma is free as long as A and B agree: thread
// (g, j) of a warp feeds logical k slots {2j,2j+1,2j+8,2j+9} from nibbles
// {0,4,1,5} / {2,6,3,7} of its own 32-bit words, which lets each thread fetch
// 32 consecutive nibbles (one 128-bit load) per row and keeps dequantisation
// at 3 ALU ops per nibble pair.
#include <mma.h>

#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

// ----------------------------------------------------------------------------- bf16 weights

struct Bf16Rows {  // the matrices of a launch: matrix b owns the CTAs first[b] .. first[b + 1] - 1
    const uint16_t *w[3];
    void *y[3];
    int n[3], first[4];
};

// One launch for all matrices of an input: at the sizes this form is for, a launch of its own costs as much as the work
// (64 x 64, q, k and v: 1.8 us each).
template <int MT, int ROWS>
__global__ void __launch_bounds__(256)
linear_bf16_kernel(const uint16_t *__restrict__ x, const __grid_constant__ Bf16Rows rows,
                   const uint16_t *__restrict__ residual, int lanes, int k, int epilogue, float scale) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int block = blockIdx.x, branch = block < rows.first[1] ? 0 : block < rows.first[2] ? 1 : 2;
    const uint16_t *__restrict__ w = rows.w[branch];
    void *__restrict__ y = rows.y[branch];
    const int n = rows.n[branch], row0 = ((block - rows.first[branch]) * 8 + warp) * ROWS;
    const int m0 = blockIdx.y * MT;
    if (row0 >= n) return;
    float acc[ROWS][MT];
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
        for (int m = 0; m < MT; m++) acc[r][m] = 0.0f;

    const int chunks = k % 8 == 0 ? k / 8 : 0;  // uint4 = 8 bf16; rows of other widths are not aligned to it
    // weights do not depend on the previous kernel: the first loads may be issued before the dependency wait
    grid_launch_dependents();
    grid_dependency_wait();
    for (int chunk = lane; chunk < chunks; chunk += 32) {
        uint4 wv[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            int row = row0 + r < n ? row0 + r : n - 1;
            wv[r] = __ldg(reinterpret_cast<const uint4 *>(w + static_cast<size_t>(row) * k) + chunk);
        }
#pragma unroll
        for (int m = 0; m < MT; m++) {
            if (m0 + m >= lanes) break;
            uint4 xv = __ldg(reinterpret_cast<const uint4 *>(x + static_cast<size_t>(m0 + m) * k) + chunk);
            const uint32_t xs[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int r = 0; r < ROWS; r++) {
                const uint32_t ws[4] = {wv[r].x, wv[r].y, wv[r].z, wv[r].w};
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    acc[r][m] = fmaf(bf16_lo(xs[i]), bf16_lo(ws[i]), acc[r][m]);
                    acc[r][m] = fmaf(bf16_hi(xs[i]), bf16_hi(ws[i]), acc[r][m]);
                }
            }
        }
    }
    // k not a multiple of 8 (tiny test shapes)
    for (int col = chunks * 8 + lane; col < k; col += 32) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            int row = row0 + r < n ? row0 + r : n - 1;
            float wf = bf16_bits_to_f32(w[static_cast<size_t>(row) * k + col]);
#pragma unroll
            for (int m = 0; m < MT; m++)
                if (m0 + m < lanes) acc[r][m] = fmaf(bf16_bits_to_f32(x[static_cast<size_t>(m0 + m) * k + col]), wf, acc[r][m]);
        }
    }
#pragma unroll
    for (int r = 0; r < ROWS; r++)
#pragma unroll
        for (int m = 0; m < MT; m++) acc[r][m] = warp_sum(acc[r][m]);
    if (lane == 0) {
#pragma unroll
        for (int r = 0; r < ROWS; r++) {
            int row = row0 + r;
            if (row >= n) break;
#pragma unroll
            for (int m = 0; m < MT; m++) {
                if (m0 + m >= lanes) break;
                size_t index = static_cast<size_t>(m0 + m) * n + row;
                float sum = acc[r][m];
                if (epilogue == EPILOGUE_F32_SCALED) {
                    reinterpret_cast<float *>(y)[index] = sum * scale;
                } else {
                    if (epilogue == EPILOGUE_RESIDUAL_ROUNDED) sum = round_bf16(sum) + bf16_bits_to_f32(residual[index]);
                    else if (epilogue == EPILOGUE_RESIDUAL_F32) sum = sum + bf16_bits_to_f32(residual[index]);
                    reinterpret_cast<uint16_t *>(y)[index] = static_cast<uint16_t>(f32_to_bf16_bits(sum));
                }
            }
        }
    }
}

bool linear_bf16_is_scalar(int lanes, int n, int k, LinearForm form) {
    return form == LINEAR_SCALAR || !linear_bf16_gemm_supported(form == LINEAR_TENSOR ? 16 : lanes, n, k);
}

cudaError_t launch_linear_bf16(const uint16_t *x, const uint16_t *w, void *y, const uint16_t *residual, int lanes,
                               int n, int k, int epilogue, float scale, cudaStream_t stream, int *error_flag, LinearForm form) {
    if (lanes <= 0) return cudaSuccess;
    // more than eight lanes: the tensor-core GEMM (weights read once instead of once per eight lanes)
    if (!linear_bf16_is_scalar(lanes, n, k, form)) return launch_linear_bf16_gemm(x, w, y, residual, lanes, n, k, epilogue, scale, error_flag, stream);
    LinearBranches branches;
    branches.add(w, nullptr, y, n);
    return launch_linear_bf16_scalar(x, branches, residual, lanes, k, epilogue, scale, stream);
}

cudaError_t launch_linear_bf16_scalar(const uint16_t *x, const LinearBranches &branches, const uint16_t *residual, int lanes, int k, int epilogue, float scale,
                                      cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    // Four rows to a warp save activation loads; a launch that would leave SMs idle then takes one (and up to four lanes), for
    // shorter chains and sums (128 rows of 2048 with 24 lanes: 24 -> 10 us).
    int ctas = 0;
    for (int b = 0; b < branches.count; b++) ctas += (branches.n[b] + 31) / 32;
    const int rows_per_warp = ctas * ((lanes + 7) / 8) < multiprocessors() ? 1 : 4;
    Bf16Rows rows = {};
    ctas = 0;
    for (int b = 0; b < 3; b++) {
        rows.first[b] = ctas;
        if (b >= branches.count) continue;
        rows.w[b] = static_cast<const uint16_t *>(branches.w[b]);
        rows.y[b] = branches.y[b];
        rows.n[b] = branches.n[b];
        ctas += (branches.n[b] + 8 * rows_per_warp - 1) / (8 * rows_per_warp);
    }
    rows.first[3] = ctas;
    for (int b = branches.count; b < 3; b++) rows.first[b] = ctas;
    if (rows_per_warp == 1) {
        if (lanes == 1) return launch_dependent(linear_bf16_kernel<1, 1>, dim3(ctas), dim3(256), 0, 1, stream, x, rows, residual, lanes, k, epilogue, scale);
        if (lanes == 2) return launch_dependent(linear_bf16_kernel<2, 1>, dim3(ctas), dim3(256), 0, 1, stream, x, rows, residual, lanes, k, epilogue, scale);
        return launch_dependent(linear_bf16_kernel<4, 1>, dim3(ctas, (lanes + 3) / 4), dim3(256), 0, 1, stream, x, rows, residual, lanes, k, epilogue, scale);
    }
    if (lanes <= 4) return launch_dependent(linear_bf16_kernel<4, 4>, dim3(ctas), dim3(256), 0, 1, stream, x, rows, residual, lanes, k, epilogue, scale);
    return launch_dependent(linear_bf16_kernel<8, 4>, dim3(ctas, (lanes + 7) / 8), dim3(256), 0, 1, stream, x, rows, residual, lanes, k, epilogue, scale);
}

// parallel_linear_silu_multiply_bf16.comp.template:58-72
template <int MT>
__global__ void __launch_bounds__(256)
linear_silu_multiply_bf16_kernel(const uint16_t *__restrict__ x, const uint16_t *__restrict__ wg,
                                 const uint16_t *__restrict__ wu, uint16_t *__restrict__ y, int lanes, int n, int k) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * 8 + warp;
    const int m0 = blockIdx.y * MT;
    if (row >= n) return;
    float gate[MT], up[MT];
#pragma unroll
    for (int m = 0; m < MT; m++) gate[m] = up[m] = 0.0f;
    grid_launch_dependents();
    grid_dependency_wait();
    for (int col = lane * 2; col < k; col += 64) {
        uint32_t g = *reinterpret_cast<const uint32_t *>(wg + static_cast<size_t>(row) * k + col);
        uint32_t u = *reinterpret_cast<const uint32_t *>(wu + static_cast<size_t>(row) * k + col);
#pragma unroll
        for (int m = 0; m < MT; m++) {
            if (m0 + m >= lanes) break;
            uint32_t xv = *reinterpret_cast<const uint32_t *>(x + static_cast<size_t>(m0 + m) * k + col);
            gate[m] = fmaf(bf16_lo(xv), bf16_lo(g), gate[m]);
            gate[m] = fmaf(bf16_hi(xv), bf16_hi(g), gate[m]);
            up[m] = fmaf(bf16_lo(xv), bf16_lo(u), up[m]);
            up[m] = fmaf(bf16_hi(xv), bf16_hi(u), up[m]);
        }
    }
#pragma unroll
    for (int m = 0; m < MT; m++) {
        gate[m] = warp_sum(gate[m]);
        up[m] = warp_sum(up[m]);
    }
    if (lane == 0)
#pragma unroll
        for (int m = 0; m < MT; m++) {
            if (m0 + m >= lanes) break;
            float value = rounded_silu(round_bf16(gate[m])) * round_bf16(up[m]);
            y[static_cast<size_t>(m0 + m) * n + row] = static_cast<uint16_t>(f32_to_bf16_bits(value));
        }
}

cudaError_t launch_linear_silu_multiply_bf16(const uint16_t *x, const uint16_t *wg, const uint16_t *wu, uint16_t *y,
                                             int lanes, int n, int k, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    dim3 grid((n + 7) / 8, (lanes + 7) / 8);
    auto kernel = lanes == 1 ? linear_silu_multiply_bf16_kernel<1> : lanes == 2 ? linear_silu_multiply_bf16_kernel<2>
                : lanes <= 4 ? linear_silu_multiply_bf16_kernel<4> : linear_silu_multiply_bf16_kernel<8>;
    return launch_dependent(kernel, grid, dim3(256), 0, 1, stream, x, wg, wu, y, lanes, n, k);
}

// ----------------------------------------------------------------------------- INT4 g128 (tensor cores)

__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                               uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Two nibbles (bits s..s+3 and s+16..s+19 of `word`) -> bf16x2 (q-8, q'-8), exact.
__device__ __forceinline__ uint32_t dequant_pair(uint32_t word, int shift) {
    uint32_t biased;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(biased) : "r"(word >> shift), "n"(0x000F000F), "n"(0x43004300));
    __nv_bfloat162 value = *reinterpret_cast<__nv_bfloat162 *>(&biased);
    const uint32_t offset_bits = 0x43084308u;  // bf16 136.0 twice
    __nv_bfloat162 offset = *reinterpret_cast<const __nv_bfloat162 *>(&offset_bits);
    value = __hsub2(value, offset);
    return *reinterpret_cast<uint32_t *>(&value);
}

struct Int4Branch {
    const uint32_t *qweight;
    const uint16_t *scales;
    uint16_t *y;
    int n;
    int first_tile;  // index of this branch's first CTA tile
};

struct Int4Launch {
    Int4Branch branch[3];
    int branches;
    const uint16_t *x;
    const uint16_t *residual;
    int lanes;
    int k;
    int epilogue;
};

constexpr int INT4_WARPS = 8;

// RT row tiles (16 rows each) per CTA; SILU_PAIR: rt 0 = gate rows, rt 1 = the same rows of the up projection,
// epilogue bf16(silu_bf16(bf16 gate) * bf16 up).  The 8 warps of a CTA split K by 128-column groups
// (warp w takes groups w, w+8, ...) and keep STAGES groups of packed weights in flight in registers: with
// ~1 us of loaded-memory latency a warp must have several KB outstanding for the SM to reach its share of HBM
// bandwidth (Little's law: ~44 KB per SM at 6.5 TB/s).
template <int RT, bool SILU_PAIR, int STAGES>
__global__ void __launch_bounds__(INT4_WARPS * 32, 2)
linear_int4_mma_kernel(const Int4Launch p) {
    __shared__ float reduce[INT4_WARPS][RT * 16][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, j = lane & 3;
    constexpr int m0 = 0;  // at most eight lanes

    int b = 0;
    if (!SILU_PAIR) {
        if (p.branches > 1 && static_cast<int>(blockIdx.x) >= p.branch[1].first_tile) b = 1;
        if (p.branches > 2 && static_cast<int>(blockIdx.x) >= p.branch[2].first_tile) b = 2;
    }
    const Int4Branch &br = p.branch[b];
    const int tile = blockIdx.x - br.first_tile;
    const int k = p.k;
    const int words_per_row = k >> 3;
    const int groups = k >> 7;

    const uint32_t *wrow[RT][2];
    const uint16_t *srow[RT][2];
#pragma unroll
    for (int rt = 0; rt < RT; rt++) {
        const Int4Branch &source = SILU_PAIR ? p.branch[rt] : br;
        int base = SILU_PAIR ? tile * 16 : (tile * RT + rt) * 16;
#pragma unroll
        for (int h = 0; h < 2; h++) {
            int row = base + g + 8 * h;
            if (row >= source.n) row = source.n - 1;  // clamped rows are computed and dropped
            wrow[rt][h] = source.qweight + static_cast<size_t>(row) * words_per_row + j * 4;
            srow[rt][h] = source.scales + static_cast<size_t>(row) * groups;
        }
    }
    const bool lane_active = m0 + g < p.lanes;
    const uint16_t *xrow = p.x + static_cast<size_t>(lane_active ? m0 + g : 0) * k + j * 32;

    float acc[RT][4];
#pragma unroll
    for (int rt = 0; rt < RT; rt++)
#pragma unroll
        for (int i = 0; i < 4; i++) acc[rt][i] = 0.0f;

    // Weights do not depend on the producer of x: the first STAGES groups are requested before the dependency wait.
    uint4 wq[STAGES][RT][2];
#pragma unroll
    for (int s = 0; s < STAGES; s++) {
        const int group = warp + s * INT4_WARPS;
        if (group < groups) {
#pragma unroll
            for (int rt = 0; rt < RT; rt++)
#pragma unroll
                for (int h = 0; h < 2; h++) wq[s][rt][h] = __ldg(reinterpret_cast<const uint4 *>(wrow[rt][h] + group * 16));
        }
    }
    grid_dependency_wait();

    for (int base = warp; base < groups; base += INT4_WARPS * STAGES) {
#pragma unroll
        for (int s = 0; s < STAGES; s++) {
            const int group = base + s * INT4_WARPS;
            if (group >= groups) break;
            // activations of lane g for this thread's 32 columns, permuted to match the nibble pairs
            uint32_t bfrag[8][2];
            if (lane_active) {
#pragma unroll
                for (int word = 0; word < 4; word++) {
                    uint4 xv = __ldg(reinterpret_cast<const uint4 *>(xrow + group * 128) + word);
                    bfrag[2 * word][0] = __byte_perm(xv.x, xv.z, 0x5410);      // (v0, v4)
                    bfrag[2 * word][1] = __byte_perm(xv.x, xv.z, 0x7632);      // (v1, v5)
                    bfrag[2 * word + 1][0] = __byte_perm(xv.y, xv.w, 0x5410);  // (v2, v6)
                    bfrag[2 * word + 1][1] = __byte_perm(xv.y, xv.w, 0x7632);  // (v3, v7)
                }
            } else {
#pragma unroll
                for (int step = 0; step < 8; step++) bfrag[step][0] = bfrag[step][1] = 0u;
            }
#pragma unroll
            for (int rt = 0; rt < RT; rt++) {
                float c[4] = {0.0f, 0.0f, 0.0f, 0.0f};
                const uint32_t wa[4] = {wq[s][rt][0].x, wq[s][rt][0].y, wq[s][rt][0].z, wq[s][rt][0].w};
                const uint32_t wb[4] = {wq[s][rt][1].x, wq[s][rt][1].y, wq[s][rt][1].z, wq[s][rt][1].w};
#pragma unroll
                for (int word = 0; word < 4; word++) {
                    mma_bf16_16816(c, dequant_pair(wa[word], 0), dequant_pair(wb[word], 0), dequant_pair(wa[word], 4),
                                   dequant_pair(wb[word], 4), bfrag[2 * word][0], bfrag[2 * word][1]);
                    mma_bf16_16816(c, dequant_pair(wa[word], 8), dequant_pair(wb[word], 8), dequant_pair(wa[word], 12),
                                   dequant_pair(wb[word], 12), bfrag[2 * word + 1][0], bfrag[2 * word + 1][1]);
                }
                float sa = bf16_bits_to_f32(srow[rt][0][group]);
                float sb = bf16_bits_to_f32(srow[rt][1][group]);
                acc[rt][0] = fmaf(c[0], sa, acc[rt][0]);
                acc[rt][1] = fmaf(c[1], sa, acc[rt][1]);
                acc[rt][2] = fmaf(c[2], sb, acc[rt][2]);
                acc[rt][3] = fmaf(c[3], sb, acc[rt][3]);
            }
            // refill this stage's registers with the group STAGES rounds ahead
            const int next = group + INT4_WARPS * STAGES;
            if (next < groups) {
#pragma unroll
                for (int rt = 0; rt < RT; rt++)
#pragma unroll
                    for (int h = 0; h < 2; h++) wq[s][rt][h] = __ldg(reinterpret_cast<const uint4 *>(wrow[rt][h] + next * 16));
            }
        }
    }
    grid_launch_dependents();

#pragma unroll
    for (int rt = 0; rt < RT; rt++) {
        reduce[warp][rt * 16 + g][2 * j] = acc[rt][0];
        reduce[warp][rt * 16 + g][2 * j + 1] = acc[rt][1];
        reduce[warp][rt * 16 + g + 8][2 * j] = acc[rt][2];
        reduce[warp][rt * 16 + g + 8][2 * j + 1] = acc[rt][3];
    }
    __syncthreads();
    const int outputs = (SILU_PAIR ? 16 : RT * 16) * 8;
    for (int index = threadIdx.x; index < outputs; index += blockDim.x) {
        int local_row = index >> 3, m = index & 7;
        if (m0 + m >= p.lanes) continue;
        if (SILU_PAIR) {
            int row = tile * 16 + local_row;
            if (row >= br.n) continue;
            float gate = 0.0f, up = 0.0f;
#pragma unroll
            for (int w = 0; w < INT4_WARPS; w++) {
                gate += reduce[w][local_row][m];
                up += reduce[w][16 + local_row][m];
            }
            float value = rounded_silu(round_bf16(gate)) * round_bf16(up);
            p.branch[2].y[static_cast<size_t>(m0 + m) * br.n + row] = static_cast<uint16_t>(f32_to_bf16_bits(value));
        } else {
            int row = tile * RT * 16 + local_row;
            if (row >= br.n) continue;
            float sum = 0.0f;
#pragma unroll
            for (int w = 0; w < INT4_WARPS; w++) sum += reduce[w][local_row][m];
            size_t out = static_cast<size_t>(m0 + m) * br.n + row;
            if (p.epilogue == EPILOGUE_F32_SCALED) {  // f32 partial sums (tensor-parallel row split)
                reinterpret_cast<float *>(br.y)[out] = sum;
                continue;
            }
            if (p.epilogue == EPILOGUE_RESIDUAL_ROUNDED) sum = round_bf16(sum) + bf16_bits_to_f32(p.residual[out]);
            else if (p.epilogue == EPILOGUE_RESIDUAL_F32) sum = sum + bf16_bits_to_f32(p.residual[out]);
            br.y[out] = static_cast<uint16_t>(f32_to_bf16_bits(sum));
        }
    }
}

cudaError_t launch_linear_int4_multi(const uint16_t *x, const void *prepared, int branches, const uint32_t *const *qweights,
                                     const uint16_t *const *scales, uint16_t *const *ys, const int *ns,
                                     const uint16_t *residual, int lanes, int k, int epilogue, cudaStream_t stream, int *error_flag) {
    if (lanes <= 0) return cudaSuccess;
    if (k % 128 != 0 || branches < 1 || branches > 3) return cudaErrorInvalidValue;
    if (linear_int4_gemm_supported(lanes, ns[0], k)) {
        // more than eight lanes: one tcgen05 GEMM launch for all the matrices that share the activations
        if (prepared == nullptr) return cudaErrorInvalidValue;
        void *outputs[3] = {ys[0], branches > 1 ? ys[1] : nullptr, branches > 2 ? ys[2] : nullptr};
        return launch_linear_int4_gemm(prepared, branches, qweights, scales, outputs, ns, branches == 1 ? residual : nullptr, lanes, k, epilogue, 1.0f, false,
                                       error_flag, stream);
    }
    Int4Launch params = {};
    params.branches = branches;
    params.x = x;
    params.residual = residual;
    params.lanes = lanes;
    params.k = k;
    params.epilogue = epilogue;
    long total_rows = 0;
    for (int b = 0; b < branches; b++) total_rows += ns[b];
    const int rt = 1;
    int tiles = 0;
    for (int b = 0; b < branches; b++) {
        params.branch[b] = Int4Branch{qweights[b], scales[b], ys[b], ns[b], tiles};
        tiles += (ns[b] + 16 * rt - 1) / (16 * rt);
    }
    dim3 grid(tiles);
    return launch_dependent(linear_int4_mma_kernel<1, false, 4>, grid, dim3(INT4_WARPS * 32), 0, 1, stream, params);
}

cudaError_t launch_linear_int4(const uint16_t *x, const void *prepared, const uint32_t *qweight, const uint16_t *scales, uint16_t *y,
                               const uint16_t *residual, int lanes, int n, int k, int group, int epilogue,
                               cudaStream_t stream, int *error_flag) {
    if (group != 128) return cudaErrorInvalidValue;
    return launch_linear_int4_multi(x, prepared, 1, &qweight, &scales, &y, &n, residual, lanes, k, epilogue, stream, error_flag);
}

// gate/up pair with the SiLU*up epilogue (gate -> bf16, SiLU -> bf16, up -> bf16, product -> bf16: the
// rounding chain of linear + linear + silu_multiply_bf16.comp.template:30-52).
cudaError_t launch_linear_int4_silu_pair(const uint16_t *x, const void *prepared, const uint32_t *gate_q, const uint16_t *gate_s,
                                         const uint32_t *up_q, const uint16_t *up_s, uint16_t *y, int lanes, int n,
                                         int k, cudaStream_t stream, int *error_flag) {
    if (lanes <= 0) return cudaSuccess;
    if (k % 128 != 0) return cudaErrorInvalidValue;
    if (linear_int4_gemm_supported(lanes, n, k)) {
        if (prepared == nullptr) return cudaErrorInvalidValue;
        const uint32_t *qweights[2] = {gate_q, up_q};
        const uint16_t *scales[2] = {gate_s, up_s};
        void *outputs[2] = {y, y};
        const int ns[2] = {n, n};
        return launch_linear_int4_gemm(prepared, 2, qweights, scales, outputs, ns, nullptr, lanes, k, EPILOGUE_BF16, 1.0f, true, error_flag, stream);
    }
    Int4Launch params = {};
    params.branches = 2;
    params.x = x;
    params.lanes = lanes;
    params.k = k;
    params.branch[0] = Int4Branch{gate_q, gate_s, nullptr, n, 0};
    params.branch[1] = Int4Branch{up_q, up_s, nullptr, n, 0};
    params.branch[2] = Int4Branch{nullptr, nullptr, y, n, 0};
    dim3 grid((n + 15) / 16);
    return launch_dependent(linear_int4_mma_kernel<2, true, 2>, grid, dim3(INT4_WARPS * 32), 0, 1, stream, params);
}

}  // namespace nerve
