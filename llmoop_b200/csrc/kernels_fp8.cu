// FP8 (e4m3, block-scaled) linears and sparse experts.
//
// Arithmetic (linear_prequant_fp8_e4m3.comp.template:69-120, sparse_moe_gate_up_fp8_e4m3.comp.template:94-198,
// sparse_moe_down_fp8_e4m3.comp.template:90-176): per 4 columns an f32 dot of e4m3 values, fma'd with
// act_scale * weight_scale.  The order of additions is fixed: column group l (columns 4 l .. 4 l + 3 of every block of
// 128) is added up over the blocks in order, then the 32 groups in a butterfly (distance 16, 8, 4, 2, 1).  The outputs
// are requantised to FP8 by the next linear and feed the choice of experts, where a last-bit difference of a sum becomes
// a step of a sixteenth or another expert, so no form of these kernels departs from that order - which leaves the work
// to the FP32 pipe (a tensor-core sum would add the groups in another order).
//
// A warp computes ROWS x M outputs: thread l owns column group l, keeps ROWS x M partial sums in registers and walks the
// blocks; weights come straight from global memory (one coalesced 128-byte row piece per warp and block, requested
// PIPE blocks ahead), the activations as fp16 from shared memory.  The products of a column group are added up with
// fp16 x fp16 + f32 multiply-adds (exact products, so the same roundings as on widened values), the scaled sums two lanes
// to a packed f32x2 operand: per weight word and lane four of the former and half of the latter, at an FP32 pipe of 25 and
// 30 TMAC/s, so about 20 TMAC/s is the bound from eight lanes on, below that the weight bytes.  1024 lanes x 4096 x 2048:
// 617 us with both operands widened to f32 (14 TMAC/s; the shared-memory loads and the conversions were at the same
// bound), now 533; x 2048 x 4096: 676 -> 509 us.
// Sparse experts are grouped: a small kernel sorts the (token, route) pairs by expert into tiles of up to eight, and an
// expert's rows are read once per tile instead of once per pair.
#include "common.cuh"
#include "kernels.cuh"
#include "launch.cuh"

namespace nerve {

namespace {

constexpr int FP8_WARPS = 8, FP8_ROWS = 8, TILE_LANES = 8;
constexpr int CHUNK = 32;  // blocks of 128 columns whose activations are staged at a time: 66 KB for eight lanes, two CTAs per SM

using pair_t = unsigned long long;  // two f32
__device__ __forceinline__ pair_t pack(float lo, float hi) {
    pair_t out;
    asm("mov.b64 %0, {%1, %2};" : "=l"(out) : "f"(lo), "f"(hi));
    return out;
}
__device__ __forceinline__ float2 unpack(pair_t v) {
    float2 out;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(out.x), "=f"(out.y) : "l"(v));
    return out;
}
__device__ __forceinline__ pair_t mul(pair_t a, pair_t b) {
    pair_t out;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(out) : "l"(a), "l"(b));
    return out;
}
// a.lo * b.lo + c and a.hi * b.hi + c of fp16 pairs in f32: the product of two e4m3 values is exact, so these round as the
// f32 multiply-add of the widened values does - without widening them, and with half the bytes in shared memory
__device__ __forceinline__ float mixed_fma_lo(uint32_t a, uint32_t b, float c) {
    asm("{\n.reg .b16 al, ah, bl, bh;\nmov.b32 {al, ah}, %1;\nmov.b32 {bl, bh}, %2;\nfma.rn.f32.f16 %0, al, bl, %0;\n}\n" : "+f"(c) : "r"(a), "r"(b));
    return c;
}
__device__ __forceinline__ float mixed_fma_hi(uint32_t a, uint32_t b, float c) {
    asm("{\n.reg .b16 al, ah, bl, bh;\nmov.b32 {al, ah}, %1;\nmov.b32 {bl, bh}, %2;\nfma.rn.f32.f16 %0, ah, bh, %0;\n}\n" : "+f"(c) : "r"(a), "r"(b));
    return c;
}
__device__ __forceinline__ pair_t fma2(pair_t a, pair_t b, pair_t c) {
    pair_t out;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(out) : "l"(a), "l"(b), "l"(c));
    return out;
}
// four e4m3 values of a word as two fp16 pairs, exact
__device__ __forceinline__ uint2 widen(uint32_t word) {
    uint2 out;
    asm("{\n.reg .b16 a, b;\nmov.b32 {a, b}, %2;\ncvt.rn.f16x2.e4m3x2 %0, a;\ncvt.rn.f16x2.e4m3x2 %1, b;\n}\n" : "=r"(out.x), "=r"(out.y) : "r"(word));
    return out;
}

// The activations of up to M lanes (rows of xq / xscale picked by `row_of`) in shared memory:
// x [block][lane pair][thread][lane of the pair][column] fp16, scales [block][M] f32.
template <int M>
constexpr size_t x_bytes() { return static_cast<size_t>(CHUNK) * 128 * M * 2; }
template <int M, typename RowOf>
__device__ __forceinline__ void stage_activations(const uint8_t *__restrict__ xq, const float *__restrict__ xscale, int k, int first, int blocks, int count, uint8_t *smem,
                                                  RowOf row_of) {
    const int words = blocks * 32, all_blocks = k >> 7;
    uint4 *x = reinterpret_cast<uint4 *>(smem);
    float *scales = reinterpret_cast<float *>(smem + x_bytes<M>());
    // (pair, word) of this thread's next item; four items' loads in flight (one after the other the staging of eight lanes
    // of 2048 took 6 of 23 us)
    int pair = threadIdx.x / words, word = threadIdx.x - pair * words;
    constexpr int BATCH = 4;
    while (pair < M / 2) {
        uint32_t lo[BATCH], hi[BATCH];
        int target[BATCH];
#pragma unroll
        for (int i = 0; i < BATCH; i++) {
            lo[i] = hi[i] = 0;
            target[i] = -1;
            if (pair < M / 2) {
                if (2 * pair < count) lo[i] = reinterpret_cast<const uint32_t *>(xq + static_cast<size_t>(row_of(2 * pair)) * k)[first * 32 + word];
                if (2 * pair + 1 < count) hi[i] = reinterpret_cast<const uint32_t *>(xq + static_cast<size_t>(row_of(2 * pair + 1)) * k)[first * 32 + word];
                target[i] = ((word >> 5) * (M / 2) + pair) * 32 + (word & 31);
            }
            word += FP8_WARPS * 32;
            while (word >= words) {
                word -= words;
                pair++;
            }
        }
#pragma unroll
        for (int i = 0; i < BATCH; i++)
            if (target[i] >= 0) {
                const uint2 a = widen(lo[i]), b = widen(hi[i]);
                x[target[i]] = make_uint4(a.x, a.y, b.x, b.y);
            }
    }
    for (int index = threadIdx.x; index < blocks * M; index += FP8_WARPS * 32) {
        const int m = index % M, block = index / M;
        scales[index] = m < count ? xscale[static_cast<size_t>(row_of(m)) * all_blocks + first + block] : 0.0f;
    }
}

// Sums of ROWS rows x M lanes over all of K; the two halves of the rows may have scale rows of their own (gate and up).
// Eight lanes take four rows at a time (the partial sums of more do not fit the registers of two CTAs per SM), fewer
// lanes eight.  On return thread t holds the outputs index(t, i) (or the one of its thread pair for M = 2).
template <int M, bool PAIRED>
struct RowSums {
    static constexpr int ROWS = M == 8 ? 4 : 8;
    static constexpr int VALUES = ROWS * M, PER_THREAD = VALUES >= 32 ? VALUES / 32 : 1;
    static constexpr int PIPE = M == 8 && PAIRED ? 2 : 4;  // blocks of weights in flight
    float sums[PER_THREAD];

    // output index = row * M + lane
    __device__ static int index(int thread, int i) {
        if (VALUES >= 32) return ((thread >> 4) & 1) * (VALUES / 2) + ((thread >> 3) & 1) * (VALUES / 4) + ((thread >> 2) & 1) * (VALUES / 8) +
                                 ((thread >> 1) & 1) * (VALUES / 16) + (thread & 1) * (VALUES / 32) + i;
        return thread >> 1;  // sixteen values: the last butterfly step leaves both threads of a pair with the same one
    }

    // stage(first, n) brings the activations of blocks first .. first + n - 1 into x (which may hold all of them already)
    template <typename RowPointer, typename Stage>
    __device__ void run(RowPointer row_pointer, const uint16_t *__restrict__ scales_a, const uint16_t *__restrict__ scales_b, int blocks, const uint8_t *smem, bool staged_already, Stage stage_blocks) {
        const uint4 *x = reinterpret_cast<const uint4 *>(smem);
        const float *x_scales = reinterpret_cast<const float *>(smem + x_bytes<M>());
        const int thread = threadIdx.x & 31;
        const uint32_t *source[ROWS];
#pragma unroll
        for (int r = 0; r < ROWS; r++) source[r] = reinterpret_cast<const uint32_t *>(row_pointer(r)) + thread;
        uint32_t words[PIPE][ROWS];
#pragma unroll
        for (int p = 0; p < PIPE; p++)
#pragma unroll
            for (int r = 0; r < ROWS; r++) words[p][r] = p < blocks ? __ldg(source[r] + p * 32) : 0u;
        pair_t acc[ROWS][M / 2];
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int p = 0; p < M / 2; p++) acc[r][p] = 0ull;
        float scale_a = 0.0f, scale_b = 0.0f;  // of block (32 i + thread)
        for (int base = 0; base < blocks; base += PIPE) {
            if (base % 32 == 0 && base + thread < blocks) {
                scale_a = bf16_bits_to_f32(__ldg(scales_a + base + thread));
                if (PAIRED) scale_b = bf16_bits_to_f32(__ldg(scales_b + base + thread));
            }
            if (base % CHUNK == 0 && (!staged_already || blocks > CHUNK)) {
                __syncthreads();
                stage_blocks(base, min(CHUNK, blocks - base));
                __syncthreads();
            }
#pragma unroll
            for (int stage = 0; stage < PIPE; stage++) {
                const int block = base + stage, staged = block % CHUNK;
                if (block >= blocks) break;
                const float wa = __shfl_sync(0xffffffffu, scale_a, block & 31), wb = PAIRED ? __shfl_sync(0xffffffffu, scale_b, block & 31) : wa;
                uint4 xv[M / 2];
                pair_t sa[M / 2], sb[M / 2];
#pragma unroll
                for (int p = 0; p < M / 2; p++) {
                    xv[p] = x[(staged * (M / 2) + p) * 32 + thread];
                    const pair_t xs = *reinterpret_cast<const pair_t *>(x_scales + staged * M + 2 * p);
                    sa[p] = mul(xs, pack(wa, wa));
                    sb[p] = PAIRED ? mul(xs, pack(wb, wb)) : sa[p];
                }
#pragma unroll
                for (int r = 0; r < ROWS; r++) {
                    const uint2 w = widen(words[stage][r]);
#pragma unroll
                    for (int p = 0; p < M / 2; p++) {
                        const float d0 = mixed_fma_hi(xv[p].y, w.y, mixed_fma_lo(xv[p].y, w.y, mixed_fma_hi(xv[p].x, w.x, mixed_fma_lo(xv[p].x, w.x, 0.0f))));
                        const float d1 = mixed_fma_hi(xv[p].w, w.y, mixed_fma_lo(xv[p].w, w.y, mixed_fma_hi(xv[p].z, w.x, mixed_fma_lo(xv[p].z, w.x, 0.0f))));
                        acc[r][p] = fma2(pack(d0, d1), r < ROWS / 2 ? sa[p] : sb[p], acc[r][p]);
                    }
                    words[stage][r] = block + PIPE < blocks ? __ldg(source[r] + (block + PIPE) * 32) : 0u;
                }
            }
        }
        // butterfly over the threads: at every step a thread keeps half of its values and passes on the other half
        float v[VALUES];
#pragma unroll
        for (int r = 0; r < ROWS; r++)
#pragma unroll
            for (int p = 0; p < M / 2; p++) {
                const float2 both = unpack(acc[r][p]);
                v[r * M + 2 * p] = both.x;
                v[r * M + 2 * p + 1] = both.y;
            }
#pragma unroll
        for (int step = 0; step < 5; step++) {
            const int offset = 16 >> step, live = VALUES >> step, half = live / 2;
            if (live > 1) {
                const bool upper = (thread & offset) != 0;
#pragma unroll
                for (int i = 0; i < half; i++) {
                    const float keep = upper ? v[half + i] : v[i], send = upper ? v[i] : v[half + i];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, offset);
                }
            } else {
                v[0] = v[0] + __shfl_xor_sync(0xffffffffu, v[0], offset);
            }
        }
#pragma unroll
        for (int i = 0; i < PER_THREAD; i++) sums[i] = v[i];
    }
};

// M lanes of a tile: the smallest form that holds them
template <typename Two, typename Four, typename Eight>
__device__ __forceinline__ void by_count(int count, Two two, Four four, Eight eight) {
    if (count <= 2) two();
    else if (count <= 4) four();
    else eight();
}

struct Fp8LinearArgs {
    const uint8_t *xq;
    const float *xscale;
    const uint8_t *w[3];  // a SiLU pair: gate, up; else matrices that share the input
    const uint16_t *wscale[3];
    uint16_t *y[3];
    int n[3];
    int first[4];  // matrix b owns the row tiles first[b] .. first[b + 1] - 1
    const uint16_t *residual;
    int lanes, k, epilogue;
    int passes;  // a CTA covers 32 x passes rows
};

template <int M>
__device__ __forceinline__ void fp8_linear_tile(const Fp8LinearArgs &a, int m0, int count, uint8_t *smem) {
    const int warp = threadIdx.x >> 5, thread = threadIdx.x & 31, blocks = a.k >> 7;
    const int tile = blockIdx.x, matrix = tile < a.first[1] ? 0 : tile < a.first[2] ? 1 : 2, rows = a.n[matrix];
    const uint8_t *const w = a.w[matrix];
    auto stage = [&](int first, int n) { stage_activations<M>(a.xq, a.xscale, a.k, first, n, count, smem, [&](int m) { return m0 + m; }); };
    const int warps = 32 * a.passes / RowSums<M, false>::ROWS;  // with rows to do in a pass
    for (int pass = 0; pass < (warps + FP8_WARPS - 1) / FP8_WARPS; pass++) {
        const int row0 = (tile - a.first[matrix]) * 32 * a.passes + (pass * FP8_WARPS + warp) * RowSums<M, false>::ROWS;
        RowSums<M, false> sums;
        const uint16_t *scale_row = a.wscale[matrix] + static_cast<size_t>(min(row0, rows - 1) >> 7) * blocks;  // eight rows lie in one block of 128
        sums.run([&](int r) { return w + static_cast<size_t>(min(row0 + r, rows - 1)) * a.k; }, scale_row, scale_row, blocks, smem, pass > 0, stage);
        if (RowSums<M, false>::VALUES < 32 && (thread & 1) != 0) continue;
#pragma unroll
        for (int i = 0; i < RowSums<M, false>::PER_THREAD; i++) {
            const int output = RowSums<M, false>::index(thread, i), row = row0 + output / M, m = output % M;
            if (row >= rows || m >= count || warp >= warps) continue;
            const size_t out = static_cast<size_t>(m0 + m) * rows + row;
            float sum = sums.sums[i];
            if (a.epilogue == EPILOGUE_RESIDUAL_F32) sum = bf16_bits_to_f32(a.residual[out]) + sum;
            else if (a.epilogue == EPILOGUE_RESIDUAL_ROUNDED) sum = round_bf16(sum) + bf16_bits_to_f32(a.residual[out]);
            a.y[matrix][out] = static_cast<uint16_t>(f32_to_bf16_bits(sum));
        }
    }
}

// grid (row tiles of 32 x passes, lane tiles of 8)
__global__ void __launch_bounds__(FP8_WARPS * 32, 2) linear_fp8_kernel(const __grid_constant__ Fp8LinearArgs a) {
    extern __shared__ __align__(16) uint8_t fp8_smem[];
    grid_launch_dependents();
    grid_dependency_wait();
    const int m0 = blockIdx.y * TILE_LANES, count = min(TILE_LANES, a.lanes - m0);
    by_count(count, [&] { fp8_linear_tile<2>(a, m0, count, fp8_smem); }, [&] { fp8_linear_tile<4>(a, m0, count, fp8_smem); },
             [&] { fp8_linear_tile<8>(a, m0, count, fp8_smem); });
}

// rounded_silu(round(gate)) * round(up) from a warp's sums: the first half of the rows is gate, the second the same rows of up
template <int M, typename Store>
__device__ __forceinline__ void silu_outputs(const RowSums<M, true> &sums, Store store) {
    const int thread = threadIdx.x & 31;
    constexpr int PER = RowSums<M, true>::PER_THREAD;
    float other[PER];
    // the up sums of a thread's gate outputs sit in the thread 16 further (the top bit of the output index)
#pragma unroll
    for (int i = 0; i < PER; i++) other[i] = __shfl_xor_sync(0xffffffffu, sums.sums[i], 16);
    if (thread >= 16 || (RowSums<M, true>::VALUES < 32 && (thread & 1) != 0)) return;
#pragma unroll
    for (int i = 0; i < PER; i++) {
        const int output = RowSums<M, true>::index(thread, i);
        store(output / M, output % M, round_bf16(sums.sums[i]), round_bf16(other[i]));
    }
}

template <int M>
__device__ __forceinline__ void fp8_silu_tile(const Fp8LinearArgs &a, int m0, int count, uint8_t *smem) {
    const int warp = threadIdx.x >> 5, blocks = a.k >> 7;
    auto stage = [&](int first, int n) { stage_activations<M>(a.xq, a.xscale, a.k, first, n, count, smem, [&](int m) { return m0 + m; }); };
    constexpr int HALF = RowSums<M, true>::ROWS / 2;
    const int warps = 32 * a.passes / RowSums<M, true>::ROWS;
    for (int pass = 0; pass < (warps + FP8_WARPS - 1) / FP8_WARPS; pass++) {
        const int row0 = blockIdx.x * 16 * a.passes + (pass * FP8_WARPS + warp) * HALF, first = min(row0, a.n[0] - 1);
        RowSums<M, true> sums;
        sums.run([&](int r) { return a.w[r / HALF] + static_cast<size_t>(min(row0 + r % HALF, a.n[0] - 1)) * a.k; }, a.wscale[0] + static_cast<size_t>(first >> 7) * blocks,
                 a.wscale[1] + static_cast<size_t>(first >> 7) * blocks, blocks, smem, pass > 0, stage);
        silu_outputs<M>(sums, [&](int r, int m, float gate, float up) {
            if (row0 + r >= a.n[0] || m >= count || warp >= warps) return;
            a.y[0][static_cast<size_t>(m0 + m) * a.n[0] + row0 + r] = static_cast<uint16_t>(f32_to_bf16_bits(rounded_silu(gate) * up));
        });
    }
}

__global__ void __launch_bounds__(FP8_WARPS * 32, 2) linear_silu_multiply_fp8_kernel(const __grid_constant__ Fp8LinearArgs a) {
    extern __shared__ __align__(16) uint8_t fp8_smem[];
    grid_launch_dependents();
    grid_dependency_wait();
    const int m0 = blockIdx.y * TILE_LANES, count = min(TILE_LANES, a.lanes - m0);
    by_count(count, [&] { fp8_silu_tile<2>(a, m0, count, fp8_smem); }, [&] { fp8_silu_tile<4>(a, m0, count, fp8_smem); },
             [&] { fp8_silu_tile<8>(a, m0, count, fp8_smem); });
}

// ---- sparse experts

// Groups the (token, route) pairs by expert: order[] = pair indices expert by expert, tiles[t] = {expert, first place in
// order, count <= 8}, tile_count.  One CTA.
constexpr int GROUP_THREADS = 1024, GROUP_MAX_EXPERTS = 1024;
__global__ void __launch_bounds__(GROUP_THREADS) moe_group_kernel(const uint32_t *__restrict__ routes, int pairs, int experts, MoeGroups groups) {
    __shared__ int counts[GROUP_MAX_EXPERTS], places[GROUP_MAX_EXPERTS], tile_places[GROUP_MAX_EXPERTS];
    __shared__ int warp_pairs[32], warp_tiles[32];
    grid_launch_dependents();
    grid_dependency_wait();
    const int e = threadIdx.x;
    counts[e] = 0;
    __syncthreads();
    auto expert_of = [&](int pair) {
        const int expert = static_cast<int>(routes[pair] & 0xffffu);
        return expert < experts ? expert : -1;
    };
    for (int pair = threadIdx.x; pair < pairs; pair += GROUP_THREADS) {
        const int expert = expert_of(pair);
        if (expert >= 0) atomicAdd(&counts[expert], 1);
    }
    __syncthreads();
    // exclusive sums of pairs and tiles over the experts
    const int own = counts[e], own_tiles = (own + TILE_LANES - 1) / TILE_LANES;
    int before = own, tiles_before = own_tiles;
    for (int offset = 1; offset < 32; offset <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, before, offset), b = __shfl_up_sync(0xffffffffu, tiles_before, offset);
        if ((e & 31) >= offset) {
            before += a;
            tiles_before += b;
        }
    }
    if ((e & 31) == 31) {
        warp_pairs[e >> 5] = before;
        warp_tiles[e >> 5] = tiles_before;
    }
    __syncthreads();
    int base = 0, tile_base = 0;
    for (int w = 0; w < (e >> 5); w++) {
        base += warp_pairs[w];
        tile_base += warp_tiles[w];
    }
    places[e] = base + before - own;
    tile_places[e] = tile_base + tiles_before - own_tiles;
    for (int t = 0; t < own_tiles; t++) groups.tiles[tile_places[e] + t] = make_int4(e, places[e] + t * TILE_LANES, min(TILE_LANES, own - t * TILE_LANES), 0);
    if (e == GROUP_MAX_EXPERTS - 1) *groups.tile_count = tile_base + tiles_before;
    __syncthreads();
    for (int pair = threadIdx.x; pair < pairs; pair += GROUP_THREADS) {
        const int expert = expert_of(pair);
        if (expert >= 0) groups.order[atomicAdd(&places[expert], 1)] = pair;
    }
}

struct MoeArgs {
    const uint8_t *xq;
    const float *xscale;
    const uint32_t *routes;
    const uint8_t *w;
    const uint16_t *wscale;
    uint16_t *out;
    MoeGroups groups;
    int hidden, inter, top_k;
    int passes;  // a CTA's rows: so many times those its warps hold at a time
};

// grid (tiles of 32 intermediate rows x passes, expert tiles); the activations of a pair are its token's row
template <int M>
__device__ __forceinline__ void moe_gate_up_tile(const MoeArgs &a, int4 tile, uint8_t *smem) {
    const int warp = threadIdx.x >> 5, k = a.hidden, blocks = k >> 7, count = tile.z;
    const int *order = a.groups.order + tile.y;
    auto stage = [&](int first, int n) { stage_activations<M>(a.xq, a.xscale, k, first, n, count, smem, [&](int m) { return order[m] / a.top_k; }); };
    constexpr int HALF = RowSums<M, true>::ROWS / 2;
    const int expert = tile.x;
    const uint8_t *w = a.w + static_cast<size_t>(expert) * 2 * a.inter * k;
    const uint16_t *ws = a.wscale + static_cast<size_t>(expert) * ((2 * a.inter + 127) >> 7) * blocks;
    for (int pass = 0; pass < a.passes * FP8_ROWS / RowSums<M, true>::ROWS; pass++) {
        const int row0 = blockIdx.x * FP8_WARPS * a.passes * (FP8_ROWS / 2) + (pass * FP8_WARPS + warp) * HALF, first = min(row0, a.inter - 1);
        RowSums<M, true> sums;
        sums.run([&](int r) { return w + static_cast<size_t>((r >= HALF ? a.inter : 0) + min(row0 + r % HALF, a.inter - 1)) * k; },
                 ws + static_cast<size_t>(first >> 7) * blocks, ws + static_cast<size_t>((a.inter + first) >> 7) * blocks, blocks, smem, pass > 0, stage);
        silu_outputs<M>(sums, [&](int r, int m, float gate, float up) {
            if (row0 + r >= a.inter || m >= count) return;
            const float value = round_bf16(round_bf16(gate / (1.0f + expf(-gate))) * up);
            a.out[static_cast<size_t>(order[m]) * a.inter + row0 + r] = static_cast<uint16_t>(f32_to_bf16_bits(value));
        });
    }
}

__global__ void __launch_bounds__(FP8_WARPS * 32, 2) moe_gate_up_fp8_kernel(const __grid_constant__ MoeArgs a) {
    extern __shared__ __align__(16) uint8_t fp8_smem[];
    grid_launch_dependents();
    grid_dependency_wait();
    if (static_cast<int>(blockIdx.y) >= *a.groups.tile_count) return;
    const int4 tile = a.groups.tiles[blockIdx.y];
    by_count(tile.z, [&] { moe_gate_up_tile<2>(a, tile, fp8_smem); }, [&] { moe_gate_up_tile<4>(a, tile, fp8_smem); }, [&] { moe_gate_up_tile<8>(a, tile, fp8_smem); });
}

// grid (tiles of 64 hidden rows x passes, expert tiles); out = bf16(bf16(sum) * route weight) per pair
template <int M>
__device__ __forceinline__ void moe_down_tile(const MoeArgs &a, int4 tile, uint8_t *smem) {
    const int warp = threadIdx.x >> 5, thread = threadIdx.x & 31, k = a.inter, blocks = k >> 7, count = tile.z;
    const int *order = a.groups.order + tile.y;
    auto stage = [&](int first, int n) { stage_activations<M>(a.xq, a.xscale, k, first, n, count, smem, [&](int m) { return order[m]; }); };
    const int expert = tile.x;
    const uint8_t *w = a.w + static_cast<size_t>(expert) * a.hidden * k;
    const uint16_t *ws = a.wscale + static_cast<size_t>(expert) * ((a.hidden + 127) >> 7) * blocks;
    for (int pass = 0; pass < a.passes * FP8_ROWS / RowSums<M, false>::ROWS; pass++) {
        const int row0 = blockIdx.x * FP8_WARPS * a.passes * FP8_ROWS + (pass * FP8_WARPS + warp) * RowSums<M, false>::ROWS;
        const uint16_t *scale_row = ws + static_cast<size_t>(min(row0, a.hidden - 1) >> 7) * blocks;
        RowSums<M, false> sums;
        sums.run([&](int r) { return w + static_cast<size_t>(min(row0 + r, a.hidden - 1)) * k; }, scale_row, scale_row, blocks, smem, pass > 0, stage);
        if (RowSums<M, false>::VALUES < 32 && (thread & 1) != 0) continue;
#pragma unroll
        for (int i = 0; i < RowSums<M, false>::PER_THREAD; i++) {
            const int output = RowSums<M, false>::index(thread, i), row = row0 + output / M, m = output % M;
            if (row >= a.hidden || m >= count) continue;
            const float weight = bf16_bits_to_f32(a.routes[order[m]] >> 16);
            a.out[static_cast<size_t>(order[m]) * a.hidden + row] = static_cast<uint16_t>(f32_to_bf16_bits(round_bf16(sums.sums[i]) * weight));
        }
    }
}

__global__ void __launch_bounds__(FP8_WARPS * 32, 2) moe_down_fp8_kernel(const __grid_constant__ MoeArgs a) {
    extern __shared__ __align__(16) uint8_t fp8_smem[];
    grid_launch_dependents();
    grid_dependency_wait();
    if (static_cast<int>(blockIdx.y) >= *a.groups.tile_count) return;
    const int4 tile = a.groups.tiles[blockIdx.y];
    by_count(tile.z, [&] { moe_down_tile<2>(a, tile, fp8_smem); }, [&] { moe_down_tile<4>(a, tile, fp8_smem); }, [&] { moe_down_tile<8>(a, tile, fp8_smem); });
}

template <typename Args>
cudaError_t launch_rows(void (*kernel)(Args), dim3 grid, int tile_lanes, cudaStream_t stream, const Args &args) {
    auto bytes = [](int m) { return static_cast<size_t>(CHUNK) * 128 * m * 2 + static_cast<size_t>(CHUNK) * m * sizeof(float); };
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(bytes(8)));
    if (status != cudaSuccess) return status;
    return launch_dependent(kernel, grid, dim3(FP8_WARPS * 32), bytes(tile_lanes <= 2 ? 2 : tile_lanes <= 4 ? 4 : 8), 1, stream, args);
}

// Rows of a CTA in units of 32: 64 save half of the staging, 32 spread a small launch over more SMs; 128 and 256 save more of
// it where some five waves of CTAs are left (1024 lanes of 2048 x 4096: 509 -> 488 us, of 5120 x 2048: 664 -> 632 us).
int fp8_passes(int row_tiles, int lanes) {  // (row tiles of 64)
    const long long ctas = static_cast<long long>(row_tiles) * ((lanes + TILE_LANES - 1) / TILE_LANES);
    int passes = ctas < 2 * multiprocessors() ? 1 : 2;
    while (passes > 1 && passes < 8 && ctas / passes >= 10 * multiprocessors()) passes *= 2;
    return passes;
}

}  // namespace

cudaError_t launch_linear_fp8(const uint8_t *xq, const float *xscale, const uint8_t *w, const uint16_t *wscale,
                              uint16_t *y, const uint16_t *residual, int lanes, int n, int k, int epilogue,
                              cudaStream_t stream) {
    LinearBranches branches;
    branches.add(w, wscale, y, n);
    return launch_linear_fp8_multi(xq, xscale, branches, residual, lanes, k, epilogue, stream);
}

cudaError_t launch_linear_fp8_multi(const uint8_t *xq, const float *xscale, const LinearBranches &branches, const uint16_t *residual, int lanes, int k,
                                    int epilogue, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (k % 128 != 0) return cudaErrorInvalidValue;
    Fp8LinearArgs args = {};
    int tiles = 0;
    for (int b = 0; b < branches.count; b++) tiles += (branches.n[b] + 63) / 64;
    args.passes = fp8_passes(tiles, lanes);
    tiles = 0;
    for (int b = 0; b < 3; b++) {
        args.first[b] = tiles;
        if (b >= branches.count) continue;
        args.w[b] = static_cast<const uint8_t *>(branches.w[b]);
        args.wscale[b] = branches.scale[b];
        args.y[b] = static_cast<uint16_t *>(branches.y[b]);
        args.n[b] = branches.n[b];
        tiles += (branches.n[b] + 32 * args.passes - 1) / (32 * args.passes);
    }
    args.first[3] = tiles;
    for (int b = branches.count; b < 3; b++) args.first[b] = tiles;
    args.xq = xq;
    args.xscale = xscale;
    args.residual = residual;
    args.lanes = lanes;
    args.k = k;
    args.epilogue = epilogue;
    return launch_rows(linear_fp8_kernel, dim3(tiles, (lanes + TILE_LANES - 1) / TILE_LANES), lanes, stream, args);
}

cudaError_t launch_linear_silu_multiply_fp8(const uint8_t *xq, const float *xscale, const uint8_t *wg,
                                            const uint16_t *wg_scale, const uint8_t *wu, const uint16_t *wu_scale,
                                            uint16_t *y, int lanes, int n, int k, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (k % 128 != 0) return cudaErrorInvalidValue;
    const int passes = fp8_passes((n + 31) / 32, lanes), rows = 16 * passes;
    Fp8LinearArgs args = {};
    args.xq = xq;
    args.xscale = xscale;
    args.w[0] = wg;
    args.w[1] = wu;
    args.wscale[0] = wg_scale;
    args.wscale[1] = wu_scale;
    args.y[0] = y;
    args.n[0] = n;
    args.lanes = lanes;
    args.k = k;
    args.epilogue = EPILOGUE_BF16;
    args.passes = passes;
    return launch_rows(linear_silu_multiply_fp8_kernel, dim3((n + rows - 1) / rows, (lanes + TILE_LANES - 1) / TILE_LANES), lanes, stream, args);
}

size_t moe_group_bytes(int lanes, int top_k, int experts) {
    const size_t pairs = static_cast<size_t>(lanes) * top_k;
    return (pairs / TILE_LANES + experts + 1) * sizeof(int4) + (pairs + 4) * sizeof(int);
}
MoeGroups moe_groups(void *scratch, int lanes, int top_k, int experts) {
    MoeGroups groups;
    const size_t pairs = static_cast<size_t>(lanes) * top_k;
    groups.tiles = static_cast<int4 *>(scratch);
    groups.order = reinterpret_cast<int *>(groups.tiles + pairs / TILE_LANES + experts + 1);
    groups.tile_count = groups.order + pairs;
    return groups;
}

cudaError_t launch_moe_group(const uint32_t *routes, const MoeGroups &groups, int lanes, int top_k, int experts, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (experts > GROUP_MAX_EXPERTS) return cudaErrorInvalidValue;
    return launch_dependent(moe_group_kernel, dim3(1), dim3(GROUP_THREADS), 0, 1, stream, routes, lanes * top_k, experts, groups);
}

static int most_tiles(int lanes, int top_k, int experts) {
    const int pairs = lanes * top_k;
    return pairs < pairs / TILE_LANES + experts ? pairs : pairs / TILE_LANES + experts;
}

// A CTA waits for its tile's entry, its pairs and their rows, one after the other, before it stages the activations: about
// half of its time when it takes 64 rows of a few pairs.  More rows per CTA pay for that once, as long as some five waves
// of CTAs are left (128 experts of 2048 x 768, 8 per token, gate and up with down: 24 tokens 186 -> 166 us with two passes,
// 1024 tokens 3090 -> 2680 us with four).
static int moe_passes(int row_tiles, int expert_tiles) {
    int passes = 1;
    while (passes < 4 && static_cast<long long>(row_tiles) * expert_tiles / (2 * passes) >= 10 * multiprocessors()) passes *= 2;
    return passes;
}

cudaError_t launch_moe_gate_up_fp8(const uint8_t *xq, const float *xscale, const MoeGroups &groups, const uint8_t *w,
                                   const uint16_t *wscale, uint16_t *intermediates, int lanes, int hidden_size,
                                   int inter, int experts, int top_k, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (hidden_size % 128 != 0) return cudaErrorInvalidValue;
    const int tiles = most_tiles(lanes, top_k, experts), passes = moe_passes((inter + 31) / 32, tiles), rows = FP8_WARPS * passes * FP8_ROWS / 2;
    const MoeArgs args{xq, xscale, nullptr, w, wscale, intermediates, groups, hidden_size, inter, top_k, passes};
    return launch_rows(moe_gate_up_fp8_kernel, dim3((inter + rows - 1) / rows, tiles), TILE_LANES, stream, args);
}

cudaError_t launch_moe_down_fp8(const uint8_t *xq, const float *xscale, const MoeGroups &groups, const uint32_t *routes, const uint8_t *w,
                                const uint16_t *wscale, uint16_t *outputs, int lanes, int hidden_size, int inter,
                                int experts, int top_k, cudaStream_t stream) {
    if (lanes <= 0) return cudaSuccess;
    if (inter % 128 != 0) return cudaErrorInvalidValue;
    const int tiles = most_tiles(lanes, top_k, experts), passes = moe_passes((hidden_size + 63) / 64, tiles), rows = FP8_WARPS * passes * FP8_ROWS;
    const MoeArgs args{xq, xscale, routes, w, wscale, outputs, groups, hidden_size, inter, top_k, passes};
    return launch_rows(moe_down_fp8_kernel, dim3((hidden_size + rows - 1) / rows, tiles), TILE_LANES, stream, args);
}

}  // namespace nerve
