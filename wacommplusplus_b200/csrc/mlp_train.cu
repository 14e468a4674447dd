// Training of the advection surrogate's MLP (388 -> 256 -> 256 -> 256 -> 3, GELU tanh form, the
// outputs multiplied by the stencil's uniformity gate) with the library's own kernels: the forward
// pass, the mean-squared loss against the targets, the backward pass through all four layers and
// an Adam update. The GEMMs of layers 1-3 (forward, input gradients) and their weight gradients run
// on the tcgen05 tensor cores with BF16 operands and FP32 accumulation; the three-output layer 4, the
// loss, GELU and its derivative, bias sums and Adam are FP32 on the CUDA cores (layer 4's weight
// gradient from BF16-rounded operands). The parameters use the flat layout of
// wacomm_b200_set_surrogate (w1 [256][388], b1, w2 [256][256], b2, w3, b3, w4 [3][256], b4), so
// trained weights go to the inference kernels unchanged.
//
// A step is four launches:
//   pack_weights_kernel  W1, W2, W3 as BF16 in the tensor cores' shared-memory layout (umma.cuh);
//   tile_kernel          128 rows of the batch through the forward pass, the loss and the input
//                        gradients of every layer, with the activations in shared memory and the
//                        accumulators in tensor memory; leaves the BF16 operands of the weight
//                        gradients (X, H1, H2, dZ1, dZ2, dZ3) as shared-memory images and the
//                        tile's bias, layer-4 and loss sums;
//   weight_grad_kernel   dW = dZ^T X of layers 1-3 over a range of tiles: the images as they are,
//                        read along the other index (MN-major operands);
//   finish_kernel        the partial sums in a fixed order, the gradients, Adam.
// Every sum runs in a fixed order: a step is reproducible bit for bit.
#include <cmath>

#include <cuda_bf16.h>

#include "engine.h"
#include "launch_rules.h"
#include "umma.cuh"

namespace wb {
namespace {

constexpr int T_HID = 256, T_STENCIL = 384, T_PARTICLE = 4, T_IN = T_STENCIL + T_PARTICLE,
              T_OUT = 3;
constexpr size_t OFF_TW1 = 0, OFF_TB1 = OFF_TW1 + (size_t)T_HID * T_IN, OFF_TW2 = OFF_TB1 + T_HID,
                 OFF_TB2 = OFF_TW2 + (size_t)T_HID * T_HID, OFF_TW3 = OFF_TB2 + T_HID,
                 OFF_TB3 = OFF_TW3 + (size_t)T_HID * T_HID, OFF_TW4 = OFF_TB3 + T_HID,
                 OFF_TB4 = OFF_TW4 + (size_t)T_OUT * T_HID, T_PARAMS = OFF_TB4 + T_OUT;

constexpr int TROWS = 128;                     // rows of a tile
constexpr int X_KB = (T_IN + 63) / 64;         // 7 K-blocks of the input (388 -> 448, zero-padded)
constexpr int H_KB = T_HID / 64;               // 4 K-blocks of a hidden layer
constexpr uint32_t A_BLOCK = TROWS * 128;      // 16 KB: 128 rows x 64 BF16
constexpr uint32_t W_BLOCK = T_HID * 128;      // 32 KB: 256 rows x 64 BF16
constexpr uint32_t X_IMAGE = X_KB * A_BLOCK, H_IMAGE = H_KB * A_BLOCK;
constexpr int W_BLOCKS = X_KB + 2 * H_KB;      // W1, W2, W3
constexpr int W2_BLOCK = X_KB, W3_BLOCK = X_KB + H_KB;

// Sums of a tile over its rows: db1, db2, db3, dW4 [3][256], db4 [3], loss.
constexpr int SUM_DB = 0, SUM_DW4 = 3 * T_HID, SUM_DB4 = 6 * T_HID, SUM_LOSS = SUM_DB4 + T_OUT,
              SUMS = SUM_LOSS + 1;

// Weight-gradient units: 128 rows (hidden units of dZ) by up to 256 columns each: W3, W2 (two row
// halves), W1 (two row halves by two column parts).
constexpr int UNITS = 8;
constexpr int X_TAIL = T_IN - T_HID;           // columns of W1's second part
constexpr int X_TAIL_N = (X_TAIL + 15) / 16 * 16;
constexpr int MAX_SPLITS = B200_SMS / UNITS;   // ranges of tiles: about one block per SM

// The work buffer: an error word (at its start), then, from the next 1024-byte boundary, the packed
// weights, the images and sums per tile and the partial weight gradients.
struct Work {
    int *err;
    uint8_t *weights;                    // [W_BLOCKS][W_BLOCK]
    uint8_t *X, *H1, *H2, *dZ1, *dZ2, *dZ3;  // [tiles] images
    float4 *slope1;                      // [tiles][T_HID / 4][TROWS]: GELU'(Z1)
    float *sums;                         // [tiles][SUMS]
    float4 *partial;                     // [UNITS][splits][T_HID / 4][TROWS]
};

size_t tiles_of(int batch) { return ((size_t)batch + TROWS - 1) / TROWS; }

size_t work_bytes(size_t tiles, Work *w, uint8_t *base) {
    size_t at = 0;
    auto take = [&](size_t bytes) {
        uint8_t *p = base ? base + at : nullptr;
        at += (bytes + 1023) / 1024 * 1024;
        return p;
    };
    Work f{};
    f.weights = take((size_t)W_BLOCKS * W_BLOCK);
    f.X = take(tiles * X_IMAGE);
    f.H1 = take(tiles * H_IMAGE);
    f.H2 = take(tiles * H_IMAGE);
    f.dZ1 = take(tiles * H_IMAGE);
    f.dZ2 = take(tiles * H_IMAGE);
    f.dZ3 = take(tiles * H_IMAGE);
    f.slope1 = reinterpret_cast<float4 *>(take(tiles * TROWS * T_HID * sizeof(float)));
    f.sums = reinterpret_cast<float *>(take(tiles * SUMS * sizeof(float)));
    f.partial = reinterpret_cast<float4 *>(
        take((size_t)UNITS * MAX_SPLITS * TROWS * T_HID * sizeof(float)));
    if (w) *w = f;
    return at;
}

__device__ __forceinline__ float gelu_exact_tanh(float x, float &derivative) {
    const float c0 = 0.7978845608028654f, c1 = 0.044715f;
    const float t = tanhf(c0 * (x + c1 * x * x * x));
    derivative = 0.5f * (1.f + t) + 0.5f * x * (1.f - t * t) * c0 * (1.f + 3.f * c1 * x * x);
    return 0.5f * x * (1.f + t);
}

__device__ __forceinline__ uint32_t pack_bf16x2(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t *>(&v);
}

__device__ __forceinline__ uint4 pack8(const float *v) {
    return make_uint4(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]), pack_bf16x2(v[4], v[5]),
                      pack_bf16x2(v[6], v[7]));
}

__device__ __forceinline__ float bf16_rounded(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

// Sum over the warp's 32 lanes of each of v[0..31]: lane l returns the sum of v[l] (v is used up).
// Each exchange halves the values a lane still carries: 31 shuffles for 32 sums.
__device__ __forceinline__ float lane_sums(float (&v)[32], int lane) {
#pragma unroll
    for (int s = 16; s >= 1; s >>= 1) {
        const bool upper = lane & s;
#pragma unroll
        for (int q = 0; q < s; q++) {
            const float send = upper ? v[q] : v[q + s], keep = upper ? v[q + s] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    }
    return v[0];
}

// ------------------------------------------------------------------ packed weights

// One thread per 16-byte chunk (8 k of one output unit) of the K-block images.
__global__ void pack_weights_kernel(const float *params, uint8_t *weights, int *err) {
    if (blockIdx.x == 0 && threadIdx.x == 0) *err = 0;
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= W_BLOCKS * T_HID * 8) return;
    const int chunk = e & 7, n = (e >> 3) % T_HID, block = (e >> 3) / T_HID;
    const int layer = block < W2_BLOCK ? 0 : block < W3_BLOCK ? 1 : 2;
    const int first = layer == 0 ? 0 : layer == 1 ? W2_BLOCK : W3_BLOCK;
    const int width = layer == 0 ? T_IN : T_HID;
    const float *row = params + (layer == 0 ? OFF_TW1 : layer == 1 ? OFF_TW2 : OFF_TW3) + (size_t)n * width;
    const int k = (block - first) * 64 + chunk * 8;
    float v[8];
#pragma unroll
    for (int q = 0; q < 8; q++) v[q] = k + q < width ? row[k + q] : 0.f;
    *reinterpret_cast<uint4 *>(weights + (size_t)block * W_BLOCK + umma::sw128_offset(n, chunk * 8)) = pack8(v);
}

// ------------------------------------------------------------------ forward and input gradients

struct TileArgs {
    const float *stencil, *particle, *gate, *target, *params;
    int batch, tiles;
    Work w;
};

constexpr int ROW_WARPS = 16, ROW_THREADS = ROW_WARPS * 32;
constexpr int PRODUCER_WARP = ROW_WARPS, MMA_WARP = ROW_WARPS + 1, TILE_THREADS = ROW_THREADS + 64;
constexpr int TRING = 3;
constexpr size_t TILE_SMEM = X_IMAGE + TRING * (size_t)W_BLOCK + 1024;
// The MMA jobs of a tile: layers 1, 2, 3 forward, then the gradients of H2 and H1.
constexpr int JOBS = 5;
__device__ __forceinline__ int job_blocks(int job) { return job == 0 ? X_KB : H_KB; }

// Bulk copy shared -> global, and the issuing thread's wait until its copies have read their source.
__device__ __forceinline__ void bulk_s2g(void *dst, const void *src, uint32_t bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(dst),
                 "r"(umma::smem_u32(src)), "r"(bytes)
                 : "memory");
    asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// A tile of 128 rows per turn, 16 row warps (TMEM lane quarter w % 4, columns 64 (w / 4) ..), one
// warp streaming weights through a ring of bulk copies, one issuing the MMAs. Operand buffer (112 KB):
// X, then H1, H2, dZ3, dZ2, dZ1 in turn, each copied out as it stands for the weight gradients.
// Tensor memory: columns 0-255 hold the accumulators of layers 1 and 3 and of both gradients,
// columns 256-511 that of layer 2, replaced by GELU'(Z2). Bound by the latency of one tile's chain of
// five GEMMs and epilogues (a precise tanhf per unit and layer) and by issue inside them: 16,384 rows,
// 128 tiles on 148 SMs, 71 us of a step of 0.107 ms (issue 39 %); with per-layer GEMMs that staged
// FP32 operands through threads the step took 0.720 ms. With the GELU unrolled over 32 columns its
// code overflowed the instruction cache: 90 us.
__global__ void __launch_bounds__(TILE_THREADS, 1) tile_kernel(const TileArgs a) {
    using namespace umma;
    extern __shared__ uint8_t dynSmem[];
    uint8_t *sA = reinterpret_cast<uint8_t *>(((uintptr_t)dynSmem + 1023) & ~(uintptr_t)1023);
    uint8_t *ring = sA + X_IMAGE;
    __shared__ __align__(8) uint64_t full[TRING], empty[TRING], aFull, accFull;
    __shared__ uint32_t tmemSlot;
    __shared__ int abortFlag, stopFlag;
    __shared__ __align__(16) float bias[3][T_HID], w4[T_OUT][T_HID];
    __shared__ float outSum[TROWS][T_OUT];
    __shared__ float colSum[4][T_HID];  // one sum over 32 rows per lane quarter
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < TRING; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&aFull, ROW_WARPS);
        mbar_init(&accFull, 1);
        abortFlag = 0;
        fence_barrier_init();
    }
    for (int c = tid; c < T_HID; c += TILE_THREADS) {
        bias[0][c] = a.params[OFF_TB1 + c];
        bias[1][c] = a.params[OFF_TB2 + c];
        bias[2][c] = a.params[OFF_TB3 + c];
        for (int o = 0; o < T_OUT; o++) w4[o][c] = a.params[OFF_TW4 + (size_t)o * T_HID + c];
    }
    if (warp == MMA_WARP) tmem_alloc(&tmemSlot, 512);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmemSlot;
    const int mine = blockIdx.x < a.tiles ? (a.tiles - 1 - blockIdx.x) / gridDim.x + 1 : 0;

    if (warp == PRODUCER_WARP) {
        if (lane == 0) {
            int issued[TRING];
            for (int s = 0; s < TRING; s++) issued[s] = -1;
            uint32_t g = 0;
            bool ok = true;
            for (int t = 0; t < mine && ok; t++)
                for (int job = 0; job < JOBS && ok; job++)
                    for (int kb = 0; kb < job_blocks(job) && ok; kb++, g++) {
                        const uint32_t s = g % TRING, n = g / TRING;
                        if (!(ok = mbar_wait(&empty[s], (n & 1) ^ 1, &abortFlag))) break;
                        mbar_expect_tx(&full[s], W_BLOCK);
                        uint8_t *dst = ring + s * W_BLOCK;
                        if (job < 3) {
                            const int block = (job == 0 ? 0 : job == 1 ? W2_BLOCK : W3_BLOCK) + kb;
                            bulk_g2s(dst, a.w.weights + (size_t)block * W_BLOCK, W_BLOCK, &full[s]);
                        } else {
                            // output units 64 kb .. of every K-block: [4][64 rows][128 bytes]
                            const int first = job == 3 ? W3_BLOCK : W2_BLOCK;
                            for (int b = 0; b < H_KB; b++)
                                bulk_g2s(dst + b * (W_BLOCK / 4),
                                         a.w.weights + (size_t)(first + b) * W_BLOCK + kb * (W_BLOCK / 4),
                                         W_BLOCK / 4, &full[s]);
                        }
                        issued[s] = (int)n;
                    }
            for (int s = 0; s < TRING; s++)  // copies still in flight land before the block exits
                if (issued[s] >= 0) mbar_wait_bounded(&full[s], (uint32_t)issued[s] & 1);
        }
        __syncwarp();
    } else if (warp == MMA_WARP) {
        if (lane == 0) {
            uint32_t g = 0, jobs = 0;
            bool ok = true;
            for (int t = 0; t < mine && ok; t++)
                for (int job = 0; job < JOBS && ok; job++, jobs++) {
                    if (!(ok = mbar_wait(&aFull, jobs & 1, &abortFlag))) break;
                    fence_after_sync();
                    const uint32_t d = tmem + (job == 1 ? T_HID : 0);
                    const uint32_t idesc = job < 3 ? idesc_bf16(TROWS, T_HID)
                                                   : idesc_bf16(TROWS, T_HID) | IDESC_B_MN_MAJOR;
                    for (int kb = 0; kb < job_blocks(job); kb++, g++) {
                        const uint32_t s = g % TRING, n = g / TRING;
                        if (!(ok = mbar_wait(&full[s], n & 1, &abortFlag))) break;
                        fence_after_sync();
                        const uint32_t A = smem_u32(sA + kb * A_BLOCK), B = smem_u32(ring + s * W_BLOCK);
#pragma unroll
                        for (int ks = 0; ks < 4; ks++)
                            mma_bf16(d, desc_sw128(A + ks * 32),
                                     job < 3 ? desc_sw128(B + ks * 32)
                                             : desc_sw128_mn(B + ks * 2048, W_BLOCK / 4),
                                     idesc, (kb | ks) != 0);
                        mma_commit(&empty[s]);
                    }
                    if (ok) mma_commit(&accFull);
                }
        }
        __syncwarp();
    } else {
        const int quarter = warp & 3, group = warp >> 2, r = quarter * 32 + lane, c0 = group * 64;
        const uint32_t acc = tmem + ((uint32_t)(quarter * 32) << 16);
        uint32_t jobs = 0;
        // Waits for a job's accumulator and for the operand buffer to have been copied out (a wait
        // that gives up raises the flag; the tile runs to its end on whatever is there).
        auto result = [&]() {
            mbar_wait(&accFull, jobs & 1, &abortFlag);
            jobs++;
            if (tid == 0) bulk_wait_read();
            __syncwarp();
            named_sync(1, ROW_THREADS);
            fence_after_sync();
        };
        // The operand buffer is written: copies it out and hands it to the tensor cores (if wanted).
        auto operand = [&](uint8_t *image, uint32_t bytes, bool more) {
            fence_async_shared();
            fence_before_sync();
            named_sync(1, ROW_THREADS);
            if (tid == 0) bulk_s2g(image, sA, bytes);
            if (more && lane == 0) mbar_arrive(&aFull);
            __syncwarp();
        };
        auto put8 = [&](int col, const float *v) {
            *reinterpret_cast<uint4 *>(sA + (col / 64) * A_BLOCK + sw128_offset(r, col % 64)) = pack8(v);
        };
        // This quarter's column sums into `out` (the tile's sums), the quarters added in order.
        auto column_sums = [&](float *out) {
            named_sync(1, ROW_THREADS);
            if (tid < T_HID)
                out[tid] = ((colSum[0][tid] + colSum[1][tid]) + colSum[2][tid]) + colSum[3][tid];
            named_sync(1, ROW_THREADS);
        };
        const bool aligned = ((reinterpret_cast<uintptr_t>(a.stencil) |
                               reinterpret_cast<uintptr_t>(a.particle)) & 15) == 0;
        for (int t = 0; t < mine; t++) {
            const size_t tile = blockIdx.x + (size_t)t * gridDim.x;
            const long long row0 = (long long)tile * TROWS;
            float *sums = a.w.sums + tile * SUMS;
            // ---- X: 16-byte chunks of 8 features, the particle features after the stencil's
            if (t > 0) {
                if (tid == 0) bulk_wait_read();
                named_sync(1, ROW_THREADS);
            }
            // (seven chunks per thread in flight)
            static_assert(TROWS * X_KB * 8 % (7 * ROW_THREADS) == 0, "whole groups of chunks");
#pragma unroll 7
            for (int turn = 0; turn < TROWS * X_KB * 8 / ROW_THREADS; turn++) {
                const int e = turn * ROW_THREADS + tid;
                const int row = e / (X_KB * 8), chunk = e % (X_KB * 8), k = chunk * 8;
                float v[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
                const long long n = row0 + row;
                if (n < a.batch && k < T_IN) {
                    const float *src = k < T_STENCIL ? a.stencil + n * T_STENCIL + k : a.particle + n * T_PARTICLE;
                    const int count = k < T_STENCIL ? 8 : T_PARTICLE;
                    if (aligned) {
                        *reinterpret_cast<float4 *>(v) = __ldg(reinterpret_cast<const float4 *>(src));
                        if (count == 8)
                            *reinterpret_cast<float4 *>(v + 4) = __ldg(reinterpret_cast<const float4 *>(src) + 1);
                    } else {
                        for (int q = 0; q < 8; q++)
                            if (q < count) v[q] = __ldg(src + q);
                    }
                }
                *reinterpret_cast<uint4 *>(sA + (k / 64) * A_BLOCK + sw128_offset(row, k % 64)) = pack8(v);
            }
            operand(a.w.X + tile * X_IMAGE, X_IMAGE, true);
            // ---- layer 1: H1 = GELU(Z1), its slope to global memory
            result();
            float4 *slope = a.w.slope1 + tile * (size_t)(T_HID / 4) * TROWS + r;
#pragma unroll 1
            for (int c = c0; c < c0 + 64; c += 8) {
                float v[8], d[8];
                tmem_ld8(acc + (uint32_t)c, v);
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = gelu_exact_tanh(v[e] + bias[0][c + e], d[e]);
                put8(c, v);
                slope[(size_t)(c / 4) * TROWS] = make_float4(d[0], d[1], d[2], d[3]);
                slope[(size_t)(c / 4 + 1) * TROWS] = make_float4(d[4], d[5], d[6], d[7]);
            }
            operand(a.w.H1 + tile * H_IMAGE, H_IMAGE, true);
            // ---- layer 2: H2 = GELU(Z2), its slope in the accumulator's place
            result();
#pragma unroll 1
            for (int c = c0; c < c0 + 64; c += 8) {
                float v[8], d[8];
                tmem_ld8(acc + (uint32_t)(T_HID + c), v);
#pragma unroll
                for (int e = 0; e < 8; e++) v[e] = gelu_exact_tanh(v[e] + bias[1][c + e], d[e]);
                put8(c, v);
                tmem_st8(acc + (uint32_t)(T_HID + c), d);
            }
            tmem_wait_st();
            operand(a.w.H2 + tile * H_IMAGE, H_IMAGE, true);
            // ---- layer 3: H3 in registers, its slope in the accumulator's place
            result();
            // (through this thread's own slots of the free operand buffer, so that one short loop
            // holds the GELU: unrolled over the registers its code overflows the instruction cache)
            float h3[64];
            float *slots = reinterpret_cast<float *>(sA) + group * 32 * TROWS + r;
#pragma unroll
            for (int half = 0; half < 2; half++) {
#pragma unroll 1
                for (int c = 0; c < 32; c += 8) {
                    const int col = c0 + 32 * half + c;
                    float v[8], d[8];
                    tmem_ld8(acc + (uint32_t)col, v);
#pragma unroll
                    for (int e = 0; e < 8; e++)
                        slots[(c + e) * TROWS] = gelu_exact_tanh(v[e] + bias[2][col + e], d[e]);
                    tmem_st8(acc + (uint32_t)col, d);
                }
#pragma unroll
                for (int e = 0; e < 32; e++) h3[32 * half + e] = slots[e * TROWS];
            }
            tmem_wait_st();
            // layer 4: each row's three sums run over the 256 units in order, so the four column
            // groups of a row take their turns
            float o[T_OUT];
#pragma unroll 1
            for (int turn = 0; turn < 4; turn++) {
                if (turn == group) {
#pragma unroll
                    for (int n = 0; n < T_OUT; n++) o[n] = turn ? outSum[r][n] : 0.f;
#pragma unroll
                    for (int e = 0; e < 64; e++)
#pragma unroll
                        for (int n = 0; n < T_OUT; n++) o[n] = fmaf(h3[e], w4[n][c0 + e], o[n]);
#pragma unroll
                    for (int n = 0; n < T_OUT; n++) outSum[r][n] = o[n];
                }
                named_sync(2 + quarter, 128);
            }
            // Y = O g; loss = mean over batch and outputs of (Y - target)^2; dO = 2 (Y - target) g / (3 batch)
            const float scale = 1.f / (3.f * a.batch);
            const long long n = row0 + r;
            float dO[T_OUT], lossSum = 0.f;
#pragma unroll
            for (int q = 0; q < T_OUT; q++) {
                dO[q] = 0.f;
                if (n < a.batch) {
                    const float g = __ldg(a.gate + n);
                    const float d = (outSum[r][q] + __ldg(a.params + OFF_TB4 + q)) * g - __ldg(a.target + n * T_OUT + q);
                    lossSum += d * d;
                    dO[q] = 2.f * d * g * scale;
                }
            }
            // dW4 from BF16-rounded operands, one output at a time
#pragma unroll 1
            for (int q = 0; q < T_OUT; q++) {
                const float dq = bf16_rounded(q == 0 ? dO[0] : q == 1 ? dO[1] : dO[2]);
#pragma unroll
                for (int half = 0; half < 2; half++) {
                    float v[32];
#pragma unroll
                    for (int e = 0; e < 32; e++) v[e] = dq * bf16_rounded(h3[32 * half + e]);
                    colSum[quarter][c0 + 32 * half + lane] = lane_sums(v, lane);
                }
                column_sums(sums + SUM_DW4 + q * T_HID);
            }
            // db4 and the loss: the first group's warps, one per lane quarter
            if (group == 0) {
                float s[T_OUT + 1] = {dO[0], dO[1], dO[2], lossSum};
#pragma unroll
                for (int q = 0; q < T_OUT + 1; q++) {
                    for (int off = 16; off > 0; off >>= 1) s[q] += __shfl_xor_sync(0xffffffffu, s[q], off);
                    if (lane == 0) colSum[quarter][q] = s[q];
                }
            }
            named_sync(1, ROW_THREADS);
            if (tid < T_OUT + 1)
                sums[SUM_DB4 + tid] = ((colSum[0][tid] + colSum[1][tid]) + colSum[2][tid]) + colSum[3][tid];
            named_sync(1, ROW_THREADS);
            // ---- dZ3 = (dO W4) GELU'(Z3)
#pragma unroll 1
            for (int c = c0; c < c0 + 64; c += 32) {
                float v[32];
                tmem_ld32(acc + (uint32_t)c, v);
#pragma unroll
                for (int e = 0; e < 32; e++) {
                    float d = fmaf(dO[0], w4[0][c + e], 0.f);
                    d = fmaf(dO[1], w4[1][c + e], d);
                    d = fmaf(dO[2], w4[2][c + e], d);
                    v[e] = d * v[e];
                }
#pragma unroll
                for (int q = 0; q < 32; q += 8) put8(c + q, v + q);
                colSum[quarter][c + lane] = lane_sums(v, lane);
            }
            operand(a.w.dZ3 + tile * H_IMAGE, H_IMAGE, true);
            column_sums(sums + SUM_DB + 2 * T_HID);
            // ---- dZ2 = (dZ3 W3) GELU'(Z2)
            result();
#pragma unroll 1
            for (int c = c0; c < c0 + 64; c += 32) {
                float v[32], d[32];
                tmem_ld32(acc + (uint32_t)c, v);
                tmem_ld32(acc + (uint32_t)(T_HID + c), d);
#pragma unroll
                for (int e = 0; e < 32; e++) v[e] *= d[e];
#pragma unroll
                for (int q = 0; q < 32; q += 8) put8(c + q, v + q);
                colSum[quarter][c + lane] = lane_sums(v, lane);
            }
            operand(a.w.dZ2 + tile * H_IMAGE, H_IMAGE, true);
            column_sums(sums + SUM_DB + T_HID);
            // ---- dZ1 = (dZ2 W2) GELU'(Z1)
            result();
#pragma unroll 1
            for (int c = c0; c < c0 + 64; c += 32) {
                float v[32];
                tmem_ld32(acc + (uint32_t)c, v);
#pragma unroll
                for (int q = 0; q < 32; q += 4) {
                    const float4 d = slope[(size_t)((c + q) / 4) * TROWS];
                    v[q] *= d.x;
                    v[q + 1] *= d.y;
                    v[q + 2] *= d.z;
                    v[q + 3] *= d.w;
                }
#pragma unroll
                for (int q = 0; q < 32; q += 8) put8(c + q, v + q);
                colSum[quarter][c + lane] = lane_sums(v, lane);
            }
            operand(a.w.dZ1 + tile * H_IMAGE, H_IMAGE, false);
            column_sums(sums + SUM_DB);
            // one thread's reading of the flag decides for all row threads, which leave together
            if (tid == 0) stopFlag = abortFlag;
            named_sync(1, ROW_THREADS);
            if (stopFlag) break;
        }
        if (tid == 0) bulk_wait_all();
    }
    fence_before_sync();
    __syncthreads();
    if (warp == MMA_WARP) {
        fence_after_sync();
        tmem_dealloc(tmem, 512);
    }
    if (tid == 0 && abortFlag) atomicOr(a.w.err, 1);
}

// ------------------------------------------------------------------ weight gradients

constexpr uint32_t G_A = 2 * A_BLOCK, G_B = H_KB * A_BLOCK;  // 128 hidden units of dZ; up to 256 columns
constexpr size_t GRAD_SMEM = 2 * (size_t)(G_A + G_B) + 1024;
constexpr int GRAD_THREADS = 128;

struct GradArgs {
    int tiles, splits;
    Work w;
};

// Unit u over the tiles of its range: partial = sum over rows of dZ[row][m] V[row][n]. Both operands
// are the tiles' images read along their rows (MN-major: 64 units per 128-byte row, 8 rows per 1024
// bytes, the next 64 units one K-block further), two tiles in flight. Bound by the copies of the
// images from L2 (96 KB for 8 MMAs): 16.5 us at 16,384 rows (four GEMMs with staged operands before:
// 169 us and their split sums 42 us).
__global__ void __launch_bounds__(GRAD_THREADS, 1) weight_grad_kernel(const GradArgs a) {
    using namespace umma;
    extern __shared__ uint8_t dynSmem[];
    uint8_t *base = reinterpret_cast<uint8_t *>(((uintptr_t)dynSmem + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t full[2], empty[2], accFull;
    __shared__ uint32_t tmemSlot;
    __shared__ int abortFlag;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int unit = blockIdx.x, split = blockIdx.y, half = unit & 1;
    const int per = (a.tiles + a.splits - 1) / a.splits;
    const int first = split * per, last = min(a.tiles, first + per), count = max(last - first, 0);
    const int kind = unit >> 1;  // 0: W3, 1: W2, 2: W1 columns 0-255, 3: the rest of W1
    const uint8_t *A = (kind == 0 ? a.w.dZ3 : kind == 1 ? a.w.dZ2 : a.w.dZ1) + half * G_A;
    const uint8_t *B = kind == 0 ? a.w.H2 : kind == 1 ? a.w.H1 : kind == 2 ? a.w.X : a.w.X + G_B;
    const size_t strideB = kind < 2 ? H_IMAGE : X_IMAGE;
    const uint32_t bytesB = kind < 3 ? G_B : X_IMAGE - G_B;
    const int N = kind < 3 ? T_HID : X_TAIL_N;
    if (tid == 0) {
        for (int s = 0; s < 2; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&accFull, 1);
        abortFlag = 0;
        fence_barrier_init();
    }
    if (warp == 0) tmem_alloc(&tmemSlot, 256);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem = tmemSlot;
    if (tid == 0) {
        const uint32_t idesc = idesc_bf16(TROWS, N) | IDESC_A_MN_MAJOR | IDESC_B_MN_MAJOR;
        int issued[2] = {-1, -1};
        auto load = [&](int t) {
            const int s = t & 1, n = t >> 1;
            if (!mbar_wait(&empty[s], (uint32_t)(n & 1) ^ 1, &abortFlag)) return false;
            uint8_t *dst = base + s * (G_A + G_B);
            mbar_expect_tx(&full[s], G_A + bytesB);
            bulk_g2s(dst, A + (size_t)(first + t) * H_IMAGE, G_A, &full[s]);
            bulk_g2s(dst + G_A, B + (size_t)(first + t) * strideB, bytesB, &full[s]);
            issued[s] = n;
            return true;
        };
        int consumed[2] = {-1, -1};
        bool ok = count == 0 || load(0);
        for (int t = 0; t < count && ok; t++) {
            if (t + 1 < count) ok = load(t + 1);
            const int s = t & 1, n = t >> 1;
            if (!ok || !(ok = mbar_wait(&full[s], (uint32_t)n & 1, &abortFlag))) break;
            consumed[s] = n;
            fence_after_sync();
            const uint32_t sA = smem_u32(base + s * (G_A + G_B)), sB = sA + G_A;
#pragma unroll
            for (int ks = 0; ks < TROWS / 16; ks++)
                mma_bf16(tmem, desc_sw128_mn(sA + ks * 2048, A_BLOCK), desc_sw128_mn(sB + ks * 2048, A_BLOCK),
                         idesc, (t | ks) != 0);
            mma_commit(&empty[s]);
        }
        mma_commit(&accFull);
        for (int s = 0; s < 2; s++)  // copies still in flight land before the block exits
            if (issued[s] > consumed[s]) mbar_wait_bounded(&full[s], (uint32_t)issued[s] & 1);
    }
    __syncwarp();
    const bool done = mbar_wait_bounded(&accFull, 0);
    __syncwarp();
    fence_after_sync();
    float4 *out = a.w.partial + ((size_t)unit * a.splits + split) * (T_HID / 4) * TROWS + warp * 32 + lane;
    for (int c = 0; c < N; c += 32) {
        float v[32];
        tmem_ld32(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c, v);
#pragma unroll
        for (int q = 0; q < 32; q += 4)
            out[(size_t)((c + q) / 4) * TROWS] =
                count ? make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (tid == 0 && (!done || abortFlag)) atomicOr(a.w.err, 1);
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        fence_after_sync();
        tmem_dealloc(tmem, 256);
    }
}

// ------------------------------------------------------------------ sums and Adam

struct Adam {
    float *params, *grads, *m, *v;
    float lr, c1, c2;
    int update;
    // gradient of parameter e, then its Adam step (beta1 0.9, beta2 0.999, eps 1e-8, bias-corrected)
    __device__ __forceinline__ void apply(size_t e, float gi) const {
        grads[e] = gi;
        if (!update) return;
        const float mi = 0.9f * m[e] + 0.1f * gi, vi = 0.999f * v[e] + 0.001f * gi * gi;
        m[e] = mi;
        v[e] = vi;
        params[e] -= lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
    }
};

constexpr int WEIGHT_ITEMS = UNITS * (T_HID / 4) * TROWS;  // float4s of the partial weight gradients
constexpr int WEIGHT_BLOCKS = WEIGHT_ITEMS / 256;
constexpr int SUM_BLOCKS = (SUMS + 31) / 32;

// The first WEIGHT_BLOCKS blocks sum the splits of four weights per thread; the others sum 32 of the
// tile sums each, 8 ranges of tiles per column added in order.
__global__ void __launch_bounds__(256) finish_kernel(const GradArgs a, const Adam adam, float lossScale,
                                                     float *loss) {
    if (blockIdx.x < WEIGHT_BLOCKS) {
        const int e = blockIdx.x * 256 + threadIdx.x;
        const int r = e % TROWS, c = e / TROWS % (T_HID / 4) * 4, unit = e / (TROWS * (T_HID / 4));
        const int kind = unit >> 1;
        if (kind == 3 && c >= X_TAIL) return;
        const float4 *p = a.w.partial + (size_t)unit * a.splits * (T_HID / 4) * TROWS + (size_t)(c / 4) * TROWS + r;
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int z = 0; z < a.splits; z++) {
            const float4 q = p[(size_t)z * (T_HID / 4) * TROWS];
            s.x += q.x;
            s.y += q.y;
            s.z += q.z;
            s.w += q.w;
        }
        const int n = (unit & 1) * TROWS + r;
        const size_t at = kind == 0   ? OFF_TW3 + (size_t)n * T_HID + c
                          : kind == 1 ? OFF_TW2 + (size_t)n * T_HID + c
                                      : OFF_TW1 + (size_t)n * T_IN + (kind == 3 ? T_HID : 0) + c;
        adam.apply(at, s.x);
        adam.apply(at + 1, s.y);
        adam.apply(at + 2, s.z);
        adam.apply(at + 3, s.w);
        return;
    }
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int c = (blockIdx.x - WEIGHT_BLOCKS) * 32 + lane;
    const int per = (a.tiles + 7) / 8, first = warp * per, last = min(a.tiles, first + per);
    float s = 0.f;
    if (c < SUMS)
        for (int t = first; t < last; t++) s += a.w.sums[(size_t)t * SUMS + c];
    part[warp][lane] = s;
    __syncthreads();
    if (warp || c >= SUMS) return;
    s = 0.f;
    for (int q = 0; q < 8; q++) s += part[q][lane];
    if (c == SUM_LOSS) *loss = s * lossScale;
    else if (c >= SUM_DB4) adam.apply(OFF_TB4 + (c - SUM_DB4), s);
    else if (c >= SUM_DW4) adam.apply(OFF_TW4 + (c - SUM_DW4), s);
    else adam.apply((c < T_HID ? OFF_TB1 : c < 2 * T_HID ? OFF_TB2 : OFF_TB3) + c % T_HID, s);
}

// Shared-memory sizes of the tensor-core kernels, once per device.
cudaError_t train_prepare() {
    static bool done[64] = {};
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (device >= 0 && device < 64 && done[device]) return cudaSuccess;
    e = cudaFuncSetAttribute(tile_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TILE_SMEM);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(weight_grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GRAD_SMEM);
    if (e == cudaSuccess && device >= 0 && device < 64) done[device] = true;
    return e;
}

}  // namespace

size_t mlp_train_work_floats(int batch) {
    // the error word and the distance to the next 1024-byte boundary, then the work areas
    return (1024 + 16 + work_bytes(tiles_of(batch), nullptr, nullptr)) / sizeof(float);
}

cudaError_t mlp_train_step(const float *stencil, const float *particle, const float *gate,
                           const float *target, int batch, float *params, float *grads, float *m,
                           float *v, float *work, float *loss, int step, float lr, bool update,
                           cudaStream_t stream) {
    cudaError_t e = train_prepare();
    if (e != cudaSuccess) return e;
    const int tiles = (int)tiles_of(batch);
    Work w;
    work_bytes((size_t)tiles, &w,
               reinterpret_cast<uint8_t *>(((uintptr_t)(work + 4) + 1023) & ~(uintptr_t)1023));
    w.err = reinterpret_cast<int *>(work);
    pack_weights_kernel<<<W_BLOCKS * T_HID * 8 / 256, 256, 0, stream>>>(params, w.weights, w.err);
    const TileArgs t{stencil, particle, gate, target, params, batch, tiles, w};
    tile_kernel<<<tiles < B200_SMS ? tiles : B200_SMS, TILE_THREADS, TILE_SMEM, stream>>>(t);
    const GradArgs g{tiles, tiles < MAX_SPLITS ? tiles : MAX_SPLITS, w};
    weight_grad_kernel<<<dim3(UNITS, g.splits), GRAD_THREADS, GRAD_SMEM, stream>>>(g);
    const Adam adam{params, grads, m, v, lr, 1.f - powf(0.9f, (float)step),
                    1.f - powf(0.999f, (float)step), update ? 1 : 0};
    finish_kernel<<<WEIGHT_BLOCKS + SUM_BLOCKS, 256, 0, stream>>>(g, adam, 1.f / (3.f * batch), loss);
    return cudaGetLastError();
}

}  // namespace wb

extern "C" size_t wacomm_b200_mlp_train_work_floats(int batch) {
    return batch > 0 ? wb::mlp_train_work_floats(batch) : 0;
}

extern "C" int wacomm_b200_mlp_train_step(const float *stencil, const float *particle,
                                          const float *gate, const float *target, int batch,
                                          float *params, float *grads, float *m, float *v,
                                          float *work, float *loss, int step, float lr, int update,
                                          void *stream) {
    if (!stencil || !particle || !gate || !target || batch <= 0 || !params || !grads || !work ||
        !loss || (update && (!m || !v || step < 1)))
        return WACOMM_B200_ERR_ARGUMENT;
    const cudaError_t e = wb::mlp_train_step(stencil, particle, gate, target, batch, params, grads,
                                             m, v, work, loss, step, lr, update != 0,
                                             static_cast<cudaStream_t>(stream));
    return e == cudaSuccess ? WACOMM_B200_OK : WACOMM_B200_ERR_CUDA;
}
