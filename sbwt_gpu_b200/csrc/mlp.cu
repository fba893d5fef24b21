// mlp.cu -- kernels of the learned prefilter (no reference counterpart):
//   * gemm_tn_kernel: D = A * B^T on the tensor cores (tcgen05.mma, BF16 in
//     shared memory, FP32 accumulators in TMEM), used by training;
//   * mlp_infer_kernel: the fused inference pass -- one-hot tile built in
//     shared memory, layer 1 on the tensor cores, bias + ReLU + BF16 written
//     back into TMEM, layer 2 with its A operand read from TMEM, bias + ReLU +
//     the 256 -> 1 dot in the epilogue; weights stay resident in shared
//     memory for the whole (persistent) launch;
//   * training helpers (one-hot batches, transposes, loss, masks, Adam),
//     k-mer sampling from the index by select walks, and the Bloom filter.
#include <algorithm>
#include <cstdio>

#include "internal.h"
#include "mlp.h"
#include "mlp_kernels.cuh"

namespace sbwt {
namespace mlp {

using namespace tc;
using u16 = uint16_t;

// ------------------------------------------------------------------ GEMM

// D[M x N] = A[M x K] * B[N x K]^T for the K range of blockIdx.z; A and B
// row-major BF16, M a multiple of 128, N of BN, K of 64.  128 threads; thread t
// ends with row m0 + t of the tile in TMEM, and EPI says what becomes of it
// (TrainEpi).  Training is bound by the number of passes over its 2-8 MB
// matrices, so every pass that works on one row or writes a transposed copy is
// done here, from TMEM, where a warp's 32 rows make both forms of a store
// coalesce: with a kernel for each of them (bias and ReLU, head, ReLU gradient,
// five transposes, FP32 intermediates between them) a step took 18 launches.
enum { kEpiAdd, kEpiRelu, kEpiHead, kEpiReluGrad };

// Column sums over a warp's 32 rows: lane l returns the sum of column l & 15 of
// the lanes' 16 values.
__device__ __forceinline__ float column_sums(float (&v)[16], u32 lane) {
#pragma unroll
    for (u32 w = 8; w; w >>= 1) {
        const bool up = lane & w;
#pragma unroll
        for (u32 i = 0; i < 8u; i++) {
            if (i >= w) break;
            const float send = up ? v[i] : v[i + w], keep = up ? v[i + w] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, w);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 16);
}

__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// 16 bf16 values of one row, and the same as a column each of the transposed matrix (`rows` rows apart).
__device__ __forceinline__ void store_row(bf16 *row, const u32 (&h)[8]) {
    *reinterpret_cast<uint4 *>(row) = make_uint4(h[0], h[1], h[2], h[3]);
    *reinterpret_cast<uint4 *>(row + 8) = make_uint4(h[4], h[5], h[6], h[7]);
}

__device__ __forceinline__ void store_columns(bf16 *first, u32 rows, const u32 (&h)[8]) {
#pragma unroll
    for (u32 i = 0; i < 16u; i++) {
        const u16 x = (u16)(h[i / 2] >> (16u * (i & 1u)));
        *reinterpret_cast<u16 *>(first + (size_t)i * rows) = x;
    }
}

__device__ __forceinline__ float bf16_of(const u32 (&h)[8], u32 i) {
    return __uint_as_float(i & 1u ? h[i / 2] & 0xffff0000u : h[i / 2] << 16);
}

template <u32 BN, int EPI>
__global__ void __launch_bounds__(128) gemm_tn_kernel(const bf16 *__restrict__ A, const bf16 *__restrict__ B, u32 M,
                                                      u32 N, u32 K, u32 kps, const TrainEpi t, int *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar;
    __shared__ u32 tmem_s;
    __shared__ float s_sum[2][BN];  // column sums of the tile
    uint8_t *sA = smem;
    uint8_t *sB = smem + 128 * 64 * 2;
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    const u32 m0 = blockIdx.x * 128u, n0 = blockIdx.y * BN;
    if constexpr (EPI == kEpiHead || EPI == kEpiReluGrad)
        for (u32 i = tid; i < BN; i += 128u) s_sum[0][i] = s_sum[1][i] = 0.0f;
    const u32 kbeg = blockIdx.z * kps, kend = min(K, kbeg + kps);
    constexpr u32 kCols = BN < 32 ? 32 : BN;
    if (warp == 0) tmem_alloc(&tmem_s, kCols);
    if (tid == 0) mbar_init(&bar, 1);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const u32 tmem = tmem_s;
    u32 phase = 0;
    bool ok = true;
    for (u32 kb = kbeg; kb < kend && ok; kb += 64) {
#pragma unroll
        for (u32 i = tid; i < 128u * 8u; i += 128u) {
            const u32 r = i >> 3, kc = i & 7u;
            const uint4 v = *reinterpret_cast<const uint4 *>(A + (size_t)(m0 + r) * K + kb + kc * 8u);
            *reinterpret_cast<uint4 *>(sA + canon_offset(128, r, kc * 8u)) = v;
        }
#pragma unroll 8
        for (u32 i = tid; i < BN * 8u; i += 128u) {
            const u32 r = i >> 3, kc = i & 7u;
            const uint4 v = *reinterpret_cast<const uint4 *>(B + (size_t)(n0 + r) * K + kb + kc * 8u);
            *reinterpret_cast<uint4 *>(sB + canon_offset(BN, r, kc * 8u)) = v;
        }
        fence_smem_to_async();
        __syncthreads();
        if (tid == 0) {
            fence_after_sync();
#pragma unroll
            for (u32 s = 0; s < 4; s++) {
                const u64 da = smem_desc(smem_addr(sA) + s * 2u * 128u * 16u, 128u * 16u, 128u);
                const u64 db = smem_desc(smem_addr(sB) + s * 2u * BN * 16u, BN * 16u, 128u);
                mma_ss(tmem, da, db, idesc_bf16(128, BN), kb > kbeg || s > 0);
            }
            mma_commit(&bar);
        }
        const bool got = mbar_wait(&bar, phase, err, kErrGemmWait);
        phase ^= 1u;
        fence_after_sync();
        ok = __syncthreads_and(got);
    }
    if (ok && kend > kbeg) {
        const u32 row = m0 + warp * 32u + lane, acc = tmem + ((warp * 32u) << 16);
        float dz = 0.0f;
        if constexpr (EPI == kEpiHead) {
            // logit of the row: h2 = bf16(ReLU(z2 + b2)), h2 . w3 + b3; BCE with logits: softplus(z) - y z,
            // d/dz = sigmoid(z) - y
            float sum = 0.0f;
            for (u32 c = 0; c < BN; c += 16) {
                u32 v[16];
                tmem_ld16(acc + c, v);
                tmem_wait_ld();
                tmem_tie(v);
#pragma unroll
                for (int j = 0; j < 16; j++)
                    sum = fmaf(bf16_round(fmaxf(__uint_as_float(v[j]) + t.bias[c + j], 0.0f)), t.w3[c + j], sum);
            }
            const float z = sum + *t.b3, y = t.labels[row];
            const float sp = z > 0 ? z + log1pf(expf(-z)) : log1pf(expf(z));
            dz = (1.0f / (1.0f + expf(-z)) - y) / (float)M;
            const float loss = warp_sum((sp - y * z) / (float)M), db3 = warp_sum(dz);
            if (lane == 0) {
                atomicAdd(t.loss, loss);
                atomicAdd(t.g_b3, db3);
            }
        }
        for (u32 c = 0; c < BN; c += 16) {
            u32 v[16], h[8];
            tmem_ld16(acc + c, v);
            tmem_wait_ld();
            tmem_tie(v);
            if constexpr (EPI == kEpiAdd) {
                float *dst = t.add + (size_t)row * N + n0 + c;
#pragma unroll
                for (int j = 0; j < 16; j += 4)
                    atomicAdd(reinterpret_cast<float4 *>(dst + j),
                              make_float4(__uint_as_float(v[j]), __uint_as_float(v[j + 1]), __uint_as_float(v[j + 2]),
                                          __uint_as_float(v[j + 3])));
            } else if constexpr (EPI == kEpiRelu) {
#pragma unroll
                for (int j = 0; j < 16; j += 2)
                    h[j / 2] = pack_bf16x2(fmaxf(__uint_as_float(v[j]) + t.bias[n0 + c + j], 0.0f),
                                           fmaxf(__uint_as_float(v[j + 1]) + t.bias[n0 + c + j + 1], 0.0f));
                store_row(t.out + (size_t)row * N + n0 + c, h);
                store_columns(t.out_t + (size_t)(n0 + c) * M + row, M, h);
            } else if constexpr (EPI == kEpiHead) {
                // dz2 = dlogit * w3 * [h2 > 0]; gradients of w3 and b2: sums over the rows
                float dw[16], db[16];
#pragma unroll
                for (int j = 0; j < 16; j++) {
                    const float x = bf16_round(fmaxf(__uint_as_float(v[j]) + t.bias[c + j], 0.0f));
                    dw[j] = dz * x;
                    db[j] = x > 0.0f ? dz * t.w3[c + j] : 0.0f;
                }
#pragma unroll
                for (int j = 0; j < 16; j += 2) h[j / 2] = pack_bf16x2(db[j], db[j + 1]);
                store_row(t.out + (size_t)row * N + c, h);
                store_columns(t.out_t + (size_t)c * M + row, M, h);
#pragma unroll
                for (int j = 0; j < 16; j++) db[j] = bf16_of(h, j);
                const float sw = column_sums(dw, lane), sb = column_sums(db, lane);
                if (lane < 16) {
                    atomicAdd(&s_sum[0][c + lane], sw);
                    atomicAdd(&s_sum[1][c + lane], sb);
                }
            } else {
                // dz1 = dh1 * [h1 > 0], only its transpose is used; gradient of b1: sums over the rows
                const uint4 *hp = reinterpret_cast<const uint4 *>(t.h + (size_t)row * N + n0 + c);
                const uint4 h0 = hp[0], h1 = hp[1];
                const u32 m[8] = {h0.x, h0.y, h0.z, h0.w, h1.x, h1.y, h1.z, h1.w};
                float g[16];
#pragma unroll
                for (int j = 0; j < 16; j++) g[j] = bf16_of(m, j) > 0.0f ? __uint_as_float(v[j]) : 0.0f;
#pragma unroll
                for (int j = 0; j < 16; j += 2) h[j / 2] = pack_bf16x2(g[j], g[j + 1]);
                store_columns(t.out_t + (size_t)(n0 + c) * M + row, M, h);
#pragma unroll
                for (int j = 0; j < 16; j++) g[j] = bf16_of(h, j);
                const float sb = column_sums(g, lane);
                if (lane < 16) atomicAdd(&s_sum[1][c + lane], sb);
            }
        }
    }
    if constexpr (EPI == kEpiHead || EPI == kEpiReluGrad) {
        __syncthreads();
        for (u32 i = tid; i < BN; i += 128u) {
            if constexpr (EPI == kEpiHead) atomicAdd(t.g_w3 + i, s_sum[0][i]);
            atomicAdd(t.g_bias + n0 + i, s_sum[1][i]);
        }
    }
    if (!ok && tid == 0) mbar_wait(&bar, phase ^ 1u, err, kErrGemmWait);  // let an MMA still in flight land
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kCols);
}

// --------------------------------------------------------- fused inference

// W1, W2, the one-hot tile and the per-column-group partial dots: 226 KiB
constexpr u32 kInferThreads = 512;
constexpr u32 kColGroups = kInferThreads / kTileM;  // 4
constexpr u32 kGroupCols = kHid / kColGroups;       // 64
constexpr u32 kInferBlock = kInferThreads + 32;     // and the warp that issues the MMAs
constexpr u32 kInferSmem = kHid * kIn * 2 + kHid * kHid * 2 + kTileM * kIn * 2 + (kColGroups - 1) * kTileM * 4;

// One-hot chunks q0..q1-1 of row r: chunk q holds inputs 8q..8q+7 = letters
// 2q and 2q+1 (4 one-hot inputs each).
__device__ __forceinline__ void onehot_chunks(uint8_t *tile, u32 R, u32 r, u64 kmer, u32 k, u32 q0, u32 q1) {
#pragma unroll
    for (u32 q = q0; q < q1; q++) {
        const u32 i0 = 2 * q, i1 = 2 * q + 1;
        const u32 c0 = i0 < k ? letter(kmer, i0) : 4u;
        const u32 c1 = i1 < k ? letter(kmer, i1) : 4u;
        // four bf16 0/1 of a letter: 1.0 shifted to its place (past the 64 bits for none)
        const u64 w0 = c0 < 4u ? 0x3F80ull << (16u * c0) : 0ull, w1 = c1 < 4u ? 0x3F80ull << (16u * c1) : 0ull;
        const uint4 w = make_uint4((u32)w0, (u32)(w0 >> 32), (u32)w1, (u32)(w1 >> 32));
        *reinterpret_cast<uint4 *>(tile + canon_offset(R, r, 8 * q)) = w;
    }
}

// BF16 pair of the ReLUs: the maximum of the rounded pair, one instruction instead of two before the rounding.
__device__ __forceinline__ u32 relu_bf16x2(float lo, float hi) {
    const __nv_bfloat162 v = __hmax2(__floats2bfloat162_rn(lo, hi), __nv_bfloat162(0.0f, 0.0f));
    return *reinterpret_cast<const u32 *>(&v);
}

// One CTA per SM (226 KiB of shared memory, all 512 TMEM columns): 16 epilogue
// warps and one that issues the MMAs.  The biases and w3 come by value in the
// parameter space (InferBias, read as float4 through the constant cache).
// Epilogue warp w reaches TMEM lanes 32*(w%4)..+31 (rows of the 128-k-mer tile);
// the four warps of a row share its columns, and layer 2's 256 -> 1 dot is summed
// over them in shared memory.
//
// Both layers go in halves of 128 hidden columns, and the TMEM columns in four
// regions of 128 that rotate by one per tile: layer 1 fills R0 and R1, its
// activations (layer 2's A operand, BF16 pairs) go to R2, layer 2 accumulates in
// R3 and, once the first half of layer 1 has been read, in R0; the next tile's
// layer 1 takes R1 and R2.  So while the epilogue works on one half of layer 1
// the tensor cores run the other half or the first half (along K) of layer 2, and
// the next tile's layer 1 runs under the layer-2 epilogue:
//   MMA:      L1a L1b | L2(k < 128)      L2(k >= 128) | L1a' L1b' | ...
//   epilogue:     | e1a     e1b   one-hot'       |  e2         | e1a' ...
// Each hand-over is an mbarrier (one phase a tile), no block-wide barrier.
//
// What bounds it are the epilogues: their ALU instructions and, before, their
// constant loads.  A prefiltered search of 10M k-mers (all but 0.13 ms of it this
// kernel) took 2.36 ms with whole layers in two halves of TMEM and block barriers;
// 2.29 as above; 2.26 with the warp's number as a uniform value, so that biases
// and w3 are loaded by the uniform path (indexed by a register, these loads kept
// the address unit and the constant cache half busy; as operands at fixed places,
// in four copies of the loop, they missed the 2 KB immediate-constant cache: 3.59);
// 2.03 with layer 2's activations rounded in pairs; 1.94 with the ReLU taken on
// the rounded pair; 1.87 with the one-hot rows made by shifts.
template <u32 COLS>
__device__ __forceinline__ void infer_epi1(u32 src, u32 dst, u32 c0, const InferBias &bias) {
    u32 v[COLS / 16][16];
#pragma unroll
    for (u32 j = 0; j < COLS / 16; j++) tmem_ld16(src + 16u * j, v[j]);
    tmem_wait_ld();
#pragma unroll
    for (u32 j = 0; j < COLS / 16; j++) {
        tmem_tie(v[j]);
        u32 packed[8];
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
            // the same 4 biases for every lane of the warp, from the parameter space
            const float4 bb = *reinterpret_cast<const float4 *>(bias.b1 + c0 + 16u * j + t);
            packed[t / 2] = relu_bf16x2(__uint_as_float(v[j][t]) + bb.x, __uint_as_float(v[j][t + 1]) + bb.y);
            packed[t / 2 + 1] = relu_bf16x2(__uint_as_float(v[j][t + 2]) + bb.z, __uint_as_float(v[j][t + 3]) + bb.w);
        }
        tmem_st8(dst + 8u * j, packed);
    }
    tmem_wait_st();
}

// Partial dot of one row's 64 layer-2 activations (bias, ReLU, BF16) with w3.
__device__ __forceinline__ float infer_epi2(u32 src, u32 c0, const InferBias &bias) {
    u32 v[4][16];
#pragma unroll
    for (u32 j = 0; j < 4; j++) tmem_ld16(src + 16u * j, v[j]);
    tmem_wait_ld();
    float acc = 0.0f;
#pragma unroll
    for (u32 j = 0; j < 4; j++) {
        tmem_tie(v[j]);
#pragma unroll
        for (int t = 0; t < 16; t += 4) {
            const u32 c = c0 + 16u * j + t;
            const float4 bb = *reinterpret_cast<const float4 *>(bias.b2 + c);
            const float4 ww = *reinterpret_cast<const float4 *>(bias.w3 + c);
            const u32 h0 = relu_bf16x2(__uint_as_float(v[j][t]) + bb.x, __uint_as_float(v[j][t + 1]) + bb.y);
            const u32 h1 = relu_bf16x2(__uint_as_float(v[j][t + 2]) + bb.z, __uint_as_float(v[j][t + 3]) + bb.w);
            acc = fmaf(__uint_as_float(h0 << 16), ww.x, acc);
            acc = fmaf(__uint_as_float(h0 & 0xffff0000u), ww.y, acc);
            acc = fmaf(__uint_as_float(h1 << 16), ww.z, acc);
            acc = fmaf(__uint_as_float(h1 & 0xffff0000u), ww.w, acc);
        }
    }
    return acc;
}

// The mbarriers of mlp_infer_kernel: layer-1 halves and layer 2 done (committed by the MMAs), activation halves,
// one-hot tile and layer-2 accumulators handed over (one arrival per epilogue warp), and the final one.
enum { kBarL1a, kBarL1b, kBarL2, kBarE1a, kBarE1b, kBarX, kBarE2, kBarEnd, kBarCount };

__global__ void __launch_bounds__(kInferBlock, 1)
    mlp_infer_kernel(const u64 *__restrict__ kmers, u64 n, u32 k, const bf16 *__restrict__ W1b,
                     const bf16 *__restrict__ W2b, const InferBias bias, const InferOut out, int *err) {
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t bar[kBarCount];
    __shared__ u32 tmem_s;
    uint8_t *sW1 = smem;
    uint8_t *sW2 = smem + kHid * kIn * 2;
    uint8_t *sX = sW2 + kHid * kHid * 2;
    float *sRed = reinterpret_cast<float *>(sX + kTileM * kIn * 2);  // [kColGroups - 1][kTileM] partial dots
    const u32 tid = threadIdx.x, warp = tid >> 5, lane = tid & 31u;
    // weights into the canonical K-major layouts (once per launch)
    for (u32 i = tid; i < kHid * (kIn / 8); i += kInferBlock) {
        const u32 r = i / (kIn / 8), kc = i % (kIn / 8);
        *reinterpret_cast<uint4 *>(sW1 + canon_offset(kHid, r, kc * 8)) =
            *reinterpret_cast<const uint4 *>(W1b + (size_t)r * kIn + kc * 8);
    }
    for (u32 i = tid; i < kHid * (kHid / 8); i += kInferBlock) {
        const u32 r = i / (kHid / 8), kc = i % (kHid / 8);
        *reinterpret_cast<uint4 *>(sW2 + canon_offset(kHid, r, kc * 8)) =
            *reinterpret_cast<const uint4 *>(W2b + (size_t)r * kHid + kc * 8);
    }
    if (warp == 0) tmem_alloc(&tmem_s, 512);
    if (tid == 0) {
        for (u32 i = 0; i < kBarCount; i++)
            mbar_init(&bar[i], i >= kBarE1a && i <= kBarE2 ? kInferThreads / 32u : 1u);
    }
    fence_smem_to_async();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const u32 T0 = tmem_s;
    // a warp's wait: all lanes see the phase, or the warp leaves its loop
    auto wait = [&](u32 b, u32 parity, int code) {
        return __all_sync(0xffffffffu, mbar_wait(&bar[b], parity, err, code));
    };
    auto region = [&](u32 i) { return T0 + (i & 3u) * 128u; };
    if (warp < kInferThreads / 32u) {
        // ---- epilogue warps
        const u32 wu = __shfl_sync(0xffffffffu, warp, 0);  // the warp's number as a uniform value
        const u32 quarter = wu & 3u, cg = wu >> 2, trow = quarter * 32u + lane;
        const u32 lane_base = (quarter * 32u) << 16;
        const u32 xr = tid & (kTileM - 1u), xg = tid / kTileM;     // one-hot: row, chunk group
        constexpr u32 kChunks = kIn / 8 / kColGroups;                // 4 of the 16 chunks of a row
        auto arrive = [&](u32 b) {
            __syncwarp();
            if (lane == 0) mbar_arrive(&bar[b]);
        };
        auto one_hot = [&](u64 kmer) {
            onehot_chunks(sX, kTileM, xr, kmer, k, xg * kChunks, (xg + 1) * kChunks);
            fence_smem_to_async();
            arrive(kBarX);
        };
        u64 tile = blockIdx.x;
        one_hot(tile * kTileM + xr < n ? kmers[tile * kTileM + xr] : 0ull);
        for (u32 it = 0;; it++) {
            const u32 ph = it & 1u;
            const u64 next = tile + gridDim.x;
            const bool has_next = next * kTileM < n;
            const u64 kmer = has_next && next * kTileM + xr < n ? __ldg(kmers + next * kTileM + xr) : 0ull;
            const u32 a2 = region(it + 2u) + lane_base + cg * 16u;
            // layer 1, bias, ReLU, BF16: this warp's 32 columns of each half
            if (!wait(kBarL1a, ph, kErrInferWait1)) break;
            fence_after_sync();
            infer_epi1<32>(region(it) + lane_base + cg * 32u, a2, cg * 32u, bias);
            fence_before_sync();
            arrive(kBarE1a);
            if (!wait(kBarL1b, ph, kErrInferWait1)) break;
            fence_after_sync();
            infer_epi1<32>(region(it + 1u) + lane_base + cg * 32u, a2 + 64u, 128u + cg * 32u, bias);
            fence_before_sync();
            arrive(kBarE1b);
            if (has_next) one_hot(kmer);  // layer 1 has read this tile's
            // layer 2: this warp's 64 columns
            if (!wait(kBarL2, ph, kErrInferWait2)) break;
            fence_after_sync();
            const float dot = infer_epi2(region(cg < 2u ? it + 3u : it) + lane_base + (cg & 1u) * 64u, cg * kGroupCols, bias);
            if (cg) sRed[(cg - 1u) * kTileM + trow] = dot;
            fence_before_sync();
            arrive(kBarE2);
            // all accumulators are read (the next activations go over them) and all partial dots written; they are
            // written again only after the next layer 2, which waits for every warp's next activations
            if (!wait(kBarE2, ph, kErrInferWait2)) break;
            fence_after_sync();
            if (cg == 0) {
                const u64 row = tile * kTileM + trow;
                float sum = dot;
#pragma unroll
                for (u32 g = 0; g + 1u < kColGroups; g++) sum += sRed[g * kTileM + trow];
                const float lg = sum + bias.b3;
                if (out.logits && row < n) out.logits[row] = lg;
                if (out.reject) {
                    // the sandwich's decision: rejected by the model at tau and by the backup Bloom filter
                    const Bloom bloom{out.bloom_bits, out.bloom_mask, out.bloom_hashes};
                    const bool rej = row < n && lg < out.tau && !bloom.probe(kmer_key(kmers[row], k));
                    const u32 bits = __ballot_sync(0xffffffffu, rej);
                    const u64 first = tile * kTileM + quarter * 32u;  // this warp's 32 rows
                    if (lane == 0 && first < n) out.reject[first >> 5] = bits;
                }
            }
            if (!has_next) break;
            tile = next;
        }
    } else {
        // ---- MMA warp: one lane issues
        constexpr u32 idesc = idesc_bf16(kTileM, 128);
        constexpr u32 half_rows = 128u / 8u * 128u;  // byte offset of rows 128.. of a weight tile
        auto layer1 = [&](u32 half, u32 dst) {
#pragma unroll
            for (u32 s = 0; s < kIn / 16; s++) {
                const u64 da = smem_desc(smem_addr(sX) + s * 2u * kTileM * 16u, kTileM * 16u, 128u);
                const u64 db = smem_desc(smem_addr(sW1) + s * 2u * kHid * 16u + half * half_rows, kHid * 16u, 128u);
                mma_ss(dst, da, db, idesc, s > 0);
            }
            mma_commit(&bar[half ? kBarL1b : kBarL1a]);
        };
        // layer 2 over the activations 128 kh .. +127, both halves of its columns
        auto layer2 = [&](u32 kh, u32 a2, u32 lo, u32 hi) {
#pragma unroll
            for (u32 s = 8u * kh; s < 8u * kh + 8u; s++) {
                const u32 b = smem_addr(sW2) + s * 2u * kHid * 16u;
                mma_ts(lo, a2 + s * 8u, smem_desc(b, kHid * 16u, 128u), idesc, s > 0);
                mma_ts(hi, a2 + s * 8u, smem_desc(b + half_rows, kHid * 16u, 128u), idesc, s > 0);
            }
        };
        bool ok = wait(kBarX, 0, kErrInferWait1);
        fence_after_sync();
        if (ok && lane == 0) {
            layer1(0, region(0));
            layer1(1, region(1));
        }
        u64 tile = blockIdx.x;
        for (u32 it = 0; ok; it++) {
            const u32 ph = it & 1u, a2 = region(it + 2u), lo = region(it + 3u), hi = region(it);
            if (!(ok = wait(kBarE1a, ph, kErrInferWait1))) break;
            fence_after_sync();
            if (lane == 0) layer2(0, a2, lo, hi);
            if (!(ok = wait(kBarE1b, ph, kErrInferWait1))) break;
            fence_after_sync();
            if (lane == 0) {
                layer2(1, a2, lo, hi);
                mma_commit(&bar[kBarL2]);
            }
            tile += gridDim.x;
            if (tile * kTileM >= n) break;
            if (!(ok = wait(kBarX, ph ^ 1u, kErrInferWait1))) break;
            fence_after_sync();
            if (lane == 0) layer1(0, region(it + 1u));  // over the second half of layer 1, which E1b handed over
            if (!(ok = wait(kBarL2, ph, kErrInferWait2))) break;
            fence_after_sync();
            if (lane == 0) layer1(1, region(it + 2u));  // over the activations, which layer 2 has read
        }
        // every MMA has landed before the columns are freed
        if (lane == 0) {
            mma_commit(&bar[kBarEnd]);
            mbar_wait(&bar[kBarEnd], 0, err, kErrInferWait2);
        }
        __syncwarp();
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(T0, 512);
}

// ------------------------------------------------------- training helpers

// Rows of 8 inputs of X[b] = one-hot of k-mer (batch_start + b) (16 a row), rows
// of 8 k-mers of its transpose XT, and Y[b] = the label; batch a multiple of 8.
__global__ void onehot_batch_kernel(const u64 *__restrict__ kmers, const uint8_t *__restrict__ labels, u64 n_train,
                                    const unsigned long long *step, u32 batch, u32 k, bf16 *__restrict__ X,
                                    bf16 *__restrict__ XT, float *__restrict__ Y) {
    const u32 t = blockIdx.x * blockDim.x + threadIdx.x, half = batch * (kIn / 8);
    const u64 start = ((u64)*step * batch) % (n_train - batch + 1);
    constexpr u32 one = 0x3F80u;  // bf16 1.0
    u32 w[4];
    if (t < half) {
        const u32 b = t / (kIn / 8), q = t % (kIn / 8);
        const u64 kmer = kmers[start + b];
        if (q == 0) Y[b] = (float)labels[start + b];
#pragma unroll
        for (u32 i = 0; i < 4u; i++) {
            const u32 l = 2u * q + i / 2u, c = l < k ? letter(kmer, l) : 4u, j = 2u * (i & 1u);
            w[i] = (c == j ? one : 0u) | (c == j + 1u ? one << 16 : 0u);
        }
        *reinterpret_cast<uint4 *>(X + (size_t)b * kIn + 8u * q) = make_uint4(w[0], w[1], w[2], w[3]);
    } else if (t < 2u * half) {
        const u32 u = t - half, i = u / (batch / 8u), b = u % (batch / 8u) * 8u, l = i / 4u, j = i & 3u;
#pragma unroll
        for (u32 x = 0; x < 4u; x++) {
            w[x] = 0;
            if (l < k)
                w[x] = (letter(kmers[start + b + 2u * x], l) == j ? one : 0u) |
                       (letter(kmers[start + b + 2u * x + 1u], l) == j ? one << 16 : 0u);
        }
        *reinterpret_cast<uint4 *>(XT + (size_t)i * batch + b) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Adam (Kingma & Ba 2015) over the whole parameter vector, then the BF16
// operand copies of W1, W2 and W2's transpose; inputs past 4k of W1 stay zero.
__global__ void adam_kernel(float *__restrict__ theta, const float *__restrict__ grad, float *__restrict__ m,
                            float *__restrict__ v, const unsigned long long *step, u32 count, float lr, u32 k,
                            bf16 *__restrict__ W1b, bf16 *__restrict__ W2b, bf16 *__restrict__ W2bT,
                            const MlpOffsets off) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float t = (float)(*step + 1);
    float g = grad[i];
    if (i < off.b1 && (i % kIn) >= 4 * k) g = 0.0f;  // padded inputs of W1
    const float mi = b1 * m[i] + (1.0f - b1) * g;
    const float vi = b2 * v[i] + (1.0f - b2) * g * g;
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.0f - powf(b1, t)), vh = vi / (1.0f - powf(b2, t));
    const float p = theta[i] - lr * mh / (sqrtf(vh) + eps);
    theta[i] = p;
    if (i < off.b1) W1b[i] = __float2bfloat16_rn(p);
    else if (i >= off.W2 && i < off.b2) {
        const u32 j = i - off.W2;
        W2b[j] = W2bT[j % kHid * kHid + j / kHid] = __float2bfloat16_rn(p);
    }
}

__global__ void step_kernel(unsigned long long *step, float *loss_hist, const float *loss_sum, u32 hist_every) {
    const unsigned long long s = *step;
    if (hist_every && s % hist_every == 0) loss_hist[s / hist_every] = *loss_sum;
    *step = s + 1;
}

// dst_t: NULL, or the transpose of src as rows of `cols`.
__global__ void to_bf16_kernel(const float *__restrict__ src, bf16 *__restrict__ dst, u32 count,
                               bf16 *__restrict__ dst_t, u32 cols) {
    const u32 i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const bf16 x = __float2bfloat16_rn(src[i]);
    dst[i] = x;
    if (dst_t) dst_t[i % cols * (count / cols) + i / cols] = x;
}

// ------------------------------------------------- k-mers from the index

// select_c(j): position of the j-th 1 (0-based) of vector c in the LINES
// layout: binary search over the line counts, then within the line.
__device__ u32 line_select(const ulonglong4 *lines_c, u32 lpc, u32 j) {
    u32 lo = 0, hi = lpc - 1;  // last line whose count <= j
    while (lo < hi) {
        const u32 mid = (lo + hi + 1) >> 1;
        const u32 cnt = (u32)(lines_c[mid].x >> 32);
        if (cnt <= j) lo = mid; else hi = mid - 1;
    }
    const ulonglong4 w = lines_c[lo];
    u32 rem = j - (u32)(w.x >> 32);
    const u64 words[4] = {w.x & 0xffffffffull, w.y, w.z, w.w};
    for (u32 wi = 0; wi < 4; wi++) {
        const u32 pc = __popcll(words[wi]);
        if (rem < pc) {
            u64 x = words[wi];
            for (int b = 63; b >= 0; b--) {
                if ((x >> b) & 1ull) {
                    if (rem == 0) return lo * dev::kLineBits + (wi * 64u + (63u - (u32)b)) - 32u;
                    rem--;
                }
            }
        }
        rem -= pc;
    }
    return 0xffffffffu;  // unreachable for j < ones(c)
}

// The k-mer of node v by k select steps back along its incoming edges;
// false for a dummy node (the walk reaches the root first).
__device__ bool node_kmer(const ulonglong4 *lines, u32 lpc, const u64 *C, u32 k, u32 v, u64 &kmer) {
    u64 x = 0;
    for (u32 t = 0; t < k; t++) {
        if (v == 0) return false;
        const u32 c = v < C[1] ? 0u : v < C[2] ? 1u : v < C[3] ? 2u : 3u;
        x |= (u64)c << (62u - 2u * (k - 1u - t));
        v = line_select(lines + (u64)c * lpc, lpc, v - (u32)C[c]);
    }
    kmer = x;
    return true;
}

// Training candidates: with probability n_pos/(n_pos+n_neg) an indexed
// k-mer (a random node, resampled if it is a dummy), else half uniform
// random k-mers and half indexed k-mers with 1-3 substitutions.
__global__ void sample_kernel(const ulonglong4 *lines, u32 lpc, C5 C5v, u32 n_nodes, u32 k, u64 n_pos, u64 n_neg,
                              u64 seed, u64 count, u64 *__restrict__ out) {
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    const u64 C[5] = {C5v.c[0], C5v.c[1], C5v.c[2], C5v.c[3], C5v.c[4]};
    u64 h = mix64(seed ^ (i * 0x9E3779B97F4A7C15ull));
    const u64 kmask = k == 32 ? ~0ull : ~((1ull << (64 - 2 * k)) - 1ull);
    const bool pos = (h % (n_pos + n_neg)) < n_pos;
    h = mix64(h);
    if (!pos && (h & 1ull)) {
        out[i] = mix64(h) & kmask;
        return;
    }
    u64 x = 0;
    for (int attempt = 0; attempt < 64; attempt++) {
        h = mix64(h);
        const u32 v = 1u + (u32)(h % (u64)(n_nodes - 1));
        if (node_kmer(lines, lpc, C, k, v, x)) break;
    }
    if (!pos) {
        h = mix64(h);
        const u32 subs = 1u + (u32)(h % 3u);
        for (u32 s = 0; s < subs; s++) {
            h = mix64(h);
            const u32 p = (u32)(h % k);
            const u32 old = letter(x, p);
            const u32 nw = (old + 1u + (u32)((h >> 32) % 3u)) & 3u;
            const u32 sh = 62u - 2u * p;
            x = (x & ~(3ull << sh)) | ((u64)nw << sh);
        }
    }
    out[i] = x;
}

// Every indexed k-mer: node v in [1, n) -> its k-mer, or ~0 for a dummy.
__global__ void enumerate_kernel(const ulonglong4 *lines, u32 lpc, C5 C5v, u32 n_nodes, u32 k, u64 *__restrict__ out) {
    const u32 v = blockIdx.x * blockDim.x + threadIdx.x + 1u;
    if (v >= n_nodes) return;
    const u64 C[5] = {C5v.c[0], C5v.c[1], C5v.c[2], C5v.c[3], C5v.c[4]};
    u64 x;
    out[v - 1] = node_kmer(lines, lpc, C, k, v, x) ? x : ~0ull;
}

// labels[i] = answers[i] found (labels == NULL: only count them, for lists
// longer than any label array).
__global__ void labels_kernel(const u64 *__restrict__ answers, u64 n, uint8_t *__restrict__ labels,
                              unsigned long long *positives) {
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const bool hit = i < n && answers[i] != ~0ull;
    if (labels && i < n) labels[i] = hit ? 1 : 0;
    const u32 m = __ballot_sync(0xffffffffu, hit);
    if ((threadIdx.x & 31u) == 0 && m) atomicAdd(positives, (unsigned long long)__popc(m));
}

// Indexed k-mers the model rejects (logit < tau) go into the Bloom filter;
// `rejected` counts them (pass 1 counts only, bits == nullptr).
__global__ void bloom_build_kernel(const u64 *__restrict__ kmers, const float *__restrict__ logits, u64 n, float tau,
                                   u32 k, u32 *bits, u64 mask, u32 hashes, unsigned long long *rejected) {
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const bool rej = i < n && kmers[i] != ~0ull && logits[i] < tau;
    if (rej && bits) bloom_insert(bits, mask, hashes, kmer_key(kmers[i], k));
    const u32 m = __ballot_sync(0xffffffffu, rej);
    if ((threadIdx.x & 31u) == 0 && m) atomicAdd(rejected, (unsigned long long)__popc(m));
}

// Accuracy of the trained model on a labelled set at threshold tau.
__global__ void accuracy_kernel(const float *__restrict__ logits, const uint8_t *__restrict__ labels, u64 n, float tau,
                                unsigned long long *correct) {
    const u64 i = (u64)blockIdx.x * blockDim.x + threadIdx.x;
    const bool ok = i < n && ((logits[i] >= tau) == (labels[i] != 0));
    const u32 m = __ballot_sync(0xffffffffu, ok);
    if ((threadIdx.x & 31u) == 0 && m) atomicAdd(correct, (unsigned long long)__popc(m));
}

// ------------------------------------------------------------ launchers

namespace {

template <u32 BN, int EPI>
int launch_gemm(const bf16 *A, const bf16 *B, u32 M, u32 N, u32 K, u32 splits, const TrainEpi &t, int *err,
                cudaStream_t s) {
    if (M % 128 || K % 64 || N % BN) return set_error("gemm: unsupported shape %ux%ux%u", M, N, K);
    const u32 ksteps = K / 64;
    splits = std::max(1u, std::min(splits, ksteps));
    const u32 kps = ((ksteps + splits - 1) / splits) * 64;
    splits = (K + kps - 1) / kps;
    constexpr u32 smem = (128 + BN) * 64 * 2;
    if (smem > 32768)  // with the static part beyond 48 KiB: the opt-in, a per-device attribute
        SBWT_CHECK_CUDA(cudaFuncSetAttribute(gemm_tn_kernel<BN, EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    gemm_tn_kernel<BN, EPI><<<dim3(M / 128, N / BN, splits), 128, smem, s>>>(A, B, M, N, K, kps, t, err);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace

// The products of a training step (prefilter.cu enqueue_step).  Tiles of 128
// columns where the rows of a result need not be whole: twice the blocks of 256.
int gemm_relu(const bf16 *A, const bf16 *B, u32 M, u32 K, const TrainEpi &t, int *err, cudaStream_t s) {
    return launch_gemm<128, kEpiRelu>(A, B, M, kHid, K, 1, t, err, s);
}
int gemm_head(const bf16 *A, const bf16 *B, u32 M, const TrainEpi &t, int *err, cudaStream_t s) {
    return launch_gemm<256, kEpiHead>(A, B, M, kHid, kHid, 1, t, err, s);
}
int gemm_relu_grad(const bf16 *A, const bf16 *B, u32 M, const TrainEpi &t, int *err, cudaStream_t s) {
    return launch_gemm<128, kEpiReluGrad>(A, B, M, kHid, kHid, 1, t, err, s);
}
int gemm_add(const bf16 *A, const bf16 *B, u32 N, u32 K, u32 splits, float *D, int *err, cudaStream_t s) {
    TrainEpi t{};
    t.add = D;
    return launch_gemm<128, kEpiAdd>(A, B, kHid, N, K, splits, t, err, s);
}

int infer(const u64 *kmers, u64 n, u32 k, const bf16 *W1b, const bf16 *W2b, const InferBias &bias,
          const InferOut &out, int *err, int num_sms, cudaStream_t s) {
    if (n == 0) return 0;
    // the shared-memory opt-in is a per-device function attribute
    int dev = 0;
    SBWT_CHECK_CUDA(cudaGetDevice(&dev));
    static bool attr_set[kMaxDevicesAttr] = {};
    if (dev < 0 || dev >= kMaxDevicesAttr) return set_error("device %d out of range", dev);
    if (!attr_set[dev]) {
        SBWT_CHECK_CUDA(cudaFuncSetAttribute(mlp_infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kInferSmem));
        attr_set[dev] = true;
    }
    const u64 tiles = (n + kTileM - 1) / kTileM;
    const u32 grid = (u32)std::min<u64>(tiles, (u64)num_sms);
    mlp_infer_kernel<<<grid, kInferBlock, kInferSmem, s>>>(kmers, n, k, W1b, W2b, bias, out, err);
    SBWT_CHECK_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace mlp
}  // namespace sbwt
