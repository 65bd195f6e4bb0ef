// The learned limiter's network: a 3-layer MLP of width 64 over 32 per-cell features, 16 outputs (5 used: one slope
// fraction per primitive variable). Weights and activations in BF16 on the tensor cores, FP32 accumulation, FP32 master
// weights. It has no counterpart in the reference.
//
// Layout of the FP32 parameter vector (kParams floats): W1 [64][32], b1 [64], W2 [64][64], b2 [64], W3 [16][64], b3 [16];
// W[n][k] maps input k to output n. Activation: ReLU after layers 1 and 2; the output o is a logit.
//
// Kernels (one warp = 16 rows, m16n8k16 BF16 MMA with FP32 accumulation; the activations of a warp stay in registers
// from layer to layer: the accumulator fragment of one layer is the A fragment of the next):
//   k_mlp_train     forward + backward of the loss sum_r sum_c w_rc (sigmoid(o_rc) - t_rc)^2 over 64 rows a block and
//                   turn, the block's gradient kept in its warps' accumulators and written to its own slot at the end
//                   (deterministic: no atomics)
//   k_mlp_reduce    the slots summed in a fixed order, scaled by the caller's factor or by 1 / sum(w)
// Inference runs forward_tc (tcgen05).
//   k_mlp_adam      Adam on the FP32 master weights
#pragma once

#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

#include "luna_b200.h"

namespace luna {
namespace mlp {

// The forward pass on the 5th-generation tensor cores (mlp_tc.cuh; defined in learned.cu): logits [n][16] of feature
// rows [n][32] on `stream`; rows (device, may be null): only the first min(n, *rows) rows, a count written earlier on the
// stream; a wait that gives up sets bit 16 of *error.
luna_status forward_tc(const float* params, const __nv_bfloat16* x, int n, const unsigned int* rows, float* logits, unsigned long long* error,
                       cudaStream_t stream);

constexpr int kIn = 32, kHidden = 64, kOut = 16, kUsed = 5;
constexpr int kW1 = 0, kB1 = kW1 + kHidden * kIn, kW2 = kB1 + kHidden, kB2 = kW2 + kHidden * kHidden, kW3 = kB2 + kHidden,
              kB3 = kW3 + kOut * kHidden, kParams = kB3 + kOut;
constexpr int kRowsPerWarp = 16, kWarps = 4, kRowsPerBlock = kRowsPerWarp * kWarps;
constexpr int kTrainBlocksPerSm = 2;  // by registers (210 a thread; 60 KB of shared memory a block)

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<const uint32_t*>(&v);
}

// D = A B + D, A 16x16 (row), B 16x8 (col), BF16 in, FP32 accumulate.
__device__ __forceinline__ void mma_bf16(float* d, const uint32_t* a, const uint32_t* b) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// Row lengths in shared memory: eight past the columns, so that the rows an 8 x 8 fragment load names start 16 B apart
// in the banks.
constexpr int kLdIn = kIn + 8, kLdHidden = kHidden + 8, kLdOut = kOut + 8;

// The block's weights in shared memory as BF16, W[n][k]: the B fragments of the forward as they lie, of the backward by
// transposing loads.
struct SmemWeights {
    __align__(16) __nv_bfloat16 w1[kHidden * kLdIn];
    __align__(16) __nv_bfloat16 w2[kHidden * kLdHidden];
    __align__(16) __nv_bfloat16 w3[kOut * kLdHidden];
    float b1[kHidden], b2[kHidden], b3[kOut];
};

__device__ __forceinline__ void load_weights(const float* __restrict__ p, SmemWeights& s) {
    for (int x = threadIdx.x; x < kHidden * kIn; x += blockDim.x) s.w1[x / kIn * kLdIn + x % kIn] = __float2bfloat16_rn(p[kW1 + x]);
    for (int x = threadIdx.x; x < kHidden * kHidden; x += blockDim.x)
        s.w2[x / kHidden * kLdHidden + x % kHidden] = __float2bfloat16_rn(p[kW2 + x]);
    for (int x = threadIdx.x; x < kOut * kHidden; x += blockDim.x)
        s.w3[x / kHidden * kLdHidden + x % kHidden] = __float2bfloat16_rn(p[kW3 + x]);
    for (int x = threadIdx.x; x < kHidden; x += blockDim.x) {
        s.b1[x] = p[kB1 + x];
        s.b2[x] = p[kB2 + x];
    }
    for (int x = threadIdx.x; x < kOut; x += blockDim.x) s.b3[x] = p[kB3 + x];
}

// Four 8 x 8 BF16 matrices, each transposed on its way: lane l names row l % 8 of matrix l / 8 (16-B aligned).
__device__ __forceinline__ void ldmatrix4_trans(const __nv_bfloat16* row, uint32_t* r) {
    const uint32_t a = static_cast<uint32_t>(__cvta_generic_to_shared(row));
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(a));
}
// The A fragment (m0..m0+15, k0..k0+15) of a matrix that lies as [k][m].
__device__ __forceinline__ void a_frag_trans(const __nv_bfloat16* m, int ld, int m0, int k0, uint32_t* a) {
    const int lane = threadIdx.x & 31;
    ldmatrix4_trans(m + (k0 + (lane >> 4) * 8 + (lane & 7)) * ld + m0 + ((lane >> 3) & 1) * 8, a);
}
// The B fragments (k0..k0+15) of columns n0..n0+7 (b[0], b[1]) and n0+8..n0+15 (b[2], b[3]) of a matrix that lies as
// [k][n].
__device__ __forceinline__ void b_frag2_trans(const __nv_bfloat16* m, int ld, int n0, int k0, uint32_t* b) {
    const int lane = threadIdx.x & 31;
    ldmatrix4_trans(m + (k0 + ((lane >> 3) & 1) * 8 + (lane & 7)) * ld + n0 + (lane >> 4) * 8, b);
}

// B fragment (k0..k0+15, n0..n0+7) of a K-contiguous matrix M[n][k] with row length ld.
__device__ __forceinline__ void b_frag(const __nv_bfloat16* m, int ld, int n0, int k0, uint32_t* b) {
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    b[0] = *reinterpret_cast<const uint32_t*>(m + (n0 + gid) * ld + k0 + 2 * tig);
    b[1] = *reinterpret_cast<const uint32_t*>(m + (n0 + gid) * ld + k0 + 8 + 2 * tig);
}

// A fragments of the next layer from the accumulators of this one (16 rows x 8 columns per tile): k-step s takes tiles
// 2s and 2s+1.
template <int Tiles>
__device__ __forceinline__ void acc_to_a(const float (&acc)[Tiles][4], uint32_t (&a)[Tiles / 2][4]) {
#pragma unroll
    for (int s = 0; s < Tiles / 2; ++s) {
        a[s][0] = pack_bf16(acc[2 * s][0], acc[2 * s][1]);
        a[s][1] = pack_bf16(acc[2 * s][2], acc[2 * s][3]);
        a[s][2] = pack_bf16(acc[2 * s + 1][0], acc[2 * s + 1][1]);
        a[s][3] = pack_bf16(acc[2 * s + 1][2], acc[2 * s + 1][3]);
    }
}

// The forward pass of one warp's 16 rows [row0, row0 + 16) from BF16 feature rows. h1, h2: the post-ReLU activations
// (FP32 accumulators), kept for the backward; out: the logits; a: the features' fragments.
__device__ __forceinline__ void forward_warp(const SmemWeights& s, const __nv_bfloat16* __restrict__ x, int n, int row0,
                                             uint32_t (&a)[kIn / 16][4], float (&h1)[kHidden / 8][4], float (&h2)[kHidden / 8][4], float (&out)[kOut / 8][4]) {
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int r0 = row0 + gid, r1 = row0 + gid + 8;
#pragma unroll
    for (int st = 0; st < kIn / 16; ++st) {
        const int k = 16 * st + 2 * tig;
        a[st][0] = r0 < n ? *reinterpret_cast<const uint32_t*>(x + static_cast<int64_t>(r0) * kIn + k) : 0u;
        a[st][1] = r1 < n ? *reinterpret_cast<const uint32_t*>(x + static_cast<int64_t>(r1) * kIn + k) : 0u;
        a[st][2] = r0 < n ? *reinterpret_cast<const uint32_t*>(x + static_cast<int64_t>(r0) * kIn + k + 8) : 0u;
        a[st][3] = r1 < n ? *reinterpret_cast<const uint32_t*>(x + static_cast<int64_t>(r1) * kIn + k + 8) : 0u;
    }
#pragma unroll
    for (int t = 0; t < kHidden / 8; ++t) {
        const float bl = s.b1[8 * t + 2 * tig], bh = s.b1[8 * t + 2 * tig + 1];
        h1[t][0] = bl;
        h1[t][1] = bh;
        h1[t][2] = bl;
        h1[t][3] = bh;
#pragma unroll
        for (int st = 0; st < kIn / 16; ++st) {
            uint32_t b[2];
            b_frag(s.w1, kLdIn, 8 * t, 16 * st, b);
            mma_bf16(h1[t], a[st], b);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) h1[t][c] = fmaxf(h1[t][c], 0.0f);
    }
    uint32_t a2[kHidden / 16][4];
    acc_to_a<kHidden / 8>(h1, a2);
#pragma unroll
    for (int t = 0; t < kHidden / 8; ++t) {
        const float bl = s.b2[8 * t + 2 * tig], bh = s.b2[8 * t + 2 * tig + 1];
        h2[t][0] = bl;
        h2[t][1] = bh;
        h2[t][2] = bl;
        h2[t][3] = bh;
#pragma unroll
        for (int st = 0; st < kHidden / 16; ++st) {
            uint32_t b[2];
            b_frag(s.w2, kLdHidden, 8 * t, 16 * st, b);
            mma_bf16(h2[t], a2[st], b);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) h2[t][c] = fmaxf(h2[t][c], 0.0f);
    }
    uint32_t a3[kHidden / 16][4];
    acc_to_a<kHidden / 8>(h2, a3);
#pragma unroll
    for (int t = 0; t < kOut / 8; ++t) {
        const float bl = s.b3[8 * t + 2 * tig], bh = s.b3[8 * t + 2 * tig + 1];
        out[t][0] = bl;
        out[t][1] = bh;
        out[t][2] = bl;
        out[t][3] = bh;
#pragma unroll
        for (int st = 0; st < kHidden / 16; ++st) {
            uint32_t b[2];
            b_frag(s.w3, kLdHidden, 8 * t, 16 * st, b);
            mma_bf16(out[t], a3[st], b);
        }
    }
}

// Stores a warp's accumulator tiles (16 rows x 8 Tiles columns) into rows of ld BF16 values.
template <int Tiles>
__device__ __forceinline__ void stage_acc(const float (&acc)[Tiles][4], __nv_bfloat16* tile, int ld) {
    const int lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int t = 0; t < Tiles; ++t) {
        const int c = 8 * t + 2 * tig;
        *reinterpret_cast<uint32_t*>(tile + gid * ld + c) = pack_bf16(acc[t][0], acc[t][1]);
        *reinterpret_cast<uint32_t*>(tile + (gid + 8) * ld + c) = pack_bf16(acc[t][2], acc[t][3]);
    }
}

// A block's 64 rows of activations and bars, one row a batch row.
struct SmemTrain {
    SmemWeights w;
    __align__(16) __nv_bfloat16 x[kRowsPerBlock * kLdIn];
    __align__(16) __nv_bfloat16 h1[kRowsPerBlock * kLdHidden];
    __align__(16) __nv_bfloat16 h2[kRowsPerBlock * kLdHidden];
    __align__(16) __nv_bfloat16 dz1[kRowsPerBlock * kLdHidden];
    __align__(16) __nv_bfloat16 dz2[kRowsPerBlock * kLdHidden];
    __align__(16) __nv_bfloat16 dout[kRowsPerBlock * kLdOut];
    float sums[2][kWarps];
};

// Forward and backward of the rows, 64 a block and turn (16 a warp); then the four warps share the block's weight
// gradients, sums over its 64 rows: warp w has the 16 rows 16 w.. of dW1 and dW2 and the 16 columns 16 w.. of dW3 in
// its accumulators from turn to turn (and the biases, as the products with a column of ones), so no partial gradient
// passes through memory. Block b's gradient goes to slot b, its loss and its sum of weights beside it. Rows beyond n or
// with zero weight add nothing.
// The batch of 16,384 rows is 256 blocks of one turn, one wave at 2 blocks an SM: what bounds it is the chain of a turn.
// Before, the four warps added their own gradients to one shared copy one after another, from fragments gathered value by
// value: 48 us for the batch, now 11. The sums over rows are the tensor core's, in FP32 from turn to turn: against 64 bits the
// gradient of 1 to 1,000,000 rows is off by what it was off before (9.2e-4, the operands' BF16; the biases' 2.1e-5).
static __global__ void __launch_bounds__(128) k_mlp_train(const float* __restrict__ params, const __nv_bfloat16* __restrict__ x,
                                                   const float* __restrict__ target, const float* __restrict__ weight, int n,
                                                   float* __restrict__ slots, float* __restrict__ loss_slots, float* __restrict__ weight_slots) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmemTrain& sm = *reinterpret_cast<SmemTrain*>(smem_raw);
    const SmemWeights& s = sm.w;
    load_weights(params, sm.w);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, gid = lane >> 2, tig = lane & 3;
    const int mine = warp * kRowsPerWarp;  // the warp's rows of the block's tiles
    float loss = 0.0f, weights = 0.0f;
    float gw1[kIn / 8][4] = {}, gw2[kHidden / 8][4] = {}, gw3[2][4] = {}, gb1[4] = {}, gb2[4] = {}, gb3[4] = {};
    const uint32_t ones = pack_bf16(1.0f, 1.0f), one_column[2] = {gid == 0 ? ones : 0u, gid == 0 ? ones : 0u};
    const int turns = (n + kRowsPerBlock - 1) / kRowsPerBlock;
    for (int turn = blockIdx.x; turn < turns; turn += gridDim.x) {
        const int row0 = turn * kRowsPerBlock + mine;
        float h1[kHidden / 8][4], h2[kHidden / 8][4], out[kOut / 8][4];
        uint32_t ax[kIn / 16][4];
        forward_warp(s, x, n, row0, ax, h1, h2, out);
        // The loss and dL/do = 2 w (sigma - t) sigma (1 - sigma); unused outputs and padded rows have w = 0.
        float dout[kOut / 8][4];
#pragma unroll
        for (int t = 0; t < kOut / 8; ++t)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int col = 8 * t + 2 * tig + (c & 1), row = row0 + gid + (c >> 1) * 8;
                float g = 0.0f;
                if (row < n && col < kUsed) {
                    const float w = weight[static_cast<int64_t>(row) * kUsed + col];
                    const float sg = 1.0f / (1.0f + __expf(-out[t][c]));
                    const float e = sg - target[static_cast<int64_t>(row) * kUsed + col];
                    loss += w * e * e;
                    weights += w;
                    g = 2.0f * w * e * sg * (1.0f - sg);
                }
                dout[t][c] = g;
            }
        if (turn != static_cast<int>(blockIdx.x)) __syncthreads();  // the last turn's tiles are read
#pragma unroll
        for (int st = 0; st < kIn / 16; ++st) {
            __nv_bfloat16* at = sm.x + (mine + gid) * kLdIn + 16 * st + 2 * tig;
            *reinterpret_cast<uint32_t*>(at) = ax[st][0];
            *reinterpret_cast<uint32_t*>(at + 8 * kLdIn) = ax[st][1];
            *reinterpret_cast<uint32_t*>(at + 8) = ax[st][2];
            *reinterpret_cast<uint32_t*>(at + 8 * kLdIn + 8) = ax[st][3];
        }
        stage_acc<kHidden / 8>(h1, sm.h1 + mine * kLdHidden, kLdHidden);
        stage_acc<kHidden / 8>(h2, sm.h2 + mine * kLdHidden, kLdHidden);
        stage_acc<kOut / 8>(dout, sm.dout + mine * kLdOut, kLdOut);
        // dH2 = dO W3 (W3 as [K = out][N = hidden]), dZ2 = dH2 where h2 > 0.
        uint32_t ao[1][4];
        acc_to_a<kOut / 8>(dout, ao);
        float dz2[kHidden / 8][4];
#pragma unroll
        for (int t = 0; t < kHidden / 8; t += 2) {
            uint32_t b[4];
            b_frag2_trans(s.w3, kLdHidden, 8 * t, 0, b);
#pragma unroll
            for (int q = 0; q < 2; ++q) {
#pragma unroll
                for (int c = 0; c < 4; ++c) dz2[t + q][c] = 0.0f;
                mma_bf16(dz2[t + q], ao[0], b + 2 * q);
#pragma unroll
                for (int c = 0; c < 4; ++c) dz2[t + q][c] = h2[t + q][c] > 0.0f ? dz2[t + q][c] : 0.0f;
            }
        }
        stage_acc<kHidden / 8>(dz2, sm.dz2 + mine * kLdHidden, kLdHidden);
        // dH1 = dZ2 W2, dZ1 = dH1 where h1 > 0.
        uint32_t az2[kHidden / 16][4];
        acc_to_a<kHidden / 8>(dz2, az2);
        float dz1[kHidden / 8][4];
#pragma unroll
        for (int t = 0; t < kHidden / 8; t += 2) {
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) dz1[t + q][c] = 0.0f;
#pragma unroll
            for (int sk = 0; sk < kHidden / 16; ++sk) {
                uint32_t b[4];
                b_frag2_trans(s.w2, kLdHidden, 8 * t, 16 * sk, b);
                mma_bf16(dz1[t], az2[sk], b);
                mma_bf16(dz1[t + 1], az2[sk], b + 2);
            }
#pragma unroll
            for (int q = 0; q < 2; ++q)
#pragma unroll
                for (int c = 0; c < 4; ++c) dz1[t + q][c] = h1[t + q][c] > 0.0f ? dz1[t + q][c] : 0.0f;
        }
        stage_acc<kHidden / 8>(dz1, sm.dz1 + mine * kLdHidden, kLdHidden);
        __syncthreads();
        // dW3[o][h] = sum_r dO[r][o] H2[r][h]; dW2[h2][h1] = sum_r dZ2[r][h2] H1[r][h1]; dW1[h1][x] = sum_r dZ1[r][h1] X[r][x].
#pragma unroll
        for (int k = 0; k < kRowsPerBlock; k += 16) {
            uint32_t a[4], b[4];
            a_frag_trans(sm.dz2, kLdHidden, 16 * warp, k, a);
            mma_bf16(gb2, a, one_column);
#pragma unroll
            for (int t = 0; t < kHidden / 8; t += 2) {
                b_frag2_trans(sm.h1, kLdHidden, 8 * t, k, b);
                mma_bf16(gw2[t], a, b);
                mma_bf16(gw2[t + 1], a, b + 2);
            }
            a_frag_trans(sm.dz1, kLdHidden, 16 * warp, k, a);
            mma_bf16(gb1, a, one_column);
#pragma unroll
            for (int t = 0; t < kIn / 8; t += 2) {
                b_frag2_trans(sm.x, kLdIn, 8 * t, k, b);
                mma_bf16(gw1[t], a, b);
                mma_bf16(gw1[t + 1], a, b + 2);
            }
            a_frag_trans(sm.dout, kLdOut, 0, k, a);
            mma_bf16(gb3, a, one_column);
            b_frag2_trans(sm.h2, kLdHidden, 16 * warp, k, b);
            mma_bf16(gw3[0], a, b);
            mma_bf16(gw3[1], a, b + 2);
        }
    }
    float* slot = slots + static_cast<int64_t>(blockIdx.x) * kParams;
    const int col = 2 * tig, row = 16 * warp + gid;
    const auto put = [&](float* at, int ld, int r, int c, const float* g) {  // a tile's accumulators at (r, c) and (r + 8, c)
        at[r * ld + c] = g[0];
        at[r * ld + c + 1] = g[1];
        at[(r + 8) * ld + c] = g[2];
        at[(r + 8) * ld + c + 1] = g[3];
    };
#pragma unroll
    for (int t = 0; t < kIn / 8; ++t) put(slot + kW1, kIn, row, 8 * t + col, gw1[t]);
#pragma unroll
    for (int t = 0; t < kHidden / 8; ++t) put(slot + kW2, kHidden, row, 8 * t + col, gw2[t]);
#pragma unroll
    for (int t = 0; t < 2; ++t) put(slot + kW3, kHidden, gid, 16 * warp + 8 * t + col, gw3[t]);
    if (tig == 0) {  // column 0 of the products with the ones
        slot[kB1 + row] = gb1[0];
        slot[kB1 + row + 8] = gb1[2];
        slot[kB2 + row] = gb2[0];
        slot[kB2 + row + 8] = gb2[2];
        if (warp == 0) {
            slot[kB3 + gid] = gb3[0];
            slot[kB3 + gid + 8] = gb3[2];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        loss += __shfl_xor_sync(0xffffffffu, loss, o);
        weights += __shfl_xor_sync(0xffffffffu, weights, o);
    }
    if (lane == 0) {
        sm.sums[0][warp] = loss;
        sm.sums[1][warp] = weights;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        loss_slots[blockIdx.x] = sm.sums[0][0] + sm.sums[0][1] + sm.sums[0][2] + sm.sums[0][3];
        if (weight_slots) weight_slots[blockIdx.x] = sm.sums[1][0] + sm.sums[1][1] + sm.sums[1][2] + sm.sums[1][3];
    }
}

// g[p] = scale * sum_b slots[b][p], loss = scale * sum_b loss_slots[b]; weight_slots given: scale is 1 / sum_b
// weight_slots[b]. Each sum in a fixed order: kReduceGroups threads a parameter take every kReduceGroups-th slot, then
// their sums in turn (5 us; one thread a parameter walked its 256 slots alone: 10 us).
constexpr int kReduceParams = 32, kReduceGroups = 8;
static __global__ void __launch_bounds__(kReduceParams * kReduceGroups) k_mlp_reduce(const float* __restrict__ slots, const float* __restrict__ loss_slots,
                                                                                     const float* __restrict__ weight_slots, int blocks, float scale,
                                                                                     float* __restrict__ g, float* __restrict__ loss) {
    __shared__ float part[kReduceGroups][kReduceParams], warp_sum[2][kReduceGroups];
    const int lane = threadIdx.x % kReduceParams, group = threadIdx.x / kReduceParams;
    const int p = blockIdx.x * kReduceParams + lane;
    float a = 0, l = 0, w = 0;
    if (p < kParams)
#pragma unroll 4
        for (int b = group; b < blocks; b += kReduceGroups) a += slots[static_cast<int64_t>(b) * kParams + p];
    for (int b = threadIdx.x; b < blocks; b += kReduceParams * kReduceGroups) {
        if (blockIdx.x == 0) l += loss_slots[b];
        if (weight_slots) w += weight_slots[b];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        l += __shfl_xor_sync(0xffffffffu, l, o);
        w += __shfl_xor_sync(0xffffffffu, w, o);
    }
    part[group][lane] = a;
    if (lane == 0) {
        warp_sum[0][group] = l;
        warp_sum[1][group] = w;
    }
    __syncthreads();
    if (group != 0) return;
    float sums[3] = {0, 0, 0};
#pragma unroll
    for (int k = 0; k < kReduceGroups; ++k) {
        sums[0] += part[k][lane];
        sums[1] += warp_sum[0][k];
        sums[2] += warp_sum[1][k];
    }
    if (weight_slots) scale = 1.0f / (sums[2] < 1e-30f ? 1e-30f : sums[2]);  // (a NaN weight stays NaN in all that it scales)
    if (p < kParams) g[p] = scale * sums[0];
    if (p == 0) *loss = scale * sums[1];
}

// Adam (Kingma and Ba) with bias correction; m, v: the moment estimates; step counts from 1.
static __global__ void k_mlp_adam(float* __restrict__ params, const float* __restrict__ g, float* __restrict__ m, float* __restrict__ v, float lr,
                           float beta1, float beta2, float eps, int step) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= kParams) return;
    const float gp = g[p];
    const float mp = beta1 * m[p] + (1.0f - beta1) * gp;
    const float vp = beta2 * v[p] + (1.0f - beta2) * gp * gp;
    m[p] = mp;
    v[p] = vp;
    const float mh = mp / (1.0f - powf(beta1, static_cast<float>(step)));
    const float vh = vp / (1.0f - powf(beta2, static_cast<float>(step)));
    params[p] -= lr * mh / (sqrtf(vh) + eps);
}

}  // namespace mlp
}  // namespace luna
