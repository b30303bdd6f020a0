// mlp.cu -- the learned refinement indicator: a 400-128-64-3 MLP with GELU
// that maps a patch's normalised conserved variables to coarsen / refine /
// keep, trained and evaluated on the GPU. Its weights are BF16, every GEMM
// accumulates in FP32 in tensor memory through tcgen05.mma (the only
// tensor-core use of the library), and the optimiser (AdamW) keeps FP32
// master weights. There is no counterpart in the reference: it stands in
// for the plain tagger (solver_tag_feature.F90:9-52 through
// hpc_amr_tag_feature, amr_external.h:92), which also labels its training
// data and judges it at run time.
//
// A training step (batch B, rows = patches) is three launches:
//   mlp_tile_kernel   per 128 rows, everything that needs only those rows:
//       Z1 = X W1^T + b1,  H1 = gelu(Z1);  Z2 = H1 W2^T + b2, H2 = gelu(Z2)
//       L  = H2 W3^T + b3 (3 logits, padded to 16), dL = softmax(L) - onehot
//       dZ2 = (dL W3) * gelu'(Z2),  dZ1 = (dZ2 W2) * gelu'(Z1)
//   mlp_wgrad_kernel  dW1 = dZ1^T X, dW2^T = H1^T dZ2, dW3^T = H2^T dL as
//       partial sums over 256 rows, db = column sums of dZ1, dZ2, dL
//   mlp_adamw_kernel  FP32 master update, BF16 copies W and W^T refreshed
// Inference is the first half of mlp_tile_kernel and an argmax.
//
// The sizes are small (2.1 GFLOP a batch of 8192), so a step is bound by
// launches, by latency and by passes over memory between them, not by the
// tensor cores. One kernel per GEMM, with operands staged chunk by chunk and
// transposed copies for the second operand's layout, took 19 launches, two
// copies and 283 us a batch; a tile that stays in shared and tensor memory,
// and operands read K-major or MN-major from the same core matrices, take
// three launches and 37 us. An epoch of 65,536 rows has 51 us beside its
// batches: the check and copy of the permutation and the read-back.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <vector>

#include "amrgpu_internal.h"
#include "device_common.cuh"
#include "mlp_internal.h"
#include "stage_kernel.cuh"
#include "umma.cuh"

namespace amrgpu {

using bf16 = __nv_bfloat16;

// gelu(x) = 0.5 x t and gelu'(x) = 0.5 t + x phi(x), with t = 1 + erf(x / sqrt 2)
__device__ __forceinline__ float gelu_t(float x) { return 1.0f + erff(x * 0.70710678118654752f); }
__device__ __forceinline__ float gelu_f(float x, float t) { return 0.5f * x * t; }
__device__ __forceinline__ float gelu_grad_f(float x, float t)
{
    return 0.5f * t + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// 16 floats -> 16 BF16 as two 16-byte pieces
__device__ __forceinline__ void pack_bf16(const float v[16], uint4 out[2])
{
    alignas(16) bf16 h[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) h[k] = __float2bfloat16_rn(v[k]);
    out[0] = reinterpret_cast<const uint4 *>(h)[0];
    out[1] = reinterpret_cast<const uint4 *>(h)[1];
}

// Arguments of mlp_tile_kernel. Row b of the batch is row perm[b] (perm null:
// b) of X and y. Training writes H1, H2, dZ1, dZ2, dL (B rows in the weight
// gradients' order, blocked_index) and per 32 rows the loss sum and the
// correct predictions; logits [B x 16] and classes [B] are written where
// given.
struct TileArgs {
    const bf16 *X;
    const int *perm;
    const int *y;
    int B;
    const bf16 *W1, *W2, *W3, *W2T, *W3T;
    const float *b1, *b2, *b3;
    float *logits;
    int *cls;
    int *counts;  // the judge's counts, set to zero (or null)
    bf16 *H1, *H2, *dZ1, *dZ2, *dL;
    double *loss;
    int *correct;
    int *err;  // error flags (a bounded wait gave up)
};

// The weights as the tile kernel reads them: K-major core matrices (umma.cuh),
// all rows of one 16-byte piece after another, so that a run of pieces is one
// bulk copy. Element (row, k) of an operand of `rows` rows:
__host__ __device__ constexpr int tiled_index(int rows, int row, int k)
{
    return (k / 8) * rows * 8 + row * 8 + k % 8;
}

// H1, H2, dZ1, dZ2 and dL as mlp_wgrad_kernel reads them: core matrices of 8
// rows, all 16-byte pieces of 8 rows after another (an MN-major operand's
// order), so that any run of rows is one bulk copy. Element (row, col), col a
// multiple of 8, of a matrix of `chunks` pieces a row:
__device__ __forceinline__ long long blocked_index(int chunks, int row, int col)
{
    return ((long long)(row >> 3) * chunks + (col >> 3)) * 64 + (row & 7) * 8;
}

// Shared memory of mlp_tile_kernel, in bytes. X and W1 fill it until the
// first GEMM is done; what comes after lives in their place. X's core
// matrices lie 144 bytes apart along a row, so that neighbouring pieces of a
// row, copied by neighbouring threads, go to different banks.
struct TileSmem {
    static constexpr int xpitch = 144, xrows = kFeatIn / 8 * xpitch;  // next piece, next 8 rows
    static constexpr int x = 0, w1 = x + 16 * xrows;
    static constexpr int bar = w1 + kH1 * kFeatIn * 2;  // MMA barrier, weight barriers, TMEM address
    static constexpr int rows = bar + 80;               // row index of each of the 128 rows
    static constexpr int total = rows + 128 * 4;
    // in X's place; t1: [column][row]
    static constexpr int h1 = x, t1 = h1 + 128 * kH1 * 2, dl = t1 + 128 * kH1 * 4;
    static constexpr int w3 = dl + 128 * kOutPad * 2, w3t = w3 + kOutPad * kH2 * 2;
    static_assert(w3t + kH2 * kOutPad * 2 <= w1, "what follows the first GEMM fits where X was");
    // in W1's place
    static constexpr int h2 = w1, t2 = h2 + 128 * kH2 * 2, dz2 = t2 + 128 * kH2 * 4;
    static constexpr int w2 = dz2 + 128 * kH2 * 2, w2t = w2 + kH2 * kH1 * 2;
    static_assert(w2t + kH1 * kH2 * 2 <= bar, "and where W1 was");
};

constexpr int kTileThreads = 512;

// A K-major operand in shared memory: where it starts, the bytes to the next
// 8 K elements and to the next 8 rows.
struct Operand {
    uint32_t at, lead, stride;
};

// D (+)= A B^T over `steps` K = 16 steps from the operands' K element 8 c0 on
__device__ __forceinline__ void issue_kmajor(uint32_t d, const Operand &a, const Operand &b, int c0, int steps,
                                             uint32_t idesc, bool first)
{
    for (int k = 0; k < steps; ++k) {
        const uint32_t c = (uint32_t)(c0 + 2 * k);
        umma_bf16_ss(d, umma_desc(a.at + c * a.lead, a.lead, a.stride), umma_desc(b.at + c * b.lead, b.lead, b.stride),
                     idesc, (first && k == 0) ? 0u : 1u);
    }
}

// One CTA = 128 rows of the batch. 16 warps: warp w reads TMEM lanes (rows)
// 32 (w % 4) .. and a quarter w / 4 of the columns; thread 0 copies the
// weights and issues the MMAs.
template <bool TRAIN>
__global__ void __launch_bounds__(kTileThreads, 1) mlp_tile_kernel(const TileArgs a)
{
    using S = TileSmem;
    constexpr uint32_t kCols = TRAIN ? 512 : 256;
    // accumulators: Z1, Z2 and the logits stay for the backward pass
    constexpr uint32_t dZ1c = 0, dZ2c = 128, dLc = 192, dB2c = 256, dB1c = 320;
    constexpr int kGroups = 5, kGroupChunks = kFeatIn / 8 / kGroups, kGroupBytes = kGroupChunks * kH1 * 16;
    extern __shared__ __align__(128) unsigned char sm[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + S::bar);
    uint64_t *wbar = bar + 1;  // W1 by groups, W2 and W3, W2^T and W3^T
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 8);
    int *srow = reinterpret_cast<int *>(sm + S::rows);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.x * 128;

    if (warp == 0) tmem_alloc(tslot, kCols);
    if (tid == 0) {
        for (int k = 0; k < 8; ++k) mbar_init(bar + k, 1);
        fence_mbar_init();
    }
    stage_launch_gate();
    if (!TRAIN && a.counts && blockIdx.x == 0 && tid < 4) a.counts[tid] = 0;
    if (tid < 128) srow[tid] = m0 + tid < a.B ? (a.perm ? a.perm[m0 + tid] : m0 + tid) : -1;
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tslot;

    // ---------------- W1 and X in K groups of 80
    if (tid == 0) {
        for (int g = 0; g < kGroups; ++g) {
            mbar_arrive_expect_tx(wbar + g, kGroupBytes);
            bulk_g2s(sm + S::w1 + g * kGroupBytes, a.W1 + g * (kGroupBytes / 2), kGroupBytes, wbar + g);
        }
    }
    constexpr int kLoads = (128 * kGroupChunks + kTileThreads - 1) / kTileThreads;
    uint4 xv[kGroups][kLoads];
#pragma unroll
    for (int g = 0; g < kGroups; ++g)
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const int t = tid + u * kTileThreads;
            xv[g][u] = make_uint4(0u, 0u, 0u, 0u);
            if (t < 128 * kGroupChunks) {
                const int r = t / kGroupChunks, c = g * kGroupChunks + t - r * kGroupChunks;
                const int row = srow[r];
                if (row >= 0) xv[g][u] = __ldg(reinterpret_cast<const uint4 *>(a.X + (long long)row * kFeatIn + 8 * c));
            }
        }
    auto store_x = [&](int g) {
#pragma unroll
        for (int u = 0; u < kLoads; ++u) {
            const int t = tid + u * kTileThreads;
            if (t < 128 * kGroupChunks) {
                const int r = t / kGroupChunks, c = g * kGroupChunks + t - r * kGroupChunks;
                *reinterpret_cast<uint4 *>(sm + S::x + (r >> 3) * S::xrows + c * S::xpitch + (r & 7) * 16) = xv[g][u];
            }
        }
    };

    unsigned phase = 0;
    int ok = 1, copies = kGroups;
    // the MMAs issued so far have finished (bounded wait); false ends the block
    auto done = [&]() -> bool {
        if (!mbar_wait_bounded(bar, phase, kWaitLimit)) ok = 0;
        phase ^= 1u;
        ok = __syncthreads_and(ok);
        tc_fence_after();
        return ok != 0;
    };
    // generic writes (and landed copies) of every thread, then the MMAs
    auto publish = [&]() {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
    };
    auto give_up = [&]() {
        // report, and release the tensor memory without writing results;
        // the MMAs in flight get another bounded wait
        if (tid == 0) atomicOr(a.err, kFlagTimeout);
        mbar_wait_bounded(bar, phase ^ 1u, kWaitLimit);
        if (tid == 0)
            for (int k = 0; k < copies; ++k) mbar_wait_bounded(wbar + k, 0, kWaitLimit);
        tc_fence_before();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, kCols);
    };
    // thread 0: weight copy k has landed
    auto landed = [&](int k) -> bool {
        if (!mbar_wait_bounded(wbar + k, 0, kWaitLimit)) ok = 0;
        return ok != 0;
    };
    const uint32_t base = smem_u32(sm);
    auto tile = [&](int at, int chunks) -> Operand { return {base + (uint32_t)at, 128u, (uint32_t)chunks * 128u}; };
    auto weights = [&](int at, int rows) -> Operand { return {base + (uint32_t)at, (uint32_t)rows * 16u, 128u}; };

    // ---------------- Z1 = X W1^T
    auto group = [&](int g) {
        publish();
        if (tid == 0 && landed(g))
            issue_kmajor(tmem + dZ1c, Operand{base + S::x, S::xpitch, S::xrows}, weights(S::w1, kH1), g * kGroupChunks,
                         kGroupChunks / 2, umma_idesc_bf16_f32(128, kH1), g == 0);
    };
    store_x(0);
    group(0);
    store_x(1);
    group(1);
    store_x(2);
    group(2);
    store_x(3);
    group(3);
    store_x(4);
    group(4);
    if (tid == 0) umma_commit(bar);
    if (!done()) return give_up();
    // the other weights into X's and W1's place, while H1 is made
    if (tid == 0) {
        mbar_arrive_expect_tx(wbar + 5, (kH2 * kH1 + kOutPad * kH2) * 2);
        bulk_g2s(sm + S::w2, a.W2, kH2 * kH1 * 2, wbar + 5);
        bulk_g2s(sm + S::w3, a.W3, kOutPad * kH2 * 2, wbar + 5);
        if (TRAIN) {
            mbar_arrive_expect_tx(wbar + 6, (kH2 * kH1 + kOutPad * kH2) * 2);
            bulk_g2s(sm + S::w2t, a.W2T, kH2 * kH1 * 2, wbar + 6);
            bulk_g2s(sm + S::w3t, a.W3T, kOutPad * kH2 * 2, wbar + 6);
        }
    }
    copies = TRAIN ? 7 : 6;

    const int r = 32 * (warp & 3) + lane, cg = warp >> 2;
    const int row = m0 + r;
    const bool rv = row < a.B;
    const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    float *t1 = reinterpret_cast<float *>(sm + S::t1), *t2 = reinterpret_cast<float *>(sm + S::t2);
    // 16 columns from nb on of a hidden layer: + bias, GELU, the next GEMM's
    // operand (and its copy for the weight gradients)
    auto hidden = [&](uint32_t dcol, const float *bias, int nb, int width, int at, float *tt, bf16 *out) {
        float v[16];
        tmem_ld16(tl + dcol + (uint32_t)nb, v);
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            v[k] += bias[nb + k];
            const float t = gelu_t(v[k]);
            if (TRAIN) tt[(nb + k) * 128 + r] = t;
            v[k] = gelu_f(v[k], t);
        }
        uint4 h[2];
        pack_bf16(v, h);
        unsigned char *dst = sm + at + ((r >> 3) * (width / 8) + nb / 8) * 128 + (r & 7) * 16;
        *reinterpret_cast<uint4 *>(dst) = h[0];
        *reinterpret_cast<uint4 *>(dst + 128) = h[1];
        if (TRAIN && rv) {
            uint4 *o = reinterpret_cast<uint4 *>(out + blocked_index(width / 8, row, nb));
            o[0] = h[0];
            o[8] = h[1];
        }
    };
#pragma unroll 1
    for (int nb = 32 * cg; nb < 32 * cg + 32; nb += 16) hidden(dZ1c, a.b1, nb, kH1, S::h1, t1, a.H1);

    // ---------------- Z2 = H1 W2^T
    publish();
    if (tid == 0) {
        if (landed(5))
            issue_kmajor(tmem + dZ2c, tile(S::h1, kH1 / 8), weights(S::w2, kH2), 0, kH1 / 16,
                         umma_idesc_bf16_f32(128, kH2), true);
        umma_commit(bar);
    }
    if (!done()) return give_up();
    hidden(dZ2c, a.b2, 16 * cg, kH2, S::h2, t2, a.H2);

    // ---------------- L = H2 W3^T
    publish();
    if (tid == 0) {
        issue_kmajor(tmem + dLc, tile(S::h2, kH2 / 8), weights(S::w3, kOutPad), 0, kH2 / 16,
                     umma_idesc_bf16_f32(128, kOutPad), true);
        umma_commit(bar);
    }
    if (!done()) return give_up();
    if (cg == 0) {
        float v[16];
        tmem_ld16(tl + dLc, v);
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] += a.b3[k];
        if (a.logits && rv) {
            float4 *dst = reinterpret_cast<float4 *>(a.logits + (long long)row * kOutPad);
#pragma unroll
            for (int k = 0; k < 4; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
        }
        const float l0 = v[0], l1 = v[1], l2 = v[2];
        const int arg = (l0 >= l1 && l0 >= l2) ? 0 : (l1 >= l2 ? 1 : 2);
        if (a.cls && rv) a.cls[row] = arg;
        if (TRAIN) {
            // softmax cross-entropy on the 3 logits: dL = softmax - onehot
            // (not divided by B; the optimiser scales), zero in the padding
            double loss = 0.0;
            int corr = 0;
            float g[16] = {};
            if (rv) {
                const float mx = fmaxf(l0, fmaxf(l1, l2));
                const float e0 = expf(l0 - mx), e1 = expf(l1 - mx), e2 = expf(l2 - mx);
                const float s = e0 + e1 + e2;
                const int yy = a.y[srow[r]];
                const float ly = yy == 0 ? l0 : yy == 1 ? l1 : l2;
                loss = (double)(mx + logf(s) - ly);
                corr = arg == yy;
                g[0] = e0 / s - (yy == 0 ? 1.0f : 0.0f);
                g[1] = e1 / s - (yy == 1 ? 1.0f : 0.0f);
                g[2] = e2 / s - (yy == 2 ? 1.0f : 0.0f);
            }
            uint4 h[2];
            pack_bf16(g, h);
            unsigned char *dst = sm + S::dl + (r >> 3) * 256 + (r & 7) * 16;
            *reinterpret_cast<uint4 *>(dst) = h[0];
            *reinterpret_cast<uint4 *>(dst + 128) = h[1];
            if (rv) {
                uint4 *o = reinterpret_cast<uint4 *>(a.dL + blocked_index(kOutPad / 8, row, 0));
                o[0] = h[0];
                o[8] = h[1];
            }
            loss = warp_sum(loss);
            corr = __reduce_add_sync(0xffffffffu, corr);
            if (lane == 0) {
                a.loss[blockIdx.x * 4 + warp] = loss;
                a.correct[blockIdx.x * 4 + warp] = corr;
            }
        }
    }
    if (TRAIN) {
        // ---------------- dZ2 = (dL W3) * gelu'(Z2)
        publish();
        if (tid == 0) {
            if (landed(6))
                issue_kmajor(tmem + dB2c, tile(S::dl, kOutPad / 8), weights(S::w3t, kH2), 0, 1,
                             umma_idesc_bf16_f32(128, kH2), true);
            umma_commit(bar);
        }
        if (!done()) return give_up();
        // 16 columns from nb on of a hidden layer's gradient
        auto back = [&](uint32_t dcol, uint32_t zcol, const float *bias, int nb, int width, int at,
                        const float *tt, bf16 *out) {
            float v[16], z[16];
            tmem_ld16(tl + dcol + (uint32_t)nb, v);
            tmem_ld16(tl + zcol + (uint32_t)nb, z);
#pragma unroll
            for (int k = 0; k < 16; ++k) v[k] *= gelu_grad_f(z[k] + bias[nb + k], tt[(nb + k) * 128 + r]);
            uint4 h[2];
            pack_bf16(v, h);
            if (at >= 0) {
                unsigned char *dst = sm + at + ((r >> 3) * (width / 8) + nb / 8) * 128 + (r & 7) * 16;
                *reinterpret_cast<uint4 *>(dst) = h[0];
                *reinterpret_cast<uint4 *>(dst + 128) = h[1];
            }
            if (rv) {
                uint4 *o = reinterpret_cast<uint4 *>(out + blocked_index(width / 8, row, nb));
                o[0] = h[0];
                o[8] = h[1];
            }
        };
        back(dB2c, dZ2c, a.b2, 16 * cg, kH2, S::dz2, t2, a.dZ2);
        // ---------------- dZ1 = (dZ2 W2) * gelu'(Z1)
        publish();
        if (tid == 0) {
            issue_kmajor(tmem + dB1c, tile(S::dz2, kH2 / 8), weights(S::w2t, kH1), 0, kH2 / 16,
                         umma_idesc_bf16_f32(128, kH1), true);
            umma_commit(bar);
        }
        if (!done()) return give_up();
#pragma unroll 1
        for (int nb = 32 * cg; nb < 32 * cg + 32; nb += 16) back(dB1c, dZ1c, a.b1, nb, kH1, -1, t1, a.dZ1);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kCols);
}

// Arguments of mlp_wgrad_kernel: the tile kernel's outputs, X as there.
struct WgradArgs {
    const bf16 *X;
    const int *perm;
    int B;
    const bf16 *H1, *H2, *dZ1, *dZ2, *dL;
    float *P1, *P2, *P3;  // per 256 rows: dW1 [128 x 400], dW2^T [128 x 64], dW3^T [64 x 16]
    float *gb;            // bias gradients, summed over the batch
    int *err;
};

constexpr int kWgradThreads = 256;
constexpr int kWgradRoles = 7;            // five fifths of dW1, dW2, dW3
constexpr int kWgradN1 = kFeatIn / 5;     // columns of a dW1 role
constexpr int kBiasBlocks = (kH1 + kH2 + kOutPad) / 8;
constexpr int kBiasRows = 4096;           // rows staged at a time
constexpr int kWgradA = kWgradK * 128 * 2, kWgradB = kWgradK * kWgradN1 * 2;
constexpr int kWgradSmem = kWgradA + kWgradB + 48 + kWgradK * 4;
static_assert(kBiasRows * 16 + 32 * 8 * 4 <= kWgradA + kWgradB, "bias rows fit the operands' space");

// The weight gradients' partial sums: one CTA per 256 rows and role, C[M x N]
// = A^T B with both operands MN-major: the leading offset goes to the next 8
// rows, the stride offset to the next 16 bytes of a row. Bulk copies bring
// what the tile kernel wrote, cp.async gathers X's columns (with cp.async for
// both, the copies took 8 of 12 us). The last kBiasBlocks CTAs sum 8 columns
// each of dZ1, dZ2, dL over the whole batch, each row in lane b % 32's sum,
// then the lanes as a shuffle tree does.
__global__ void __launch_bounds__(kWgradThreads, 2) mlp_wgrad_kernel(const WgradArgs a)
{
    extern __shared__ __align__(128) unsigned char sm[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int splits = (a.B + kWgradK - 1) / kWgradK;
    if ((int)blockIdx.x >= splits * kWgradRoles) {
        stage_launch_gate();
        const int u0 = 8 * ((int)blockIdx.x - splits * kWgradRoles);
        const bf16 *src;
        int chunks, col;
        if (u0 < kH1) { src = a.dZ1; chunks = kH1 / 8; col = u0; }
        else if (u0 < kH1 + kH2) { src = a.dZ2; chunks = kH2 / 8; col = u0 - kH1; }
        else { src = a.dL; chunks = kOutPad / 8; col = u0 - kH1 - kH2; }
        const int u = tid & 7, l = tid >> 3;
        float s = 0.0f;
        for (int b0 = 0; b0 < a.B; b0 += kBiasRows) {
            const int nb = min(kBiasRows, a.B - b0);
            for (int k = tid; k < nb; k += kWgradThreads)
                cp_async16(sm + k * 16, src + blocked_index(chunks, b0 + k, col));
            cp_async_commit();
            cp_async_wait_all();
            __syncthreads();
            const bf16 *rows = reinterpret_cast<const bf16 *>(sm);
#pragma unroll 8
            for (int k = l; k < nb; k += 32) s += __bfloat162float(rows[k * 8 + u]);
            __syncthreads();
        }
        float *p = reinterpret_cast<float *>(sm + kBiasRows * 16);
        p[l * 8 + u] = s;
        for (int o = 16; o > 0; o >>= 1) {
            __syncthreads();
            if (l < o) p[l * 8 + u] += p[(l + o) * 8 + u];
        }
        if (l == 0) a.gb[u0 + u] = p[u];
        return;
    }

    constexpr uint32_t kCols = 128;
    uint64_t *bar = reinterpret_cast<uint64_t *>(sm + kWgradA + kWgradB);
    uint64_t *cbar = bar + 1;  // the bulk copies of each group of 64 rows
    uint32_t *tslot = reinterpret_cast<uint32_t *>(bar + 5);
    int *srow = reinterpret_cast<int *>(bar + 6);  // the rows of X
    const int z = blockIdx.x / kWgradRoles, role = blockIdx.x % kWgradRoles;
    const int k0 = z * kWgradK, kc = min(kWgradK, a.B - k0), kr = (kc + 15) / 16 * 16;
    // A and B in 16-byte pieces a row; dW3 has 64 rows: the other half of the
    // tile multiplies what follows in shared memory and is not stored
    const int ma = role < 6 ? kH1 / 8 : kH2 / 8, nb = role < 5 ? kWgradN1 / 8 : role == 5 ? kH2 / 8 : kOutPad / 8;
    const bf16 *A = role < 5 ? a.dZ1 : role == 5 ? a.H1 : a.H2;
    const bf16 *Bm = role == 5 ? a.dZ2 : a.dL;
    if (warp == 0) tmem_alloc(tslot, kCols);
    if (tid == 0) {
        for (int k = 0; k < 5; ++k) mbar_init(bar + k, 1);
        fence_mbar_init();
    }
    stage_launch_gate();
    unsigned char *sA = sm, *sB = sm + kWgradA;
    if (tid == 0) {
        for (int g = 0; 64 * g < kc; ++g) {
            const int rows = min(64, kc - 64 * g), na = rows * ma * 16, nbytes = role < 5 ? 0 : rows * nb * 16;
            mbar_arrive_expect_tx(cbar + g, (unsigned)(na + nbytes));
            bulk_g2s(sA + 64 * g * ma * 16, A + (long long)(k0 + 64 * g) * ma * 8, (unsigned)na, cbar + g);
            if (nbytes)
                bulk_g2s(sB + 64 * g * nb * 16, Bm + (long long)(k0 + 64 * g) * nb * 8, (unsigned)nbytes, cbar + g);
        }
    }
    if (role < 5) {
        // (one load for all: read where it is used, the copies waited for it)
        if (tid < kc) srow[tid] = a.perm ? a.perm[k0 + tid] : k0 + tid;
        __syncthreads();
    }
    // rows past the batch, up to a whole K step, are zero
    for (int t = tid; t < (kr - kc) * (ma + nb); t += kWgradThreads) {
        const int k = kc + t / (ma + nb), c = t % (ma + nb);
        unsigned char *dst = c < ma ? sA + ((k >> 3) * ma + c) * 128 : sB + ((k >> 3) * nb + c - ma) * 128;
        *reinterpret_cast<uint4 *>(dst + (k & 7) * 16) = make_uint4(0u, 0u, 0u, 0u);
    }
    // X's columns of the role, in the same four groups; neighbouring threads
    // take the two halves of a 32-byte sector, then the next row
    for (int g = 0; g < 4; ++g) {
        if (role < 5) {
            constexpr int np = kWgradN1 / 16;
            for (int t = tid; t < 64 * kWgradN1 / 8; t += kWgradThreads) {
                const int k = 64 * g + (t >> 1 & 7) + 8 * ((t >> 4) / np), c = (t & 1) + 2 * ((t >> 4) % np);
                if (k >= kc) continue;
                const int row = srow[k];
                cp_async16(sB + ((k >> 3) * (kWgradN1 / 8) + c) * 128 + (k & 7) * 16,
                           a.X + (long long)row * kFeatIn + role * kWgradN1 + 8 * c);
            }
        }
        cp_async_commit();
    }
    const uint32_t idesc = umma_idesc_bf16_f32(128, 8 * nb) | kUmmaMnMajorA | kUmmaMnMajorB;
    uint32_t tmem = 0;
    int ok = 1;
    auto group = [&](int g) {
        fence_async_smem();
        tc_fence_before();
        __syncthreads();
        tc_fence_after();
        tmem = *tslot;
        if (tid == 0 && 64 * g < kc) {
            if (!mbar_wait_bounded(cbar + g, 0, kWaitLimit)) ok = 0;
            for (int k = 64 * g; ok && k < min(kr, 64 * (g + 1)); k += 16)
                umma_bf16_ss(tmem, umma_desc(smem_u32(sA) + (uint32_t)((k >> 3) * ma) * 128u, (uint32_t)ma * 128u, 128),
                             umma_desc(smem_u32(sB) + (uint32_t)((k >> 3) * nb) * 128u, (uint32_t)nb * 128u, 128),
                             idesc, k > 0 ? 1u : 0u);
        }
    };
    cp_async_wait_group<3>();
    group(0);
    cp_async_wait_group<2>();
    group(1);
    cp_async_wait_group<1>();
    group(2);
    cp_async_wait_group<0>();
    group(3);
    if (tid == 0) umma_commit(bar);
    if (!mbar_wait_bounded(bar, 0, kWaitLimit)) ok = 0;
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (!ok) {
        // report; the copies and MMAs in flight get another bounded wait
        if (tid == 0) {
            atomicOr(a.err, kFlagTimeout);
            for (int g = 0; 64 * g < kc; ++g) mbar_wait_bounded(cbar + g, 0, kWaitLimit);
        }
        mbar_wait_bounded(bar, 0, kWaitLimit);
    } else {
        const int row = 32 * (warp & 3) + lane;
        float *out;
        int ldo;
        if (role < 5) { out = a.P1 + ((long long)z * kH1 + row) * kFeatIn + role * kWgradN1; ldo = kH1; }
        else if (role == 5) { out = a.P2 + ((long long)z * kH1 + row) * kH2; ldo = kH1; }
        else { out = a.P3 + ((long long)z * kH2 + row) * kOutPad; ldo = kH2; }
        for (int c = 16 * (warp >> 2); c < 8 * nb; c += 32) {
            float v[16];
            tmem_ld16(tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)c, v);
            if (row < ldo) {
                float4 *dst = reinterpret_cast<float4 *>(out + c);
#pragma unroll
                for (int k = 0; k < 4; ++k) dst[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, kCols);
}

// ---------------------------------------------------------------- features

// Patch features: the quad's n x n patch box-averaged to 8 x 8 (n = 8: as
// is, n = 16: 2 x 2 means) plus a one-cell ring from the neighbour cells
// its edge fluxes pair with (the flux kernels' index pairing; a coarse
// hanging side averages its two fine neighbours, a boundary side repeats
// the edge cells, the four ring corners repeat the patch corners), each
// field normalised by the patch's own mean state:
//   x0 = S (rho - mean rho) / mean rho
//   x1 = S (rho u - mean rho u) / (mean rho * a),   x2 likewise for rho v
//   x3 = S (rho E - mean rho E) / mean rho E
// with a the sound speed of the mean state and S = kFeatScale; layout
// X[q][c*100 + (J+1)*10 + (I+1)], I, J = -1..8.
//
// One warp per quad, a patch in shared memory: 64 cells (two a lane) and the
// 32 ring cells (one a lane). Bound by the latency of a quad's loads and of
// its divisions and root, which one warp now does once for the quad: a block
// of four warps and three barriers per quad took 27 us for 6802 quads of 8x8
// (14 MB read), this takes 12 us.
constexpr int kFeatWarps = 4;

template <int N>
__global__ void __launch_bounds__(32 * kFeatWarps) features_kernel(const double *q, long long stride,
                                                                   const QuadDesc *quads, int nquad, bf16 *X)
{
    constexpr int R = N / 8;
    constexpr int NN = N * N;
    __shared__ double sP[kFeatWarps][4][100];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int quad = blockIdx.x * kFeatWarps + w;
    if (quad >= nquad) return;
    double(*P)[100] = sP[w];
    const int sd = lane >> 3, M = lane & 7;
    const SideDesc d = quads[quad].side[sd];
    const double inv = 1.0 / (double)(R * R);
    double v[4][2];
#pragma unroll
    for (int f = 0; f < 4; ++f)
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int I = lane & 7, J = (lane >> 3) + 4 * k;
            double s = 0.0;
#pragma unroll
            for (int dj = 0; dj < R; ++dj)
#pragma unroll
                for (int di = 0; di < R; ++di)
                    s += q[f * stride + (long long)quad * NN + (R * J + dj) * N + (R * I + di)];
            v[f][k] = s * inv;
            P[f][(J + 1) * 10 + I + 1] = v[f][k];
        }
    {
        // box mean over the R cells facing this ring cell (own edge cells
        // for a boundary side are averaged across the edge only)
        const double rinv = 1.0 / (double)R;
        const int at = sd == 0 ? (M + 1) * 10 : sd == 1 ? (M + 1) * 10 + 9 : sd == 2 ? M + 1 : 90 + M + 1;
        const bool own = !(d.kind == kSideFull || d.kind == kSideFineHang || d.kind == kSideCoarseHang);
        const long long b0 = (long long)(own ? quad : d.nbr0) * NN;
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            double s = 0.0;
#pragma unroll
            for (int dm = 0; dm < R; ++dm) {
                const int m = R * M + dm;
                const int oc = (sd == 0) ? m * N : (sd == 1) ? m * N + N - 1 : (sd == 2) ? m : (N - 1) * N + m;
                const int fc = facing_cell<N>(sd, m);
                double x = q[f * stride + b0 + (own ? oc : fc)];
                if (d.kind == kSideCoarseHang) x = 0.5 * (x + q[f * stride + (long long)d.nbr1 * NN + fc]);
                s += x;
            }
            P[f][at] = s * rinv;
        }
    }
    // means of the 8 x 8 patch, in a fixed order
    double m4[4];
#pragma unroll
    for (int f = 0; f < 4; ++f) m4[f] = (warp_sum(v[f][0]) + warp_sum(v[f][1])) / 64.0;
    __syncwarp();
    if (lane < 16) {
        const int f = lane >> 2, cj = lane & 2 ? 9 : 0, ci = lane & 1 ? 9 : 0;
        P[f][cj * 10 + ci] = P[f][(lane & 2 ? 8 : 1) * 10 + (lane & 1 ? 8 : 1)];
    }
    const double mr = m4[0], mu = m4[1], mv = m4[2], me = m4[3];
    const double pbar = 0.4 * (me - 0.5 * (mu * mu + mv * mv) / mr);
    const double c2 = 1.4 * pbar / mr;
    const double abar = sqrt(c2 > 1e-24 ? c2 : 1e-24);
    const double sc[4] = {kFeatScale / mr, kFeatScale / (mr * abar), kFeatScale / (mr * abar), kFeatScale / me};
    __syncwarp();
    __nv_bfloat162 *out = reinterpret_cast<__nv_bfloat162 *>(X + (long long)quad * kFeatIn);
#pragma unroll
    for (int f = 0; f < 4; ++f)
        for (int k = lane; k < 50; k += 32) {
            const double x0 = (P[f][2 * k] - m4[f]) * sc[f], x1 = (P[f][2 * k + 1] - m4[f]) * sc[f];
            out[50 * f + k] = __nv_bfloat162(__float2bfloat16_rn((float)x0), __float2bfloat16_rn((float)x1));
        }
}

// Largest relative density jump of a quad (the plain indicator's method 5
// quantity, as in tag_kernel): between adjacent cells of the patch and
// between an edge cell and the neighbour cell(s) its face flux pairs it
// with. By one warp, whose lanes all get it.
template <int N>
__device__ __forceinline__ double jump_of(const double *rho, const QuadDesc *quads, int quad, int lane)
{
    constexpr int NN = N * N;
    const double *p = rho + (long long)quad * NN;
    auto rj = [](double x, double y) { return fabs(x - y) / fmin(x, y); };
    double J = 0.0;
    for (int c = lane; c < NN; c += 32) {
        const int i = c % N, j = c / N;
        if (i + 1 < N) J = fmax(J, rj(p[c + 1], p[c]));
        if (j + 1 < N) J = fmax(J, rj(p[c + N], p[c]));
    }
    for (int e = lane; e < 4 * N; e += 32) {
        const int s = e / N, mm = e % N;
        const SideDesc &d = quads[quad].side[s];
        const int own = (s == 0) ? mm * N : (s == 1) ? mm * N + N - 1 : (s == 2) ? mm : (N - 1) * N + mm;
        const int fc = facing_cell<N>(s, mm);
        if (d.kind == kSideFull || d.kind == kSideFineHang || d.kind == kSideCoarseHang)
            J = fmax(J, rj(p[own], rho[(long long)d.nbr0 * NN + fc]));
        if (d.kind == kSideCoarseHang) J = fmax(J, rj(p[own], rho[(long long)d.nbr1 * NN + fc]));
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) J = fmax(J, __shfl_xor_sync(0xffffffffu, J, o));
    return J;
}

template <int N>
__global__ void jump_kernel(const double *rho, const QuadDesc *quads, int nquad, double *jump)
{
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= nquad) return;
    const double J = jump_of<N>(rho, quads, w, lane);
    if (lane == 0) jump[w] = J;
}

// plain three-class label of a jump: refine (1) when J >= tol, coarsen (0)
// when J < lo_frac * tol, keep (2) in between
__device__ __forceinline__ int class_of(double j, double tol, double lo_frac)
{
    return j >= tol ? kClassRefine : (j < lo_frac * tol ? kClassCoarsen : kClassKeep);
}

// Labels of n jumps. cover: merged into the label already there, keeping the
// finer demand (refine if either asks for it, coarsen only if both do, keep
// otherwise)
__global__ void label_kernel(const double *J, int n, double tol, double lo_frac, int *cls, int cover)
{
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    int c = class_of(J[k], tol, lo_frac);
    if (cover) {
        const int old = cls[k];
        c = (old == kClassRefine || c == kClassRefine) ? kClassRefine
            : (old == kClassCoarsen && c == kClassCoarsen) ? kClassCoarsen : kClassKeep;
    }
    cls[k] = c;
}

// The judge: the plain class of the quads that a hash of (seed, quad) puts
// below `fraction`, against the learned class, one warp per quad. counts[0]:
// judged, [1]: the classes differ, [2]: the learned one is coarser (the tile
// kernel has set them to zero). On the host the sampling loop and the two
// copies of the sample cost 30-40 us at 7000 quads, most of a call.
template <int N>
__global__ void __launch_bounds__(256) judge_kernel(const double *rho, const QuadDesc *quads, int nquad,
                                                    unsigned long long seed, double fraction, double tol,
                                                    double lo_frac, const int *cls, int *counts)
{
    const int quad = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (quad >= nquad) return;
    unsigned long long z = seed * 0x9E3779B97F4A7C15ull + (unsigned long long)quad * 0xD1B54A32D192ED03ull +
                           0x8CB92BA72F3D8DD7ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    if (!((double)(z >> 11) * (1.0 / 9007199254740992.0) < fraction)) return;
    const int p = class_of(jump_of<N>(rho, quads, quad, lane), tol, lo_frac), t = cls[quad];
    if (lane == 0) {
        atomicAdd(counts, 1);
        if (p != t) atomicAdd(counts + 1, 1);
        if ((p == kClassRefine && t != kClassRefine) || (t == kClassCoarsen && p != kClassCoarsen))
            atomicAdd(counts + 2, 1);
    }
}

// ---------------------------------------------------------------- optimiser

// The parameter tensors in flat order (W1, b1, W2, b2, W3, b3) and where
// each one's gradient is after the weight-gradient kernel.
struct GradArgs {
    const float *P1, *P2, *P3, *gb;
    int splits;
    float inv_b;  // the loss kernel leaves dL unscaled
};

constexpr int kOffB1 = kH1 * kFeatIn, kOffW2 = kOffB1 + kH1, kOffB2 = kOffW2 + kH2 * kH1, kOffW3 = kOffB2 + kH2,
              kOffB3 = kOffW3 + kOut * kH2;

// Thread t's flat parameter: W2 and W3 in the order of their partials, which
// hold the transposes, so that neighbouring threads read neighbours.
__device__ __forceinline__ int param_of(int t)
{
    if (t >= kOffW2 && t < kOffB2) {
        const int k = t - kOffW2;
        return kOffW2 + (k % kH2) * kH1 + k / kH2;
    }
    if (t >= kOffW3 && t < kOffB3) {
        const int k = t - kOffW3;
        return kOffW3 + (k % kOut) * kH2 + k / kOut;
    }
    return t;
}

// Gradient of flat parameter idx: a weight's is the sum over the partials in
// order, read transposed where they hold W^T.
__device__ __forceinline__ float grad_of(const GradArgs &g, int idx)
{
    const float *p;
    int step;
    if (idx < kOffB1) {
        p = g.P1 + idx;
        step = kH1 * kFeatIn;
    } else if (idx < kOffW2) {
        return g.gb[idx - kOffB1] * g.inv_b;
    } else if (idx < kOffB2) {
        const int k = idx - kOffW2, o = k / kH1, i = k % kH1;
        p = g.P2 + i * kH2 + o;
        step = kH1 * kH2;
    } else if (idx < kOffW3) {
        return g.gb[kH1 + idx - kOffB2] * g.inv_b;
    } else if (idx < kOffB3) {
        const int k = idx - kOffW3, o = k / kH2, i = k % kH2;
        p = g.P3 + i * kOutPad + o;
        step = kH2 * kOutPad;
    } else {
        return g.gb[kH1 + kH2 + idx - kOffB3] * g.inv_b;
    }
    float s = 0.0f;
#pragma unroll 32
    for (int k = 0; k < g.splits; ++k) s += p[(long long)k * step];
    return s * g.inv_b;
}

// AdamW (decoupled weight decay, on weights only) on the FP32 master
// parameters; refreshes the BF16 copies of W and W^T (tiled_index) and the
// padded FP32 b3 that the tile kernel reads.
struct AdamArgs {
    GradArgs g;
    float *w, *m, *v;
    bf16 *W1, *W2, *W3, *W2T, *W3T;
    float *b3p;
    float lr, wd, b1, b2, eps, c1, c2;  // c1 = 1/(1-b1^t), c2 = 1/(1-b2^t)
};

__global__ void __launch_bounds__(128) mlp_adamw_kernel(const AdamArgs a)
{
    stage_launch_gate();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kMlpParams) return;
    const int idx = param_of(t);
    const bool weight = idx < kOffB1 || (idx >= kOffW2 && idx < kOffB2) || (idx >= kOffW3 && idx < kOffB3);
    const float m0 = a.m[idx], v0 = a.v[idx];
    float w = a.w[idx];
    const float g = grad_of(a.g, idx);
    const float m = a.b1 * m0 + (1.0f - a.b1) * g;
    const float v = a.b2 * v0 + (1.0f - a.b2) * g * g;
    a.m[idx] = m;
    a.v[idx] = v;
    const float wd = weight ? a.wd : 0.0f;
    w -= a.lr * ((m * a.c1) / (sqrtf(v * a.c2) + a.eps) + wd * w);
    a.w[idx] = w;
    const bf16 wb = __float2bfloat16_rn(w);
    if (idx < kOffB1) {
        a.W1[tiled_index(kH1, idx / kFeatIn, idx % kFeatIn)] = wb;
    } else if (idx >= kOffW2 && idx < kOffB2) {
        const int k = idx - kOffW2, o = k / kH1, i = k % kH1;
        a.W2[tiled_index(kH2, o, i)] = wb;
        a.W2T[tiled_index(kH1, i, o)] = wb;
    } else if (idx >= kOffW3 && idx < kOffB3) {
        const int k = idx - kOffW3, o = k / kH2, i = k % kH2;
        a.W3[tiled_index(kOutPad, o, i)] = wb;
        a.W3T[tiled_index(kH2, i, o)] = wb;
    } else if (idx >= kOffB3) {
        a.b3p[idx - kOffB3] = w;
    }
}

__global__ void __launch_bounds__(256) mlp_grad_kernel(const GradArgs g, float *out)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= kMlpParams) return;
    const int idx = param_of(t);
    out[idx] = grad_of(g, idx);
}

// ---------------------------------------------------------------- host side

cudaError_t mlp_launch_features(int n, const double *q, long long stride, const QuadDesc *quads, int nquad, bf16 *X,
                                cudaStream_t st)
{
    if (nquad <= 0) return cudaSuccess;
    const int blocks = (nquad + kFeatWarps - 1) / kFeatWarps;
    switch (n) {
    case 8: features_kernel<8><<<blocks, 32 * kFeatWarps, 0, st>>>(q, stride, quads, nquad, X); break;
    case 16: features_kernel<16><<<blocks, 32 * kFeatWarps, 0, st>>>(q, stride, quads, nquad, X); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t mlp_launch_jump(int n, const double *rho, const QuadDesc *quads, int nquad, double *J, cudaStream_t st)
{
    if (nquad <= 0) return cudaSuccess;
    const int blocks = (nquad * 32 + 255) / 256;
    switch (n) {
    case 2: jump_kernel<2><<<blocks, 256, 0, st>>>(rho, quads, nquad, J); break;
    case 4: jump_kernel<4><<<blocks, 256, 0, st>>>(rho, quads, nquad, J); break;
    case 8: jump_kernel<8><<<blocks, 256, 0, st>>>(rho, quads, nquad, J); break;
    case 16: jump_kernel<16><<<blocks, 256, 0, st>>>(rho, quads, nquad, J); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t mlp_launch_judge(int n, const double *rho, const QuadDesc *quads, int nquad, unsigned long long seed,
                             double fraction, double tol, double lo_frac, const int *cls, int *counts, cudaStream_t st)
{
    if (nquad <= 0) return cudaSuccess;
    const int blocks = (nquad * 32 + 255) / 256;
    switch (n) {
    case 8: judge_kernel<8><<<blocks, 256, 0, st>>>(rho, quads, nquad, seed, fraction, tol, lo_frac, cls, counts); break;
    case 16: judge_kernel<16><<<blocks, 256, 0, st>>>(rho, quads, nquad, seed, fraction, tol, lo_frac, cls, counts); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t mlp_launch_labels(const double *J, int n, double tol, double lo_frac, int *cls, cudaStream_t st,
                              bool cover)
{
    if (n <= 0) return cudaSuccess;
    label_kernel<<<(n + 255) / 256, 256, 0, st>>>(J, n, tol, lo_frac, cls, cover ? 1 : 0);
    return cudaGetLastError();
}

namespace {

template <typename T>
bool dalloc(T **p, size_t n, std::vector<void *> &own)
{
    if (cudaMalloc((void **)p, sizeof(T) * std::max<size_t>(n, 1)) != cudaSuccess) return false;
    own.push_back((void *)*p);
    return true;
}

// Offsets of the flat FP32 parameter vector: W1 [128x400], b1, W2 [64x128],
// b2, W3 [3x64], b3.
const int kParamOff[7] = {0, kOffB1, kOffW2, kOffB2, kOffW3, kOffB3, kMlpParams};

// A launch that may be scheduled while its predecessor in the stream drains
// (the kernel waits on the device, stage_launch_gate).
template <class Args>
cudaError_t launch_after(const void *kernel, int grid, int threads, size_t smem, const Args &a, cudaStream_t st)
{
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3((unsigned)grid);
    lc.blockDim = dim3((unsigned)threads);
    lc.dynamicSmemBytes = smem;
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    void *args[] = {const_cast<Args *>(&a)};
    return cudaLaunchKernelExC(&lc, kernel, args);
}

}  // namespace

MlpState::~MlpState() { release(); }

void MlpState::release()
{
    for (void *p : batch_owned) cudaFree(p);
    for (void *p : fixed_owned) cudaFree(p);
    batch_owned.clear();
    fixed_owned.clear();
    cudaFree(Xall);
    cudaFree(yall);
    cudaFree(perm);
    cudaFree(jump);
    cudaFree(stats);
    cudaFreeHost(h_back);
    h_back = nullptr;
    cap_back = 0;
    cap_stats = 0;
    stats = nullptr;
    Xall = nullptr;
    yall = nullptr;
    perm = nullptr;
    jump = nullptr;
    cap_batch = cap_train = 0;
    cap_data = n_data = cap_perm = 0;
    cap_jump = 0;
}

bool MlpState::init(uint64_t seed)
{
    auto &o = fixed_owned;
    if (!dalloc(&w, kMlpParams, o) || !dalloc(&m, kMlpParams, o) || !dalloc(&v, kMlpParams, o) ||
        !dalloc(&W1, size_t(kH1) * kFeatIn, o) || !dalloc(&W2, size_t(kH2) * kH1, o) ||
        !dalloc(&W3, size_t(kOutPad) * kH2, o) || !dalloc(&W2T, size_t(kH1) * kH2, o) ||
        !dalloc(&W3T, size_t(kH2) * kOutPad, o) || !dalloc(&b3p, kOutPad, o) || !dalloc(&err, 1, o))
        return false;
    // deterministic init: U(-1/sqrt(fan_in), 1/sqrt(fan_in)) for weights and
    // biases, from splitmix64 of the seed and the element index
    std::vector<float> h(kMlpParams);
    auto u01 = [&](uint64_t k) {
        uint64_t z = seed * 0x9E3779B97F4A7C15ULL + k + 0x632BE59BD9B4E019ULL;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ULL;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBULL;
        z ^= z >> 31;
        return (double)(z >> 11) * (1.0 / 9007199254740992.0);
    };
    const int fan[6] = {kFeatIn, kFeatIn, kH1, kH1, kH2, kH2};
    for (int t = 0; t < 6; ++t)
        for (int k = kParamOff[t]; k < kParamOff[t + 1]; ++k)
            h[size_t(k)] = (float)((2.0 * u01(uint64_t(k)) - 1.0) / std::sqrt((double)fan[t]));
    return set_params(h.data());
}

bool MlpState::set_params(const float *h)
{
    if (cudaMemcpy(w, h, sizeof(float) * kMlpParams, cudaMemcpyHostToDevice) != cudaSuccess) return false;
    if (cudaMemset(m, 0, sizeof(float) * kMlpParams) != cudaSuccess) return false;
    if (cudaMemset(v, 0, sizeof(float) * kMlpParams) != cudaSuccess) return false;
    step = 0;
    return refresh_bf16();
}

// BF16 GEMM copies of the FP32 master weights (host round trip; set-up only)
bool MlpState::refresh_bf16()
{
    using bf = __nv_bfloat16;
    std::vector<float> h(kMlpParams);
    if (cudaMemcpy(h.data(), w, sizeof(float) * kMlpParams, cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    const bf zero = __float2bfloat16(0.0f);
    std::vector<bf> w1(size_t(kH1) * kFeatIn), w2(size_t(kH2) * kH1), w3(size_t(kOutPad) * kH2, zero),
        w2t(size_t(kH1) * kH2), w3t(size_t(kH2) * kOutPad, zero);
    std::vector<float> b3(kOutPad, 0.0f);
    // piece by piece of 8 in a row: element by element through tiled_index,
    // two divisions and a scattered store each, it takes 200 us more (set_params
    // 450 us, so 252 us)
    auto pieces = [](const float *src, int rows, int cols, bf *dst) {
        for (int c = 0; c < cols / 8; ++c)
            for (int o = 0; o < rows; ++o)
                for (int k = 0; k < 8; ++k)
                    dst[tiled_index(rows, o, 8 * c) + k] = __float2bfloat16(src[o * cols + 8 * c + k]);
    };
    pieces(h.data() + kParamOff[0], kH1, kFeatIn, w1.data());
    pieces(h.data() + kParamOff[2], kH2, kH1, w2.data());
    for (int o = 0; o < kH2; ++o)
        for (int i = 0; i < kH1; ++i) w2t[size_t(tiled_index(kH1, i, o))] = w2[size_t(tiled_index(kH2, o, i))];
    for (int o = 0; o < kOut; ++o) {
        for (int i = 0; i < kH2; ++i) {
            const bf b = __float2bfloat16(h[size_t(kParamOff[4] + o * kH2 + i)]);
            w3[size_t(tiled_index(kOutPad, o, i))] = b;
            w3t[size_t(tiled_index(kH2, i, o))] = b;
        }
        b3[size_t(o)] = h[size_t(kParamOff[5] + o)];
    }
    return cudaMemcpy(W1, w1.data(), w1.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemcpy(W2, w2.data(), w2.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemcpy(W3, w3.data(), w3.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemcpy(W2T, w2t.data(), w2t.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemcpy(W3T, w3t.data(), w3t.size() * 2, cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemcpy(b3p, b3.data(), b3.size() * 4, cudaMemcpyHostToDevice) == cudaSuccess &&
           cudaMemset(err, 0, sizeof(int)) == cudaSuccess;
}

// Buffers for batches of B rows: features, labels, logits and classes, and
// with `train` what the weight gradients are made from.
bool MlpState::ensure_batch(int B, bool train)
{
    if (B <= cap_batch && (!train || B <= cap_train)) return true;
    // twice the old capacity at least (rows stay a multiple of 128): a mesh
    // that grows a few quads per regrid reallocates rarely
    if (B > cap_batch) B = std::max(B, 2 * cap_batch);
    else B = cap_batch;
    train = train || cap_train > 0;
    cudaStreamSynchronize(stream);
    for (void *p : batch_owned) cudaFree(p);
    batch_owned.clear();
    cap_batch = cap_train = 0;
    auto &o = batch_owned;
    const size_t b = size_t(B);
    const size_t splits = (b + kWgradK - 1) / kWgradK;
    bool ok = dalloc(&X, b * kFeatIn, o) && dalloc(&y, b, o) && dalloc(&Lg, b * kOutPad, o) && dalloc(&cls, b + 4, o);
    if (ok && train)
        ok = dalloc(&H1, b * kH1, o) && dalloc(&H2, b * kH2, o) && dalloc(&dZ1, b * kH1, o) &&
             dalloc(&dZ2, b * kH2, o) && dalloc(&dL, b * kOutPad, o) && dalloc(&P1, splits * kH1 * kFeatIn, o) &&
             dalloc(&P2, splits * kH1 * kH2, o) && dalloc(&P3, splits * kH2 * kOutPad, o) &&
             dalloc(&gb, size_t(kH1 + kH2 + kOutPad), o) && dalloc(&gflat, size_t(kMlpParams), o);
    if (ok) cap_batch = B;
    if (ok && train) cap_train = B;
    return ok;
}

bool MlpState::ensure_stats(long long groups)
{
    if (groups <= cap_stats) return true;
    cudaStreamSynchronize(stream);
    cudaFree(stats);
    stats = nullptr;
    cap_stats = 0;
    groups = std::max<long long>(groups, 1024);
    if (cudaMalloc((void **)&stats, (sizeof(double) + sizeof(int)) * size_t(groups) + sizeof(double)) != cudaSuccess)
        return false;
    cap_stats = groups;
    return true;
}

bool MlpState::ensure_data(long long n)
{
    if (n <= cap_data) return true;
    long long cap = std::max<long long>(n, cap_data * 2);
    __nv_bfloat16 *nx = nullptr;
    int *ny = nullptr;
    if (cudaMalloc(&nx, sizeof(__nv_bfloat16) * size_t(cap) * kFeatIn) != cudaSuccess) return false;
    if (cudaMalloc(&ny, sizeof(int) * size_t(cap)) != cudaSuccess) {
        cudaFree(nx);
        return false;
    }
    if (n_data > 0) {
        cudaMemcpyAsync(nx, Xall, sizeof(__nv_bfloat16) * size_t(n_data) * kFeatIn, cudaMemcpyDeviceToDevice, stream);
        cudaMemcpyAsync(ny, yall, sizeof(int) * size_t(n_data), cudaMemcpyDeviceToDevice, stream);
    }
    cudaStreamSynchronize(stream);
    cudaFree(Xall);
    cudaFree(yall);
    Xall = nx;
    yall = ny;
    cap_data = cap;
    return true;
}

bool MlpState::ensure_jump(int n)
{
    if (n <= cap_jump) return true;
    n = std::max(2 * n, 1024);  // headroom: a mesh that grows reallocates rarely
    cudaStreamSynchronize(stream);
    cudaFree(jump);
    jump = nullptr;
    cap_jump = 0;
    if (cudaMalloc(&jump, sizeof(double) * size_t(n)) != cudaSuccess) return false;
    cap_jump = n;
    return true;
}

bool MlpState::ensure_back(size_t bytes)
{
    if (bytes <= cap_back) return true;
    cudaStreamSynchronize(stream);
    cudaFreeHost(h_back);
    h_back = nullptr;
    cap_back = 0;
    bytes = std::max<size_t>(2 * bytes, 4096);
    if (cudaMallocHost(&h_back, bytes) != cudaSuccess) return false;
    cap_back = bytes;
    return true;
}

namespace {

TileArgs tile_args(const MlpState &s, const RowSource &r, int B)
{
    TileArgs a{};
    a.X = r.X;
    a.perm = r.perm;
    a.y = r.y;
    a.B = B;
    a.W1 = s.W1; a.W2 = s.W2; a.W3 = s.W3; a.W2T = s.W2T; a.W3T = s.W3T;
    a.b1 = s.w + kOffB1; a.b2 = s.w + kOffB2; a.b3 = s.b3p;
    a.err = s.err;
    return a;
}

GradArgs grad_args(const MlpState &s, int B)
{
    GradArgs g{};
    g.P1 = s.P1; g.P2 = s.P2; g.P3 = s.P3; g.gb = s.gb;
    g.splits = (B + kWgradK - 1) / kWgradK;
    g.inv_b = 1.0f / (float)B;
    return g;
}

// The kernels' shared-memory opt-in, once per device.
cudaError_t opt_in()
{
    static std::mutex mu;
    static std::vector<int> done;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    std::lock_guard<std::mutex> lk(mu);
    if (std::find(done.begin(), done.end(), dev) != done.end()) return cudaSuccess;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if ((e = cudaFuncSetAttribute((const void *)mlp_tile_kernel<false>, attr, TileSmem::total)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute((const void *)mlp_tile_kernel<true>, attr, TileSmem::total)) != cudaSuccess) return e;
    if ((e = cudaFuncSetAttribute((const void *)mlp_wgrad_kernel, attr, kWgradSmem)) != cudaSuccess) return e;
    done.push_back(dev);
    return cudaSuccess;
}

}  // namespace

// Forward pass of B rows: logits [B x 16] and classes where given; the
// judge's counts, where given, set to zero.
cudaError_t MlpState::infer(const RowSource &r, int B, float *logits, int *classes, int *counts, cudaStream_t st)
{
    cudaError_t e = opt_in();
    if (e != cudaSuccess) return e;
    TileArgs a = tile_args(*this, r, B);
    a.logits = logits;
    a.cls = classes;
    a.counts = counts;
    return launch_after((const void *)mlp_tile_kernel<false>, (B + 127) / 128, kTileThreads, TileSmem::total, a, st);
}

// Forward and backward pass of B rows (a multiple of 8): the weight-gradient
// partials P1..P3, the bias sums gb, and per 32 rows the loss sum and the
// correct predictions.
cudaError_t MlpState::gradients(const RowSource &r, int B, float *logits, double *loss, int *correct, cudaStream_t st)
{
    cudaError_t e = opt_in();
    if (e != cudaSuccess) return e;
    TileArgs a = tile_args(*this, r, B);
    a.logits = logits;
    a.H1 = H1; a.H2 = H2; a.dZ1 = dZ1; a.dZ2 = dZ2; a.dL = dL;
    a.loss = loss;
    a.correct = correct;
    e = launch_after((const void *)mlp_tile_kernel<true>, (B + 127) / 128, kTileThreads, TileSmem::total, a, st);
    if (e != cudaSuccess) return e;
    WgradArgs w{};
    w.X = r.X;
    w.perm = r.perm;
    w.B = B;
    w.H1 = H1; w.H2 = H2; w.dZ1 = dZ1; w.dZ2 = dZ2; w.dL = dL;
    w.P1 = P1; w.P2 = P2; w.P3 = P3; w.gb = gb;
    w.err = err;
    const int splits = (B + kWgradK - 1) / kWgradK;
    return launch_after((const void *)mlp_wgrad_kernel, splits * kWgradRoles + kBiasBlocks, kWgradThreads, kWgradSmem,
                        w, st);
}

cudaError_t MlpState::update(int B, float lr, float wd, cudaStream_t st)
{
    ++step;
    const float b1 = 0.9f, b2 = 0.999f;
    AdamArgs a{};
    a.g = grad_args(*this, B);
    a.w = w; a.m = m; a.v = v;
    a.W1 = W1; a.W2 = W2; a.W3 = W3; a.W2T = W2T; a.W3T = W3T;
    a.b3p = b3p;
    a.lr = lr;
    a.wd = wd;
    a.b1 = b1;
    a.b2 = b2;
    a.eps = 1e-8f;
    a.c1 = (float)(1.0 / (1.0 - std::pow((double)b1, (double)step)));
    a.c2 = (float)(1.0 / (1.0 - std::pow((double)b2, (double)step)));
    return launch_after((const void *)mlp_adamw_kernel, (kMlpParams + 127) / 128, 128, 0, a, st);
}

cudaError_t MlpState::flat_grad(int B, cudaStream_t st)
{
    mlp_grad_kernel<<<(kMlpParams + 255) / 256, 256, 0, st>>>(grad_args(*this, B), gflat);
    return cudaGetLastError();
}

}  // namespace amrgpu
