// mlp.cu — the warm-start network: parameters, pair set, training on the tensor cores, inference entry.
//
// Training step (one launch per minibatch, whose last CTA applies AdamW). Each CTA (one per SM) takes tiles of 128
// pairs. Per tile, on the tensor cores (tcgen05.mma, M = 128, BF16 operands in shared memory, FP32 accumulators in
// TMEM):
//   Z1  = X  W1^T            (K = 16)    TMEM cols   0..63
//   Z2  = A1 W2^T            (K = 64)    TMEM cols  64..127     A1 = relu(Z1 + b1)
//   dA1 = dZ2 W2             (K = 64)    TMEM cols   0..63      dZ2 = dy w3 [Z2 + b2 > 0]
//   G  += [dZ2 dZ1]^T [A1 X 1]  (K = 128 pairs, N = 80)  TMEM cols 128..207, summed over tiles
// so G holds dW2 (rows 0-63, cols 0-63), db2 (rows 0-63, col 76), dW1 (rows 64-127, cols 64-75) and db1
// (rows 64-127, col 76); the 64 -> 1 output layer and its gradient are FP32 on the CUDA cores. At the end the
// CTA adds G into the global gradient with atomics.
//
// A minibatch is one tile per CTA, so a step lasts as long as one tile's chain of four products and the work
// between them. 512 threads share a tile: warp w holds 32 of its rows (w mod 4) and a quarter of every row's columns
// (w div 4), so each thread passes 16 columns a product and four warps per scheduler cover one another's latencies
// (one thread a row, unrolled over 64 columns: 29 us a step of 8,192 pairs and 2.4 us for AdamW; now 14.4 us for both).
// The weight-gradient product reads the operands of the other products in place, as M- and N-major operands (the
// 8 x 8 core matrices of a K-major [pair][column] tile are those of the M-major [column][pair] one), where
// transposed copies took 204 two-byte stores a thread with four-way bank conflicts.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "gpe_internal.h"
#include "mlp.cuh"

struct gpe_mlp {
    int device = 0;
    gpe::MlpDev* dev = nullptr; // network image read by the kernels
    float* master    = nullptr; // FP32 parameter vector (GPE_MLP_NUM_WEIGHTS)
    float* grad      = nullptr; // gradient accumulator, [NW] = loss sum, [NW+1] = epoch loss sum
    float* adam_m    = nullptr;
    float* adam_v    = nullptr;
    double* stats    = nullptr; // standardisation sums
    uint32_t* status = nullptr;
    float* X         = nullptr; // pair set
    float* T         = nullptr;
    int32_t* idx     = nullptr;
    int32_t* cnt     = nullptr;
    int32_t* order   = nullptr; // shuffled pair indices of an epoch
    uint32_t* sh_target = nullptr; // the shuffle's scratch: each swap's target and its rank among the target's swaps,
    uint32_t* sh_rank   = nullptr; // the swaps per target (zero between shuffles), their first places, and the swaps by
    uint32_t* sh_count  = nullptr; // target
    uint32_t* sh_start  = nullptr;
    uint32_t* sh_swaps  = nullptr;
    uint32_t* sh_bsum   = nullptr;
    uint32_t* done      = nullptr; // CTAs of the running training step that have added their gradient
    int64_t cap      = 0;
    int64_t adam_t   = 0;
    int32_t pair_iters = 20;    // iterations of the plain solve that produced the pairs
    float mu[GPE_MLP_FEATURES], sd[GPE_MLP_FEATURES], ymu = 0.f, ysd = 1.f;
    void* base       = nullptr;
};

namespace gpe {

const MlpDev* mlp_device(const gpe_mlp* m) { return m->dev; }
MlpData mlp_data(gpe_mlp* m) { return MlpData{m->X, m->T, m->idx, m->cnt, m->cap}; }
int32_t mlp_pair_iters(const gpe_mlp* m) { return m->pair_iters; }
void mlp_set_pair_iters(gpe_mlp* m, int32_t iters) { m->pair_iters = iters; }

namespace {

constexpr int TRAIN_T = 512;           // threads a CTA: four a row of the tile
constexpr int AX_N    = 80;            // columns of [A1 X 1]: hidden layer 1 (0-63), features (64-75), ones, zeros
constexpr int AX_X    = 64;
constexpr int AX_ONES = 76;
constexpr int DZ_N    = 128;           // columns of [dZ2 dZ1]
constexpr uint32_t TRAIN_TMEM_COLS = 256;

struct __align__(128) MlpTrainSmem {
    uint16_t ax[MLP_TILE * AX_N]; // [A1 X 1]
    uint16_t dz[MLP_TILE * DZ_N]; // [dZ2 dZ1]
    uint16_t w1[MLP_H * MLP_FP];
    uint16_t w2[MLP_H * MLP_H];
    uint16_t w2t[MLP_H * MLP_H];
    float b1[MLP_H], b2[MLP_H], w3[MLP_H], mu[MLP_FP], isd[MLP_FP];
    float y[MLP_TILE];        // outputs
    float tn[MLP_TILE];       // standardised targets
    float dw3[MLP_H];
    float dw3q[4][MLP_H];     // a tile's sums over 32 rows each
    float db3, loss, b3, ymu, iysd;
    uint64_t bar;
    uint32_t tmem;
    uint32_t last;
};

// AdamW's state and constants (Loshchilov & Hutter 2019): decoupled weight decay on W1, W2 and w3; bc1, bc2 =
// 1 - beta^t. net is null where the gradient alone is asked for.
struct AdamW {
    MlpDev* net;
    float* master;
    float* m;
    float* v;
    uint32_t* done;
    float lr, wd, b1, b2, eps, bc1, bc2;
};

__device__ __forceinline__ uint16_t bf16_bits(float v)
{
    const __nv_bfloat16 h = __float2bfloat16_rn(v);
    return *reinterpret_cast<const uint16_t*>(&h);
}

__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) { v += __shfl_xor_sync(0xffffffffu, v, o); }
    return v;
}

__device__ __forceinline__ uint4 pack8(const float (&a)[16], int c)
{
    return make_uint4(tc::pack_bf16(a[8 * c + 0], a[8 * c + 1]), tc::pack_bf16(a[8 * c + 2], a[8 * c + 3]),
                      tc::pack_bf16(a[8 * c + 4], a[8 * c + 5]), tc::pack_bf16(a[8 * c + 6], a[8 * c + 7]));
}

// Sums of 16 values over a warp's lanes: each exchange halves the values a lane still carries (16 shuffles instead of
// 80); lanes 2c and 2c + 1 return the sum of value c (with the bits of c in the order 8, 4, 2, 1 of the lane's
// 16, 8, 4, 2).
__device__ __forceinline__ float warp_sum16(float (&v)[16])
{
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int h = 8; h > 0; h >>= 1) {
        const bool up = (lane & (uint32_t)(2 * h)) != 0u;
#pragma unroll
        for (int k = 0; k < h; ++k) {
            const float send = up ? v[k] : v[k + h];
            const float keep = up ? v[k + h] : v[k];
            v[k]             = keep + __shfl_xor_sync(0xffffffffu, send, 2 * h);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__device__ __forceinline__ void put_param(MlpDev* m, int p, float w);

// All threads of one CTA: every parameter's step. A thread loads all of its parameters' state before it writes any, so
// that the update costs one memory latency instead of ten. The fused and unfused forms are explicit: the first steps
// divide a small gradient by its own size, so a last bit of the moments is worth 1e-4 of some weights after an epoch,
// and the kernel that this is compiled into must not choose it.
__device__ __forceinline__ void adamw(const AdamW& ad, float* grad)
{
    constexpr int PER = (MLP_NW + TRAIN_T - 1) / TRAIN_T;
    float g[PER], mm[PER], vv[PER], w[PER];
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int p = q * TRAIN_T + (int)threadIdx.x;
        if (p < MLP_NW) {
            g[q]  = __ldcg(&grad[p]);
            mm[q] = ad.m[p];
            vv[q] = ad.v[p];
            w[q]  = ad.master[p];
        }
    }
#pragma unroll
    for (int q = 0; q < PER; ++q) {
        const int p = q * TRAIN_T + (int)threadIdx.x;
        if (p < MLP_NW) {
            grad[p] = 0.f;
            mm[q]   = fmaf(1.f - ad.b1, g[q], __fmul_rn(ad.b1, mm[q]));
            vv[q]   = fmaf((1.f - ad.b2) * g[q], g[q], __fmul_rn(ad.b2, vv[q]));
            ad.m[p] = mm[q];
            ad.v[p] = vv[q];
            const bool decay = (p < MLP_OFF_B1) || (p >= MLP_OFF_W2 && p < MLP_OFF_B2) ||
                               (p >= MLP_OFF_W3 && p < MLP_OFF_B3);
            float step = (mm[q] / ad.bc1) / (sqrtf(vv[q] / ad.bc2) + ad.eps);
            if (decay) { step = __fadd_rn(step, __fmul_rn(ad.wd, w[q])); }
            w[q] = fmaf(-ad.lr, step, w[q]);
            ad.master[p] = w[q];
            put_param(ad.net, p, w[q]);
        }
    }
}

// X and grad 16-byte aligned. grad[NW] is the loss sum, grad[NW + 1] (with AdamW) the epoch's.
__global__ void __launch_bounds__(TRAIN_T, 1)
    k_mlp_train(const MlpDev* m, const float* __restrict__ X, const float* __restrict__ T,
                const int32_t* __restrict__ order, int32_t n, float inv_n, float* grad, uint32_t* __restrict__ status,
                const AdamW adam)
{
    extern __shared__ uint8_t smem_raw[];
    MlpTrainSmem& S = *reinterpret_cast<MlpTrainSmem*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) &
                                                        ~static_cast<uintptr_t>(127));
    const uint32_t t    = threadIdx.x;
    const uint32_t quad = (t >> 5) & 3u, part = t >> 7; // 32 rows of the tile, a quarter of their columns
    const uint32_t r    = quad * 32u + (t & 31u);
    const uint32_t c0   = part * 16u;
    const int32_t ntiles = (n + MLP_TILE - 1) / MLP_TILE; // at least gridDim.x
    // this thread's part of pair r of a tile: four features, or (the row's fourth thread) the target; loaded a tile
    // ahead, the first beside the network
    float4 in   = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch  = [&](int32_t tile) {
        const int64_t q = (int64_t)tile * MLP_TILE + r;
        if (q >= n) { return; }
        const int32_t s = order ? __ldg(&order[q]) : (int32_t)q;
        if (part < 3u) {
            in = __ldg(reinterpret_cast<const float4*>(X) + (size_t)s * (MLP_F / 4) + part);
        } else {
            in.x = __ldg(&T[s]);
        }
    };
    fetch((int32_t)blockIdx.x);

    // ---- stage the network, clear the accumulators ----
    {
        const uint4* s1 = reinterpret_cast<const uint4*>(m->w1);
        const uint4* s2 = reinterpret_cast<const uint4*>(m->w2);
        const uint4* s3 = reinterpret_cast<const uint4*>(m->w2t);
        if (t < MLP_H * MLP_FP / 8) { reinterpret_cast<uint4*>(S.w1)[t] = s1[t]; }
        static_assert(MLP_H * MLP_H / 8 == TRAIN_T, "one 16-byte word of W2 a thread");
        reinterpret_cast<uint4*>(S.w2)[t]  = s2[t];
        reinterpret_cast<uint4*>(S.w2t)[t] = s3[t];
        if (t < MLP_H) {
            S.b1[t] = m->b1[t];
            S.b2[t] = m->b2[t];
            S.w3[t] = m->w3[t];
        }
        if (t < MLP_H) { S.dw3[t] = 0.f; }
        if (t < MLP_FP) {
            S.mu[t]  = m->mu[t];
            S.isd[t] = m->isd[t];
        }
        if (t == 0) {
            S.db3  = 0.f;
            S.loss = 0.f;
            S.b3   = m->b3;
            S.ymu  = m->ymu;
            S.iysd = m->ysd > 0.f ? 1.f / m->ysd : 0.f;
            tc::mbar_init(&S.bar, 1);
        }
        if (t < 32) { tc::tmem_alloc(&S.tmem, TRAIN_TMEM_COLS); }
        tc::fence_async_smem();
        tc::fence_before();
        __syncthreads();
        tc::fence_after();
    }
    const uint32_t tm   = S.tmem;
    const uint32_t mine = tm + ((quad * 32u) << 16); // this warp's TMEM lanes
    constexpr uint32_t ID64 = tc::idesc_bf16(128, 64);
    constexpr uint32_t IDG  = tc::idesc_bf16(128, AX_N) | (1u << 15) | (1u << 16); // A is M-major, B is N-major
    constexpr uint32_t AX_ROWS = AX_N * 16, DZ_ROWS = DZ_N * 16; // bytes from one group of 8 rows to the next
    uint32_t phase      = 0;
    bool ok             = true;
    bool first          = true;
    float my_loss = 0.f, my_db3 = 0.f;

    for (int32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const bool valid = (int64_t)tile * MLP_TILE + r < n;
        // ---- standardised features, four a thread; the fourth thread of a row: ones column and target ----
        if (part < 3u) {
            const float* mu = &S.mu[4u * part];
            const float* sd = &S.isd[4u * part];
            uint2 u         = make_uint2(0u, 0u);
            if (valid) {
                u = make_uint2(tc::pack_bf16((in.x - mu[0]) * sd[0], (in.y - mu[1]) * sd[1]),
                               tc::pack_bf16((in.z - mu[2]) * sd[2], (in.w - mu[3]) * sd[3]));
            }
            *reinterpret_cast<uint2*>(&S.ax[kmajor(r, AX_X + 4u * part, AX_N)]) = u;
        } else {
            *reinterpret_cast<uint2*>(&S.ax[kmajor(r, AX_ONES, AX_N)]) = make_uint2(valid ? bf16_bits(1.f) : 0u, 0u);
            S.tn[r] = valid ? (in.x - S.ymu) * S.iysd : 0.f;
        }
        if (tile < ntiles - (int32_t)gridDim.x) { fetch(tile + (int32_t)gridDim.x); }
        tc::fence_async_smem();
        __syncthreads();
        if (t == 0) {
            tc::fence_after();
            // the ones column meets a zero weight
            tc::mma(tm, tc::sdesc(tc::saddr(S.ax) + (AX_X / 8) * 128u, 128, AX_ROWS),
                    tc::sdesc(tc::saddr(S.w1), 128, MLP_FP * 16), ID64, 0u);
            tc::commit(&S.bar);
        }
        ok = tc::mbar_wait(&S.bar, phase) && ok;
        phase ^= 1u;
        tc::fence_after();
        // ---- hidden layer 1 ----
        uint32_t mask1 = 0u;
        {
            float z[16];
            tc::ld16(mine + c0, z);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const float v = z[c] + S.b1[c0 + c];
                mask1 |= v > 0.f ? 1u << c : 0u;
                z[c] = fmaxf(v, 0.f);
            }
            *reinterpret_cast<uint4*>(&S.ax[kmajor(r, c0, AX_N)])      = pack8(z, 0);
            *reinterpret_cast<uint4*>(&S.ax[kmajor(r, c0 + 8u, AX_N)]) = pack8(z, 1);
        }
        tc::fence_before();
        tc::fence_async_smem();
        __syncthreads();
        if (t == 0) {
            tc::fence_after();
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                tc::mma(tm + 64u, tc::sdesc(tc::saddr(S.ax) + 256u * k, 128, AX_ROWS),
                        tc::sdesc(tc::saddr(S.w2) + 256u * k, 128, MLP_H * 16), ID64, k > 0 ? 1u : 0u);
            }
            tc::commit(&S.bar);
        }
        ok = tc::mbar_wait(&S.bar, phase) && ok;
        phase ^= 1u;
        tc::fence_after();
        // ---- output, loss, dZ2 ----
        {
            float v[16];
            tc::ld16(mine + 64u + c0, v);
#pragma unroll
            for (int c = 0; c < 16; ++c) { v[c] += S.b2[c0 + c]; }
            // the output as one chain over the 64 columns, quarter by quarter (the inference kernels' order)
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) {
                if (part == k) {
                    float y = k == 0u ? S.b3 : S.y[r];
#pragma unroll
                    for (int c = 0; c < 16; ++c) { y = fmaf(fmaxf(v[c], 0.f), S.w3[c0 + c], y); }
                    S.y[r] = y;
                }
                __syncthreads();
            }
            const float y  = S.y[r];
            const float e  = valid ? y - S.tn[r] : 0.f;
            const float dy = 2.f * e * inv_n;
            if (part == 0u) {
                my_loss = fmaf(e, e, my_loss);
                my_db3 += dy;
            }
            float d[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                d[c] = v[c] > 0.f ? dy * S.w3[c0 + c] : 0.f;
                v[c] = dy * fmaxf(v[c], 0.f);
            }
            *reinterpret_cast<uint4*>(&S.dz[kmajor(r, c0, DZ_N)])      = pack8(d, 0);
            *reinterpret_cast<uint4*>(&S.dz[kmajor(r, c0 + 8u, DZ_N)]) = pack8(d, 1);
            const float sum = warp_sum16(v);
            if ((t & 1u) == 0u) { S.dw3q[quad][c0 + ((t & 31u) >> 1)] = sum; }
        }
        tc::fence_before();
        tc::fence_async_smem();
        __syncthreads();
        if (t == 0) {
            tc::fence_after();
#pragma unroll
            for (uint32_t k = 0; k < 4; ++k) {
                tc::mma(tm, tc::sdesc(tc::saddr(S.dz) + 256u * k, 128, DZ_ROWS),
                        tc::sdesc(tc::saddr(S.w2t) + 256u * k, 128, MLP_H * 16), ID64, k > 0 ? 1u : 0u);
            }
            tc::commit(&S.bar);
        }
        if (t >= 64u && t < 64u + MLP_H) { // while the product runs: one sum, 32 rows after 32 rows
            const uint32_t c = t - 64u;
            S.dw3[c] = (((S.dw3[c] + S.dw3q[0][c]) + S.dw3q[1][c]) + S.dw3q[2][c]) + S.dw3q[3][c];
        }
        ok = tc::mbar_wait(&S.bar, phase) && ok;
        phase ^= 1u;
        tc::fence_after();
        // ---- dZ1 ----
        {
            float z[16];
            tc::ld16(mine + c0, z);
#pragma unroll
            for (int c = 0; c < 16; ++c) { z[c] = ((mask1 >> c) & 1u) ? z[c] : 0.f; }
            *reinterpret_cast<uint4*>(&S.dz[kmajor(r, 64u + c0, DZ_N)])      = pack8(z, 0);
            *reinterpret_cast<uint4*>(&S.dz[kmajor(r, 64u + c0 + 8u, DZ_N)]) = pack8(z, 1);
        }
        tc::fence_before();
        tc::fence_async_smem();
        __syncthreads();
        if (t == 0) {
            tc::fence_after();
            // M- and N-major: the leading byte offset leads from 8 pairs to the next 8, the stride byte offset from 8
            // columns to the next 8; 16 pairs an instruction
#pragma unroll
            for (uint32_t k = 0; k < MLP_TILE / 16; ++k) {
                tc::mma(tm + 128u, tc::sdesc(tc::saddr(S.dz) + 2u * DZ_ROWS * k, DZ_ROWS, 128),
                        tc::sdesc(tc::saddr(S.ax) + 2u * AX_ROWS * k, AX_ROWS, 128), IDG, (first && k == 0) ? 0u : 1u);
            }
            tc::commit(&S.bar);
        }
        ok = tc::mbar_wait(&S.bar, phase) && ok; // the next tile overwrites the operands
        phase ^= 1u;
        tc::fence_after();
        first = false;
    }

    // ---- the CTA's sums into the global gradient ----
    if (part == 0u) {
        my_loss = warp_sum(my_loss);
        my_db3  = warp_sum(my_db3);
        if ((t & 31u) == 0u) {
            atomicAdd(&S.loss, my_loss);
            atomicAdd(&S.db3, my_db3);
        }
    }
    if (quad < 2u) { // rows 0-63: dW2, and db2 in the ones column
        float z[16];
        tc::ld16(mine + 128u + c0, z);
#pragma unroll
        for (int c = 0; c < 16; c += 4) {
            atomicAdd(reinterpret_cast<float4*>(&grad[MLP_OFF_W2 + r * MLP_H + c0 + c]),
                      make_float4(z[c], z[c + 1], z[c + 2], z[c + 3]));
        }
        if (part == 0u) {
            tc::ld16(mine + 128u + AX_X, z);
            atomicAdd(&grad[MLP_OFF_B2 + r], z[AX_ONES - AX_X]);
        }
    } else if (part == 0u) { // rows 64-127: dW1, db1
        float z[16];
        tc::ld16(mine + 128u + AX_X, z);
        const uint32_t i = r - 64u;
#pragma unroll
        for (int c = 0; c < MLP_F; c += 4) {
            atomicAdd(reinterpret_cast<float4*>(&grad[MLP_OFF_W1 + i * MLP_F + c]),
                      make_float4(z[c], z[c + 1], z[c + 2], z[c + 3]));
        }
        atomicAdd(&grad[MLP_OFF_B1 + i], z[AX_ONES - AX_X]);
    }
    tc::fence_before();
    __syncthreads();
    if (t < MLP_H) { atomicAdd(&grad[MLP_OFF_W3 + t], S.dw3[t]); }
    if (t == 0) {
        atomicAdd(&grad[MLP_OFF_B3], S.db3);
        atomicAdd(&grad[MLP_NW], S.loss);
    }
    if (!ok) { atomicOr(status, GPE_STATUS_TIMEOUT); }
    if (t < 32) {
        tc::fence_after();
        tc::tmem_dealloc(tm, TRAIN_TMEM_COLS);
    }
    // ---- the last CTA to get here applies the sum ----
    if (adam.net) {
        __threadfence();
        __syncthreads();
        if (t == 0) {
            S.last = atomicAdd(adam.done, 1u) == gridDim.x - 1u ? 1u : 0u;
            __threadfence();
        }
        __syncthreads();
        if (S.last) {
            adamw(adam, grad);
            if (t == 0) {
                grad[MLP_NW + 1] += __ldcg(&grad[MLP_NW]);
                grad[MLP_NW] = 0.f;
                *adam.done   = 0u;
            }
        }
    }
}

// Writes parameter p of the FP32 vector into the kernels' image (BF16 layouts and FP32 vectors).
__device__ __forceinline__ void put_param(MlpDev* m, int p, float w)
{
    if (p < MLP_OFF_B1) {
        const int i = p / MLP_F, f = p % MLP_F;
        m->w1[kmajor(i, f, MLP_FP)] = bf16_bits(w);
    } else if (p < MLP_OFF_W2) {
        m->b1[p - MLP_OFF_B1] = w;
    } else if (p < MLP_OFF_B2) {
        const int j = (p - MLP_OFF_W2) / MLP_H, i = (p - MLP_OFF_W2) % MLP_H;
        m->w2[kmajor(j, i, MLP_H)]  = bf16_bits(w);
        m->w2t[kmajor(i, j, MLP_H)] = bf16_bits(w);
    } else if (p < MLP_OFF_W3) {
        m->b2[p - MLP_OFF_B2] = w;
    } else if (p < MLP_OFF_B3) {
        m->w3[p - MLP_OFF_W3] = w;
    } else {
        m->b3 = w;
    }
}

__global__ void k_mlp_pack(MlpDev* __restrict__ m, const float* __restrict__ master)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < MLP_NW) { put_param(m, p, master[p]); }
}

// Sums of x, x^2 per feature and of t, t^2 over pairs [0, n) (FP64). Warp w of a block sums features 4w..4w+3 (the
// fourth the targets), 32 pairs at a time; one atomic per sum and block (with one per warp and sum on 26 addresses,
// 126 us for 472,000 pairs).
__global__ void __launch_bounds__(128) k_mlp_stats(const float* __restrict__ X, const float* __restrict__ T, int32_t n,
                                                   double* __restrict__ acc)
{
    const uint32_t w = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    double s[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0}; // four sums, four sums of squares
    for (int32_t i = (int32_t)(blockIdx.x * 32u + lane); i < n; i += (int32_t)(gridDim.x * 32u)) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (w < 3u) {
            v = __ldg(reinterpret_cast<const float4*>(X) + (size_t)i * (MLP_F / 4) + w);
        } else {
            v.x = __ldg(&T[i]);
        }
        const double a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            s[q] += a[q];
            s[4 + q] += a[q] * a[q];
            if (w == 3u) { break; }
        }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        double v = s[q];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) { v += __shfl_xor_sync(0xffffffffu, v, o); }
        if (lane == 0u && (w < 3u || (q & 3) == 0)) {
            const uint32_t at = w < 3u ? (q < 4 ? 4u * w + q : MLP_F + 4u * w + (q - 4)) : 2u * MLP_F + (q >> 2);
            atomicAdd(&acc[at], v);
        }
    }
}

// ----- the epoch's order ---------------------------------------------------------------------------------
// The Fisher-Yates shuffle of 0..n-1 driven by SplitMix64 (Steele, Lea & Flood 2014): for q = n-1 down to 1, swap places
// q and j_q = draw % (q + 1). Draw t of the generator is a function of its start and t, so every target j_q is known at
// once. Place q is final after swap q, and holds what lay at j_q just before it. Swap q puts at j_q what lay at q, so
// what lies at place p just before swap q was put there by the last swap before it with target p, the smallest r > q
// with j_r = p: it is what lay at place r just before swap r; or p itself where there is no such r. The same question
// asked again and again, now always for the smallest r of all, ends after about log n steps. So with the swaps sorted
// by target every place of the result is found independently: four short kernels (and a scan) instead of a walk
// over the host's memory, 2.6 ms of a 5.4 ms epoch of 472,000 pairs.
__device__ __forceinline__ uint64_t splitmix_at(uint64_t start, uint64_t t)
{
    uint64_t z = start + t * 0x9E3779B97F4A7C15ull;
    z          = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z          = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__global__ void k_shuffle_draw(uint64_t start, uint32_t n, uint32_t* __restrict__ target, uint32_t* __restrict__ rank,
                               uint32_t* __restrict__ count)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) { return; }
    const uint32_t j = q == 0u ? 0u : (uint32_t)(splitmix_at(start, (uint64_t)(n - q)) % (uint64_t)(q + 1u));
    target[q]        = j;
    if (j != q) { rank[q] = atomicAdd(&count[j], 1u); } // (a swap of a place with itself moves nothing)
}

__global__ void k_shuffle_place(uint32_t n, const uint32_t* __restrict__ target, const uint32_t* __restrict__ rank,
                                const uint32_t* __restrict__ start, uint32_t* __restrict__ swaps)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) { return; }
    const uint32_t j = target[q];
    if (j != q) { swaps[start[j] + rank[q]] = q; }
}

__global__ void k_shuffle_order(uint32_t n, const uint32_t* __restrict__ target, const uint32_t* __restrict__ start,
                                const uint32_t* __restrict__ swaps, int32_t* __restrict__ order)
{
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= n) { return; }
    uint32_t p = target[q], after = q; // what lies at p just before swap `after`
    for (;;) {
        uint32_t r = 0xffffffffu;
        for (uint32_t t = start[p]; t < start[p + 1u]; ++t) {
            const uint32_t s = swaps[t];
            if (s > after || p == after) { r = min(r, s); }
        }
        if (r == 0xffffffffu) { break; }
        p = after = r; // r > p: the walk ends
    }
    order[q] = (int32_t)p;
}

__global__ void __launch_bounds__(MLP_TILE)
    k_mlp_infer(const MlpDev* __restrict__ m, const float* __restrict__ X, float* __restrict__ out, int32_t n,
                uint32_t* __restrict__ status)
{
    __shared__ MlpFwdSmem S;
    const int32_t ntiles = (n + MLP_TILE - 1) / MLP_TILE;
    if ((int32_t)blockIdx.x >= ntiles) { return; }
    mlp_fwd_setup(S, m);
    const float ymu = m->ymu, ysd = m->ysd;
    uint32_t phase  = 0;
    bool ok         = true;
    for (int32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int32_t q  = tile * MLP_TILE + (int32_t)threadIdx.x;
        const bool valid = q < n;
        float f[MLP_F];
#pragma unroll
        for (int k = 0; k < MLP_F; ++k) { f[k] = valid ? __ldg(&X[(size_t)q * MLP_F + k]) : 0.f; }
        const float y = mlp_fwd_tile(S, f, phase, ok);
        if (valid) { out[q] = fmaf(y, ysd, ymu); }
    }
    if (!ok) { atomicOr(status, GPE_STATUS_TIMEOUT); }
    mlp_fwd_teardown(S);
}

// ----- host helpers -------------------------------------------------------------------------------------
uint64_t splitmix64(uint64_t& s)
{
    // SplitMix64 (Steele, Lea & Flood 2014)
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z          = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z          = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

double uniform01(uint64_t& s) { return (double)(splitmix64(s) >> 11) * (1.0 / 9007199254740992.0); }

int32_t upload_norm(gpe_mlp* m, cudaStream_t st)
{
    float mu[MLP_FP] = {0}, isd[MLP_FP] = {0};
    for (int f = 0; f < MLP_F; ++f) {
        mu[f]  = m->mu[f];
        isd[f] = m->sd[f] > 0.f ? 1.f / m->sd[f] : 0.f;
    }
    const float y[2] = {m->ymu, m->ysd};
    GPE_TRY_CUDA(cudaMemcpyAsync(m->dev->mu, mu, sizeof(mu), cudaMemcpyHostToDevice, st));
    GPE_TRY_CUDA(cudaMemcpyAsync(m->dev->isd, isd, sizeof(isd), cudaMemcpyHostToDevice, st));
    GPE_TRY_CUDA(cudaMemcpyAsync(&m->dev->ymu, y, sizeof(y), cudaMemcpyHostToDevice, st));
    GPE_TRY_CUDA(cudaStreamSynchronize(st));
    return GPE_OK;
}

int32_t read_status(gpe_mlp* m, cudaStream_t st)
{
    uint32_t v = 0;
    GPE_TRY_CUDA(cudaMemcpyAsync(&v, m->status, sizeof(v), cudaMemcpyDeviceToHost, st));
    GPE_TRY_CUDA(cudaStreamSynchronize(st));
    if (v) {
        GPE_TRY_CUDA(cudaMemsetAsync(m->status, 0, sizeof(uint32_t), st));
        if (v & GPE_STATUS_TIMEOUT) {
            gpe::set_error(GPE_ERR_TIMEOUT, "a tensor-core wait of the network kernels gave up");
            return GPE_ERR_TIMEOUT;
        }
    }
    return GPE_OK;
}

int32_t pair_count(const gpe_mlp* m, cudaStream_t st, int64_t* n)
{
    int32_t c[2] = {0, 0};
    GPE_TRY_CUDA(cudaMemcpyAsync(c, m->cnt, sizeof(c), cudaMemcpyDeviceToHost, st));
    GPE_TRY_CUDA(cudaStreamSynchronize(st));
    *n = std::min<int64_t>(c[1], m->cap);
    return GPE_OK;
}

int train_grid(int32_t n) { return std::max(1, std::min((n + MLP_TILE - 1) / MLP_TILE, gpe::sm_count())); }

size_t train_smem() { return sizeof(MlpTrainSmem) + 128; }

// m->order = the shuffle of 0..n-1 (n >= 1) from the generator's state rs
int32_t shuffle_order(gpe_mlp* m, uint32_t n, uint64_t rs, cudaStream_t st)
{
    const unsigned g = (n + 255u) / 256u;
    k_shuffle_draw<<<g, 256, 0, st>>>(rs, n, m->sh_target, m->sh_rank, m->sh_count);
    GPE_CHECK_LAUNCH("k_shuffle_draw");
    const int32_t rc = launch_exclusive_scan(m->sh_count, n, m->sh_bsum, m->sh_start, {st, false});
    if (rc) { return rc; }
    k_shuffle_place<<<g, 256, 0, st>>>(n, m->sh_target, m->sh_rank, m->sh_start, m->sh_swaps);
    GPE_CHECK_LAUNCH("k_shuffle_place");
    k_shuffle_order<<<g, 256, 0, st>>>(n, m->sh_target, m->sh_start, m->sh_swaps, m->order);
    GPE_CHECK_LAUNCH("k_shuffle_order");
    return GPE_OK;
}

} // namespace
} // namespace gpe

using namespace gpe;

extern "C" {

int32_t gpe_mlp_create(int64_t max_pairs, uint64_t seed, gpe_mlp** out)
{
    gpe::clear_error();
    if (!out || max_pairs < 0 || max_pairs > (int64_t)INT32_MAX / 2) { return GPE_ERR_BAD_ARG; }
    *out    = nullptr;
    int dev = 0;
    int32_t rc = gpe::current_device(&dev);
    if (rc) { return rc; }
    gpe_mlp* m = new gpe_mlp();
    m->device  = dev;
    m->cap     = max_pairs;
    const size_t P = (size_t)std::max<int64_t>(max_pairs, 1);
    Carver c;
    const size_t o_dev  = c.take<MlpDev>(1);
    const size_t o_mas  = c.take<float>(MLP_NW);
    const size_t o_grad = c.take<float>(MLP_NW + 8);
    const size_t o_am   = c.take<float>(MLP_NW);
    const size_t o_av   = c.take<float>(MLP_NW);
    const size_t o_st   = c.take<double>(64);
    const size_t o_stat = c.take<uint32_t>(4);
    const size_t o_cnt  = c.take<int32_t>(4);
    const size_t o_X    = c.take<float>(P * MLP_F);
    const size_t o_T    = c.take<float>(P);
    const size_t o_idx  = c.take<int32_t>(P);
    const size_t o_ord  = c.take<int32_t>(P);
    const size_t o_sht  = c.take<uint32_t>(P);
    const size_t o_shr  = c.take<uint32_t>(P);
    const size_t o_shc  = c.take<uint32_t>(P);
    const size_t o_shs  = c.take<uint32_t>(P + 1);
    const size_t o_shw  = c.take<uint32_t>(P);
    const size_t o_shb  = c.take<uint32_t>(scan_blocks((uint32_t)P) + 1);
    const size_t o_done = c.take<uint32_t>(1);
    cudaError_t e       = cudaMalloc(&m->base, c.off);
    if (e == cudaSuccess) { e = cudaMemset(m->base, 0, c.off); }
    if (e == cudaSuccess) {
        e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)train_smem());
    }
    if (e != cudaSuccess) {
        gpe::set_cuda_error(e, "gpe_mlp_create");
        if (m->base) { cudaFree(m->base); }
        delete m;
        return GPE_ERR_CUDA;
    }
    uint8_t* b  = static_cast<uint8_t*>(m->base);
    m->dev      = reinterpret_cast<MlpDev*>(b + o_dev);
    m->master   = reinterpret_cast<float*>(b + o_mas);
    m->grad     = reinterpret_cast<float*>(b + o_grad);
    m->adam_m   = reinterpret_cast<float*>(b + o_am);
    m->adam_v   = reinterpret_cast<float*>(b + o_av);
    m->stats    = reinterpret_cast<double*>(b + o_st);
    m->status   = reinterpret_cast<uint32_t*>(b + o_stat);
    m->cnt      = reinterpret_cast<int32_t*>(b + o_cnt);
    m->X        = reinterpret_cast<float*>(b + o_X);
    m->T        = reinterpret_cast<float*>(b + o_T);
    m->idx      = reinterpret_cast<int32_t*>(b + o_idx);
    m->order    = reinterpret_cast<int32_t*>(b + o_ord);
    m->sh_target = reinterpret_cast<uint32_t*>(b + o_sht);
    m->sh_rank   = reinterpret_cast<uint32_t*>(b + o_shr);
    m->sh_count  = reinterpret_cast<uint32_t*>(b + o_shc);
    m->sh_start  = reinterpret_cast<uint32_t*>(b + o_shs);
    m->sh_swaps  = reinterpret_cast<uint32_t*>(b + o_shw);
    m->sh_bsum   = reinterpret_cast<uint32_t*>(b + o_shb);
    m->done      = reinterpret_cast<uint32_t*>(b + o_done);
    // uniform He initialisation (He et al. 2015): U(-sqrt(6/fan_in), sqrt(6/fan_in)); the output layer
    // starts small so that an untrained network stays close to the previous-step warm start
    std::vector<float> w(MLP_NW, 0.f);
    uint64_t s = seed ^ 0x6A09E667F3BCC909ull;
    const double a1 = std::sqrt(6.0 / MLP_F), a2 = std::sqrt(6.0 / MLP_H), a3 = 0.1 * std::sqrt(6.0 / MLP_H);
    for (int p = MLP_OFF_W1; p < MLP_OFF_B1; ++p) { w[p] = (float)((2.0 * uniform01(s) - 1.0) * a1); }
    for (int p = MLP_OFF_W2; p < MLP_OFF_B2; ++p) { w[p] = (float)((2.0 * uniform01(s) - 1.0) * a2); }
    for (int p = MLP_OFF_W3; p < MLP_OFF_B3; ++p) { w[p] = (float)((2.0 * uniform01(s) - 1.0) * a3); }
    for (int f = 0; f < MLP_F; ++f) {
        m->mu[f] = 0.f;
        m->sd[f] = 1.f;
    }
    m->ymu = 0.f;
    m->ysd = 1.f;
    *out   = m;
    float blob[GPE_MLP_BLOB_FLOATS];
    std::memcpy(blob, w.data(), sizeof(float) * MLP_NW);
    for (int f = 0; f < MLP_F; ++f) {
        blob[MLP_NW + f]         = 0.f;
        blob[MLP_NW + MLP_F + f] = 1.f;
    }
    blob[MLP_NW + 2 * MLP_F]     = 0.f;
    blob[MLP_NW + 2 * MLP_F + 1] = 1.f;
    rc = gpe_mlp_set_blob(m, blob, GPE_MLP_BLOB_FLOATS);
    if (rc) {
        gpe_mlp_destroy(m);
        *out = nullptr;
    }
    return rc;
}

int32_t gpe_mlp_destroy(gpe_mlp* m)
{
    if (!m) { return GPE_ERR_BAD_ARG; }
    if (m->base) { cudaFree(m->base); }
    delete m;
    return GPE_OK;
}

int32_t gpe_mlp_get_blob(const gpe_mlp* m, float* blob, int64_t n)
{
    gpe::clear_error();
    if (!m || !blob || n != GPE_MLP_BLOB_FLOATS) { return GPE_ERR_BAD_ARG; }
    GPE_TRY_CUDA(cudaMemcpy(blob, m->master, sizeof(float) * MLP_NW, cudaMemcpyDeviceToHost));
    for (int f = 0; f < MLP_F; ++f) {
        blob[MLP_NW + f]         = m->mu[f];
        blob[MLP_NW + MLP_F + f] = m->sd[f];
    }
    blob[MLP_NW + 2 * MLP_F]     = m->ymu;
    blob[MLP_NW + 2 * MLP_F + 1] = m->ysd;
    return GPE_OK;
}

int32_t gpe_mlp_set_blob(gpe_mlp* m, const float* blob, int64_t n)
{
    gpe::clear_error();
    if (!m || !blob || n != GPE_MLP_BLOB_FLOATS) { return GPE_ERR_BAD_ARG; }
    for (int64_t q = 0; q < n; ++q) {
        if (!std::isfinite(blob[q])) {
            gpe::set_error(GPE_ERR_BAD_ARG, "gpe_mlp_set_blob: entry %lld is not finite", (long long)q);
            return GPE_ERR_BAD_ARG;
        }
    }
    for (int f = 0; f < MLP_F; ++f) {
        m->mu[f] = blob[MLP_NW + f];
        m->sd[f] = blob[MLP_NW + MLP_F + f];
    }
    m->ymu = blob[MLP_NW + 2 * MLP_F];
    m->ysd = blob[MLP_NW + 2 * MLP_F + 1];
    GPE_TRY_CUDA(cudaMemcpy(m->master, blob, sizeof(float) * MLP_NW, cudaMemcpyHostToDevice));
    GPE_TRY_CUDA(cudaMemset(m->adam_m, 0, sizeof(float) * MLP_NW));
    GPE_TRY_CUDA(cudaMemset(m->adam_v, 0, sizeof(float) * MLP_NW));
    m->adam_t = 0;
    k_mlp_pack<<<(MLP_NW + 255) / 256, 256>>>(m->dev, m->master);
    GPE_CHECK_LAUNCH("k_mlp_pack");
    int32_t rc = upload_norm(m, nullptr);
    if (rc) { return rc; }
    GPE_TRY_CUDA(cudaDeviceSynchronize());
    return GPE_OK;
}

int32_t gpe_mlp_num_pairs(const gpe_mlp* m, int64_t* n)
{
    if (!m || !n) { return GPE_ERR_BAD_ARG; }
    return pair_count(m, nullptr, n);
}

int32_t gpe_mlp_get_pairs(const gpe_mlp* m, float* features, float* targets, int32_t* index, int64_t n,
                          int32_t mem, void* stream)
{
    gpe::clear_error();
    if (!m || (mem != GPE_MEM_HOST && mem != GPE_MEM_DEVICE)) { return GPE_ERR_BAD_ARG; }
    cudaStream_t st = as_stream(stream);
    int64_t have    = 0;
    int32_t rc      = pair_count(m, st, &have);
    if (rc) { return rc; }
    if (n != have) {
        gpe::set_error(GPE_ERR_BAD_ARG, "gpe_mlp_get_pairs: n must equal the pair count (%lld)", (long long)have);
        return GPE_ERR_BAD_ARG;
    }
    const cudaMemcpyKind k = mem == GPE_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    if (n > 0) {
        if (features) { GPE_TRY_CUDA(cudaMemcpyAsync(features, m->X, sizeof(float) * MLP_F * (size_t)n, k, st)); }
        if (targets) { GPE_TRY_CUDA(cudaMemcpyAsync(targets, m->T, sizeof(float) * (size_t)n, k, st)); }
        if (index) { GPE_TRY_CUDA(cudaMemcpyAsync(index, m->idx, sizeof(int32_t) * (size_t)n, k, st)); }
    }
    GPE_TRY_CUDA(cudaStreamSynchronize(st));
    return GPE_OK;
}

int32_t gpe_mlp_set_pairs(gpe_mlp* m, const float* features, const float* targets, int64_t n, int32_t mem,
                          void* stream)
{
    gpe::clear_error();
    if (!m || n < 0 || (n > 0 && (!features || !targets)) || (mem != GPE_MEM_HOST && mem != GPE_MEM_DEVICE)) {
        return GPE_ERR_BAD_ARG;
    }
    if (n > m->cap) {
        gpe::set_error(GPE_ERR_CAPACITY, "gpe_mlp_set_pairs: %lld pairs exceed the capacity %lld", (long long)n,
                       (long long)m->cap);
        return GPE_ERR_CAPACITY;
    }
    cudaStream_t st        = as_stream(stream);
    const cudaMemcpyKind k = mem == GPE_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    if (n > 0) {
        GPE_TRY_CUDA(cudaMemcpyAsync(m->X, features, sizeof(float) * MLP_F * (size_t)n, k, st));
        GPE_TRY_CUDA(cudaMemcpyAsync(m->T, targets, sizeof(float) * (size_t)n, k, st));
        GPE_TRY_CUDA(cudaMemsetAsync(m->idx, 0xff, sizeof(int32_t) * (size_t)n, st));
    }
    const int32_t c[2] = {(int32_t)n, (int32_t)n};
    GPE_TRY_CUDA(cudaMemcpyAsync(m->cnt, c, sizeof(c), cudaMemcpyHostToDevice, st));
    GPE_TRY_CUDA(cudaStreamSynchronize(st));
    return GPE_OK;
}

int32_t gpe_mlp_train(gpe_mlp* m, const gpe_mlp_train_params* tp, float* train_loss, float* val_loss, void* stream)
{
    gpe::clear_error();
    if (!m || !tp || tp->epochs < 0 || tp->batch <= 0 || !(tp->lr >= 0.f) || !(tp->val_fraction >= 0.f) ||
        !(tp->val_fraction < 1.f) || !(tp->beta1 >= 0.f && tp->beta1 < 1.f) || !(tp->beta2 >= 0.f && tp->beta2 < 1.f) ||
        tp->lr_schedule < 0 || tp->lr_schedule > 1) {
        return GPE_ERR_BAD_ARG;
    }
    cudaStream_t st = as_stream(stream);
    int64_t n       = 0;
    int32_t rc      = pair_count(m, st, &n);
    if (rc) { return rc; }
    const int64_t n_val   = (int64_t)std::floor((double)n * tp->val_fraction);
    const int64_t n_train = n - n_val;
    if (n_train <= 0) {
        gpe::set_error(GPE_ERR_NOT_READY, "gpe_mlp_train: no training pairs");
        return GPE_ERR_NOT_READY;
    }
    // standardisation from the training pairs
    GPE_TRY_CUDA(cudaMemsetAsync(m->stats, 0, sizeof(double) * 64, st));
    k_mlp_stats<<<std::min<int64_t>((n_train + 31) / 32, 4 * gpe::sm_count()), 128, 0, st>>>(m->X, m->T,
                                                                                         (int32_t)n_train, m->stats);
    GPE_CHECK_LAUNCH("k_mlp_stats");
    double acc[2 * MLP_F + 2];
    GPE_TRY_CUDA(cudaMemcpyAsync(acc, m->stats, sizeof(acc), cudaMemcpyDeviceToHost, st));
    GPE_TRY_CUDA(cudaStreamSynchronize(st));
    const double nn = (double)n_train;
    for (int f = 0; f < MLP_F; ++f) {
        const double mu = acc[f] / nn;
        const double va = std::max(acc[MLP_F + f] / nn - mu * mu, 0.0);
        const double sd = std::sqrt(va);
        m->mu[f]        = (float)mu;
        m->sd[f]        = sd > 1e-12 * std::max(1.0, std::fabs(mu)) ? (float)sd : 0.f;
    }
    {
        const double mu = acc[2 * MLP_F] / nn;
        const double sd = std::sqrt(std::max(acc[2 * MLP_F + 1] / nn - mu * mu, 0.0));
        m->ymu          = (float)mu;
        m->ysd          = sd > 0.0 ? (float)sd : 1.f;
    }
    rc = upload_norm(m, st);
    if (rc) { return rc; }
    GPE_TRY_CUDA(cudaMemsetAsync(m->grad, 0, sizeof(float) * (MLP_NW + 8), st));
    // epochs
    uint64_t rs      = tp->seed ^ 0xBB67AE8584CAA73Bull;
    const int32_t B  = tp->batch;
    float last_epoch = 0.f;
    const double steps_total = (double)tp->epochs * (double)((n_train + B - 1) / B);
    int64_t step             = 0;
    for (int32_t ep = 0; ep < tp->epochs; ++ep) {
        rc = shuffle_order(m, (uint32_t)n_train, rs, st);
        if (rc) { return rc; }
        rs += (uint64_t)(n_train - 1) * 0x9E3779B97F4A7C15ull; // the generator after the epoch's draws
        GPE_TRY_CUDA(cudaMemsetAsync(m->grad + MLP_NW + 1, 0, sizeof(float), st));
        for (int64_t b0 = 0; b0 < n_train; b0 += B) {
            const int32_t nb = (int32_t)std::min<int64_t>(B, n_train - b0);
            ++m->adam_t;
            const float bc1 = 1.f - (float)std::pow((double)tp->beta1, (double)m->adam_t);
            const float bc2 = 1.f - (float)std::pow((double)tp->beta2, (double)m->adam_t);
            const float lr = tp->lr_schedule == 1
                                 ? (float)(0.5 * (double)tp->lr *
                                           (1.0 + std::cos(3.141592653589793 * (double)step / steps_total)))
                                 : tp->lr;
            ++step;
            const AdamW adam{m->dev, m->master, m->adam_m, m->adam_v, m->done, lr, tp->weight_decay, tp->beta1,
                             tp->beta2, tp->adam_eps, bc1, bc2};
            k_mlp_train<<<train_grid(nb), TRAIN_T, train_smem(), st>>>(m->dev, m->X, m->T, m->order + b0, nb,
                                                                      1.f / (float)nb, m->grad, m->status, adam);
            GPE_CHECK_LAUNCH("k_mlp_train");
            if (m->adam_t == 1) {
                rc = read_status(m, st); // a first step that timed out stops the run at once
                if (rc) { return rc; }
            }
        }
        float el = 0.f;
        GPE_TRY_CUDA(cudaMemcpyAsync(&el, m->grad + MLP_NW + 1, sizeof(float), cudaMemcpyDeviceToHost, st));
        GPE_TRY_CUDA(cudaStreamSynchronize(st));
        last_epoch = el / (float)n_train;
        rc         = read_status(m, st);
        if (rc) { return rc; }
    }
    if (train_loss) { *train_loss = last_epoch; }
    if (val_loss) {
        float vl = 0.f;
        if (n_val > 0) {
            GPE_TRY_CUDA(cudaMemsetAsync(m->grad, 0, sizeof(float) * (MLP_NW + 8), st));
            k_mlp_train<<<train_grid((int32_t)n_val), TRAIN_T, train_smem(), st>>>(
                m->dev, m->X + (size_t)n_train * MLP_F, m->T + n_train, nullptr, (int32_t)n_val, 1.f / (float)n_val,
                m->grad, m->status, AdamW{});
            GPE_CHECK_LAUNCH("k_mlp_train");
            GPE_TRY_CUDA(cudaMemcpyAsync(&vl, m->grad + MLP_NW, sizeof(float), cudaMemcpyDeviceToHost, st));
            GPE_TRY_CUDA(cudaMemsetAsync(m->grad, 0, sizeof(float) * (MLP_NW + 8), st));
            GPE_TRY_CUDA(cudaStreamSynchronize(st));
            vl /= (float)n_val;
        }
        *val_loss = vl;
    }
    return read_status(m, st);
}

int32_t gpe_mlp_infer(const gpe_mlp* m, const float* features, float* out, int64_t n, int32_t mem, void* stream)
{
    gpe::clear_error();
    if (!m || n < 0 || (n > 0 && (!features || !out)) || (mem != GPE_MEM_HOST && mem != GPE_MEM_DEVICE) ||
        n > (int64_t)INT32_MAX / MLP_F) {
        return GPE_ERR_BAD_ARG;
    }
    if (n == 0) { return GPE_OK; }
    cudaStream_t st = as_stream(stream);
    const float* dX = features;
    float* dY       = out;
    void* tmp       = nullptr;
    if (mem == GPE_MEM_HOST) {
        GPE_TRY_CUDA(cudaMalloc(&tmp, sizeof(float) * (size_t)n * (MLP_F + 1)));
        dX = static_cast<float*>(tmp);
        dY = static_cast<float*>(tmp) + (size_t)n * MLP_F;
        cudaError_t e = cudaMemcpyAsync(const_cast<float*>(dX), features, sizeof(float) * (size_t)n * MLP_F,
                                        cudaMemcpyHostToDevice, st);
        if (e != cudaSuccess) {
            cudaFree(tmp);
            gpe::set_cuda_error(e, "gpe_mlp_infer");
            return GPE_ERR_CUDA;
        }
    }
    const int32_t ntiles = (int32_t)((n + MLP_TILE - 1) / MLP_TILE);
    k_mlp_infer<<<std::min(ntiles, 6 * gpe::sm_count()), MLP_TILE, 0, st>>>(m->dev, dX, dY, (int32_t)n, m->status);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess && mem == GPE_MEM_HOST) {
        e = cudaMemcpyAsync(out, dY, sizeof(float) * (size_t)n, cudaMemcpyDeviceToHost, st);
    }
    if (e == cudaSuccess) { e = cudaStreamSynchronize(st); }
    if (tmp) { cudaFree(tmp); }
    if (e != cudaSuccess) {
        gpe::set_cuda_error(e, "gpe_mlp_infer");
        return GPE_ERR_CUDA;
    }
    return read_status(const_cast<gpe_mlp*>(m), st);
}

int32_t gpe_mlp_gradient(gpe_mlp* m, const float* features, const float* targets, int64_t n, float* grad,
                         float* loss, int32_t mem, void* stream)
{
    gpe::clear_error();
    if (!m || n <= 0 || !features || !targets || !grad || (mem != GPE_MEM_HOST && mem != GPE_MEM_DEVICE) ||
        n > (int64_t)INT32_MAX / MLP_F) {
        return GPE_ERR_BAD_ARG;
    }
    cudaStream_t st = as_stream(stream);
    void* tmp       = nullptr;
    constexpr size_t G = (MLP_NW + 8 + 3) / 4 * 4; // features and gradient start on 16-byte boundaries
    GPE_TRY_CUDA(cudaMalloc(&tmp, sizeof(float) * (G + (size_t)n * (MLP_F + 1))));
    float* dG = static_cast<float*>(tmp);
    float* dX = dG + G;
    float* dT = dX + (size_t)n * MLP_F;
    const cudaMemcpyKind k = mem == GPE_MEM_HOST ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToDevice;
    cudaError_t e          = cudaMemcpyAsync(dX, features, sizeof(float) * (size_t)n * MLP_F, k, st);
    if (e == cudaSuccess) { e = cudaMemcpyAsync(dT, targets, sizeof(float) * (size_t)n, k, st); }
    if (e == cudaSuccess) { e = cudaMemsetAsync(dG, 0, sizeof(float) * (MLP_NW + 8), st); }
    if (e == cudaSuccess) {
        k_mlp_train<<<train_grid((int32_t)n), TRAIN_T, train_smem(), st>>>(m->dev, dX, dT, nullptr, (int32_t)n,
                                                                          1.f / (float)n, dG, m->status, AdamW{});
        e = cudaGetLastError();
    }
    const cudaMemcpyKind ko = mem == GPE_MEM_HOST ? cudaMemcpyDeviceToHost : cudaMemcpyDeviceToDevice;
    if (e == cudaSuccess) { e = cudaMemcpyAsync(grad, dG, sizeof(float) * MLP_NW, ko, st); }
    float l = 0.f;
    if (e == cudaSuccess) { e = cudaMemcpyAsync(&l, dG + MLP_NW, sizeof(float), cudaMemcpyDeviceToHost, st); }
    if (e == cudaSuccess) { e = cudaStreamSynchronize(st); }
    cudaFree(tmp);
    if (e != cudaSuccess) {
        gpe::set_cuda_error(e, "gpe_mlp_gradient");
        return GPE_ERR_CUDA;
    }
    if (loss) { *loss = l / (float)n; }
    return read_status(m, st);
}

} // extern "C"
