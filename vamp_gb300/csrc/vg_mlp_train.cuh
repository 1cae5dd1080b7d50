// One training step of the learned order's network in two kernels (included by vg_mlp.cu).
//
//   mlp_rows_kernel     a CTA per 128 rows: features, both layers, head, loss, and the gradient
//                       back to the first layer's activations, with the activations in shared
//                       memory throughout.  It leaves the operands of the weight gradients
//                       (features, H1, H2, dH2, dH1) transposed, in the core-matrix layout the
//                       tensor core reads.
//   mlp_weights_kernel  dW2 in 2 x 8 tiles of 128 x 32 and dW1 in 2, each a chain over all rows
//                       (bulk copies into a ring of stages), the bias and head gradients as
//                       fixed-order column sums, and Adam on the spot.
//
// What bounds a step is latency: 0.9 GFLOP at 1,024 rows are 0.5 us of tensor time, but layer 1,
// layer 2, the head and the way back wait for one another, and dW2 is a chain of K = rows.  As
// 19 launches of general kernels (8 CTAs or fewer each, operands staged by plain loads) a step of
// 1,024 rows took 456 us; now 27 (rows 14, weights 9, the rest the hand-over between them).  Every
// rounding point and every order of accumulation is that of those
// launches (K in steps of 16, lane-strided head sums, 32-phase column sums), so the
// trained weights are the same bits.
#pragma once

#include <cuda_bf16.h>

#include "vg_tc.cuh"

namespace vg
{
    constexpr int kTrainThreads = 512;
    // bytes of one 128-row tile of a 256-wide operand, transposed: 32 column groups x 16 row groups
    // x 128-byte core matrices
    constexpr int kTileT = 128 * kHidden * 2;

    // Buffers of the step, one tile after another: xt kin x 128, the others kTileT each.
    struct StepBuffers
    {
        unsigned char *xt, *h1t, *h2t, *dh2t, *dh1t;
        float *dz;  // [rows]
    };

    // W1 [256][kin], W2 [256][256] and W2^T as the tensor core reads them (tc::tile_offset), for
    // bulk copies into shared memory.
    struct CoreWeights
    {
        unsigned char *w1, *w2, *w2t;
    };

    struct RowsParams
    {
        const float *q;        // [n][dim]
        const uint8_t *valid;  // [n]
        int n, dim, kin;
        const unsigned char *w1, *w2, *w2t;  // BF16 weights in core-matrix layout (CoreWeights)
        const float *b1, *b2, *w3, *b3;
        StepBuffers out;
        __nv_bfloat16 *x;  // [rows][kin] features, row-major (null: not wanted)
        float *loss;
        int *err;
        uint32_t wait_limit;
    };

    inline size_t rows_smem_bytes()
    {
        return kHidden * kHidden * 2 + 128 * kHidden * 2 + 3 * kHidden * 4;
    }

    // The 8 x 8 core matrices of row group `rg` (rows 8 rg .. 8 rg + 7) of a shared-memory tile of
    // kc columns, transposed (ldmatrix.trans) to a global tile: column group major, 16 row groups
    // each.  One warp; 128 bytes per store.
    __device__ __forceinline__ void store_transposed(const unsigned char *tile, int kc, int rg, unsigned char *out)
    {
        const int lane = threadIdx.x & 31;
        const int groups = kc >> 3;
        for (int c0 = 0; c0 < groups; c0 += 4)
        {
            // lanes 8 i .. 8 i + 7 give the rows of matrix i (the last ones again past the end)
            const int c = min(c0 + (lane >> 3), groups - 1);
            uint32_t r[4];
            tc::ldmatrix_x4_trans(tile + (rg * groups + c) * 128 + (lane & 7) * 16, r);
#pragma unroll
            for (int i = 0; i < 4; ++i)
            {
                if (c0 + i < groups)
                    *reinterpret_cast<uint32_t *>(out + ((c0 + i) * 16 + rg) * 128 + 4 * lane) = r[i];
            }
        }
    }

    __global__ void __launch_bounds__(kTrainThreads, 1) mlp_rows_kernel(const RowsParams p)
    {
        extern __shared__ __align__(1024) unsigned char rows_smem[];
        __shared__ uint64_t bar, wbar[2];  // MMAs; W1, then W2 and W2^T
        __shared__ uint32_t tmem_slot;
        __shared__ int skip;
        unsigned char *sw2 = rows_smem;                   // W2, later W2^T: 256 x 256
        unsigned char *sh = sw2 + kHidden * kHidden * 2;  // the activations: 128 x 256
        unsigned char *sx = sh;                           // features and W1 until layer 1 is done
        unsigned char *sw1 = sx + 128 * p.kin * 2;
        float *sb1 = reinterpret_cast<float *>(sh + 128 * kHidden * 2);
        float *sb2 = sb1 + kHidden;
        float *sw3 = sb2 + kHidden;
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        const int row0 = blockIdx.x * 128;
        if (warp == 0)
            tc::tmem_alloc(&tmem_slot, 512);
        if (tid == 0)
        {
            tc::mbar_init(&bar, 1);
            tc::mbar_init(&wbar[0], 1);
            tc::mbar_init(&wbar[1], 1);
        }
        const int kin = p.kin;
        // nothing is read or written before this: the inputs may be the kernel before's outputs, and
        // the step before writes the weights and reads the buffers that this one writes
        tc::wait_previous_kernel();
        tc::start_next_kernel();
        if (tid == 0)
            skip = *static_cast<volatile int *>(p.err);
        // The weights come whole, by bulk copies (16-byte copies by the threads, 16 each, cost 6,400
        // cycles a matrix); W2 lands while layer 1 runs.
        auto load_weights = [&](unsigned char *dst, const unsigned char *src, uint32_t bytes, uint64_t *b) {
            tc::mbar_expect(b, bytes);
            tc::bulk_load(dst, src, bytes, b);
        };
        constexpr uint32_t kW2 = kHidden * kHidden * 2;
        const uint32_t w1_bytes = static_cast<uint32_t>(kHidden * kin) * 2u;
        if (tid == 0)
        {
            load_weights(sw1, p.w1, w1_bytes, &wbar[0]);
            load_weights(sw2, p.w2, kW2, &wbar[1]);
        }
        for (int j = tid; j < kHidden; j += kTrainThreads)
        {
            sb1[j] = p.b1[j];
            sb2[j] = p.b2[j];
            sw3[j] = p.w3[j];
        }
        // features: sin and cos of each joint, zeros in the padding and past row n
        for (int u = tid; u < 128 * (kin / 2); u += kTrainThreads)
        {
            const int r = u & 127, d = u >> 7;
            __nv_bfloat162 f = __floats2bfloat162_rn(0.0f, 0.0f);
            if (row0 + r < p.n && d < p.dim)
            {
                const float a = p.q[static_cast<size_t>(row0 + r) * p.dim + d];
                f = __floats2bfloat162_rn(sinf(a), cosf(a));
            }
            *reinterpret_cast<__nv_bfloat162 *>(sx + tc::tile_offset(r, 2 * d, kin)) = f;
            if (p.x)
                *reinterpret_cast<__nv_bfloat162 *>(p.x + static_cast<size_t>(row0 + r) * kin + 2 * d) = f;
        }
        tc::fence_smem_to_async();
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        const uint32_t tmem = tmem_slot;
        const uint32_t idesc = tc::idesc_bf16_f32(128, kHidden);
        uint32_t phase = 0;
        bool pending = false;
        // thread 0 waits for B's copy (its barrier's phase `ph`), then issues the MMAs; if the copy does
        // not come in time nothing is committed, and the wait for the MMAs gives up in turn
        auto issue = [&](const unsigned char *a, const unsigned char *b, int kc, uint32_t acc, uint64_t *wb, uint32_t ph) {
            if (tid == 0 && tc::mbar_wait(wb, ph, kWaitLimit))
            {
                tc::fence_after_sync();
                const uint32_t a0 = tc::smem_u32(a), b0 = tc::smem_u32(b), sbo = static_cast<uint32_t>(kc / 8) * 128u;
                for (int kk = 0; kk < kc / 16; ++kk)
                    tc::mma_bf16(tmem + acc, tc::smem_desc(a0 + kk * 256, 128, sbo), tc::smem_desc(b0 + kk * 256, 128, sbo), idesc,
                                 kk > 0);
                tc::mma_commit(&bar);
                pending = true;
            }
        };
        // bounded wait for the MMAs committed last; every thread takes the same decision
        auto finished = [&]() {
            const bool ok = __syncthreads_and(tc::mbar_wait(&bar, phase, p.wait_limit)) != 0;
            if (ok)
            {
                phase ^= 1u;
                pending = false;
                tc::fence_after_sync();
            }
            return ok;
        };
        // epilogue threads: warp w reads TMEM lane quarter w % 4 and columns 64 (w / 4) ..
        const int erow = 32 * (warp & 3) + lane, c_lo = 64 * (warp >> 2);
        const uint32_t lanes = tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16);
        auto publish = [&]() {
            tc::fence_smem_to_async();
            tc::fence_before_sync();
            __syncthreads();
        };
        // activations bf16(max(D + bias, 0)) of this thread's row and columns; the bits that are > 0
        auto activate = [&](uint32_t acc, const float *bias) {
            unsigned long long positive = 0ull;
#pragma unroll 1
            for (int c0 = c_lo; c0 < c_lo + 64; c0 += 32)
            {
                float v[32];
                tc::tmem_load32(lanes + acc + static_cast<uint32_t>(c0), v);
                uint32_t bits = 0u;
#pragma unroll
                for (int j = 0; j < 32; j += 8)
                {
                    __align__(16) __nv_bfloat162 h[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                    {
                        h[k] = __floats2bfloat162_rn(fmaxf(__fadd_rn(v[j + 2 * k], bias[c0 + j + 2 * k]), 0.0f),
                                                     fmaxf(__fadd_rn(v[j + 2 * k + 1], bias[c0 + j + 2 * k + 1]), 0.0f));
                        const uint32_t w = *reinterpret_cast<const uint32_t *>(&h[k]);
                        bits |= (w & 0x7fffu ? 1u : 0u) << (j + 2 * k) | (w & 0x7fff0000u ? 1u : 0u) << (j + 2 * k + 1);
                    }
                    *reinterpret_cast<uint4 *>(sh + tc::tile_offset(erow, c0 + j, kHidden)) = *reinterpret_cast<const uint4 *>(h);
                }
                positive |= static_cast<unsigned long long>(bits) << (c0 - c_lo);
            }
            return positive;
        };
        auto tile_of = [&](unsigned char *base, int bytes) { return base + static_cast<size_t>(blockIdx.x) * bytes; };

        bool ok = true, w2t_coming = false;
        do
        {
            if (skip)  // an earlier kernel gave up
                break;
            // layer 1, the transposed features meanwhile
            issue(sx, sw1, kin, 0, &wbar[0], 0);
            if (warp < 16)
                store_transposed(sx, kin, warp, tile_of(p.out.xt, 128 * kin * 2));
            if (!(ok = finished()))
                break;
            const unsigned long long h1_positive = activate(0, sb1);
            publish();
            // layer 2
            issue(sh, sw2, kHidden, kHidden, &wbar[1], 0);
            store_transposed(sh, kHidden, warp, tile_of(p.out.h1t, kTileT));
            if (!(ok = finished()))
                break;
            if (tid == 0)
            {
                load_weights(sw2, p.w2t, kW2, &wbar[1]);  // W2 has been read
                w2t_coming = true;
            }
            activate(kHidden, sb2);
            __syncthreads();
            // Head, four threads a row: thread g of a row holds the columns 8 g + 32 k + i (lanes
            // 8 g + i of a warp that strides the row by 32).  dH2 takes the place of H2, row group by
            // row group, each in one warp.
            {
                store_transposed(sh, kHidden, warp, tile_of(p.out.h2t, kTileT));
                __syncwarp();
                const int r = 8 * warp + (lane & 7), g = lane >> 3;
                unsigned char *at = sh + (warp * 32 + g) * 128 + (lane & 7) * 16;
                uint4 h[8];
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    v[i] = 0.0f;
#pragma unroll
                for (int k = 0; k < 8; ++k)
                {
                    h[k] = *reinterpret_cast<const uint4 *>(at + 4 * k * 128);
                    const uint32_t *w = reinterpret_cast<const uint32_t *>(&h[k]);
                    const float *w3 = sw3 + 8 * (g + 4 * k);
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        v[i] = fmaf(__uint_as_float(i & 1 ? w[i >> 1] & 0xffff0000u : w[i >> 1] << 16), w3[i], v[i]);
                }
                // the butterfly of a warp sum: lanes 16 and 8 apart in other threads, 4, 2, 1 in this one
#pragma unroll
                for (int o = 16; o >= 8; o >>= 1)
                {
#pragma unroll
                    for (int i = 0; i < 8; ++i)
                        v[i] += __shfl_xor_sync(0xffffffffu, v[i], o);
                }
                const float s0 = v[0] + v[4], s1 = v[1] + v[5], s2 = v[2] + v[6], s3 = v[3] + v[7];
                const float z = ((s0 + s2) + (s1 + s3)) + p.b3[0];
                const float prob = 1.0f / (1.0f + expf(-z));
                float d = 0.0f, l = 0.0f;
                if (row0 + r < p.n)
                {
                    const float y = p.valid[row0 + r] ? 0.0f : 1.0f;  // label: 1 = in collision
                    d = (prob - y) / static_cast<float>(p.n);
                    // log(1 + exp(z)) - y z, evaluated stably
                    l = (fmaxf(z, 0.0f) - z * y + log1pf(expf(-fabsf(z)))) / static_cast<float>(p.n);
                }
                if (g == 0)
                {
                    p.out.dz[row0 + r] = d;
                    // one addition a row: the epoch's sum rounds as it would row by row
                    if (row0 + r < p.n)
                        atomicAdd(p.loss, l);
                }
#pragma unroll
                for (int k = 0; k < 8; ++k)
                {
                    const uint32_t *w = reinterpret_cast<const uint32_t *>(&h[k]);
                    const float *w3 = sw3 + 8 * (g + 4 * k);
                    __align__(16) __nv_bfloat162 o[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        o[i] = __floats2bfloat162_rn(__uint_as_float(w[i] << 16) > 0.0f ? d * w3[2 * i] : 0.0f,
                                                     __uint_as_float(w[i] & 0xffff0000u) > 0.0f ? d * w3[2 * i + 1] : 0.0f);
                    *reinterpret_cast<uint4 *>(at + 4 * k * 128) = *reinterpret_cast<const uint4 *>(o);
                }
                __syncwarp();
                store_transposed(sh, kHidden, warp, tile_of(p.out.dh2t, kTileT));
            }
            publish();
            // back through layer 2
            issue(sh, sw2, kHidden, 0, &wbar[1], 1);
            if (!(ok = finished()))
                break;
            // dH1 = bf16(dH2 W2) where H1 > 0
#pragma unroll 1
            for (int c0 = c_lo; c0 < c_lo + 64; c0 += 32)
            {
                float v[32];
                tc::tmem_load32(lanes + static_cast<uint32_t>(c0), v);
                const uint32_t on = static_cast<uint32_t>(h1_positive >> (c0 - c_lo));
#pragma unroll
                for (int j = 0; j < 32; j += 8)
                {
                    __align__(16) __nv_bfloat162 h[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k)
                        h[k] = __floats2bfloat162_rn(on >> (j + 2 * k) & 1u ? v[j + 2 * k] : 0.0f,
                                                     on >> (j + 2 * k + 1) & 1u ? v[j + 2 * k + 1] : 0.0f);
                    *reinterpret_cast<uint4 *>(sh + tc::tile_offset(erow, c0 + j, kHidden)) = *reinterpret_cast<const uint4 *>(h);
                }
            }
            __syncthreads();
            store_transposed(sh, kHidden, warp, tile_of(p.out.dh1t, kTileT));
        } while (false);
        if ((!ok || skip) && tid == 0)
        {
            atomicExch(p.err, 1);
            // let the MMAs and copies still in flight finish before their memory is released
            if (pending)
                tc::mbar_wait(&bar, phase, kWaitLimit);
            tc::mbar_wait(&wbar[0], 0, kWaitLimit);
            tc::mbar_wait(&wbar[1], w2t_coming ? 1 : 0, kWaitLimit);
        }
        tc::fence_before_sync();
        __syncthreads();
        if (warp == 0)
        {
            tc::fence_after_sync();
            tc::tmem_free(tmem, 512);
        }
    }

    // ------------------------------------------------------------------------------ weights

    struct WeightsParams
    {
        StepBuffers in;
        int rows, kin;
        float *w, *grad, *m1, *m2;  // parameter order: W1, b1, W2, b2, w3, b3
        int adam;                   // 0: gradients to grad; 1: Adam on w, m1, m2
        float lr, b1, b2, eps, c1, c2;
        CoreWeights core;
        int *err;
        uint32_t wait_limit;
    };

    constexpr int kStages = 4;
    constexpr int kTileN = 32;          // columns of a dW2 tile
    constexpr int kStageA = 128 * 256;  // bytes of a 128 x 128 operand chunk
    constexpr int kStageB = 64 * 256;   // of a chunk of at most 64 columns
    constexpr int kWeightsThreads = 256;
    constexpr int kSumWarps = kWeightsThreads / 32;

    inline size_t weights_smem_bytes()
    {
        return kStages * (kStageA + kStageB);
    }

    inline int weights_grid()
    {
        return 2 * (kHidden / kTileN) + 2 + (3 * kHidden / 8 + 1 + kSumWarps - 1) / kSumWarps;
    }

    // K parameters' steps (indices i[k], gradients g[k]): the gradients stored, or Adam, all loads
    // before the first store; the new weights to w.
    template <int K>
    __device__ __forceinline__ void weight_steps(const WeightsParams &p, const size_t *i, const float *g, float *w)
    {
        if (!p.adam)
        {
#pragma unroll
            for (int k = 0; k < K; ++k)
                p.grad[i[k]] = g[k];
            return;
        }
        float m[K], v[K];
        bool still[K];
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            w[k] = p.w[i[k]];
            m[k] = p.m1[i[k]];
            v[k] = p.m2[i[k]];
        }
#pragma unroll
        for (int k = 0; k < K; ++k)
        {
            // a weight that has never had a gradient stays (padded inputs, dead units): its zeros
            // would take the slow paths of the divisions and the root, for the whole warp
            still[k] = g[k] == 0.0f && m[k] == 0.0f && v[k] == 0.0f;
            m[k] = p.b1 * m[k] + (1.0f - p.b1) * g[k];
            v[k] = p.b2 * v[k] + (1.0f - p.b2) * g[k] * g[k];
            const float ms = still[k] ? 1.0f : m[k], vs = still[k] ? 1.0f : v[k];
            const float wi = w[k] - p.lr * (ms / p.c1) / (sqrtf(vs / p.c2) + p.eps);
            w[k] = still[k] ? w[k] : wi;
            p.m1[i[k]] = m[k];
            p.m2[i[k]] = v[k];
            p.w[i[k]] = w[k];
        }
    }

    __device__ __forceinline__ void weight_step(const WeightsParams &p, size_t i, float g)
    {
        float w;
        weight_steps<1>(p, &i, &g, &w);
    }

    __global__ void __launch_bounds__(kWeightsThreads, 1) mlp_weights_kernel(const WeightsParams p)
    {
        extern __shared__ __align__(1024) unsigned char weights_smem[];
        __shared__ uint64_t full[kStages], empty[kStages], done;
        __shared__ uint32_t tmem_slot;
        __shared__ int failed;
        __shared__ float red[kSumWarps][8][33];
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
        const size_t o_b1 = static_cast<size_t>(kHidden) * p.kin, o_w2 = o_b1 + kHidden, o_b2 = o_w2 + kHidden * kHidden,
                     o_w3 = o_b2 + kHidden, o_b3 = o_w3 + kHidden;
        constexpr int kTiles2 = 2 * (kHidden / kTileN);
        const int tiles = p.rows / 128;
        if (tid == 0)
            failed = 0;
        if (static_cast<int>(blockIdx.x) >= kTiles2 + 2)
        {
            // Column sums, a warp per 8 columns of db2, db1 and dw3 (and one for db3): 32 phases of
            // rows y, y + 32, ... summed apart, then phase by phase.
            const int job = (static_cast<int>(blockIdx.x) - kTiles2 - 2) * kSumWarps + warp;
            tc::wait_previous_kernel();
            tc::start_next_kernel();
            if (*static_cast<volatile int *>(p.err))
                return;
            if (job == 3 * kHidden / 8)
            {
                float acc = 0.0f;
                for (int r = lane; r < p.rows; r += 32)
                    acc = fmaf(p.in.dz[r], 1.0f, acc);
                float sum = 0.0f;
                for (int k = 0; k < 32; ++k)
                    sum += __shfl_sync(0xffffffffu, acc, k);
                if (lane == 0)
                    weight_step(p, o_b3, sum);
            }
            else if (job < 3 * kHidden / 8)
            {
                const int kind = job / (kHidden / 8), jg = job % (kHidden / 8);
                const unsigned char *src = kind == 0 ? p.in.dh2t : kind == 1 ? p.in.dh1t : p.in.h2t;
                // lane: column jg * 8 + lane / 4, rows 2 (lane % 4) and the next of each 8-row group
                float acc[4][2] = {};
                for (int t = 0; t < tiles; ++t)
                {
                    const unsigned char *at = src + static_cast<size_t>(t) * kTileT + jg * 16 * 128 + 4 * lane;
                    const float *dz = p.in.dz + 128 * t + 2 * (lane & 3);
                    uint32_t v[16];
                    float2 d[16];
#pragma unroll
                    for (int g = 0; g < 16; ++g)
                    {
                        v[g] = *reinterpret_cast<const uint32_t *>(at + g * 128);
                        d[g] = kind == 2 ? *reinterpret_cast<const float2 *>(dz + 8 * g) : make_float2(1.0f, 1.0f);
                    }
#pragma unroll
                    for (int g = 0; g < 16; ++g)
                    {
                        acc[g & 3][0] = fmaf(__uint_as_float(v[g] << 16), d[g].x, acc[g & 3][0]);
                        acc[g & 3][1] = fmaf(__uint_as_float(v[g] & 0xffff0000u), d[g].y, acc[g & 3][1]);
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
                {
                    red[warp][lane >> 2][8 * k + 2 * (lane & 3)] = acc[k][0];
                    red[warp][lane >> 2][8 * k + 2 * (lane & 3) + 1] = acc[k][1];
                }
                __syncwarp();
                if (lane < 8)
                {
                    float sum = 0.0f;
                    for (int k = 0; k < 32; ++k)
                        sum += red[warp][lane][k];
                    weight_step(p, (kind == 0 ? o_b2 : kind == 1 ? o_b1 : o_w3) + 8 * jg + lane, sum);
                }
            }
            return;
        }
        // a 128 x N tile: rows 128 mt .. of dW2 (N = 32 columns from n0) or of dW1 (all kin columns)
        const bool second = static_cast<int>(blockIdx.x) < kTiles2;
        const int mt = blockIdx.x & 1, n0 = second ? (blockIdx.x >> 1) * kTileN : 0;
        const int N = second ? kTileN : p.kin;
        const unsigned char *ga = (second ? p.in.dh2t : p.in.dh1t) + mt * kStageA;
        const unsigned char *gb = second ? p.in.h1t + n0 * 256 : p.in.xt;
        const size_t b_tile = second ? kTileT : static_cast<size_t>(p.kin) * 256;
        const uint32_t b_bytes = static_cast<uint32_t>(N) * 256u;
        const uint32_t tcols = N <= 32 ? 32u : 64u;
        if (warp == 0)
            tc::tmem_alloc(&tmem_slot, tcols);
        if (tid == 0)
        {
            for (int s = 0; s < kStages; ++s)
            {
                tc::mbar_init(&full[s], 1);
                tc::mbar_init(&empty[s], 1);
            }
            tc::mbar_init(&done, 1);
        }
        tc::fence_before_sync();
        __syncthreads();
        tc::fence_after_sync();
        const uint32_t tmem = tmem_slot;
        tc::wait_previous_kernel();
        tc::start_next_kernel();
        if (tid == 0)
        {
            auto load = [&](int t) {
                const int s = t % kStages;
                unsigned char *at = weights_smem + s * (kStageA + kStageB);
                tc::mbar_expect(&full[s], kStageA + b_bytes);
                tc::bulk_load(at, ga + static_cast<size_t>(t) * kTileT, kStageA, &full[s]);
                tc::bulk_load(at + kStageA, gb + static_cast<size_t>(t) * b_tile, b_bytes, &full[s]);
            };
            const uint32_t idesc = tc::idesc_bf16_f32(128, N);
            int loaded = 0, used = 0;  // chunks whose copies were issued; whose MMAs were
            bool ok = *static_cast<volatile int *>(p.err) == 0;
            for (; ok && loaded < tiles && loaded < kStages; ++loaded)
                load(loaded);
            for (; used < tiles && ok; ++used)
            {
                const int s = used % kStages;
                ok = tc::mbar_wait(&full[s], used / kStages & 1, p.wait_limit);
                if (!ok)
                    break;
                const uint32_t a0 = tc::smem_u32(weights_smem + s * (kStageA + kStageB)), b0 = a0 + kStageA;
                for (int kk = 0; kk < 8; ++kk)
                    tc::mma_bf16(tmem, tc::smem_desc(a0 + kk * 256, 128, 2048), tc::smem_desc(b0 + kk * 256, 128, 2048), idesc,
                                 used > 0 || kk > 0);
                tc::mma_commit(&empty[s]);
                // the chunk before has been read: its stage takes the next one
                if (used > 0 && loaded < tiles)
                {
                    ok = tc::mbar_wait(&empty[(used - 1) % kStages], (used - 1) / kStages & 1, p.wait_limit);
                    if (ok)
                        load(loaded++);
                }
            }
            tc::mma_commit(&done);
            ok = ok && tc::mbar_wait(&done, 0, p.wait_limit);
            if (!ok)
            {
                // let the copies and MMAs still in flight finish before their memory is released
                atomicExch(p.err, 1);
                failed = 1;
                for (int t = used; t < loaded; ++t)
                    tc::mbar_wait(&full[t % kStages], t / kStages & 1, kWaitLimit);
                tc::mbar_wait(&done, 0, kWaitLimit);
            }
        }
        __syncthreads();
        tc::fence_after_sync();
        if (!failed)
        {
            // Through shared memory (the stages are free), so that a warp takes a row's 32 columns:
            // its weights and moments are then whole 128-byte lines (with each thread on a row of
            // its own, one column after another, this took most of the kernel's 47 us).  The new
            // weights go out in core-matrix layout, 16 bytes a thread.
            float *acc = reinterpret_cast<float *>(weights_smem);                               // [128][33]
            __nv_bfloat16 *wr = reinterpret_cast<__nv_bfloat16 *>(weights_smem + 128 * 33 * 4);  // [128][40]
            __nv_bfloat16 *wt = wr + 128 * 40;                                                   // [32][136]
            constexpr int kRows = 8;  // rows of a warp in flight together
            constexpr int kWarps = kWeightsThreads / 32;
            for (int c0 = 0; c0 < N; c0 += 32)
            {
                if (warp < 4)
                {
                    float v[32];
                    tc::tmem_load32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c0), v);
#pragma unroll
                    for (int c = 0; c < 32; ++c)
                        acc[tid * 33 + c] = v[c];
                }
                __syncthreads();
                const int c = n0 + c0 + lane;
                if (c0 + lane < N)
                {
#pragma unroll 1
                    for (int r0 = warp * kRows; r0 < 128; r0 += kWarps * kRows)
                    {
                        size_t at[kRows];
                        float g[kRows], w[kRows];
#pragma unroll
                        for (int k = 0; k < kRows; ++k)
                        {
                            const size_t j = static_cast<size_t>(128 * mt + r0 + k);
                            at[k] = second ? o_w2 + j * kHidden + c : j * p.kin + c;
                            g[k] = acc[(r0 + k) * 33 + lane];
                        }
                        weight_steps<kRows>(p, at, g, w);
                        if (p.adam)
                        {
#pragma unroll
                            for (int k = 0; k < kRows; ++k)
                            {
                                const __nv_bfloat16 wb = __float2bfloat16_rn(w[k]);
                                wr[(r0 + k) * 40 + lane] = wb;
                                if (second)
                                    wt[lane * 136 + r0 + k] = wb;
                            }
                        }
                    }
                }
                __syncthreads();
                if (p.adam)
                {
                    const int groups = min(N - c0, 32) / 8;
                    for (int u = tid; u < 128 * groups; u += kWeightsThreads)
                    {
                        // row r, columns 8 g ..: eight threads fill a core matrix
                        const int r = (u & 7) + 8 * ((u >> 3) / groups), g = (u >> 3) % groups;
                        *reinterpret_cast<uint4 *>((second ? p.core.w2 : p.core.w1) +
                                                   tc::tile_offset(128 * mt + r, n0 + c0 + 8 * g, second ? kHidden : p.kin)) =
                            *reinterpret_cast<const uint4 *>(wr + r * 40 + 8 * g);
                    }
                    for (int u = tid; second && u < 32 * 16; u += kWeightsThreads)
                    {
                        const int r = (u & 7) + 8 * (u >> 7), g = u >> 3 & 15;
                        *reinterpret_cast<uint4 *>(p.core.w2t + tc::tile_offset(n0 + r, 128 * mt + 8 * g, kHidden)) =
                            *reinterpret_cast<const uint4 *>(wt + r * 136 + 8 * g);
                    }
                    __syncthreads();
                }
            }
        }
        tc::fence_before_sync();
        __syncthreads();
        if (warp == 0)
        {
            tc::fence_after_sync();
            tc::tmem_free(tmem, tcols);
        }
    }
}  // namespace vg
