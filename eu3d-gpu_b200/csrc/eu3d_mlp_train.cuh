// eu3d_mlp_train.cuh — a training step of the learned-chemistry ensemble in
// three kernels over all members: rows (forward, loss and the gradients'
// way back to the first layer), weight gradients, Adam.
//
// A batch's rows are independent up to the weight gradients, so k_train_rows
// gives each 128-row tile of each member to one CTA, which runs every layer
// forward and back on the tensor cores with the tile's activations, and on the
// way back its layer gradients, in shared memory as the next MMA's A operand
// (two CTAs per SM: one's epilogue under the other's MMAs). What the weight
// gradients need, the bf16 inputs and gradients of every layer, goes to global
// memory as K slabs with the rows along K, in the layout the MMAs read, tile by
// tile. The pre-activations (fp32, for SiLU') are kept a column at a time and
// read back by the same thread. k_train_dw then forms every layer's dW = dZ^T H
// of every member in one launch, split along the rows to fill the chip.
// k_train_adam updates the parameters, packs the bf16 weights for the next step
// and clears the gradients.
//
// Rounding points are the layer-wise path's: bf16 inputs, weights, activations
// and layer gradients, fp32 accumulation, bias gradients from the fp32 layer
// gradients. Launched layer by layer, with transposes, column sums and
// one-value-a-lane epilogues of their own, a step of three members at batch
// 16384 took 3.2 ms (about 165 launches); in three kernels, with the planes
// transposed row by row and staged into the MMAs' layout by k_train_dw, 0.35 ms
// (rows 0.25, weight gradients 0.10); with the planes written in that layout
// 0.26 ms.
#pragma once

#include <cuda_bf16.h>

#include "eu3d_gemm.cuh"
#include "eu3d_mlp_kernels.hpp"
#include "eu3d_tc.cuh"

namespace eu3d {

// three slabs in flight: two CTAs' shared memory then just fits an SM
constexpr int kTrainThreads = 256, kTrainSlots = 3, kTrainSlabBytes = 256 * kFusedSlabK * 2;
constexpr size_t kTrainSmem = size_t(kTrainRows) * 256 * 2 + kTrainSlots * kTrainSlabBytes + 64;

__device__ __forceinline__ unsigned long long train_row(unsigned long long key, int i, long long n)
{
    // uniform index in [0, n) from a counter-based hash (splitmix64) of the key
    // and the batch position: batches drawn on the device, no host copies
    unsigned long long z = key + 0x9E3779B97F4A7C15ull * (unsigned long long)(i + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return z % (unsigned long long)n;
}

// Sum over the warp's lanes of each of 32 values: lane q returns value q's sum.
__device__ __forceinline__ float column_sum(float (&v)[32], int lane)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < o; ++q) {
            const bool hi = (lane & o) != 0;
            const float send = hi ? v[q] : v[q + o], keep = hi ? v[q + o] : v[q];
            v[q] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    return v[0];
}

// 8 bf16 of one row into an A operand (core-matrix layout).
__device__ __forceinline__ void put_operand(unsigned char *act, int col, int row, const __nv_bfloat16 *v)
{
    *reinterpret_cast<uint4 *>(act + ((col / 8) * kTrainRows + row) * 16) = *reinterpret_cast<const uint4 *>(v);
}

__global__ void __launch_bounds__(kTrainThreads, 2) k_train_rows(const __grid_constant__ TrainParams p)
{
    extern __shared__ __align__(128) unsigned char smem[];
    unsigned char *act = smem;                                    // [256 / 8][128][16 B]
    unsigned char *ring = smem + kTrainRows * 256 * 2;            // weight slabs
    uint64_t *full = reinterpret_cast<uint64_t *>(ring + kTrainSlots * kTrainSlabBytes), *empty = full + kTrainSlots;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(empty + kTrainSlots);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tslot + 1);

    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, quad = warp % 4, half = warp / 4;
    const int e = p.first + blockIdx.y;
    const TrainMember &mem = p.member[e];
    const int lrow = quad * 32 + lane, row = blockIdx.x * kTrainRows + lrow;
    const bool valid = row < p.n;
    const long long src = !valid ? 0 : p.drawn ? (long long)train_row(mem.key, row, p.rows) : row;
    // this tile's part of a plane of `cols` columns: as K slabs (K = rows) in the
    // core-matrix layout, and of the fp32 pre-activations, columns outermost
    const size_t tiles = gridDim.x, tile = blockIdx.x;
    auto slab_rows = [&](__nv_bfloat16 *plane, int layer, int cols) {
        return plane + (layer * tiles + tile) * size_t(cols) * kTrainRows + (size_t(lrow / 8) * cols) * 8 + lrow % 8;
    };
    auto z_rows = [&](int layer) { return mem.ZT + (layer * tiles + tile) * size_t(p.width) * kTrainRows + lrow; };

    if (warp == 0) {
        tc::tmem_alloc(tslot, 256);
        tc::tmem_relinquish();
    }
    if (tid == 0) {
        for (int q = 0; q < kTrainSlots; ++q) {
            tc::mbar_init(&full[q], 1);
            tc::mbar_init(&empty[q], 1);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // features -> first A operand and, transposed, the first layer's input
    __nv_bfloat16 *xt = slab_rows(mem.XT, 0, p.in_pad);
    for (int kc = half; kc < p.in_pad / 8; kc += 2) {
        __align__(16) __nv_bfloat16 v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = kc * 8 + q;
            float f = 0.0f;
            if (valid && c < p.n_in)
                f = (p.X[src * p.n_in + c] - p.in_shift[c]) * p.in_scale[c];
            v[q] = __float2bfloat16_rn(f);
            xt[c * 8] = v[q];
        }
        put_operand(act, kc * 8, lrow, v);
    }
    tc::fence_proxy_async();
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tslot;
    const uint32_t trow = tmem + (uint32_t(quad * 32) << 16);
    const int L = p.hidden;       // hidden layers; GEMMs 0 .. L forward, then L .. 1 back
    const int ngemm = 2 * L + 1;
    int issued = 0, done = 0;     // weight slabs requested and consumed (thread 0)
    bool ok = true;

    // GEMM q: its weights, K and N
    auto shape = [&](int q, const __nv_bfloat16 *&w, int &K, int &N) {
        if (q <= L) {
            K = q == 0 ? p.in_pad : p.width;
            N = q == L ? p.out_pad : p.width;
            w = mem.slabs[q];
        } else {
            const int l = L - (q - L - 1); // back through layer l
            K = l == L ? p.out_pad : p.width;
            N = p.width;
            w = mem.slabs_t[l];
        }
    };
    auto request = [&](int q, int s) { // slab s of GEMM q into the next slot
        const __nv_bfloat16 *w;
        int K, N;
        shape(q, w, K, N);
        const int slot = issued % kTrainSlots;
        if (issued >= kTrainSlots && !tc::mbar_wait(&empty[slot], uint32_t((issued / kTrainSlots - 1) & 1)))
            return false;
        const uint32_t bytes = uint32_t(N) * min(kFusedSlabK, K - s * kFusedSlabK) * 2;
        tc::mbar_arrive_expect_tx(&full[slot], bytes);
        tc::bulk_g2s(ring + slot * kTrainSlabBytes, w + (size_t)s * N * kFusedSlabK, bytes, &full[slot]);
        ++issued;
        return true;
    };
    auto slabs_of = [&](int q) {
        const __nv_bfloat16 *w;
        int K, N;
        shape(q, w, K, N);
        return (K + kFusedSlabK - 1) / kFusedSlabK;
    };

    // 32 pre-activations of this thread's row, columns c0 ..
    float zz[32];
    auto load_z = [&](const float *z, int c0) {
        z += c0 * kTrainRows;
        if (c0 + 32 <= p.width) {
#pragma unroll
            for (int u = 0; u < 32; ++u) zz[u] = z[u * kTrainRows];
        } else {
#pragma unroll
            for (int u = 0; u < 32; ++u) zz[u] = c0 + u < p.width ? z[u * kTrainRows] : 0.0f;
        }
    };

    for (int q = 0; q < ngemm; ++q) {
        // the way back: the first pre-activations come while the MMAs run
        if (q > L)
            load_z(z_rows(2 * L - q), half * 32);
        // ------------------------------------------------------------ MMAs
        if (tid == 0) {
            const __nv_bfloat16 *w;
            int K, N;
            shape(q, w, K, N);
            const int ns = slabs_of(q), first = done;
            const uint32_t idesc = tc::idesc_bf16_f32(kTrainRows, N);
            bool good = true;
            while (good && issued < first + min(ns, kTrainSlots)) good = request(q, issued - first);
            for (int s = 0; good && s < ns; ++s) {
                const int slot = done % kTrainSlots;
                good = good && tc::mbar_wait(&full[slot], uint32_t((done / kTrainSlots) & 1));
                if (!good)
                    break;
                tc::tc_fence_after();
                const int kw = min(kFusedSlabK, K - s * kFusedSlabK);
                const uint32_t a0 = tc::smem_u32(act), b0 = tc::smem_u32(ring + slot * kTrainSlabBytes);
                for (int kk = 0; kk < kw / 16; ++kk) {
                    const int kg = s * (kFusedSlabK / 16) + kk;
                    tc::mma_bf16(tmem, tc::smem_desc(a0 + kg * 2 * kTrainRows * 16, kTrainRows * 16, 128),
                                 tc::smem_desc(b0 + kk * 2 * N * 16, N * 16, 128), idesc, (s > 0 || kk > 0) ? 1u : 0u);
                }
                tc::mma_commit(&empty[slot]);
                ++done;
                // refill the slot of the MMAs before these, which run meanwhile
                if (s >= 1 && issued < first + ns)
                    good = request(q, issued - first);
            }
            // the last slab's commit follows every MMA of the GEMM
            if (good)
                good = tc::mbar_wait(&empty[(done - 1) % kTrainSlots], uint32_t(((done - 1) / kTrainSlots) & 1));
            // the next GEMM's first slabs arrive under this one's epilogue
            if (q + 1 < ngemm)
                for (int s = 0; good && s < min(slabs_of(q + 1), kTrainSlots); ++s) good = request(q + 1, s);
            if (!good) {
                *abort_flag = 1;
                atomicExch(p.err, 1);
            }
        }
        __syncthreads();
        tc::tc_fence_after();
        if (*abort_flag) {
            ok = false;
            break;
        }
        // -------------------------------------------------------- epilogue
        if (q < L) { // hidden layer: z, silu(z) as bf16
            float *z0 = z_rows(q);
            __nv_bfloat16 *ht0 = slab_rows(mem.HT, q, p.width);
            const float *bias = mem.bias[q];
            for (int c0 = half * 32; c0 < p.width; c0 += 64) {
                float v[32];
                tc::tmem_ld32(trow + c0, v);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = c0 + j * 8;
                    if (c < p.width) {
                        __align__(16) __nv_bfloat16 h[8];
                        const float4 b0 = __ldg(reinterpret_cast<const float4 *>(bias + c)),
                                     b1 = __ldg(reinterpret_cast<const float4 *>(bias + c + 4));
                        const float bb[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            v[j * 8 + u] += bb[u];
                            h[u] = __float2bfloat16_rn(silu(v[j * 8 + u]));
                        }
                        put_operand(act, c, lrow, h);
                        __nv_bfloat16 *ht = ht0 + c * 8;
                        float *z = z0 + c * kTrainRows;
#pragma unroll
                        for (int u = 0; u < 8; ++u) {
                            ht[u * 8] = h[u];
                            z[u * kTrainRows] = v[j * 8 + u];
                        }
                    }
                }
            }
        } else if (q == L) { // output: loss and its gradient
            float sq = 0.0f;
            __nv_bfloat16 *yt = slab_rows(mem.dYT, 0, p.out_pad);
            for (int c0 = half * 32; c0 < p.out_pad; c0 += 64) {
                float v[32];
                tc::tmem_ld32(trow + c0, v);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = c0 + j * 8;
                    __align__(16) __nv_bfloat16 g[8];
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        float d = 0.0f;
                        if (valid && c + u < p.n_out) {
                            const float target = (p.T[src * p.n_out + c + u] - p.out_shift[c + u]) * p.out_scale[c + u];
                            d = v[j * 8 + u] + __ldg(mem.bias[L] + c + u) - target;
                            sq += d * d;
                            d = 2.0f * d / float((long long)p.n * p.n_out);
                        }
                        g[u] = __float2bfloat16_rn(d);
                        v[j * 8 + u] = __bfloat162float(g[u]);
                        if (c + u < p.out_pad)
                            yt[(c + u) * 8] = g[u];
                    }
                    if (c < p.out_pad)
                        put_operand(act, c, lrow, g);
                }
                const float s = column_sum(v, lane);
                if (c0 + lane < p.out_pad)
                    atomicAdd(&mem.gb[L][c0 + lane], s);
            }
            for (int o = 16; o > 0; o >>= 1) sq += __shfl_down_sync(0xffffffffu, sq, o);
            if (lane == 0 && sq != 0.0f)
                atomicAdd(&p.loss[e], sq);
        } else { // back through layer l into hidden layer l - 1
            const int l = L - (q - L - 1);
            const float *z = z_rows(l - 1);
            __nv_bfloat16 *zt0 = slab_rows(mem.dZT, l - 1, p.width);
            for (int c0 = half * 32; c0 < p.width; c0 += 64) {
                if (c0 > half * 32)
                    load_z(z, c0);
                float v[32];
                tc::tmem_ld32(trow + c0, v);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int c = c0 + j * 8;
                    __align__(16) __nv_bfloat16 g[8];
                    // (rows past the batch have zero gradients: no loss)
#pragma unroll
                    for (int u = 0; u < 8; ++u) {
                        const float d = c < p.width ? v[j * 8 + u] * silu_grad(zz[j * 8 + u]) : 0.0f;
                        v[j * 8 + u] = d;
                        g[u] = __float2bfloat16_rn(d);
                    }
                    if (c < p.width) {
                        __nv_bfloat16 *zt = zt0 + c * 8;
#pragma unroll
                        for (int u = 0; u < 8; ++u) zt[u * 8] = g[u];
                        put_operand(act, c, lrow, g);
                    }
                }
                const float s = column_sum(v, lane);
                if (c0 + lane < p.width)
                    atomicAdd(&mem.gb[l - 1][c0 + lane], s);
            }
        }
        tc::fence_proxy_async();
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
    }
    if (!ok && tid == 0) {
        // copies in flight land and MMAs issued finish (bounded) before the
        // CTA's memory goes away
        for (int s = issued > kTrainSlots ? issued - kTrainSlots : 0; s < issued; ++s)
            tc::mbar_wait(&full[s % kTrainSlots], uint32_t((s / kTrainSlots) & 1));
        if (done > 0)
            tc::mbar_wait(&empty[(done - 1) % kTrainSlots], uint32_t(((done - 1) / kTrainSlots) & 1));
    }
    tc::tc_fence_before();
    __syncthreads();
    if (warp == 0)
        tc::tmem_dealloc(tmem, 256);
}

// dW = dZ^T H of every layer of every member. The batch's 64-row slabs are cut into
// pieces; a CTA takes every `splits`-th piece of one layer (all its outputs and
// inputs, two 128 x 256 accumulators at most) and adds each piece's sums to the fp32
// gradient four values at a time. The operands lie in global memory as the MMAs
// read them, so a slab is one bulk copy each, three of them in flight.
//
// The pieces are the layer-wise training's splits of K (one below 512 rows, 4 below
// 2048, else 16), so every piece's sum is bitwise that one's and only the order in
// which the pieces are added is open: with other pieces a batch of 256 rows, 24
// steps a pass, was 1e-2 of its gradients' norm off in the second pass (Adam divides
// a gradient by its size; the layer-wise code is 7e-3 off itself). Where 16 pieces would
// leave the chip idle (few layers and members, more than 24 CTAs for each) or make a
// CTA come back often (fewer than 16), there is a piece for each CTA.
constexpr int kDwThreads = 256, kDwK = 64, kDwSlots = 3, kDwOperand = 256 * kDwK * 2;
constexpr size_t kDwSmem = size_t(kDwSlots) * 2 * kDwOperand + 8 * (2 * kDwSlots + 1) + 16;

__global__ void __launch_bounds__(kDwThreads, 1) k_train_dw(const __grid_constant__ TrainParams p, int unit)
{
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + size_t(kDwSlots) * 2 * kDwOperand), *empty = full + kDwSlots;
    uint64_t *acc = empty + kDwSlots;
    uint32_t *tslot = reinterpret_cast<uint32_t *>(acc + 1);
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const TrainMember &mem = p.member[p.first + blockIdx.y];
    // the job: `unit` CTAs for the first layer and for the outputs (one narrow
    // operand), twice as many for each layer between
    const int L = p.hidden;
    const int l = int(blockIdx.x) < unit ? 0 : min(L, (int(blockIdx.x) - unit) / (2 * unit) + 1);
    const int splits = l == 0 || l == L ? unit : 2 * unit, split = int(blockIdx.x) - (l == 0 ? 0 : unit + (l - 1) * 2 * unit);
    const int M = l == L ? p.out_pad : p.width, N = l == 0 ? p.in_pad : p.width;
    const int tiles = (p.n + kTrainRows - 1) / kTrainRows, slabs = (p.n + kDwK - 1) / kDwK;
    const __nv_bfloat16 *A = l == L ? mem.dYT : mem.dZT + size_t(l) * tiles * p.width * kTrainRows;
    const __nv_bfloat16 *B = l == 0 ? mem.XT : mem.HT + size_t(l - 1) * tiles * p.width * kTrainRows;
    const int pieces = p.n < 512 ? 1 : p.n < 2048 ? 4 : 2 * unit >= 16 && 2 * unit <= 24 ? 16 : splits;
    const int per = (slabs + pieces - 1) / pieces;
    if (split >= pieces || split * per >= slabs)
        return;
    if (warp == 0) {
        tc::tmem_alloc(tslot, 512);
        tc::tmem_relinquish();
    }
    if (threadIdx.x == 0) {
        for (int q = 0; q < kDwSlots; ++q) {
            tc::mbar_init(&full[q], 1);
            tc::mbar_init(&empty[q], 1);
        }
        tc::mbar_init(acc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tmem = *tslot;
    bool ok = true;
    int done = 0; // slabs of the pieces before: the ring goes on from piece to piece
    for (int piece = split, turn = 0; ok && piece < pieces && piece * per < slabs; piece += splits, ++turn) {
        const int k0 = piece * per, end = done + min(slabs - k0, per);
        if (threadIdx.x == 0) { // copies
            int k = done;
            for (; k < end; ++k) {
                const int slot = k % kDwSlots;
                if (k >= kDwSlots && !tc::mbar_wait(&empty[slot], uint32_t((k / kDwSlots - 1) & 1))) {
                    ok = false;
                    break;
                }
                unsigned char *a = smem + size_t(slot) * 2 * kDwOperand;
                const size_t at = size_t(k0 + k - done);
                tc::mbar_arrive_expect_tx(&full[slot], uint32_t(M + N) * kDwK * 2);
                tc::bulk_g2s(a, A + at * M * kDwK, uint32_t(M) * kDwK * 2, &full[slot]);
                tc::bulk_g2s(a + kDwOperand, B + at * N * kDwK, uint32_t(N) * kDwK * 2, &full[slot]);
            }
            // copies in flight land before the CTA's memory goes away
            for (int q = max(done, k - kDwSlots); q < k; ++q)
                ok = tc::mbar_wait(&full[q % kDwSlots], uint32_t((q / kDwSlots) & 1)) && ok;
        } else if (threadIdx.x == 32) { // MMAs
            const uint32_t idesc = tc::idesc_bf16_f32(128, N);
            for (int k = done; k < end; ++k) {
                const int slot = k % kDwSlots;
                ok = tc::mbar_wait(&full[slot], uint32_t((k / kDwSlots) & 1));
                if (!ok)
                    break;
                tc::tc_fence_after();
                const uint32_t a0 = tc::smem_u32(smem + size_t(slot) * 2 * kDwOperand), b0 = a0 + kDwOperand;
#pragma unroll
                for (int kk = 0; kk < kDwK / 16; ++kk)
                    for (int h = 0; h * 128 < M; ++h) // (rows past M are accumulated from what lies there and not read)
                        tc::mma_bf16(tmem + 256 * h, tc::smem_desc(a0 + kk * 2 * M * 16 + h * 128 * 16, M * 16, 128),
                                     tc::smem_desc(b0 + kk * 2 * N * 16, N * 16, 128), idesc,
                                     (k > done || kk > 0) ? 1u : 0u);
                tc::mma_commit(&empty[slot]);
            }
            tc::mma_commit(acc); // every MMA issued so far
            ok = tc::mbar_wait(acc, uint32_t(turn & 1)) && ok;
        }
        ok = __syncthreads_and(ok);
        tc::tc_fence_after();
        if (ok) {
            const int h = warp / 4, m = warp * 32 + lane;
            float *g = mem.gW[l] + size_t(m) * N;
            if (h * 128 < M)
                for (int c0 = 0; c0 < N; c0 += 32) {
                    float v[32];
                    tc::tmem_ld32(tmem + 256 * h + (uint32_t((warp % 4) * 32) << 16) + c0, v);
                    if (m < M)
#pragma unroll
                        for (int j = 0; j < 8; ++j)
                            if (c0 + j * 4 < N)
                                asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(g + c0 + j * 4),
                                             "f"(v[j * 4]), "f"(v[j * 4 + 1]), "f"(v[j * 4 + 2]), "f"(v[j * 4 + 3])
                                             : "memory");
                }
        } else if (threadIdx.x == 0) {
            atomicExch(p.err, 1);
        }
        // the accumulators are read before the next piece's MMAs overwrite them
        tc::tc_fence_before();
        __syncthreads();
        tc::tc_fence_after();
        done = end;
    }
    if (warp == 0)
        tc::tmem_dealloc(tmem, 512);
}

// Position of element (n, k) of an [N x K] operand in its K-slabs of kFusedSlabK
// columns, each in the core-matrix layout, slabs back to back.
__device__ __forceinline__ size_t slab_at(int n, int k, int N)
{
    const int s = k / kFusedSlabK, kl = k % kFusedSlabK;
    return (size_t)s * N * kFusedSlabK + ((size_t)(kl / 8) * N + n) * 8 + kl % 8;
}

// Adam on every parameter of the members (pads have zero gradients and stay
// zero), or with lr == 0 the packing of the weights alone; the gradients are
// cleared for the next step.
__global__ void k_train_adam(const __grid_constant__ TrainParams p, float lr, float b1, float b2, float eps, float c1, float c2)
{
    const TrainMember &mem = p.member[p.first + blockIdx.y];
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < p.params; t += gridDim.x * blockDim.x) {
        int l = 0, base = 0, in = 0, out = 0;
        for (l = 0; l <= p.hidden; ++l) {
            in = l == 0 ? p.in_pad : p.width;
            out = l == p.hidden ? p.out_pad : p.width;
            if (t < base + out * in + out)
                break;
            base += out * in + out;
        }
        const int at = t - base;
        float w = mem.P[t];
        if (lr > 0.0f) {
            const float g = mem.G[t];
            const float mi = b1 * mem.M[t] + (1.0f - b1) * g;
            const float vi = b2 * mem.V[t] + (1.0f - b2) * g * g;
            mem.M[t] = mi;
            mem.V[t] = vi;
            w -= lr * (mi * c1) / (sqrtf(vi * c2) + eps);
            mem.P[t] = w;
            mem.G[t] = 0.0f;
        }
        if (at < out * in) {
            const int o = at / in, i = at % in;
            const __nv_bfloat16 b = __float2bfloat16_rn(w);
            mem.Wb[l][at] = b;
            mem.slabs[l][slab_at(o, i, out)] = b;
            mem.slabs_t[l][slab_at(i, o, in)] = b;
        }
    }
}

} // namespace eu3d
