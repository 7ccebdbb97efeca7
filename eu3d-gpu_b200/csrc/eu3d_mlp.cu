// eu3d_mlp.cu — launchers of the learned-chemistry model's kernels: the BF16 GEMM
// (eu3d_gemm.cuh), the fused inference (eu3d_mlp_fused.cuh), the training step
// (eu3d_mlp_train.cuh), feature packing and output unscaling.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include "eu3d.h"
#include "eu3d_attr.hpp"
#include "eu3d_gemm.cuh"
#include "eu3d_mlp_fused.cuh"
#include "eu3d_mlp_kernels.hpp"
#include "eu3d_mlp_train.cuh"

using namespace eu3d;

namespace {

template <int BN>
cudaError_t gemm_launch(const __nv_bfloat16 *A, int lda, const __nv_bfloat16 *B, int ldb, int M, int N, int K,
                        const float *bias, int act, float *Cf, __nv_bfloat16 *Cb, float *Cpre, int ldc, int *err,
                        cudaStream_t s)
{
    const size_t smem = gemm_smem_bytes<BN>();
    static SmemLimit limit; // per instantiation, per device
    const cudaError_t e = limit.ensure(k_gemm_bf16<BN>, smem);
    if (e != cudaSuccess)
        return e;
    const dim3 grid((M + kGemmBM - 1) / kGemmBM, (N + BN - 1) / BN);
    k_gemm_bf16<BN><<<grid, kGemmThreads, smem, s>>>(A, lda, B, ldb, M, N, K, bias, act, Cf, Cb, Cpre, ldc, err);
    return cudaGetLastError();
}

// rows of n_in fp32 features -> (x - shift) * scale as bf16, zero padded to ld
__global__ void k_pack_features(const float *__restrict__ X, long long n, int n_in, const float *__restrict__ shift,
                                const float *__restrict__ scale, __nv_bfloat16 *__restrict__ out, int ld)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * ld)
        return;
    const long long r = t / ld;
    const int c = int(t % ld);
    float v = 0.0f;
    if (c < n_in)
        v = (X[r * n_in + c] - shift[c]) * scale[c];
    out[t] = __float2bfloat16_rn(v);
}

// Y [n x ld] normalised outputs of member e -> denormalised fp32 out[e][n][n_out]
__global__ void k_unscale(const float *__restrict__ Y, long long n, int ld, int n_out, const float *__restrict__ shift,
                          const float *__restrict__ scale, float *__restrict__ out)
{
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n * n_out)
        return;
    const long long r = t / n_out;
    const int c = int(t % n_out);
    out[t] = Y[r * ld + c] / scale[c] + shift[c];
}

inline unsigned blocks(long long n, int t) { return unsigned((n + t - 1) / t); }

} // namespace

namespace eu3d {

cudaError_t gemm_bf16(const void *A, int lda, const void *B, int ldb, int M, int N, int K, const float *bias, int act,
                      float *Cf, void *Cb, float *Cpre, int ldc, int *err, cudaStream_t s)
{
    auto a = static_cast<const __nv_bfloat16 *>(A);
    auto b = static_cast<const __nv_bfloat16 *>(B);
    auto cb = static_cast<__nv_bfloat16 *>(Cb);
    if (N > 128)
        return gemm_launch<256>(a, lda, b, ldb, M, N, K, bias, act, Cf, cb, Cpre, ldc, err, s);
    if (N > 64)
        return gemm_launch<128>(a, lda, b, ldb, M, N, K, bias, act, Cf, cb, Cpre, ldc, err, s);
    return gemm_launch<64>(a, lda, b, ldb, M, N, K, bias, act, Cf, cb, Cpre, ldc, err, s);
}

cudaError_t pack_features(const float *X, long long n, int n_in, const float *shift, const float *scale, void *out,
                          int ld, cudaStream_t s)
{
    k_pack_features<<<blocks(n * ld, 256), 256, 0, s>>>(X, n, n_in, shift, scale, static_cast<__nv_bfloat16 *>(out), ld);
    return cudaGetLastError();
}

cudaError_t train_rows(const TrainParams &p, cudaStream_t s)
{
    static SmemLimit limit; // per device
    const cudaError_t e = limit.ensure(k_train_rows, kTrainSmem);
    if (e != cudaSuccess)
        return e;
    k_train_rows<<<dim3(unsigned((p.n + kTrainRows - 1) / kTrainRows), unsigned(p.members)), kTrainThreads, kTrainSmem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t train_weights(const TrainParams &p, int sms, cudaStream_t s)
{
    static SmemLimit limit; // per device
    const cudaError_t e = limit.ensure(k_train_dw, kDwSmem);
    if (e != cudaSuccess)
        return e;
    // one CTA per SM: `unit` for the narrow first layer and outputs, twice that for
    // the layers between
    const int parts = 2 * p.hidden * p.members, unit = sms / parts > 1 ? sms / parts : 1;
    k_train_dw<<<dim3(unsigned(2 * p.hidden * unit), unsigned(p.members)), kDwThreads, kDwSmem, s>>>(p, unit);
    return cudaGetLastError();
}

cudaError_t train_adam(const TrainParams &p, float lr, float b1, float b2, float eps, float c1, float c2, cudaStream_t s)
{
    k_train_adam<<<dim3(blocks(p.params, 256), unsigned(p.members)), 256, 0, s>>>(p, lr, b1, b2, eps, c1, c2);
    return cudaGetLastError();
}

cudaError_t mlp_fused(const FusedMlpParams &p, const float *feat, int ld_feat, int count_host, const int *count_dev,
                      int max_rows, float *out, long long s_row, long long s_mem, int *err, int grid, cudaStream_t s)
{
    if (!fused_supported(p.in_pad, p.width, p.out_pad, p.members, p.layers))
        return cudaErrorInvalidValue;
    const size_t smem = fused_smem_bytes(p.in_pad, p.width, p.out_pad, p.layers, p.members);
    static SmemLimit limit; // per device: the largest size set so far
    const cudaError_t e = limit.ensure(k_mlp_fused, smem);
    if (e != cudaSuccess)
        return e;
    if (grid < 1)
        return cudaSuccess;
    k_mlp_fused<<<grid, kFusedThreads, smem, s>>>(p, feat, ld_feat, count_host, count_dev, max_rows, out, s_row, s_mem,
                                                  err);
    return cudaGetLastError();
}

cudaError_t unscale_outputs(const float *Y, long long n, int ld, int n_out, const float *shift, const float *scale,
                            float *out, cudaStream_t s)
{
    k_unscale<<<blocks(n * n_out, 256), 256, 0, s>>>(Y, n, ld, n_out, shift, scale, out);
    return cudaGetLastError();
}

} // namespace eu3d
