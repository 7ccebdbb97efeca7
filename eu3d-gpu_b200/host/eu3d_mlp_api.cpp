// eu3d_mlp_api.cpp — the learned-chemistry model (include/eu3d.h, eu_mlp_*):
// an ensemble of MLPs (n_in -> width x hidden SiLU layers -> n_out) trained and
// evaluated with the BF16 tensor-core GEMM (fp32 accumulation, fp32 master
// weights, Adam). All tensors stay on the device; training batches are drawn
// on the device from caller-provided fp32 arrays.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <random>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "eu3d.h"
#include "eu3d_mlp_kernels.hpp"
#include "mlp_internal.hpp"

namespace {

struct Layer {
    int in = 0, out = 0, in_pad = 0, out_pad = 0;
    long long at = 0;                   // of W in the member's parameters; b follows
    float *W = nullptr, *b = nullptr;   // fp32 master, padded [out_pad x in_pad], [out_pad]
    float *gW = nullptr, *gb = nullptr; // gradients
    __nv_bfloat16 *Wb = nullptr;        // [out_pad x in_pad]
    __nv_bfloat16 *slabs = nullptr, *slabs_t = nullptr; // its K-slabs and its transpose's
};

int pad16(int n) { return (n + 15) / 16 * 16; }

} // namespace

struct eu_mlp {
    int device = 0;
    cudaStream_t stream = nullptr;
    int *d_err = nullptr;
    std::string err;
    bool ready = false;
    int n_in = 0, width = 0, hidden = 0, n_out = 0, members = 0, max_batch = 0;
    int in_pad = 0, out_pad = 0;
    std::vector<std::vector<Layer>> net;
    float *in_shift = nullptr, *in_scale = nullptr, *out_shift = nullptr, *out_scale = nullptr;
    // fp32 parameters, gradients and Adam's moments: `params` padded values a member
    float *P = nullptr, *G = nullptr, *M = nullptr, *V = nullptr;
    long long params = 0;
    void *X = nullptr;    // bf16 [B x in_pad]
    std::vector<void *> H; // bf16 [B x width]
    float *Y = nullptr;   // fp32 [B x out_pad]
    float *loss = nullptr; // [members]
    long long adam_t = 0;
    std::vector<void *> allocs;
    // training scratch (allocated by the first training call, grown with the
    // batch and the members that run together, kept)
    void *train = nullptr;
    size_t train_bytes = 0;
    // inference in one persistent kernel (eu3d_mlp_fused.cuh), on the K-slabs
    bool fused = false;
    __nv_bfloat16 *slabs = nullptr;
    long long slab_off[eu3d::kFusedMaxMembers][eu3d::kFusedMaxLayers] = {};
    int sms = 0;
};

namespace {

eu_status mfail(eu_mlp *m, eu_status s, const char *fmt, ...)
{
    if (m) {
        char buf[512];
        va_list ap;
        va_start(ap, fmt);
        std::vsnprintf(buf, sizeof buf, fmt, ap);
        va_end(ap);
        m->err = buf;
    }
    return s;
}

#define MCK(m, call)                                                                               \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            return mfail((m), e_ == cudaErrorMemoryAllocation ? EU_ERR_OUT_OF_MEMORY : EU_ERR_CUDA, "%s: %s", #call, \
                         cudaGetErrorString(e_));                                                  \
    } while (0)

template <typename T>
cudaError_t malloc_zero(eu_mlp *m, T **p, size_t bytes)
{
    void *q = nullptr;
    cudaError_t e = cudaMalloc(&q, bytes);
    if (e != cudaSuccess)
        return e;
    m->allocs.push_back(q);
    *p = static_cast<T *>(q);
    return cudaMemsetAsync(q, 0, bytes, m->stream);
}

void free_all(eu_mlp *m)
{
    for (void *p : m->allocs) cudaFree(p);
    m->allocs.clear();
    if (m->train)
        cudaFree(m->train);
    m->train = nullptr;
    m->train_bytes = 0;
    m->net.clear();
    m->H.clear();
    m->ready = false;
}

long long params_per_member(const eu_mlp *m)
{
    long long n = 0;
    for (const Layer &L : m->net[0]) n += (long long)L.out * L.in + L.out;
    return n;
}

// layer-wise inference of member e over n packed rows in m->X (on stream s), with
// the fused kernel's activation, so that the two predictions agree bitwise
eu_status forward(eu_mlp *m, int e, int n, cudaStream_t s = nullptr)
{
    if (!s)
        s = m->stream;
    auto &net = m->net[e];
    for (int l = 0; l < m->hidden; ++l) {
        const void *A = l == 0 ? m->X : m->H[l - 1];
        const int lda = l == 0 ? m->in_pad : m->width;
        const Layer &L = net[l];
        MCK(m, eu3d::gemm_bf16(A, lda, L.Wb, L.in_pad, n, L.out_pad, L.in_pad, L.b, 4, nullptr, m->H[l], nullptr,
                               m->width, m->d_err, s));
    }
    const Layer &L = net[m->hidden];
    MCK(m, eu3d::gemm_bf16(m->H[m->hidden - 1], m->width, L.Wb, L.in_pad, n, L.out_pad, L.in_pad, L.b, 0, m->Y, nullptr,
                           nullptr, m->out_pad, m->d_err, s));
    return EU_OK;
}

// The training kernels' parameters for members [first, first + count), without a
// batch.
eu3d::TrainParams train_params(const eu_mlp *m, int first, int count)
{
    eu3d::TrainParams p{};
    p.n_in = m->n_in;
    p.in_pad = m->in_pad;
    p.width = m->width;
    p.hidden = m->hidden;
    p.n_out = m->n_out;
    p.out_pad = m->out_pad;
    p.params = int(m->params);
    p.first = first;
    p.members = count;
    p.in_shift = m->in_shift;
    p.in_scale = m->in_scale;
    p.out_shift = m->out_shift;
    p.out_scale = m->out_scale;
    p.loss = m->loss;
    p.err = m->d_err;
    for (int e = 0; e < m->members; ++e) {
        eu3d::TrainMember &t = p.member[e];
        t.P = m->P + e * m->params;
        t.G = m->G + e * m->params;
        t.M = m->M + e * m->params;
        t.V = m->V + e * m->params;
        for (int l = 0; l <= m->hidden; ++l) {
            const Layer &L = m->net[e][l];
            t.bias[l] = L.b;
            t.gW[l] = L.gW;
            t.gb[l] = L.gb;
            t.Wb[l] = L.Wb;
            t.slabs[l] = L.slabs;
            t.slabs_t[l] = L.slabs_t;
        }
    }
    return p;
}

// A batch of n rows of the caller's arrays, with scratch for `group` members: all
// of them (6.2 KB a row and member at 256 x 3), or, where memory is short, one, on
// which they run one at a time. (A gradient of one member takes all of them's too:
// a second allocation for the training that follows costs 0.4 ms.)
eu_status train_batch(eu_mlp *m, eu3d::TrainParams &p, const float *X, const float *T, long long rows, int n, bool drawn,
                      int &group)
{
    group = m->members;
    // whole tiles: every piece a multiple of 128 values
    const size_t rows_pad = size_t(n + eu3d::kTrainRows - 1) / eu3d::kTrainRows * eu3d::kTrainRows;
    const size_t wide = size_t(m->hidden) * m->width * rows_pad;
    const size_t bytes = wide * (4 + 2 + 2) + rows_pad * (m->in_pad + m->out_pad) * 2;
    if (m->train_bytes < bytes * group) {
        auto drop = [&] { // nothing of an earlier call uses it any more
            cudaStreamSynchronize(m->stream);
            cudaFree(m->train);
            m->train = nullptr;
            m->train_bytes = 0;
        };
        if (m->train && m->train_bytes < bytes)
            drop();
        void *fresh = nullptr;
        cudaError_t e = cudaMalloc(&fresh, bytes * group);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError(); // the launches' own check starts clean
            e = cudaSuccess;
            group = 1;
            if (!m->train && (e = cudaMalloc(&fresh, bytes)) != cudaSuccess)
                cudaGetLastError();
        }
        if (e != cudaSuccess)
            return mfail(m, e == cudaErrorMemoryAllocation ? EU_ERR_OUT_OF_MEMORY : EU_ERR_CUDA, "training scratch: %s",
                         cudaGetErrorString(e));
        if (fresh) {
            if (m->train)
                drop();
            m->train = fresh;
            m->train_bytes = bytes * group;
        }
    }
    p.X = X;
    p.T = T;
    p.rows = rows;
    p.n = n;
    p.drawn = drawn;
    for (int e = 0; e < m->members; ++e) {
        eu3d::TrainMember &t = p.member[e];
        unsigned char *at = static_cast<unsigned char *>(m->train) + e % group * bytes;
        t.ZT = reinterpret_cast<float *>(at);
        t.HT = reinterpret_cast<__nv_bfloat16 *>(at + wide * 4);
        t.dZT = t.HT + wide;
        t.XT = t.dZT + wide;
        t.dYT = t.XT + rows_pad * m->in_pad;
    }
    return EU_OK;
}

// The bf16 weights of members [first, first + count) from the fp32 masters.
eu_status refresh(eu_mlp *m, int first, int count)
{
    MCK(m, eu3d::train_adam(train_params(m, first, count), 0.0f, 0, 0, 0, 0, 0, m->stream));
    return EU_OK;
}

eu_status check_err(eu_mlp *m)
{
    int herr = 0;
    MCK(m, cudaMemcpyAsync(&herr, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    if (herr) {
        cudaMemsetAsync(m->d_err, 0, sizeof(int), m->stream);
        return mfail(m, EU_ERR_TIMEOUT, "a tensor-core pipeline wait gave up");
    }
    return EU_OK;
}

} // namespace

namespace eu3d {
bool mlp_shape(const eu_mlp *m, int *n_in, int *n_out, int *members)
{
    if (!m || !m->ready)
        return false;
    *n_in = m->n_in;
    *n_out = m->n_out;
    *members = m->members;
    return true;
}

int mlp_layers(const eu_mlp *m) { return m && m->ready ? m->hidden + 1 : 0; }

int mlp_batches(const eu_mlp *m, long long n)
{
    return m && m->ready && m->max_batch > 0 ? int((n + m->max_batch - 1) / m->max_batch) : 0;
}

bool mlp_view(const eu_mlp *m, MlpView *v)
{
    if (!m || !m->ready || !v)
        return false;
    *v = MlpView{m->device, m->n_in,  m->width,    m->hidden,   m->n_out,    m->members,  m->in_pad,
                 m->out_pad, m->stream, m->in_shift, m->in_scale, m->out_shift, m->out_scale};
    return true;
}

bool mlp_layer_view(const eu_mlp *m, int member, int layer, MlpLayerView *v)
{
    if (!m || !m->ready || !v || member < 0 || member >= m->members || layer < 0 || layer > m->hidden)
        return false;
    const Layer &L = m->net[member][layer];
    *v = MlpLayerView{L.in_pad, L.out_pad, L.Wb, L.b};
    return true;
}

eu_status mlp_fail(eu_mlp *m, eu_status s, const char *msg) { return mfail(m, s, "%s", msg); }

bool mlp_fused_params(const eu_mlp *m, FusedMlpParams *p)
{
    if (!m || !m->ready || !m->fused || !p)
        return false;
    *p = FusedMlpParams{};
    p->members = m->members;
    p->layers = m->hidden + 1;
    p->n_in = m->n_in;
    p->in_pad = m->in_pad;
    p->width = m->width;
    p->out_pad = m->out_pad;
    p->n_out = m->n_out;
    p->slabs = m->slabs;
    for (int e = 0; e < m->members; ++e)
        for (int l = 0; l <= m->hidden; ++l) {
            p->off[e][l] = m->slab_off[e][l];
            p->bias[e][l] = m->net[e][l].b;
        }
    p->in_shift = m->in_shift;
    p->in_scale = m->in_scale;
    p->out_shift = m->out_shift;
    p->out_scale = m->out_scale;
    return true;
}

eu_status mlp_predict_queue(eu_mlp *m, const float *feat, const int *count_dev, int max_rows, float *out,
                            long long s_row, long long s_mem, cudaStream_t s)
{
    FusedMlpParams p;
    if (!mlp_fused_params(m, &p))
        return mfail(m, EU_ERR_UNSUPPORTED, "the model's shape has no fused inference kernel");
    const int tiles = (max_rows + 127) / 128;
    const int grid = eu3d::fused_grid(tiles, m->sms);
    MCK(m, eu3d::mlp_fused(p, feat, m->n_in, 0, count_dev, max_rows, out, s_row, s_mem, m->d_err, grid, s));
    return EU_OK;
}

bool mlp_has_fused(const eu_mlp *m) { return m && m->ready && m->fused; }

int *mlp_error_flag(eu_mlp *m) { return m ? m->d_err : nullptr; }

cudaStream_t mlp_stream(const eu_mlp *m) { return m ? m->stream : nullptr; }

eu_status mlp_predict_stream(eu_mlp *m, const float *X, long long n, float *out, cudaStream_t s)
{
    for (long long r0 = 0; r0 < n; r0 += m->max_batch) {
        const int nb = int(n - r0 < m->max_batch ? n - r0 : m->max_batch);
        MCK(m, eu3d::pack_features(X + r0 * m->n_in, nb, m->n_in, m->in_shift, m->in_scale, m->X, m->in_pad,
                                   s));
        for (int e = 0; e < m->members; ++e) {
            eu_status st = forward(m, e, nb, s);
            if (st != EU_OK)
                return st;
            MCK(m, eu3d::unscale_outputs(m->Y, nb, m->out_pad, m->n_out, m->out_shift, m->out_scale,
                                         out + ((long long)e * n + r0) * m->n_out, s));
        }
    }
    return EU_OK;
}
} // namespace eu3d

extern "C" {

eu_status eu_mlp_create(int device, eu_mlp **out)
{
    if (!out)
        return EU_ERR_INVALID_ARGUMENT;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev)
        return EU_ERR_CUDA;
    eu_mlp *m = new (std::nothrow) eu_mlp;
    if (!m)
        return EU_ERR_OUT_OF_MEMORY;
    m->device = device;
    if (cudaSetDevice(device) != cudaSuccess ||
        cudaDeviceGetAttribute(&m->sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess ||
        cudaMalloc(&m->d_err, sizeof(int)) != cudaSuccess || cudaMemset(m->d_err, 0, sizeof(int)) != cudaSuccess) {
        eu_mlp_destroy(m);
        return EU_ERR_CUDA;
    }
    *out = m;
    return EU_OK;
}

eu_status eu_mlp_destroy(eu_mlp *m)
{
    if (!m)
        return EU_ERR_INVALID_ARGUMENT;
    cudaSetDevice(m->device);
    if (m->stream)
        cudaStreamSynchronize(m->stream);
    free_all(m);
    if (m->d_err)
        cudaFree(m->d_err);
    if (m->stream)
        cudaStreamDestroy(m->stream);
    delete m;
    return EU_OK;
}

const char *eu_mlp_last_error(const eu_mlp *m) { return m ? m->err.c_str() : "null handle"; }

eu_status eu_mlp_gemm(eu_mlp *m, const void *A, int lda, const void *B, int ldb, int M, int N, int K, const float *bias,
                      int act, float *Cf, void *Cb, float *Cpre, int ldc, void *stream)
{
    if (!m)
        return EU_ERR_INVALID_ARGUMENT;
    if (!A || !B || M < 0 || N <= 0 || K <= 0 || (K % 16) != 0 || (lda % 8) != 0 || (ldb % 8) != 0 || lda < K ||
        ldb < K || ldc < N || (!Cf && !Cb && !Cpre) || (act != 0 && act != 1))
        return mfail(m, EU_ERR_INVALID_ARGUMENT, "gemm: K %% 16, lda/ldb %% 8 and an output are required");
    if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15)
        return mfail(m, EU_ERR_INVALID_ARGUMENT, "gemm: operands must be 16-byte aligned");
    if (M == 0)
        return EU_OK;
    cudaSetDevice(m->device);
    cudaStream_t s = stream ? static_cast<cudaStream_t>(stream) : m->stream;
    cudaError_t e = eu3d::gemm_bf16(A, lda, B, ldb, M, N, K, bias, act, Cf, Cb, Cpre, ldc, m->d_err, s);
    if (e != cudaSuccess)
        return mfail(m, EU_ERR_CUDA, "gemm launch: %s", cudaGetErrorString(e));
    int herr = 0;
    e = cudaMemcpyAsync(&herr, m->d_err, sizeof(int), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess)
        e = cudaStreamSynchronize(s);
    if (e != cudaSuccess)
        return mfail(m, EU_ERR_CUDA, "gemm: %s", cudaGetErrorString(e));
    if (herr) {
        cudaMemsetAsync(m->d_err, 0, sizeof(int), s);
        return mfail(m, EU_ERR_TIMEOUT, "gemm: a tensor-core pipeline wait gave up");
    }
    return EU_OK;
}

eu_status eu_mlp_init(eu_mlp *m, int n_in, int width, int hidden_layers, int n_out, int members, int max_batch,
                      unsigned seed)
{
    if (!m)
        return EU_ERR_INVALID_ARGUMENT;
    if (n_in < 1 || n_in > 256 || width < 16 || width > 256 || (width % 16) || hidden_layers < 1 || hidden_layers > 8 ||
        n_out < 1 || n_out > 256 || members < 1 || members > 8 || max_batch < 16 || (max_batch % 16))
        return mfail(m, EU_ERR_INVALID_ARGUMENT, "mlp sizes out of range");
    cudaSetDevice(m->device);
    free_all(m);
    m->n_in = n_in;
    m->width = width;
    m->hidden = hidden_layers;
    m->n_out = n_out;
    m->members = members;
    m->max_batch = max_batch;
    m->in_pad = pad16(n_in);
    m->out_pad = pad16(n_out);
    m->adam_t = 0;
    std::mt19937_64 rng(seed);
    m->net.assign(members, std::vector<Layer>(hidden_layers + 1));
    m->params = 0;
    long long slab_values = 0;
    for (int l = 0; l <= hidden_layers; ++l) {
        const long long in = pad16(l == 0 ? n_in : width), out = pad16(l == hidden_layers ? n_out : width);
        m->params += out * in + out;
        slab_values += out * in;
    }
    const size_t all = size_t(m->params) * members * 4;
    __nv_bfloat16 *Wb = nullptr, *slabs_t = nullptr;
    MCK(m, malloc_zero(m, &m->P, all));
    MCK(m, malloc_zero(m, &m->G, all));
    MCK(m, malloc_zero(m, &m->M, all));
    MCK(m, malloc_zero(m, &m->V, all));
    MCK(m, malloc_zero(m, &Wb, size_t(slab_values) * members * 2));
    MCK(m, malloc_zero(m, &m->slabs, size_t(slab_values) * members * 2));
    MCK(m, malloc_zero(m, &slabs_t, size_t(slab_values) * members * 2));
    std::vector<float> init(size_t(m->params) * members, 0.0f);
    long long slab = 0;
    for (int e = 0; e < members; ++e) {
        long long at = 0;
        for (int l = 0; l <= hidden_layers; ++l) {
            Layer &L = m->net[e][l];
            L.in = l == 0 ? n_in : width;
            L.out = l == hidden_layers ? n_out : width;
            L.in_pad = pad16(L.in);
            L.out_pad = pad16(L.out);
            const long long nw = (long long)L.out_pad * L.in_pad, base = e * m->params + at;
            L.at = at;
            L.W = m->P + base;
            L.b = L.W + nw;
            L.gW = m->G + base;
            L.gb = L.gW + nw;
            L.Wb = Wb + slab;
            L.slabs = m->slabs + slab;
            L.slabs_t = slabs_t + slab;
            m->slab_off[e][l] = slab;
            slab += nw;
            at += nw + L.out_pad;
            // He-uniform initialisation (SiLU layers), zero biases
            const double bound = std::sqrt(6.0 / L.in) * (l == hidden_layers ? 0.5 : 1.0);
            std::uniform_real_distribution<double> u(-bound, bound);
            for (int o = 0; o < L.out; ++o)
                for (int i = 0; i < L.in; ++i) init[size_t(base) + size_t(o) * L.in_pad + i] = float(u(rng));
        }
    }
    MCK(m, cudaMemcpyAsync(m->P, init.data(), all, cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    const int B = max_batch;
    MCK(m, malloc_zero(m, &m->in_shift, size_t(m->in_pad) * 4));
    MCK(m, malloc_zero(m, &m->in_scale, size_t(m->in_pad) * 4));
    MCK(m, malloc_zero(m, &m->out_shift, size_t(m->out_pad) * 4));
    MCK(m, malloc_zero(m, &m->out_scale, size_t(m->out_pad) * 4));
    {
        std::vector<float> one(256, 1.0f);
        MCK(m, cudaMemcpyAsync(m->in_scale, one.data(), size_t(m->in_pad) * 4, cudaMemcpyHostToDevice, m->stream));
        MCK(m, cudaMemcpyAsync(m->out_scale, one.data(), size_t(m->out_pad) * 4, cudaMemcpyHostToDevice, m->stream));
        MCK(m, cudaStreamSynchronize(m->stream));
    }
    MCK(m, malloc_zero(m, &m->X, size_t(B) * m->in_pad * 2));
    m->H.assign(hidden_layers, nullptr);
    for (int l = 0; l < hidden_layers; ++l) MCK(m, malloc_zero(m, &m->H[l], size_t(B) * width * 2));
    MCK(m, malloc_zero(m, &m->Y, size_t(B) * m->out_pad * 4));
    MCK(m, malloc_zero(m, &m->loss, eu3d::kFusedMaxMembers * sizeof(float)));
    m->fused = eu3d::fused_supported(m->in_pad, width, m->out_pad, members, hidden_layers + 1);
    {
        eu_status s = refresh(m, 0, members);
        if (s != EU_OK)
            return s;
    }
    MCK(m, cudaStreamSynchronize(m->stream));
    // the no-allocation entry point's fixed array is loaded on this device now,
    // before the caller can hand its free memory to a pool of its own
    MCK(m, eu3d::noalloc_setup(m->device));
    m->ready = true;
    return EU_OK;
}

eu_status eu_mlp_set_scaling(eu_mlp *m, const float *in_shift, const float *in_scale, const float *out_shift,
                             const float *out_scale)
{
    if (!m || !in_shift || !in_scale || !out_shift || !out_scale)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    cudaSetDevice(m->device);
    MCK(m, cudaMemcpyAsync(m->in_shift, in_shift, size_t(m->n_in) * 4, cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaMemcpyAsync(m->in_scale, in_scale, size_t(m->n_in) * 4, cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaMemcpyAsync(m->out_shift, out_shift, size_t(m->n_out) * 4, cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaMemcpyAsync(m->out_scale, out_scale, size_t(m->n_out) * 4, cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    return EU_OK;
}

long long eu_mlp_num_params(const eu_mlp *m)
{
    if (!m || !m->ready)
        return 0;
    return params_per_member(m) * m->members;
}

namespace {
// The member's values without the layers' padding, in the order of the flat
// parameters, and back.
long long unpad(const eu_mlp *m, const float *padded, float *out)
{
    long long n = 0;
    for (const Layer &L : m->net[0]) {
        const float *w = padded + L.at, *b = w + (long long)L.out_pad * L.in_pad;
        for (int o = 0; o < L.out; ++o, n += L.in) std::memcpy(out + n, w + (long long)o * L.in_pad, size_t(L.in) * 4);
        std::memcpy(out + n, b, size_t(L.out) * 4);
        n += L.out;
    }
    return n;
}

long long pad(const eu_mlp *m, const float *in, float *padded)
{
    long long n = 0;
    for (const Layer &L : m->net[0]) {
        float *w = padded + L.at, *b = w + (long long)L.out_pad * L.in_pad;
        for (int o = 0; o < L.out; ++o, n += L.in) std::memcpy(w + (long long)o * L.in_pad, in + n, size_t(L.in) * 4);
        std::memcpy(b, in + n, size_t(L.out) * 4);
        n += L.out;
    }
    return n;
}
} // namespace

eu_status eu_mlp_get_params(eu_mlp *m, float *out)
{
    if (!m || !out)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    cudaSetDevice(m->device);
    std::vector<float> all(size_t(m->params) * m->members);
    MCK(m, cudaMemcpyAsync(all.data(), m->P, all.size() * 4, cudaMemcpyDeviceToHost, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    for (int e = 0; e < m->members; ++e) out += unpad(m, all.data() + e * m->params, out);
    return EU_OK;
}

eu_status eu_mlp_set_params(eu_mlp *m, const float *in)
{
    if (!m || !in)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    cudaSetDevice(m->device);
    std::vector<float> all(size_t(m->params) * m->members, 0.0f);
    for (int e = 0; e < m->members; ++e) in += pad(m, in, all.data() + e * m->params);
    MCK(m, cudaMemcpyAsync(m->P, all.data(), all.size() * 4, cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    const eu_status s = refresh(m, 0, m->members);
    if (s != EU_OK)
        return s;
    MCK(m, cudaStreamSynchronize(m->stream));
    return EU_OK;
}

eu_status eu_mlp_loss_grad(eu_mlp *m, int member, const float *X, const float *T, int n, float *loss_out,
                           float *grads_out)
{
    if (!m || !X || !T || !loss_out)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    if (member < 0 || member >= m->members || n < 16 || n > m->max_batch || (n % 16))
        return mfail(m, EU_ERR_INVALID_ARGUMENT, "member or batch size (multiple of 16 up to max_batch)");
    cudaSetDevice(m->device);
    eu3d::TrainParams p = train_params(m, member, 1);
    int group;
    eu_status s = train_batch(m, p, X, T, n, n, false, group);
    if (s != EU_OK)
        return s;
    float *g = m->G + member * m->params;
    MCK(m, cudaMemsetAsync(g, 0, size_t(m->params) * 4, m->stream));
    MCK(m, cudaMemsetAsync(m->loss + member, 0, sizeof(float), m->stream));
    MCK(m, eu3d::train_rows(p, m->stream));
    MCK(m, eu3d::train_weights(p, m->sms, m->stream));
    float sq = 0;
    std::vector<float> all(grads_out ? size_t(m->params) : 0);
    MCK(m, cudaMemcpyAsync(&sq, m->loss + member, sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if (grads_out)
        MCK(m, cudaMemcpyAsync(all.data(), g, all.size() * 4, cudaMemcpyDeviceToHost, m->stream));
    if ((s = check_err(m)) != EU_OK)
        return s;
    *loss_out = sq / float((long long)n * m->n_out);
    if (grads_out)
        unpad(m, all.data(), grads_out);
    return EU_OK;
}

eu_status eu_mlp_train(eu_mlp *m, const float *X, const float *T, long long n, int batch, int steps, float lr,
                       unsigned seed, float *mean_loss)
{
    if (!m || !X || !T)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    if (batch < 16 || batch > m->max_batch || (batch % 16) || n < batch || steps < 0 || !(lr > 0))
        return mfail(m, EU_ERR_INVALID_ARGUMENT, "batch must be a multiple of 16, <= max_batch and <= n");
    cudaSetDevice(m->device);
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    eu3d::TrainParams p = train_params(m, 0, m->members);
    int group; // members that run together
    eu_status s = train_batch(m, p, X, T, n, batch, true, group);
    if (s != EU_OK)
        return s;
    MCK(m, cudaMemsetAsync(m->G, 0, size_t(m->params) * m->members * 4, m->stream));
    for (int it = 0; it < steps; ++it) {
        ++m->adam_t;
        const float c1 = 1.0f / (1.0f - std::pow(b1, float(m->adam_t)));
        const float c2 = 1.0f / (1.0f - std::pow(b2, float(m->adam_t)));
        for (int e = 0; e < m->members; ++e)
            p.member[e].key = (unsigned long long)seed * 0x100000001B3ull + (unsigned long long)m->adam_t * 131ull + e;
        if (it + 1 == steps) // the last batch's loss is the one returned
            MCK(m, cudaMemsetAsync(m->loss, 0, size_t(m->members) * sizeof(float), m->stream));
        for (p.first = 0; p.first < m->members; p.first += group) {
            p.members = std::min(group, m->members - p.first);
            MCK(m, eu3d::train_rows(p, m->stream));
            MCK(m, eu3d::train_weights(p, m->sms, m->stream));
        }
        p.first = 0;
        p.members = m->members;
        MCK(m, eu3d::train_adam(p, lr, b1, b2, eps, c1, c2, m->stream));
    }
    std::vector<float> sq(m->members, 0.0f);
    if (steps > 0)
        MCK(m, cudaMemcpyAsync(sq.data(), m->loss, sq.size() * sizeof(float), cudaMemcpyDeviceToHost, m->stream));
    if ((s = check_err(m)) != EU_OK)
        return s;
    if (mean_loss)
        for (int e = 0; e < m->members; ++e) mean_loss[e] = float(sq[e] / double((long long)batch * m->n_out));
    return EU_OK;
}

eu_status eu_mlp_predict_fused(eu_mlp *m, const float *X, long long n, float *out)
{
    if (!m || !X || !out || n < 0 || n > 0x7fffffffLL)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    if (!m->fused)
        return mfail(m, EU_ERR_UNSUPPORTED, "the model's shape has no fused inference kernel");
    cudaSetDevice(m->device);
    eu3d::FusedMlpParams p;
    eu3d::mlp_fused_params(m, &p);
    const long long tiles = (n + 127) / 128;
    const int grid = eu3d::fused_grid(tiles, m->sms);
    MCK(m, eu3d::mlp_fused(p, X, m->n_in, int(n), nullptr, int(n), out, m->n_out, n * m->n_out, m->d_err, grid,
                           m->stream));
    return check_err(m);
}

eu_status eu_mlp_predict_fused_async(eu_mlp *m, const float *X, long long n, float *out)
{
    if (!m || !X || !out || n < 0 || n > 0x7fffffffLL)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    if (!m->fused)
        return mfail(m, EU_ERR_UNSUPPORTED, "the model's shape has no fused inference kernel");
    cudaSetDevice(m->device);
    eu3d::FusedMlpParams p;
    eu3d::mlp_fused_params(m, &p);
    const long long tiles = (n + 127) / 128;
    const int grid = eu3d::fused_grid(tiles, m->sms);
    MCK(m, eu3d::mlp_fused(p, X, m->n_in, int(n), nullptr, int(n), out, m->n_out, n * m->n_out, m->d_err, grid,
                           m->stream));
    return EU_OK;
}

eu_status eu_mlp_sync(eu_mlp *m)
{
    if (!m)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    cudaSetDevice(m->device);
    return check_err(m);
}

eu_status eu_mlp_stream(eu_mlp *m, void **stream)
{
    if (!m || !stream)
        return EU_ERR_INVALID_ARGUMENT;
    *stream = m->stream;
    return EU_OK;
}

eu_status eu_mlp_predict(eu_mlp *m, const float *X, long long n, float *out)
{
    if (!m || !X || !out || n < 0)
        return EU_ERR_INVALID_ARGUMENT;
    if (!m->ready)
        return mfail(m, EU_ERR_NOT_READY, "eu_mlp_init first");
    cudaSetDevice(m->device);
    for (long long r0 = 0; r0 < n; r0 += m->max_batch) {
        const int nb = int(n - r0 < m->max_batch ? n - r0 : m->max_batch);
        MCK(m, eu3d::pack_features(X + r0 * m->n_in, nb, m->n_in, m->in_shift, m->in_scale, m->X, m->in_pad,
                                   m->stream));
        for (int e = 0; e < m->members; ++e) {
            eu_status s = forward(m, e, nb);
            if (s != EU_OK)
                return s;
            MCK(m, eu3d::unscale_outputs(m->Y, nb, m->out_pad, m->n_out, m->out_shift, m->out_scale,
                                         out + ((long long)e * n + r0) * m->n_out, m->stream));
        }
    }
    return check_err(m);
}

} // extern "C"
