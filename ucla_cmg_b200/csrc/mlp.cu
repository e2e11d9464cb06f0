// mlp.cu -- trainer for the learned ionic step: a tanh MLP with FP32 master
// weights, trained on the GPU by the kernels in this file (tiled SGEMM for
// the forward and backward products, with the bias, tanh, tanh gradient and
// loss in their epilogues and the weight gradients split over the batch, and
// Adam).  Inference in the time loop uses the BF16 tensor-core
// kernel in surrogate.cu; these kernels are for training only.
#include <cstring>
#include <vector>
#include <random>
#include <cmath>
#include <algorithm>

#include "kernels.cuh"

namespace ep {

constexpr int GT = 64, GK = 16;   // 64x64 output tile, 16-deep k slices, 4x4 per thread

// what the product's epilogue does
enum { E_BIAS = 0, E_TANH = 1, E_DTANH = 2, E_MSE = 3, E_PART = 4 };

// Arguments beyond the operands, by epilogue:
//   E_BIAS, E_TANH  bias[n]
//   E_DTANH         h: the layer's activations, C = (A B) (1 - h^2)
//   E_MSE           bias[n]; C = 2 w (P - Y) / rows, loss += sum w (P - Y)^2 / rows
//   E_PART          C += z * cz: this k chunk's partial product; bsum (+ z * cz):
//                   the column sums of A over the chunk
struct GemmEpi {
    const float *bias, *h, *Y, *w;
    double *loss;
    float *bsum;
    long long cz;
    int kchunk;
};

// C = op(A) op(B); A: M x K (TA: K x M), B: K x N (TB: N x K).  The next k
// slice is loaded into registers while the current one is multiplied; the
// products of a network step are small (K 23 .. 128 for the activations), so
// a slice's load latency, not the multiply rate, is what a CTA would wait on.
template <bool TA, bool TB, int EPI>
__global__ void __launch_bounds__(256) k_sgemm(int M, int N, int K, const float *__restrict__ A, int lda,
                                               const float *__restrict__ B, int ldb, float *C, int ldc, GemmEpi ep) {
    __shared__ __align__(16) float As[2][GK][GT + 4];
    __shared__ __align__(16) float Bs[2][GK][GT + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * GT, n0 = blockIdx.x * GT;
    int k0 = 0, k1 = K;
    if (EPI == E_PART) {
        k0 = (int)blockIdx.z * ep.kchunk;
        k1 = min(K, k0 + ep.kchunk);
        C += (long long)blockIdx.z * ep.cz;
    }
    // a thread's four elements of a slice of either operand, neighbouring
    // threads along the operand's rows
    const int ka = TA ? tid >> 6 : tid & 15, ma = TA ? tid & 63 : tid >> 4;
    const int kb = TB ? tid & 15 : tid >> 6, nb = TB ? tid >> 4 : tid & 63;
    float ra[4], rb[4];
    auto load = [&](int k) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int gk = k + ka + (TA ? 4 * i : 0), gm = m0 + ma + (TA ? 0 : 16 * i);
            ra[i] = gm < M && gk < k1 ? __ldg(A + (TA ? (size_t)gk * lda + gm : (size_t)gm * lda + gk)) : 0.f;
            const int hk = k + kb + (TB ? 0 : 4 * i), gn = n0 + nb + (TB ? 16 * i : 0);
            rb[i] = gn < N && hk < k1 ? __ldg(B + (TB ? (size_t)gn * ldb + hk : (size_t)hk * ldb + gn)) : 0.f;
        }
    };
    auto put = [&](int buf) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            As[buf][ka + (TA ? 4 * i : 0)][ma + (TA ? 0 : 16 * i)] = ra[i];
            Bs[buf][kb + (TB ? 0 : 4 * i)][nb + (TB ? 16 * i : 0)] = rb[i];
        }
    };
    float acc[4][4] = {{0.f}}, col[4] = {0.f, 0.f, 0.f, 0.f};
    load(k0);
    int buf = 0;
    for (int k = k0; k < k1; k += GK, buf ^= 1) {
        put(buf);
        __syncthreads();                      // the slice before last is no longer read
        if (k + GK < k1) load(k + GK);
#pragma unroll
        for (int kk = 0; kk < GK; kk++) {
            const float4 a4 = *reinterpret_cast<const float4 *>(&As[buf][kk][ty * 4]);
            const float4 b4 = *reinterpret_cast<const float4 *>(&Bs[buf][kk][tx * 4]);
            const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
            if (EPI == E_PART && blockIdx.x == 0)
#pragma unroll
                for (int i = 0; i < 4; i++) col[i] += a[i];
        }
    }
    double l = 0.0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
        if (EPI == E_PART && blockIdx.x == 0 && tx == 0) ep.bsum[(long long)blockIdx.z * ep.cz + gm] = col[i];
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            const size_t at = (size_t)gm * ldc + gn;
            float v = acc[i][j];
            if (EPI == E_BIAS || EPI == E_TANH || EPI == E_MSE) v += ep.bias[gn];
            if (EPI == E_TANH) v = tanhf(v);
            if (EPI == E_DTANH) { const float h = ep.h[at]; v *= 1.f - h * h; }
            if (EPI == E_MSE) {
                const float d = v - ep.Y[at], wj = ep.w ? ep.w[gn] : 1.f;
                v = 2.f * wj * d / (float)M;
                l += (double)wj * (double)d * (double)d / (double)M;
            }
            C[at] = v;
        }
    }
    if (EPI == E_MSE) {
        for (int o = 16; o > 0; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
        if ((tid & 31) == 0 && l != 0.0) atomicAdd(ep.loss, l);
    }
}

template <bool TA, bool TB, int EPI>
static void sgemm(int M, int N, int K, const float *A, int lda, const float *B, int ldb, float *C, int ldc,
                  const GemmEpi &ep, cudaStream_t s) {
    dim3 grid((N + GT - 1) / GT, (M + GT - 1) / GT, EPI == E_PART ? (K + ep.kchunk - 1) / ep.kchunk : 1);
    k_sgemm<TA, TB, EPI><<<grid, 256, 0, s>>>(M, N, K, A, lda, B, ldb, C, ldc, ep);
}

// the weight gradients' partial products summed over the chunks, in order
__global__ void k_sum_parts(int n, int parts, const float *__restrict__ p, float *out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float s = 0.f;
#pragma unroll 8
    for (int z = 0; z < parts; z++) s += __ldg(p + (size_t)z * n + i);
    out[i] = s;
}

__global__ void k_adam(int n, float *p, const float *g, float *m, float *v, float lr, float b1, float b2,
                       float eps, float c1, float c2) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi;
    const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    p[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
}

}  // namespace ep

using namespace ep;

struct ep_mlp {
    int device = 0;
    int L = 0;                       // number of weight layers
    std::vector<int> dims;           // L + 1
    std::vector<size_t> woff, boff;  // offsets into the flat parameter vector
    size_t np = 0;
    float *p = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
    float *act = nullptr;            // activations of the largest batch (layers 1..L); the workspace's start
    float *dlt = nullptr, *dlt2 = nullptr;
    float *w_out = nullptr;
    float *part = nullptr;           // the gradients of each chunk of a batch's rows
    double *loss = nullptr;
    int cap = 0;                     // batch capacity of act/dlt
    long long t = 0;                 // Adam step
    int maxw = 0;
};

// Chunks that a batch's rows are cut into for the weight gradients, whose
// products are small (128 x 128) and deep (the batch): with one CTA per 64 x 64
// tile four CTAs walked all 8192 rows.  At least 32 rows a chunk, at most 64
// chunks, and 16M floats of partial gradients.
static int grad_parts(const ep_mlp *m, int B) {
    const long long most = std::max<long long>(1, (16ll << 20) / (long long)m->np);
    return (int)std::min<long long>(std::min<long long>(64, most), (B + 31) / 32);
}

// one allocation for the activations, the two deltas and the partial gradients
static int mlp_reserve(ep_mlp *m, int batch) {
    if (batch <= m->cap) return EP_OK;
    size_t tot = 0;
    for (int l = 1; l <= m->L; l++) tot += (size_t)m->dims[l];
    const size_t act = tot * batch, dlt = (size_t)m->maxw * batch, part = m->np * (size_t)grad_parts(m, batch);
    cudaFree(m->act);
    m->act = m->dlt = m->dlt2 = m->part = nullptr;
    m->cap = 0;
    if (cudaMalloc(&m->act, sizeof(float) * (act + 2 * dlt + part)) != cudaSuccess) {
        cudaGetLastError();
        set_error("MLP workspace allocation failed (batch %d)", batch);
        return EP_ERR_NOMEM;
    }
    m->dlt = m->act + act;
    m->dlt2 = m->dlt + dlt;
    m->part = m->dlt2 + dlt;
    m->cap = batch;
    return EP_OK;
}

// activation of layer l (1..L) for a batch of `cap` rows
static float *act_of(ep_mlp *m, int l) {
    size_t off = 0;
    for (int k = 1; k < l; k++) off += (size_t)m->dims[k] * m->cap;
    return m->act + off;
}

// hidden layers 1 .. L-1
static void forward_hidden(ep_mlp *m, const float *X, int B, cudaStream_t s) {
    const float *h = X;
    for (int l = 1; l < m->L; l++) {
        float *z = act_of(m, l);
        GemmEpi ep{};
        ep.bias = m->p + m->boff[l - 1];
        sgemm<false, true, E_TANH>(B, m->dims[l], m->dims[l - 1], h, m->dims[l - 1], m->p + m->woff[l - 1],
                                   m->dims[l - 1], z, m->dims[l], ep, s);
        h = z;
    }
}
static const float *last_hidden(ep_mlp *m, const float *X) { return m->L > 1 ? act_of(m, m->L - 1) : X; }

extern "C" {

int ep_mlp_create(int32_t n_layers, const int32_t *dims, uint64_t seed, int device, ep_mlp **out) {
    EP_CHECK_ARG(out && dims && n_layers >= 1 && n_layers <= 8, "bad MLP shape");
    for (int l = 0; l <= n_layers; l++) EP_CHECK_ARG(dims[l] > 0 && dims[l] <= 4096, "bad MLP width");
    EP_CUDA(cudaSetDevice(device));
    ep_mlp *m = new ep_mlp();
    m->device = device;
    m->L = n_layers;
    m->dims.assign(dims, dims + n_layers + 1);
    for (int l = 0; l < n_layers; l++) {
        m->woff.push_back(m->np);
        m->np += (size_t)dims[l + 1] * dims[l];
        m->boff.push_back(m->np);
        m->np += (size_t)dims[l + 1];
        m->maxw = std::max(m->maxw, std::max(dims[l], dims[l + 1]));
    }
    // Xavier-uniform weights, zero biases
    std::vector<float> h(m->np, 0.f);
    std::mt19937_64 rng(seed);
    for (int l = 0; l < n_layers; l++) {
        const float a = std::sqrt(6.f / (float)(dims[l] + dims[l + 1]));
        std::uniform_real_distribution<float> U(-a, a);
        for (size_t k = 0; k < (size_t)dims[l + 1] * dims[l]; k++) h[m->woff[l] + k] = U(rng);
    }
    if (cudaMalloc(&m->p, sizeof(float) * m->np) != cudaSuccess ||
        cudaMalloc(&m->g, sizeof(float) * m->np) != cudaSuccess ||
        cudaMalloc(&m->m, sizeof(float) * m->np) != cudaSuccess ||
        cudaMalloc(&m->v, sizeof(float) * m->np) != cudaSuccess ||
        cudaMalloc(&m->w_out, sizeof(float) * dims[n_layers]) != cudaSuccess ||
        cudaMalloc(&m->loss, sizeof(double)) != cudaSuccess) {
        cudaGetLastError();
        ep_mlp_destroy(m);
        set_error("MLP allocation failed");
        return EP_ERR_NOMEM;
    }
    cudaMemcpy(m->p, h.data(), sizeof(float) * m->np, cudaMemcpyHostToDevice);
    cudaMemset(m->g, 0, sizeof(float) * m->np);
    cudaMemset(m->m, 0, sizeof(float) * m->np);
    cudaMemset(m->v, 0, sizeof(float) * m->np);
    *out = m;
    return EP_OK;
}

void ep_mlp_destroy(ep_mlp *m) {
    if (!m) return;
    cudaFree(m->p); cudaFree(m->g); cudaFree(m->m); cudaFree(m->v);
    cudaFree(m->act); cudaFree(m->w_out); cudaFree(m->loss);
    delete m;
}

int ep_mlp_num_params(const ep_mlp *m) { return m ? (int)m->np : EP_ERR_ARG; }

int ep_mlp_get_params(ep_mlp *m, float *out) {
    EP_CHECK_ARG(m && out, "null argument");
    EP_CUDA(cudaMemcpy(out, m->p, sizeof(float) * m->np, cudaMemcpyDeviceToHost));
    return EP_OK;
}

int ep_mlp_set_params(ep_mlp *m, const float *in) {
    EP_CHECK_ARG(m && in, "null argument");
    EP_CUDA(cudaMemcpy(m->p, in, sizeof(float) * m->np, cudaMemcpyHostToDevice));
    EP_CUDA(cudaMemset(m->m, 0, sizeof(float) * m->np));
    EP_CUDA(cudaMemset(m->v, 0, sizeof(float) * m->np));
    m->t = 0;
    return EP_OK;
}

int ep_mlp_forward(ep_mlp *m, const float *X, float *Y, int32_t B, void *stream) {
    EP_CHECK_ARG(m && X && Y && B > 0, "bad arguments");
    int rc = mlp_reserve(m, B);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    forward_hidden(m, X, B, s);
    const int L = m->L, nin = m->dims[L - 1], nout = m->dims[L];
    GemmEpi ep{};
    ep.bias = m->p + m->boff[L - 1];
    // a single layer goes through the workspace: Y may be X
    float *out = L > 1 ? Y : act_of(m, 1);
    sgemm<false, true, E_BIAS>(B, nout, nin, last_hidden(m, X), nin, m->p + m->woff[L - 1], nin, out, nout, ep, s);
    if (L == 1) EP_CUDA(cudaMemcpyAsync(Y, out, sizeof(float) * (size_t)B * nout, cudaMemcpyDeviceToDevice, s));
    EP_CUDA(cudaGetLastError());
    return EP_OK;
}

int ep_mlp_loss_grad(ep_mlp *m, const float *X, const float *Y, const float *w_out_host, int32_t B,
                     double *loss, float *grad_host, void *stream) {
    EP_CHECK_ARG(m && X && Y && B > 0, "bad arguments");
    int rc = mlp_reserve(m, B);
    if (rc) return rc;
    cudaStream_t s = (cudaStream_t)stream;
    const int L = m->L, dout = m->dims[L];
    if (w_out_host) EP_CUDA(cudaMemcpyAsync(m->w_out, w_out_host, sizeof(float) * dout, cudaMemcpyHostToDevice, s));
    const int parts = grad_parts(m, B);
    forward_hidden(m, X, B, s);
    EP_CUDA(cudaMemsetAsync(m->loss, 0, sizeof(double), s));
    float *d = m->dlt, *d2 = m->dlt2;
    {
        // the output layer with the loss and its gradient
        GemmEpi ep{};
        ep.bias = m->p + m->boff[L - 1];
        ep.Y = Y;
        ep.w = w_out_host ? m->w_out : nullptr;
        ep.loss = m->loss;
        const int nin = m->dims[L - 1];
        sgemm<false, true, E_MSE>(B, dout, nin, last_hidden(m, X), nin, m->p + m->woff[L - 1], nin, d, dout, ep, s);
    }
    for (int l = L; l >= 1; l--) {
        const float *hprev = l > 1 ? act_of(m, l - 1) : X;
        const int nout = m->dims[l], nin = m->dims[l - 1];
        // dW_l = delta^T hprev  (nout x nin), db_l = colsum(delta), a part per chunk of rows
        GemmEpi ep{};
        ep.bsum = m->part + m->boff[l - 1];
        ep.cz = (long long)m->np;
        ep.kchunk = (B + parts - 1) / parts;
        sgemm<true, false, E_PART>(nout, nin, B, d, nout, hprev, nin, m->part + m->woff[l - 1], nin, ep, s);
        if (l > 1) {
            // delta_{l-1} = (delta W_l) * (1 - h_{l-1}^2)
            GemmEpi eb{};
            eb.h = hprev;
            sgemm<false, false, E_DTANH>(B, nin, nout, d, nout, m->p + m->woff[l - 1], nin, d2, nin, eb, s);
            std::swap(d, d2);
        }
    }
    const int used = (B + (B + parts - 1) / parts - 1) / ((B + parts - 1) / parts);    // chunks that have rows
    k_sum_parts<<<(int)((m->np + 255) / 256), 256, 0, s>>>((int)m->np, used, m->part, m->g);
    EP_CUDA(cudaGetLastError());
    if (loss) {
        EP_CUDA(cudaMemcpyAsync(loss, m->loss, sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    if (grad_host) EP_CUDA(cudaMemcpyAsync(grad_host, m->g, sizeof(float) * m->np, cudaMemcpyDeviceToHost, s));
    if (loss || grad_host) EP_CUDA(cudaStreamSynchronize(s));
    return EP_OK;
}

int ep_mlp_adam_step(ep_mlp *m, float lr, float beta1, float beta2, float eps) {
    EP_CHECK_ARG(m, "null trainer");
    m->t++;
    const float c1 = 1.f - std::pow(beta1, (float)m->t), c2 = 1.f - std::pow(beta2, (float)m->t);
    k_adam<<<(int)((m->np + 255) / 256), 256>>>((int)m->np, m->p, m->g, m->m, m->v, lr, beta1, beta2, eps, c1, c2);
    EP_CUDA(cudaGetLastError());
    return EP_OK;
}

}  // extern "C"
