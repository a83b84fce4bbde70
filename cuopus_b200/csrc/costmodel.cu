// Learned cost model of the decode scheduler: per-chain features from the
// packets' TOC bytes, and an FP32 multilayer perceptron (16 -> 64 -> 64 -> 1,
// ReLU) that predicts the log decode time of a chain, trained and evaluated
// with the kernels below.  The queue schedule of the decoder visits chains in
// decreasing predicted cost (longest first); the packet-count order is the
// fallback.  None of this changes a decoded sample: it only orders the work.
//
// Parameter layout (floats, one contiguous device buffer of MLP_NPARAM):
//   W1[16][64] | b1[64] | W2[64][64] | b2[64] | w3[64] | b3
// Training is full-batch Adam on the mean squared error.  Gradients are
// reduced deterministically: one kernel stores each sample's activations and
// back-propagated signals, a second sums them over samples in index order
// for every parameter (no atomics), so a training run is reproducible.
#include <cuda_runtime.h>
#include <stdint.h>
#include <string.h>

#include <vector>

#include "../../include/cuopus.h"

namespace {

constexpr int F = CUOPUS_MLP_FEATURES;   // 16
constexpr int H = CUOPUS_MLP_HIDDEN;     // 64
constexpr int OFF_W1 = 0;
constexpr int OFF_B1 = OFF_W1 + F * H;
constexpr int OFF_W2 = OFF_B1 + H;
constexpr int OFF_B2 = OFF_W2 + H * H;
constexpr int OFF_W3 = OFF_B2 + H;
constexpr int OFF_B3 = OFF_W3 + H;
constexpr int NPARAM = OFF_B3 + 1;
static_assert(NPARAM == CUOPUS_MLP_NPARAM, "parameter layout");
// per-sample record of the training forward/backward pass
constexpr int R_X = 0, R_H1 = R_X + F, R_G1 = R_H1 + H, R_H2 = R_G1 + H, R_G2 = R_H2 + H, R_D = R_G2 + H;
constexpr int REC = R_D + 1;

// ------------------------------------------------------------------ features

// TOC of RFC 6716 section 3.1: config = toc >> 3.
__device__ __forceinline__ int toc_mode(int config) { return config < 12 ? 0 : (config < 16 ? 1 : 2); }
__device__ __forceinline__ int toc_qms(int config)   // frame duration in quarter milliseconds
{
    if (config < 12) return (config & 3) == 0 ? 40 : (config & 3) == 1 ? 80 : (config & 3) == 2 ? 160 : 240;
    if (config < 16) return (config & 1) ? 80 : 40;
    return 10 << (config & 3);
}
__device__ __forceinline__ int toc_bw(int config)   // 0 NB, 1 MB, 2 WB, 3 SWB, 4 FB
{
    if (config < 12) return config >> 2;
    if (config < 16) return config < 14 ? 3 : 4;
    int b = (config - 16) >> 2;          // NB, WB, SWB, FB
    return b == 0 ? 0 : b + 1;
}

// Features of 32 chains a block, G lanes for each; feat[c * 16 + k].  A packet
// costs two dependent loads (offset and length, then its TOC bytes), so a chain's
// packets go to its lanes, 2 G in flight; one thread per chain walked them one
// after the other (4096 chains of 0.5-2 s, features and predictions: 617 us, 66
// now).  The sums are whole numbers, so their order does not matter.  Then each
// warp works out one feature of all 32 chains at a time: with a chain's sixteen
// in a warp of its own, five lanes of which took logarithms, 40,000 chains of one
// packet took 64 us a call, one thread per chain 28, this 28.
template <int G>
__global__ void __launch_bounds__(32 * G)
k_chain_features(const uint8_t *__restrict__ data, const uint64_t *__restrict__ off, const uint32_t *__restrict__ len,
                 const uint32_t *__restrict__ first, const uint32_t *__restrict__ npkts,
                 const uint8_t *__restrict__ channels, int nchains, float *__restrict__ feat)
{
    enum { BYTES, FRAMES, Q, SILK, HYBRID, CELT, F25, F5, F10, F20, F40, BW, STEREO, SUMS };
    __shared__ unsigned long long sums[SUMS][32];
    const int lane = threadIdx.x % G, own = threadIdx.x / G;
    const long long c0 = (long long)blockIdx.x * 32, c = c0 + own;
    unsigned long long sum[SUMS] = {};
    const uint32_t n = c < nchains ? npkts[c] : 0;
    const uint64_t p0 = n ? first[c] : 0;
    // two packets a step, their loads side by side
    for (uint64_t k = lane; k < n; k += 2 * G) {
        uint32_t L[2], toc[2], count[2];
        uint64_t at[2];
#pragma unroll
        for (int u = 0; u < 2; u++) {
            const bool in = k + u * G < n;
            L[u] = in ? len[p0 + k + u * G] : 0;
            at[u] = in ? off[p0 + k + u * G] : 0;
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            toc[u] = L[u] > 0 ? data[at[u]] : 0;
            count[u] = L[u] > 1 ? data[at[u] + 1] & 63 : 0;
        }
#pragma unroll
        for (int u = 0; u < 2; u++) {
            if (!L[u]) continue;
            const int cfg = toc[u] >> 3, code = toc[u] & 3;
            const int nf = code == 0 ? 1 : code < 3 ? 2 : count[u];
            const int qms = toc_qms(cfg), mode = toc_mode(cfg);
            sum[BYTES] += L[u];
            sum[FRAMES] += nf;
            sum[Q] += (unsigned)(nf * qms);
            sum[SILK] += mode == 0 ? nf : 0;
            sum[HYBRID] += mode == 1 ? nf : 0;
            sum[CELT] += mode == 2 ? nf : 0;
            sum[F25] += qms == 10 ? nf : 0;
            sum[F5] += qms == 20 ? nf : 0;
            sum[F10] += qms == 40 ? nf : 0;
            sum[F20] += qms == 80 ? nf : 0;
            sum[F40] += qms > 80 ? nf : 0;
            sum[BW] += (unsigned)(nf * toc_bw(cfg));
            sum[STEREO] += (toc[u] >> 2) & 1;
        }
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < SUMS; i++) {
#pragma unroll
        for (int o = G / 2; o > 0; o >>= 1) sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], o);
        if (lane == 0) sums[i][own] = sum[i];
    }
    __syncthreads();
    // feature k (the same on all lanes of the warp) of chain c0 + j: a logarithm, the
    // channels, or a fraction
    for (int i = threadIdx.x; i < 32 * F; i += 32 * G) {
        const int k = i >> 5, j = i & 31;
        if (c0 + j >= nchains) continue;
        float v;
        if (k < 4 || k == 15) {
            const double bytes = (double)sums[BYTES][j], secs = (double)sums[Q][j] / 4000.0;
            const double x = k == 0 ? (double)npkts[c0 + j] : k == 1 ? bytes : k == 2 ? (double)sums[FRAMES][j]
                           : k == 3 ? secs : secs > 0 ? bytes / secs : 0.0;
            v = (float)log1p(x);
        } else if (k == 4) {
            v = (float)(channels[c0 + j] - 1);
        } else if (k < 14) {
            const double frames = (double)sums[FRAMES][j], fr = frames > 0 ? 1.0 / frames : 0.0;
            v = k < 13 ? (float)((double)sums[SILK + k - 5][j] * fr) : (float)((double)sums[BW][j] * fr * 0.25);
        } else {
            const uint32_t pk = npkts[c0 + j];
            v = (float)(pk ? (double)sums[STEREO][j] / pk : 0.0);
        }
        feat[(size_t)(c0 + j) * F + k] = v;
    }
}

// ------------------------------------------------------------------ network

// Forward pass of one sample with the weights staged in shared memory.
// Returns the output; h1 / h2 receive the post-ReLU activations.
__device__ __forceinline__ float mlp_forward(const float *w, const float *x, float *h1, float *h2)
{
#pragma unroll 4
    for (int j = 0; j < H; j++) {
        float a = w[OFF_B1 + j];
#pragma unroll
        for (int i = 0; i < F; i++) a = fmaf(x[i], w[OFF_W1 + i * H + j], a);
        h1[j] = a > 0.f ? a : 0.f;
    }
    for (int j = 0; j < H; j++) {
        float a = w[OFF_B2 + j];
#pragma unroll 8
        for (int k = 0; k < H; k++) a = fmaf(h1[k], w[OFF_W2 + k * H + j], a);
        h2[j] = a > 0.f ? a : 0.f;
    }
    float y = w[OFF_B3];
#pragma unroll 8
    for (int j = 0; j < H; j++) y = fmaf(h2[j], w[OFF_W3 + j], y);
    return y;
}

__device__ void stage_weights(float *ws, const float *__restrict__ params)
{
    for (int i = threadIdx.x; i < NPARAM; i += blockDim.x) ws[i] = params[i];
    __syncthreads();
}

// Predictions of PRED_SAMPLES samples per block, one thread per hidden neuron:
// the neuron's weights are read once, coalesced, into registers and serve all
// of the block's samples, whose activations are exchanged through shared
// memory.  Every sum runs in mlp_forward's order.  (One thread per sample, with
// the activations in local memory and 21 KB of weights staged per 128
// samples, was most of the chip idle at the sizes of a batch.)
enum { PRED_SAMPLES = 16 };
__global__ void __launch_bounds__(H) k_mlp_predict(const float *__restrict__ params, const float *__restrict__ X, int n,
                                                   float *__restrict__ y)
{
    __shared__ float xs[PRED_SAMPLES][F], h1[PRED_SAMPLES][H + 1], h2[PRED_SAMPLES][H + 1];
    const int j = threadIdx.x, s0 = blockIdx.x * PRED_SAMPLES;
    const int cnt = n - s0 < PRED_SAMPLES ? n - s0 : PRED_SAMPLES;
    for (int i = j; i < PRED_SAMPLES * F; i += H) xs[i / F][i % F] = i < cnt * F ? X[(size_t)s0 * F + i] : 0.f;
    float w1[F], w2[H];
#pragma unroll
    for (int i = 0; i < F; i++) w1[i] = params[OFF_W1 + i * H + j];
#pragma unroll
    for (int k = 0; k < H; k++) w2[k] = params[OFF_W2 + k * H + j];
    const float b1 = params[OFF_B1 + j], b2 = params[OFF_B2 + j];
    __syncthreads();
#pragma unroll 4
    for (int s = 0; s < PRED_SAMPLES; s++) {
        float a = b1;
#pragma unroll
        for (int i = 0; i < F; i++) a = fmaf(xs[s][i], w1[i], a);
        h1[s][j] = a > 0.f ? a : 0.f;
    }
    __syncthreads();
#pragma unroll 4
    for (int s = 0; s < PRED_SAMPLES; s++) {
        float a = b2;
#pragma unroll
        for (int k = 0; k < H; k++) a = fmaf(h1[s][k], w2[k], a);
        h2[s][j] = a > 0.f ? a : 0.f;
    }
    __syncthreads();
    if (j < cnt) {
        float v = params[OFF_B3];
#pragma unroll 8
        for (int k = 0; k < H; k++) v = fmaf(h2[j][k], params[OFF_W3 + k], v);
        y[s0 + j] = v;
    }
}

// Forward + back-propagated signals of one sample for the loss
// L = mean_s (y_s - t_s)^2: rec[s] = {x, h1, g1, h2, g2, dL/dy}, with
// g2 = dL/d(pre-activation 2) and g1 = dL/d(pre-activation 1).
__global__ void k_mlp_backprop(const float *__restrict__ params, const float *__restrict__ X,
                               const float *__restrict__ T, int n, float *__restrict__ rec, float *__restrict__ sqerr)
{
    extern __shared__ float ws[];
    stage_weights(ws, params);
    int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    float x[F], h1[H], h2[H];
#pragma unroll
    for (int i = 0; i < F; i++) x[i] = X[(size_t)s * F + i];
    float y = mlp_forward(ws, x, h1, h2);
    float e = y - T[s];
    float d = 2.f * e / (float)n;
    float *r = rec + (size_t)s * REC;
#pragma unroll
    for (int i = 0; i < F; i++) r[R_X + i] = x[i];
    float g2[H];
    for (int j = 0; j < H; j++) {
        g2[j] = h2[j] > 0.f ? d * ws[OFF_W3 + j] : 0.f;
        r[R_H1 + j] = h1[j];
        r[R_H2 + j] = h2[j];
        r[R_G2 + j] = g2[j];
    }
    for (int k = 0; k < H; k++) {
        float a = 0.f;
        if (h1[k] > 0.f) {
#pragma unroll 8
            for (int j = 0; j < H; j++) a = fmaf(ws[OFF_W2 + k * H + j], g2[j], a);
        }
        r[R_G1 + k] = a;
    }
    r[R_D] = d;
    sqerr[s] = e * e;
}

// One thread per parameter: its gradient summed over samples in index order.
// Thread NPARAM also sums the squared errors into *loss.
__global__ void k_mlp_reduce(const float *__restrict__ rec, const float *__restrict__ sqerr, int n,
                             float *__restrict__ grad, float *__restrict__ loss)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p > NPARAM) return;
    if (p == NPARAM) {
        float a = 0.f;
        for (int s = 0; s < n; s++) a += sqerr[s];
        *loss = a / (float)n;
        return;
    }
    int ca, cb;   // gradient = sum_s rec[s][ca] * rec[s][cb] (cb < 0: rec[s][ca] alone)
    if (p < OFF_B1) { ca = R_X + p / H; cb = R_G1 + p % H; }
    else if (p < OFF_W2) { ca = R_G1 + (p - OFF_B1); cb = -1; }
    else if (p < OFF_B2) { ca = R_H1 + (p - OFF_W2) / H; cb = R_G2 + (p - OFF_W2) % H; }
    else if (p < OFF_W3) { ca = R_G2 + (p - OFF_B2); cb = -1; }
    else if (p < OFF_B3) { ca = R_H2 + (p - OFF_W3); cb = R_D; }
    else { ca = R_D; cb = -1; }
    float a = 0.f;
    if (cb < 0)
        for (int s = 0; s < n; s++) a += rec[(size_t)s * REC + ca];
    else
        for (int s = 0; s < n; s++) a = fmaf(rec[(size_t)s * REC + ca], rec[(size_t)s * REC + cb], a);
    grad[p] = a;
}

// Adam (beta1 0.9, beta2 0.999, eps 1e-8).  `t` counts the steps taken on
// the device (k_tick advances it after each update), so a captured graph of
// several steps stays correct on replay.
__global__ void k_adam(float *__restrict__ params, const float *__restrict__ grad, float *__restrict__ m,
                       float *__restrict__ v, const int *__restrict__ t, float lr)
{
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= NPARAM) return;
    float step = (float)(*t + 1);
    float g = grad[p];
    float mi = 0.9f * m[p] + 0.1f * g;
    float vi = 0.999f * v[p] + 0.001f * g * g;
    m[p] = mi;
    v[p] = vi;
    float mh = mi / (1.f - powf(0.9f, step));
    float vh = vi / (1.f - powf(0.999f, step));
    params[p] -= lr * mh / (sqrtf(vh) + 1e-8f);
}

__global__ void k_tick(int *t) { *t += 1; }

const int THREADS = 128;
const size_t SMEM = NPARAM * sizeof(float);

int set_err(char *errbuf, size_t errcap, int rc, const char *msg, cudaError_t e)
{
    if (errbuf && errcap) {
        size_t n = strlen(msg);
        const char *es = cudaGetErrorString(e);
        size_t m = strlen(es);
        size_t k = 0;
        for (size_t i = 0; i < n && k + 1 < errcap; i++) errbuf[k++] = msg[i];
        if (k + 2 < errcap) { errbuf[k++] = ':'; errbuf[k++] = ' '; }
        for (size_t i = 0; i < m && k + 1 < errcap; i++) errbuf[k++] = es[i];
        errbuf[k] = 0;
    }
    return rc;
}

#define CKM(call, what)                                                                                \
    do {                                                                                               \
        cudaError_t e_ = (call);                                                                       \
        if (e_ != cudaSuccess) return set_err(errbuf, errcap, 2, what, e_);                            \
    } while (0)

int grid_of(int n) { return (n + THREADS - 1) / THREADS; }

cudaError_t smem_attr()
{
    static bool done = false;
    if (done) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_mlp_backprop, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM);
    done = e == cudaSuccess;
    return e;
}

cudaError_t grad_launches(const float *params, const float *X, const float *T, int n, float *rec, float *sqerr,
                          float *grad, float *loss, cudaStream_t st)
{
    k_mlp_backprop<<<grid_of(n), THREADS, SMEM, st>>>(params, X, T, n, rec, sqerr);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    k_mlp_reduce<<<grid_of(NPARAM + 1), THREADS, 0, st>>>(rec, sqerr, n, grad, loss);
    return cudaGetLastError();
}

} // namespace

extern "C" int cuopus_chain_features(const cuopus_batch *b, float *feat_dev, void *cuda_stream, char *errbuf,
                                     size_t errcap)
{
    if (!b || !feat_dev || !b->data || !b->off || !b->len || !b->first || !b->npkts || !b->channels)
        return set_err(errbuf, errcap, 3, "chain_features: NULL argument", cudaSuccess);
    if (b->nchains <= 0) return 0;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    int dev = 0, sms = 0;
    CKM(cudaGetDevice(&dev), "cudaGetDevice");
    CKM(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "SM count");
    const unsigned blocks = (unsigned)(((long long)b->nchains + 31) / 32);
    // Lanes per chain: as many as keep all chains on the GPU at once.  Microseconds
    // a call at 32 / 16 / 8 / 4 / 2 lanes:
    //    4,096 chains of 60 packets 32 / 32 / 34 / 38 / 47, of 400 60 / 74 / 110 / 149 / 268;
    //    9,472 of 1                 37 / 31 / 29 / 30 / 31, of 60 38 / 34 / 35 / 38 / 47;
    //   16,384 of 1                 42 / 31 / 27 / 26 / 27, of 60 51 / 42 / 38 / 45 / 61;
    //   40,000 of 1                 67 / 41 / 32 / 29 / 29, of 60 91 / 80 / 72 / 69 / 78;
    //  200,000 of 1                240 / 109 / 59 / 47 / 44, of 16 278 / 138 / 94 / 89 / 95.
    const auto launch = [&](auto kernel, int lanes) {
        kernel<<<blocks, 32 * lanes, 0, st>>>(b->data, b->off, b->len, b->first, b->npkts, b->channels, b->nchains,
                                              feat_dev);
    };
    if (b->nchains <= 32ll * sms) launch(k_chain_features<32>, 32);
    else if (b->nchains <= 64ll * sms) launch(k_chain_features<16>, 16);
    else if (b->nchains <= 128ll * sms) launch(k_chain_features<8>, 8);
    else if (b->nchains <= 512ll * sms) launch(k_chain_features<4>, 4);
    else launch(k_chain_features<2>, 2);
    CKM(cudaGetLastError(), "chain_features launch");
    CKM(cudaStreamSynchronize(st), "chain_features");
    return 0;
}

extern "C" int cuopus_mlp_init(float *params_dev, uint64_t seed, void *cuda_stream, char *errbuf, size_t errcap)
{
    if (!params_dev) return set_err(errbuf, errcap, 3, "mlp_init: NULL params", cudaSuccess);
    // He-uniform weights from a 64-bit LCG, zero biases
    std::vector<float> p(NPARAM, 0.f);
    uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto uni = [&]() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (float)((double)(s >> 11) * (1.0 / 9007199254740992.0)) * 2.f - 1.f;
    };
    float a1 = sqrtf(6.f / F), a2 = sqrtf(6.f / H), a3 = sqrtf(3.f / H);
    for (int i = 0; i < F * H; i++) p[OFF_W1 + i] = a1 * uni();
    for (int i = 0; i < H * H; i++) p[OFF_W2 + i] = a2 * uni();
    for (int i = 0; i < H; i++) p[OFF_W3 + i] = a3 * uni();
    cudaStream_t st = (cudaStream_t)cuda_stream;
    CKM(cudaMemcpyAsync(params_dev, p.data(), NPARAM * sizeof(float), cudaMemcpyHostToDevice, st), "mlp_init copy");
    CKM(cudaStreamSynchronize(st), "mlp_init");
    return 0;
}

extern "C" int cuopus_mlp_predict(const float *params_dev, const float *x_dev, int n, float *y_dev,
                                  void *cuda_stream, char *errbuf, size_t errcap)
{
    if (!params_dev || (n > 0 && (!x_dev || !y_dev)))
        return set_err(errbuf, errcap, 3, "mlp_predict: NULL argument", cudaSuccess);
    if (n <= 0) return 0;
    cudaStream_t st = (cudaStream_t)cuda_stream;
    k_mlp_predict<<<(unsigned)(((long long)n + PRED_SAMPLES - 1) / PRED_SAMPLES), H, 0, st>>>(params_dev, x_dev, n, y_dev);
    CKM(cudaGetLastError(), "mlp_predict launch");
    CKM(cudaStreamSynchronize(st), "mlp_predict");
    return 0;
}

extern "C" int cuopus_mlp_grad(const float *params_dev, const float *x_dev, const float *t_dev, int n,
                               float *grad_dev, float *loss_dev, void *cuda_stream, char *errbuf, size_t errcap)
{
    if (!params_dev || !x_dev || !t_dev || !grad_dev || !loss_dev || n <= 0)
        return set_err(errbuf, errcap, 3, "mlp_grad: bad argument", cudaSuccess);
    cudaStream_t st = (cudaStream_t)cuda_stream;
    CKM(smem_attr(), "mlp smem");
    float *rec = nullptr, *sq = nullptr;
    CKM(cudaMalloc(&rec, (size_t)n * REC * sizeof(float)), "mlp_grad alloc");
    cudaError_t e = cudaMalloc(&sq, (size_t)n * sizeof(float));
    if (e == cudaSuccess) e = grad_launches(params_dev, x_dev, t_dev, n, rec, sq, grad_dev, loss_dev, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    cudaFree(rec);
    cudaFree(sq);
    if (e != cudaSuccess) return set_err(errbuf, errcap, 2, "mlp_grad", e);
    return 0;
}

// Full-batch Adam at learning rate lr; the step (gradient kernels + update)
// is captured once as a CUDA graph of 50 steps and replayed, so the steps run
// are `steps` rounded up to a multiple of 50.  losses (host, may be NULL,
// `steps` entries) receives the loss before each step.
extern "C" int cuopus_mlp_train(float *params_dev, const float *x_dev, const float *t_dev, int n, int steps,
                                float lr, float *losses, void *cuda_stream, char *errbuf, size_t errcap)
{
    if (!params_dev || !x_dev || !t_dev || n <= 0 || steps < 0)
        return set_err(errbuf, errcap, 3, "mlp_train: bad argument", cudaSuccess);
    cudaStream_t st = (cudaStream_t)cuda_stream;
    CKM(smem_attr(), "mlp smem");
    const int chunk = 50;
    float *rec = nullptr, *work = nullptr;
    int *tstep = nullptr;
    // work: sqerr[n] | grad | m | v | loss[chunk]
    size_t wn = (size_t)n + 3 * NPARAM + chunk;
    cudaError_t e = cudaMalloc(&rec, (size_t)n * REC * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&work, wn * sizeof(float));
    if (e == cudaSuccess) e = cudaMalloc(&tstep, sizeof(int));
    if (e == cudaSuccess) e = cudaMemsetAsync(work, 0, wn * sizeof(float), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(tstep, 0, sizeof(int), st);
    float *sq = work, *grad = sq + n, *m = grad + NPARAM, *v = m + NPARAM, *lossv = v + NPARAM;
    cudaStream_t cs = nullptr;
    cudaGraphExec_t exec = nullptr;
    if (e == cudaSuccess) e = cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking);
    if (e == cudaSuccess) {
        cudaGraph_t g = nullptr;
        e = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        if (e == cudaSuccess) {
            cudaError_t e1 = cudaSuccess;
            for (int k = 0; k < chunk && e1 == cudaSuccess; k++) {
                e1 = grad_launches(params_dev, x_dev, t_dev, n, rec, sq, grad, lossv + k, cs);
                if (e1 == cudaSuccess) {
                    k_adam<<<grid_of(NPARAM), THREADS, 0, cs>>>(params_dev, grad, m, v, tstep, lr);
                    k_tick<<<1, 1, 0, cs>>>(tstep);
                    e1 = cudaGetLastError();
                }
            }
            e = cudaStreamEndCapture(cs, &g);
            if (e == cudaSuccess) e = e1;
        }
        if (e == cudaSuccess) e = cudaGraphInstantiate(&exec, g, 0);
        if (g) cudaGraphDestroy(g);
    }
    std::vector<float> lv(chunk);
    for (int done = 0; e == cudaSuccess && done < steps; done += chunk) {
        e = cudaGraphLaunch(exec, st);
        if (e == cudaSuccess && losses) {
            e = cudaMemcpyAsync(lv.data(), lossv, chunk * sizeof(float), cudaMemcpyDeviceToHost, st);
            if (e == cudaSuccess) e = cudaStreamSynchronize(st);
            for (int k = 0; k < chunk && done + k < steps; k++) losses[done + k] = lv[k];
        }
    }
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (exec) cudaGraphExecDestroy(exec);
    if (cs) cudaStreamDestroy(cs);
    cudaFree(rec);
    cudaFree(work);
    cudaFree(tstep);
    if (e != cudaSuccess) return set_err(errbuf, errcap, 2, "mlp_train", e);
    return 0;
}
