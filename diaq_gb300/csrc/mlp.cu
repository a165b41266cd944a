// The learned (s, m) proposer: a small FP32 MLP, 16 features -> 64 -> 64 -> 21 + 30 logits
// (s in 0..20, m in 1..30), with hand-written forward, softmax cross-entropy, backward and Adam
// kernels.  No counterpart in the reference, whose expm picks s by the norm bound alone
// (src/spME.cpp:256-262) and m by a Frobenius stop test.
//
// Parameters live in one flat float buffer: W1[16][64] b1[64] W2[64][64] b2[64] W3[64][51] b3[51]
// (W[i][j] maps input i to output j).  Every reduction over the batch runs in an order fixed by the
// batch size, so gradients are deterministic.
#include <algorithm>
#include <cmath>
#include <random>
#include <vector>

#include "diaq_internal.cuh"

namespace diaq_gb300 {

constexpr int kIn = 16, kH1 = 64, kH2 = 64, kOutS = 21, kOutM = 30, kOut = kOutS + kOutM;
constexpr int oW1 = 0, oB1 = oW1 + kIn * kH1, oW2 = oB1 + kH1, oB2 = oW2 + kH1 * kH2, oW3 = oB2 + kH2,
              oB3 = oW3 + kH2 * kOut, kParams = oB3 + kOut;

struct Mlp {
    float *p = nullptr, *m = nullptr, *v = nullptr;  // params, Adam moments
    float *work = nullptr;                           // weight gradients of `cap` blocks' rows
    int cap = 0;
    int64_t t = 0;  // Adam step
    ~Mlp() {
        cudaFree(p);
        cudaFree(work);
    }
};

// One pass over the batch.  The network is small (8,563 parameters, 34 KB) and a row's forward and
// backward pass touches nothing but the weights, so a block keeps the weights in shared memory and
// takes kRows rows at a time through the forward pass, the softmax, the backward pass and the
// products that make up the weight gradient; every activation stays in shared memory.  The weight
// gradient of the block's rows is held in registers (37 values per thread: a 4 x 4 tile of W2, one
// of W3, a strip of W1, a bias) and written once per block; mlp_reduce_kernel then sums the blocks'
// parts.  The sum over the batch is split over up to 2 blocks per SM this way: one thread per weight
// walking the whole batch left a chain of B dependent loads on 34 blocks: a training step of 1,024
// rows took 544 us that way (450 of them in those launches) and takes 21 us now.  What bounds it now
// is latency: two dependent launches (chained, 26 -> 21 us) with one round of 8 rows per block.
constexpr int kRows = 8;                       // rows per block and round: one per warp in the softmax
constexpr int kMlpThreads = 256;
constexpr int kLd2 = kH2 + 1;                  // W2 rows padded: read along both indices, conflict-free
constexpr int kOutPad = 52;                    // logits rows padded to whole float4s

struct MlpShared {  // 45 KB
    float w1[kIn * kH1], b1[kH1], w2[kH1 * kLd2], b2[kH2], w3[kH2 * kOut], b3[kOut];
    alignas(16) float x[kRows][kIn], a1[kRows][kH1], a2[kRows][kH2], lg[kRows][kOutPad], d2[kRows][kH2], d1[kRows][kH1];
};

__device__ __forceinline__ void mlp_load_weights(MlpShared &S, const float *p) {
    const int t = threadIdx.x;
    for (int i = t; i < kIn * kH1; i += kMlpThreads) S.w1[i] = p[oW1 + i];
    for (int i = t; i < kH1 * kH2; i += kMlpThreads) S.w2[(i / kH2) * kLd2 + i % kH2] = p[oW2 + i];
    for (int i = t; i < kH2 * kOut; i += kMlpThreads) S.w3[i] = p[oW3 + i];
    if (t < kH1) S.b1[t] = p[oB1 + t];
    if (t < kH2) S.b2[t] = p[oB2 + t];
    if (t < kOut) S.b3[t] = p[oB3 + t];
}

// Logits of rows row0 .. row0 + kRows - 1 into S.lg (rows past B read as zeros).  Thread t works on
// unit t % 64 of rows t / 64 and t / 64 + 4; each unit's sum runs over its inputs in order.
__device__ __forceinline__ void mlp_forward_rows(MlpShared &S, const float *X, int64_t row0, int B) {
    const int t = threadIdx.x, j = t & 63, q = t >> 6;
    if (t < kRows * kIn) {
        const int64_t b = row0 + t / kIn;
        S.x[t / kIn][t % kIn] = b < B ? X[row0 * kIn + t] : 0.f;
    }
    __syncthreads();
    float s0 = S.b1[j], s1 = s0;
#pragma unroll
    for (int i = 0; i < kIn; ++i) {
        const float w = S.w1[i * kH1 + j];
        s0 = fmaf(S.x[q][i], w, s0);
        s1 = fmaf(S.x[q + 4][i], w, s1);
    }
    S.a1[q][j] = fmaxf(s0, 0.f);
    S.a1[q + 4][j] = fmaxf(s1, 0.f);
    __syncthreads();
    s0 = s1 = S.b2[j];
#pragma unroll 16
    for (int i = 0; i < kH1; ++i) {
        const float w = S.w2[i * kLd2 + j];
        s0 = fmaf(S.a1[q][i], w, s0);
        s1 = fmaf(S.a1[q + 4][i], w, s1);
    }
    S.a2[q][j] = fmaxf(s0, 0.f);
    S.a2[q + 4][j] = fmaxf(s1, 0.f);
    __syncthreads();
    if (j < kOut) {
        s0 = s1 = S.b3[j];
#pragma unroll 16
        for (int i = 0; i < kH2; ++i) {
            const float w = S.w3[i * kOut + j];
            s0 = fmaf(S.a2[q][i], w, s0);
            s1 = fmaf(S.a2[q + 4][i], w, s1);
        }
        S.lg[q][j] = s0;
        S.lg[q + 4][j] = s1;
    } else if (j == kOut) {
        S.lg[q][j] = S.lg[q + 4][j] = 0.f;
    }
    __syncthreads();
}

// Logits[B][51], or the argmax of each head (s_out, m_out), for every row.
__global__ void __launch_bounds__(kMlpThreads)
    mlp_forward_kernel(const float *__restrict__ p, const float *__restrict__ X, int B, float *__restrict__ logits,
                       int32_t *__restrict__ s_out, int32_t *__restrict__ m_out) {
    __shared__ MlpShared S;
    mlp_load_weights(S, p);
    for (int64_t row0 = (int64_t)blockIdx.x * kRows; row0 < B; row0 += (int64_t)gridDim.x * kRows) {
        __syncthreads();
        mlp_forward_rows(S, X, row0, B);
        const int n = (int)min((int64_t)kRows, B - row0);
        if (logits)
            for (int i = threadIdx.x; i < n * kOut; i += kMlpThreads)
                logits[row0 * kOut + i] = S.lg[i / kOut][i % kOut];
        if (s_out && threadIdx.x < n) {
            const float *l = S.lg[threadIdx.x];
            int bs = 0, bm = 0;
            for (int j = 1; j < kOutS; ++j)
                if (l[j] > l[bs]) bs = j;
            for (int j = 1; j < kOutM; ++j)
                if (l[kOutS + j] > l[kOutS + bm]) bm = j;
            s_out[row0 + threadIdx.x] = bs;
            m_out[row0 + threadIdx.x] = bm + 1;
        }
    }
}

// One head of one row, a lane per logit: CE(softmax(l), lab) to every lane, and l replaced by
// (softmax - onehot) / B.  A label outside the head gives loss 0 and no gradient.
__device__ __forceinline__ float softmax_ce_head(float *l, int n, int lab, int lane, float B) {
    const float v = lane < n ? l[lane] : 0.f;
    float mx = lane < n ? v : -INFINITY;
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    const float e = lane < n ? expf(v - mx) : 0.f;
    float se = e;
    for (int o = 16; o > 0; o >>= 1) se += __shfl_xor_sync(0xffffffffu, se, o);
    const bool ok = lab >= 0 && lab < n;
    const float vl = __shfl_sync(0xffffffffu, v, ok ? lab : 0);
    if (lane < n) l[lane] = ok ? (e / se - (lane == lab ? 1.f : 0.f)) / B : 0.f;
    return ok ? -(vl - mx - logf(se)) : 0.f;
}

// acc[4][4] += u (4 values) x v (4 values)
__device__ __forceinline__ void outer4(float (&acc)[4][4], const float4 &u, const float4 &v) {
    const float a[4] = {u.x, u.y, u.z, u.w}, b[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
}

// Per-row losses (loss may be NULL) and, per block, the gradient of the mean loss over the block's
// rows: part[block][kParams].
__global__ void __launch_bounds__(kMlpThreads)
    mlp_grad_kernel(const float *p, const float *X, const int32_t *ys, const int32_t *ym, int B, float *loss, float *part) {
    __shared__ MlpShared S;
    dependency_wait();   // launched while the previous step's reduction drains
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    mlp_load_weights(S, p);
    const int i4 = (t >> 4) * 4, j4 = (t & 15) * 4;       // tile of W2 (and of W3, j4 < 52); column strip of W1
    float g1[4] = {0.f, 0.f, 0.f, 0.f}, g2[4][4], g3[4][4], gb = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) g2[i][j] = g3[i][j] = 0.f;
    for (int64_t row0 = (int64_t)blockIdx.x * kRows; row0 < B; row0 += (int64_t)gridDim.x * kRows) {
        __syncthreads();
        mlp_forward_rows(S, X, row0, B);
        const int64_t b = row0 + wid;
        const bool live = b < B;
        const float l = softmax_ce_head(S.lg[wid], kOutS, live ? ys[b] : -1, lane, (float)B) +
                        softmax_ce_head(S.lg[wid] + kOutS, kOutM, live ? ym[b] - 1 : -1, lane, (float)B);
        if (loss && live && lane == 0) loss[b] = l;
        __syncthreads();
        {   // dL/da2, dL/da1 (masked by the ReLUs): thread t on unit t % 64 of two rows
            const int i = t & 63, q = t >> 6;
            float s0 = 0.f, s1 = 0.f;
#pragma unroll 17
            for (int j = 0; j < kOut; ++j) {
                const float w = S.w3[i * kOut + j];
                s0 = fmaf(S.lg[q][j], w, s0);
                s1 = fmaf(S.lg[q + 4][j], w, s1);
            }
            S.d2[q][i] = S.a2[q][i] > 0.f ? s0 : 0.f;
            S.d2[q + 4][i] = S.a2[q + 4][i] > 0.f ? s1 : 0.f;
            __syncthreads();
            s0 = s1 = 0.f;
#pragma unroll 16
            for (int j = 0; j < kH2; ++j) {
                const float w = S.w2[i * kLd2 + j];
                s0 = fmaf(S.d2[q][j], w, s0);
                s1 = fmaf(S.d2[q + 4][j], w, s1);
            }
            S.d1[q][i] = S.a1[q][i] > 0.f ? s0 : 0.f;
            S.d1[q + 4][i] = S.a1[q + 4][i] > 0.f ? s1 : 0.f;
            __syncthreads();
        }
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const float4 d1 = *reinterpret_cast<const float4 *>(&S.d1[r][j4]);
            const float x = S.x[r][i4 >> 2];
            g1[0] = fmaf(x, d1.x, g1[0]);
            g1[1] = fmaf(x, d1.y, g1[1]);
            g1[2] = fmaf(x, d1.z, g1[2]);
            g1[3] = fmaf(x, d1.w, g1[3]);
            outer4(g2, *reinterpret_cast<const float4 *>(&S.a1[r][i4]), *reinterpret_cast<const float4 *>(&S.d2[r][j4]));
            if (j4 < kOutPad)
                outer4(g3, *reinterpret_cast<const float4 *>(&S.a2[r][i4]), *reinterpret_cast<const float4 *>(&S.lg[r][j4]));
            gb += t < kH1 ? S.d1[r][t] : t < kH1 + kH2 ? S.d2[r][t - kH1] : t < kH1 + kH2 + kOut ? S.lg[r][t - kH1 - kH2] : 0.f;
        }
    }
    float *o = part + (int64_t)blockIdx.x * kParams;
#pragma unroll
    for (int j = 0; j < 4; ++j) o[oW1 + (i4 >> 2) * kH1 + j4 + j] = g1[j];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            o[oW2 + (i4 + i) * kH2 + j4 + j] = g2[i][j];
            if (j4 + j < kOut) o[oW3 + (i4 + i) * kOut + j4 + j] = g3[i][j];
        }
    if (t < kH1) o[oB1 + t] = gb;
    else if (t < kH1 + kH2) o[oB2 + t - kH1] = gb;
    else if (t < kH1 + kH2 + kOut) o[oB3 + t - kH1 - kH2] = gb;
    dependents_go();
}

// Sums the blocks' parts per parameter in a fixed order (8 slices of the blocks, then the slices),
// into g (may be NULL) and, with adam, straight into the Adam step of p, m, v.
struct AdamStep {
    float *p, *m, *v;
    float lr, b1, b2, eps, bc1, bc2;
};
constexpr int kSlices = 8;
__global__ void __launch_bounds__(32 * kSlices)
    mlp_reduce_kernel(const float *part, int nblk, float *g, int adam, AdamStep A) {
    __shared__ float red[kSlices][32];
    dependency_wait();   // launched while the gradient kernel drains
    const int lane = threadIdx.x & 31, sl = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < kParams) {
#pragma unroll 8
        for (int b = sl; b < nblk; b += kSlices) s += part[(int64_t)b * kParams + i];
    }
    red[sl][lane] = s;
    dependents_go();
    __syncthreads();
    if (sl != 0 || i >= kParams) return;
    float gi = red[0][lane];
#pragma unroll
    for (int k = 1; k < kSlices; ++k) gi += red[k][lane];
    if (g) g[i] = gi;
    if (!adam) return;
    const float mi = A.b1 * A.m[i] + (1.f - A.b1) * gi;
    const float vi = A.b2 * A.v[i] + (1.f - A.b2) * gi * gi;
    A.m[i] = mi;
    A.v[i] = vi;
    A.p[i] -= A.lr * (mi / A.bc1) / (sqrtf(vi / A.bc2) + A.eps);
}

// Blocks of a pass over B rows: at most two per SM (the shared memory would hold four).
static int grad_blocks(int B) { return (int)std::min<int64_t>(((int64_t)B + kRows - 1) / kRows, 2 * num_sms()); }

static int ensure_work(Mlp &M, int nblk) {
    if (nblk <= M.cap) return DIAQ_OK;
    if (M.work) cudaFree(M.work);
    M.work = nullptr;
    M.cap = 0;
    DQ_CUDA(dev_malloc(&M.work, sizeof(float) * kParams * (size_t)nblk));
    M.cap = nblk;
    return DIAQ_OK;
}

static int forward(Mlp &M, const float *X, int B, float *logits, int32_t *s_out, int32_t *m_out, cudaStream_t s) {
    mlp_forward_kernel<<<grad_blocks(B), kMlpThreads, 0, s>>>(M.p, X, B, logits, s_out, m_out);
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

// The batch's gradient into g (may be NULL) and, with adam, into an Adam step.
static int gradient(Mlp &M, const float *X, const int32_t *ys, const int32_t *ym, int B, float *loss, float *g,
                    const AdamStep *adam, cudaStream_t s) {
    const int nblk = grad_blocks(B);
    DQ_TRY(ensure_work(M, nblk));
    launch_chained(true, mlp_grad_kernel, (unsigned)nblk, kMlpThreads, s, M.p, X, ys, ym, B, loss, M.work);
    launch_chained(true, mlp_reduce_kernel, (kParams + 31) / 32, 32 * kSlices, s, M.work, nblk, g, adam ? 1 : 0,
                   adam ? *adam : AdamStep{});
    DQ_CUDA(cudaGetLastError());
    return DIAQ_OK;
}

}  // namespace diaq_gb300

using namespace diaq_gb300;

struct diaq_mlp_s : public Mlp {};

extern "C" {

int diaq_mlp_num_params(void) { return kParams; }

int diaq_mlp_create(uint64_t seed, diaq_mlp_t *out) {
    if (!out) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    std::vector<float> h(kParams, 0.f);
    std::mt19937_64 rng(seed);
    auto init = [&](int off, int fan_in, int n) {  // He initialisation, biases stay 0
        std::normal_distribution<double> nd(0.0, std::sqrt(2.0 / fan_in));
        for (int i = 0; i < n; ++i) h[off + i] = (float)nd(rng);
    };
    init(oW1, kIn, kIn * kH1);
    init(oW2, kH1, kH1 * kH2);
    init(oW3, kH2, kH2 * kOut);
    diaq_mlp_s *M = new diaq_mlp_s();
    cudaError_t e = dev_malloc(&M->p, sizeof(float) * 3 * kParams);
    if (e == cudaSuccess) {
        M->m = M->p + kParams;
        M->v = M->p + 2 * kParams;
        e = cudaMemset(M->p, 0, sizeof(float) * 3 * kParams);
    }
    if (e == cudaSuccess) e = cudaMemcpy(M->p, h.data(), sizeof(float) * kParams, cudaMemcpyHostToDevice);
    if (e != cudaSuccess) {
        delete M;
        return cuda_status(e, "mlp create", __FILE__, __LINE__);
    }
    *out = M;
    return DIAQ_OK;
}

int diaq_mlp_destroy(diaq_mlp_t M) {
    delete M;
    return DIAQ_OK;
}

int diaq_mlp_get_params(diaq_mlp_t M, float *host_out) {
    if (!M || !host_out) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    DQ_CUDA(cudaMemcpy(host_out, M->p, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    return DIAQ_OK;
}

int diaq_mlp_set_params(diaq_mlp_t M, const float *host_in) {
    if (!M || !host_in) return set_error(DIAQ_ERR_INVALID, "NULL argument");
    DQ_CUDA(cudaMemcpy(M->p, host_in, sizeof(float) * kParams, cudaMemcpyHostToDevice));
    DQ_CUDA(cudaMemset(M->m, 0, sizeof(float) * 2 * kParams));
    M->t = 0;
    return DIAQ_OK;
}

int diaq_mlp_forward(diaq_mlp_t M, const float *X, int B, float *logits, void *stream) {
    if (!M || !X || !logits || B < 0) return set_error(DIAQ_ERR_INVALID, "mlp forward: bad argument");
    if (B == 0) return DIAQ_OK;
    return forward(*M, X, B, logits, nullptr, nullptr, (cudaStream_t)stream);
}

int diaq_mlp_gradient(diaq_mlp_t M, const float *X, const int32_t *s_label, const int32_t *m_label, int B,
                      float *grad_out, float *loss_out, void *stream) {
    if (!M || !X || !s_label || !m_label || B <= 0) return set_error(DIAQ_ERR_INVALID, "mlp gradient: bad argument");
    return gradient(*M, X, s_label, m_label, B, loss_out, grad_out, nullptr, (cudaStream_t)stream);
}

int diaq_mlp_train_step(diaq_mlp_t M, const float *X, const int32_t *s_label, const int32_t *m_label, int B,
                        float lr, float *loss_out, void *stream) {
    if (!M || !X || !s_label || !m_label || B <= 0) return set_error(DIAQ_ERR_INVALID, "mlp gradient: bad argument");
    const float b1 = 0.9f, b2 = 0.999f;
    const int64_t t = M->t + 1;
    const AdamStep A{M->p, M->m, M->v, lr, b1, b2, 1e-8f, 1.f - (float)std::pow((double)b1, (double)t),
                     1.f - (float)std::pow((double)b2, (double)t)};
    DQ_TRY(gradient(*M, X, s_label, m_label, B, loss_out, nullptr, &A, (cudaStream_t)stream));
    M->t = t;
    return DIAQ_OK;
}

int diaq_mlp_propose(diaq_mlp_t M, const float *X, int B, int32_t *s_out, int32_t *m_out, void *stream) {
    if (!M || !X || !s_out || !m_out || B < 0) return set_error(DIAQ_ERR_INVALID, "mlp propose: bad argument");
    if (B == 0) return DIAQ_OK;
    return forward(*M, X, B, nullptr, s_out, m_out, (cudaStream_t)stream);
}

}  // extern "C"
