// Small multilayer perceptron for the learned continuation predictor:
// in -> width (GELU) -> ... -> width (GELU) -> out, trained online with Adam.
//
// Weights are kept as FP32 master copies and used in BF16 (rounded to
// nearest even) in the forward and backward products, with FP32
// accumulation; activations, gradients and the optimiser state are FP32.
// GELU is the erf form, 0.5 x (1 + erf(x / sqrt 2)).  The loss is the mean
// squared error over all outputs.  The products run on the tensor cores
// (mma.sync BF16 with FP32 accumulation; FP32 operands as exact sums of three
// BF16 terms, see k_linear_mma); training iterations (forward, backward, Adam)
// are captured in CUDA graphs and replayed.
//
// An iteration is latency: 24 small kernels one after the other took 60 us.  Of
// these only the forward pass, the gradients of the layers' inputs and the last
// weight gradient depend on each other (9 kernels for 3 hidden layers): the loss
// and the other weight gradients run on a second stream, the loss gradient and
// the activations' derivatives are epilogues, one Adam kernel updates every
// layer, the kernels of the chain are linked by programmatic dependent launch (a
// kernel is resident, with its weights loaded, while its predecessor still
// runs), and a graph holds TRAIN_UNROLL iterations.  An iteration on 40 rows of
// the predictor's network: 59.7 -> 30.5 us (300 rows: 82.3 -> 60.8).  The order of
// every sum is untouched: the same bits.  (One cooperative launch with barriers
// between the stages was slower, 66 us: a barrier over 152 SMs is some 4 us.)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "vefem.h"
#include "vefem_early.cuh"
#include "vefem_internal.h"

namespace {

struct Layer {
    int in, out;
    float *W = nullptr, *b = nullptr;          // FP32 master [out][in], [out]
    __nv_bfloat16 *Wb = nullptr;               // BF16 copy used by the products
    float *mW = nullptr, *vW = nullptr, *mb = nullptr, *vb = nullptr;   // Adam moments
    float *gW = nullptr, *gb = nullptr;        // gradients
    float *Z = nullptr, *A = nullptr;          // pre-activation, activation [n][out]
    float *dA = nullptr;                       // gradient w.r.t. A [n][out]
};

// ---- products on the tensor cores: mma.sync m16n8k16, BF16 x BF16 -> FP32
//
// The weights enter as their BF16 copy.  The activations and gradients are
// FP32; each is split exactly into three BF16 terms (x = h + m + l: h the
// nearest BF16, m the nearest BF16 of x - h, l of what is left; 8 + 8 + 8
// significand bits cover FP32's 24), so with the exact BF16 x BF16 products
// and FP32 accumulation a product X W^T is the FP32 product of the FP32
// activations with the BF16 weights, as on the CUDA cores.  For the weight
// gradient dZ^T X both operands are FP32: the six split products whose
// magnitude exceeds 2^-24 of the leading one are summed (h h, h m, m h, h l,
// l h, m m).  No atomics: every output is owned by one CTA, results are the
// same on every run.
//
// The products are small (a few hundred rows by 256) and run once per
// training iteration, so they are latency-bound: a CTA computes one 16 x 8
// output tile, its four warps split K and their partial tiles are added in
// warp order through shared memory.  Fragment layouts of m16n8k16
// (g = lane / 4, t = lane % 4): A registers (g, 2t..2t+1), (g+8, 2t..),
// (g, 2t+8..), (g+8, 2t+8..); B registers (k = 2t..2t+1, n = g),
// (k = 2t+8.., n = g); C (g, 2t..2t+1), (g+8, 2t..2t+1).  Two BF16 per 32-bit
// register, the lower index in the low half.
constexpr int MMA_WARPS = 4;

__device__ __forceinline__ uint32_t pack2(__nv_bfloat16 lo, __nv_bfloat16 hi)
{
    return (uint32_t)__bfloat16_as_ushort(lo) | ((uint32_t)__bfloat16_as_ushort(hi) << 16);
}

__device__ __forceinline__ void split3(float x, __nv_bfloat16 (&p)[3])
{
    p[0] = __float2bfloat16_rn(x);
    const float r1 = x - __bfloat162float(p[0]);
    p[1] = __float2bfloat16_rn(r1);
    p[2] = __float2bfloat16_rn(r1 - __bfloat162float(p[1]));
}

__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 "
        "{%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

enum { LIN_FWD = 0, LIN_BWD_X = 1, LIN_BWD_W = 2 };

// Programmatic dependent launch inside an iteration.  A kernel first waits for
// its predecessor (at once, without a programmatic dependency), then lets its
// successor start; so whatever runs before a kernel's wait may read what the
// predecessor's own predecessors wrote, with load_early (vefem_early.cuh), but
// nothing of the predecessor's.  What it reads after the wait was written while
// it was resident: no operand is const __restrict__, whose loads are for data
// that does not change while a kernel runs.
__device__ __forceinline__ void pdl_link()
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Operand element loaders (zero outside the matrix).
//   forward  Y = X W^T:   A(m, k) = X[m][k]   (n x in),  B(k, c) = W[c][k]
//   backward dX = dZ W:   A(m, k) = dZ[m][k]  (n x out), B(k, c) = W[k][c]
//   weights  gW = dZ^T X: A(m, k) = dZ[k][m]  (out x n), B(k, c) = X[k][c], and
//                         column c = in the constant 1 (its output is gb)
template <int MODE>
__device__ __forceinline__ float load_a(const float *A, int M, int K, int lda, int m, int k)
{
    if (m >= M || k >= K) return 0.0f;
    return MODE == LIN_BWD_W ? A[(size_t)k * lda + m] : A[(size_t)m * lda + k];
}

// d * gelu'(z)
__device__ __forceinline__ float gelu_bwd(float d, float z)
{
    const float cdf = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
    const float pdf = 0.39894228040143268f * expf(-0.5f * z * z);
    return d * (cdf + z * pdf);
}

// The operands of MMA_AHEAD k-steps are loaded before their first product, so a
// warp's loads are in flight together, and those of the weights before the
// wait for the predecessor unless that is the Adam kernel (early = 0).
constexpr int MMA_AHEAD = 4;

// FWD: out0 pre-activation, out1 activation (gelu) or output; with target T, out2 = the gradient
// 2 (Y - T) / count of the mean squared error.  BWD_X: out0 = dX times gelu'(aux).
// BWD_W: out0 weight gradient, out2 bias gradient.
template <int MODE>
__global__ void __launch_bounds__(MMA_WARPS * 32)
k_linear_mma(int M, int N, int K, const float *A, int lda, const __nv_bfloat16 *Wb, const float *Bf, int ldb,
             const float *bias, const float *aux, float *out0, float *out1, float *out2, int ldo, int gelu, int early)
{
    __shared__ float s_part[MMA_WARPS - 1][32][4];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int g = lane >> 2, t = lane & 3;
    const int m0 = blockIdx.y * 16, n0 = blockIdx.x * 8;
    const int ksteps = (K + 15) / 16;
    const int per = (ksteps + MMA_WARPS - 1) / MMA_WARPS;
    const int ks0 = warp * per, ks1 = min(ksteps, (warp + 1) * per);
    const int c = n0 + g;                  // the B column this thread loads
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    __nv_bfloat16 wb[MMA_AHEAD][4];
    auto load_weights = [&](int ks) {
#pragma unroll
        for (int h = 0; h < MMA_AHEAD; h++)
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int k = (ks + h) * 16 + 2 * t + (u & 1) + 8 * (u >> 1);
                const bool in = ks + h < ks1 && c < N && k < K;
                wb[h][u] = in ? load_early(MODE == LIN_FWD ? Wb + (size_t)c * ldb + k : Wb + (size_t)k * ldb + c)
                              : __float2bfloat16_rn(0.0f);
            }
    };
    if (MODE != LIN_BWD_W && early) load_weights(ks0);
    pdl_link();
    for (int ks = ks0; ks < ks1; ks += MMA_AHEAD) {
        if (MODE != LIN_BWD_W && (!early || ks > ks0)) load_weights(ks);
        float fa[MMA_AHEAD][8], fb[MMA_AHEAD][4];
#pragma unroll
        for (int h = 0; h < MMA_AHEAD; h++) {
            if (ks + h >= ks1) continue;
            const int k0 = (ks + h) * 16;
#pragma unroll
            for (int r = 0; r < 4; r++) {
                const int row = m0 + g + 8 * (r & 1), col = k0 + 2 * t + 8 * (r >> 1);
                fa[h][2 * r] = load_a<MODE>(A, M, K, lda, row, col);
                fa[h][2 * r + 1] = load_a<MODE>(A, M, K, lda, row, col + 1);
            }
            if (MODE == LIN_BWD_W) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const int k = k0 + 2 * t + (u & 1) + 8 * (u >> 1);
                    fb[h][u] = k < K && c < N ? (c < N - 1 ? Bf[(size_t)k * ldb + c] : 1.0f) : 0.0f;
                }
            }
        }
#pragma unroll
        for (int h = 0; h < MMA_AHEAD; h++) {
            if (ks + h >= ks1) continue;
            // A fragments of the three split terms
            uint32_t af[3][4];
#pragma unroll
            for (int r = 0; r < 4; r++) {
                __nv_bfloat16 lo[3], hi[3];
                split3(fa[h][2 * r], lo);
                split3(fa[h][2 * r + 1], hi);
#pragma unroll
                for (int q = 0; q < 3; q++) af[q][r] = pack2(lo[q], hi[q]);
            }
            if (MODE != LIN_BWD_W) {
                const uint32_t b0 = pack2(wb[h][0], wb[h][1]), b1 = pack2(wb[h][2], wb[h][3]);
                // small terms first
                mma_bf16(acc, af[2], b0, b1);
                mma_bf16(acc, af[1], b0, b1);
                mma_bf16(acc, af[0], b0, b1);
            } else {
                __nv_bfloat16 x[4][3];
#pragma unroll
                for (int u = 0; u < 4; u++) split3(fb[h][u], x[u]);
                uint32_t bf[3][2];
#pragma unroll
                for (int q = 0; q < 3; q++) {
                    bf[q][0] = pack2(x[0][q], x[1][q]);
                    bf[q][1] = pack2(x[2][q], x[3][q]);
                }
                mma_bf16(acc, af[1], bf[1][0], bf[1][1]);
                mma_bf16(acc, af[2], bf[0][0], bf[0][1]);
                mma_bf16(acc, af[0], bf[2][0], bf[2][1]);
                mma_bf16(acc, af[1], bf[0][0], bf[0][1]);
                mma_bf16(acc, af[0], bf[1][0], bf[1][1]);
                mma_bf16(acc, af[0], bf[0][0], bf[0][1]);
            }
        }
    }
    // partial tiles of warps 1..3 added to warp 0's, in warp order
    if (warp > 0) {
#pragma unroll
        for (int u = 0; u < 4; u++) s_part[warp - 1][lane][u] = acc[u];
    }
    __syncthreads();
    if (warp != 0) return;
#pragma unroll
    for (int w = 0; w < MMA_WARPS - 1; w++)
#pragma unroll
        for (int u = 0; u < 4; u++) acc[u] += s_part[w][lane][u];
    // epilogue
#pragma unroll
    for (int u = 0; u < 4; u++) {
        const int m = m0 + g + (u >= 2 ? 8 : 0);
        const int cc = n0 + 2 * t + (u & 1);
        if (m >= M || cc >= N) continue;
        const float v = acc[u];
        const size_t o = (size_t)m * ldo + cc;
        if (MODE == LIN_FWD) {
            const float z = v + bias[cc];
            out0[o] = z;
            out1[o] = gelu ? 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)) : z;
            if (aux) {
                const float d = z - aux[o];
                out2[o] = 2.0f * d / (float)(M * N);
            }
        } else if (MODE == LIN_BWD_X) {
            out0[o] = gelu_bwd(v, aux[o]);
        } else {
            if (cc < N - 1) out0[o] = v;
            else out2[m] = v;
        }
    }
}

dim3 mma_grid(int M, int N)
{
    return dim3((unsigned)((N + 7) / 8), (unsigned)((M + 15) / 16));
}

// MSE loss, *loss = mean (Y - T)^2.  One block: each thread sums its strided share
// in order, then a fixed tree in shared memory -- the same bits on every run (no
// atomics).  step: Adam's iteration count, if any, goes up by one.
constexpr int MSE_THREADS = 1024;
__global__ void __launch_bounds__(MSE_THREADS) k_mse(int count, const float *__restrict__ Y,
                                                     const float *__restrict__ T, float *__restrict__ loss, int *step)
{
    __shared__ float red[MSE_THREADS];
    pdl_link();
    if (step && threadIdx.x == 0) *step += 1;
    float acc = 0.0f;
    for (int i = threadIdx.x; i < count; i += MSE_THREADS) {
        const float d = Y[i] - T[i];
        acc += d * d;
    }
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = MSE_THREADS / 2; s > 0; s >>= 1) {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) *loss = red[0] / (float)count;
}

// Adam on the FP32 masters of every weight and bias array, then the BF16 copy;
// t is read from device memory.  An array's first block is seg.block0.
struct AdamSeg {
    float *p;
    const float *g;
    float *m, *v;
    __nv_bfloat16 *pb;
    int count, block0;
};

__global__ void k_adam(const AdamSeg *__restrict__ segs, int nseg, float lr, const int *__restrict__ step)
{
    pdl_link();
    int s = 0;
    while (s + 1 < nseg && (int)blockIdx.x >= segs[s + 1].block0) s++;
    const AdamSeg a = segs[s];
    float *__restrict__ p = a.p;
    const float *__restrict__ g = a.g;
    float *__restrict__ m = a.m;
    float *__restrict__ v = a.v;
    const int i = (blockIdx.x - a.block0) * blockDim.x + threadIdx.x;
    if (i >= a.count) return;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    const float t = (float)(*step);
    const float mi = b1 * m[i] + (1.0f - b1) * g[i];
    const float vi = b2 * v[i] + (1.0f - b2) * g[i] * g[i];
    m[i] = mi;
    v[i] = vi;
    const float mh = mi / (1.0f - powf(b1, t));
    const float vh = vi / (1.0f - powf(b2, t));
    const float np = p[i] - lr * mh / (sqrtf(vh) + eps);
    p[i] = np;
    if (a.pb) a.pb[i] = __float2bfloat16_rn(np);
}

__global__ void k_to_bf16(int count, const float *__restrict__ p, __nv_bfloat16 *pb)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < count) pb[i] = __float2bfloat16_rn(p[i]);
}

}  // namespace


struct vefem_mlp {
    int device = 0;
    int in = 0, width = 0, out = 0, hidden = 0;
    std::vector<Layer> L;
    int cap = 0;                  // rows the activation buffers hold
    float *X = nullptr, *T = nullptr, *loss = nullptr;
    int *step = nullptr;
    cudaStream_t s = nullptr, s2 = nullptr;   // s2: weight gradients beside the backward chain
    cudaEvent_t fork = nullptr, join = nullptr;
    AdamSeg *segs = nullptr;
    int nseg = 0, adam_blocks = 0;
    cudaGraphExec_t graph[2] = {nullptr, nullptr};   // TRAIN_UNROLL iterations, and one
    int graph_n = -1;
    float graph_lr = 0.0f;
    std::string err;
};

namespace {

int mlp_fail(vefem_mlp *m, int code, const std::string &msg)
{
    if (m)
        m->err = msg;
    else
        vefem::set_global_error(msg);
    return code;
}

#define MCK(call)                                                                   \
    do {                                                                            \
        cudaError_t _e = (call);                                                    \
        if (_e != cudaSuccess)                                                      \
            return mlp_fail(m, VEFEM_ERR_CUDA, std::string(#call) + ": " + cudaGetErrorString(_e)); \
    } while (0)

int64_t nparams(const vefem_mlp *m)
{
    int64_t n = 0;
    for (const Layer &l : m->L) n += (int64_t)l.in * l.out + l.out;
    return n;
}

void drop_graphs(vefem_mlp *m)
{
    for (cudaGraphExec_t &g : m->graph) {
        if (g) cudaGraphExecDestroy(g);
        g = nullptr;
    }
}

int ensure_rows(vefem_mlp *m, int n)
{
    if (n <= m->cap) return VEFEM_OK;
    for (Layer &l : m->L) {
        cudaFree(l.Z);
        cudaFree(l.A);
        cudaFree(l.dA);
        MCK(cudaMalloc(&l.Z, sizeof(float) * n * l.out));
        MCK(cudaMalloc(&l.A, sizeof(float) * n * l.out));
        MCK(cudaMalloc(&l.dA, sizeof(float) * n * l.out));
    }
    cudaFree(m->X);
    cudaFree(m->T);
    MCK(cudaMalloc(&m->X, sizeof(float) * n * m->in));
    MCK(cudaMalloc(&m->T, sizeof(float) * n * m->out));
    m->cap = n;
    drop_graphs(m);
    return VEFEM_OK;
}

// A launch on stream st; pdl: it may begin while the stream's previous kernel
// still runs (every kernel here waits for it before it reads anything).
template <typename... Args, typename... Act>
void go(bool pdl, void (*kern)(Args...), dim3 grid, int threads, cudaStream_t st, Act... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = pdl ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, args...);
}

// Forward pass; with train the last layer also leaves the loss gradient in its dA.
// first: its first kernel follows no kernel of a chain.
void launch_forward(vefem_mlp *m, int n, bool train, bool pdl, bool first)
{
    const float *x = m->X;
    for (size_t i = 0; i < m->L.size(); i++) {
        Layer &l = m->L[i];
        const bool last = i + 1 == m->L.size();
        // Y[n][out] = X[n][in] W^T + b (GELU but on the last layer); Z keeps the pre-activation
        go(pdl && !(first && i == 0), k_linear_mma<LIN_FWD>, mma_grid(n, l.out), MMA_WARPS * 32, m->s, n, l.out, l.in,
           x, l.in, (const __nv_bfloat16 *)l.Wb, (const float *)nullptr, l.in, (const float *)l.b,
           last && train ? (const float *)m->T : (const float *)nullptr, l.Z, l.A, l.dA, l.out, last ? 0 : 1,
           pdl && i > 0 ? 1 : 0);
        x = l.A;
    }
}

// gW[out][in] = dZ^T X and gb[out] = dZ^T 1 (the extra column)
void launch_weight_gradient(vefem_mlp *m, int n, int i, bool pdl, cudaStream_t st)
{
    Layer &l = m->L[i];
    const float *xin = i == 0 ? m->X : m->L[i - 1].A;
    go(pdl, k_linear_mma<LIN_BWD_W>, mma_grid(l.out, l.in + 1), MMA_WARPS * 32, st, l.out, l.in + 1, n,
       (const float *)l.dA, l.out, (const __nv_bfloat16 *)nullptr, xin, l.in, (const float *)nullptr,
       (const float *)nullptr, l.gW, (float *)nullptr, l.gb, l.in, 0, 0);
}

// Loss and backward pass: the gradients of the layers' inputs and the first
// layer's weight gradient on s, the loss and the other weight gradients on
// side (joined at the end).
void launch_backward(vefem_mlp *m, int n, bool pdl, cudaStream_t side, int *step)
{
    // dA of the output layer holds dLoss/dY; the others' dA are dLoss/dZ
    Layer &o = m->L.back();
    for (int i = (int)m->L.size() - 1; i > 0; i--) {
        Layer &l = m->L[i], &below = m->L[i - 1];
        cudaEventRecord(m->fork, m->s);
        cudaStreamWaitEvent(side, m->fork, 0);
        // dZ[n][in] = (dZ[n][out] W[out][in]) gelu'(Z) of the layer below
        go(pdl, k_linear_mma<LIN_BWD_X>, mma_grid(n, l.in), MMA_WARPS * 32, m->s, n, l.in, l.out, (const float *)l.dA,
           l.out, (const __nv_bfloat16 *)l.Wb, (const float *)nullptr, l.in, (const float *)nullptr,
           (const float *)below.Z, below.dA, (float *)nullptr, (float *)nullptr, l.in, 0, pdl ? 1 : 0);
        if (&l == &o)
            go(false, k_mse, dim3(1), MSE_THREADS, side, n * o.out, (const float *)o.A, (const float *)m->T, m->loss, step);
        launch_weight_gradient(m, n, i, false, side);
    }
    launch_weight_gradient(m, n, 0, pdl, m->s);
    cudaEventRecord(m->join, side);
    cudaStreamWaitEvent(m->s, m->join, 0);
}

constexpr int TRAIN_UNROLL = 8;     // iterations of the longer graph

cudaError_t capture_training(vefem_mlp *m, int n, float lr, int iters, cudaGraphExec_t *out)
{
    cudaGraph_t g = nullptr;
    cudaError_t e = cudaStreamBeginCapture(m->s, cudaStreamCaptureModeThreadLocal);
    if (e != cudaSuccess) return e;
    for (int it = 0; it < iters; it++) {
        launch_forward(m, n, true, true, it == 0);
        launch_backward(m, n, true, m->s2, m->step);
        k_adam<<<m->adam_blocks, 256, 0, m->s>>>(m->segs, m->nseg, lr, m->step);
    }
    const cudaError_t le = cudaGetLastError();
    e = cudaStreamEndCapture(m->s, &g);
    if (le != cudaSuccess) e = le;
    if (e == cudaSuccess) e = cudaGraphInstantiate(out, g, 0);
    if (g) cudaGraphDestroy(g);
    return e;
}

}  // namespace

namespace {

int mlp_init(vefem_mlp *m, uint64_t seed)
{
    const int hidden_layers = m->hidden;
    MCK(cudaSetDevice(m->device));
    MCK(cudaStreamCreateWithFlags(&m->s, cudaStreamNonBlocking));
    MCK(cudaStreamCreateWithFlags(&m->s2, cudaStreamNonBlocking));
    MCK(cudaEventCreateWithFlags(&m->fork, cudaEventDisableTiming));
    MCK(cudaEventCreateWithFlags(&m->join, cudaEventDisableTiming));
    // Kaiming-uniform-like init from a 64-bit LCG (deterministic for a seed)
    uint64_t st = seed * 6364136223846793005ULL + 1442695040888963407ULL;
    auto uni = [&st]() {
        st = st * 6364136223846793005ULL + 1442695040888963407ULL;
        return (double)(st >> 11) * (1.0 / 9007199254740992.0);
    };
    for (int i = 0; i <= hidden_layers; i++) {
        Layer l;
        l.in = i == 0 ? m->in : m->width;
        l.out = i == hidden_layers ? m->out : m->width;
        m->L.push_back(l);
    }
    for (Layer &l : m->L) {
        const size_t nw = (size_t)l.in * l.out;
        std::vector<float> w(nw), b(l.out, 0.0f);
        const double bound = std::sqrt(1.0 / l.in);
        for (size_t k = 0; k < nw; k++) w[k] = (float)((2.0 * uni() - 1.0) * bound);
        float **f[] = {&l.W, &l.mW, &l.vW, &l.gW};
        for (float **p : f) MCK(cudaMalloc(p, sizeof(float) * nw));
        float **g[] = {&l.b, &l.mb, &l.vb, &l.gb};
        for (float **p : g) MCK(cudaMalloc(p, sizeof(float) * l.out));
        MCK(cudaMalloc(&l.Wb, sizeof(__nv_bfloat16) * nw));
        MCK(cudaMemcpy(l.W, w.data(), sizeof(float) * nw, cudaMemcpyHostToDevice));
        MCK(cudaMemcpy(l.b, b.data(), sizeof(float) * l.out, cudaMemcpyHostToDevice));
        MCK(cudaMemset(l.mW, 0, sizeof(float) * nw));
        MCK(cudaMemset(l.vW, 0, sizeof(float) * nw));
        MCK(cudaMemset(l.mb, 0, sizeof(float) * l.out));
        MCK(cudaMemset(l.vb, 0, sizeof(float) * l.out));
        k_to_bf16<<<(int)((nw + 255) / 256), 256, 0, m->s>>>((int)nw, l.W, l.Wb);
    }
    std::vector<AdamSeg> segs;
    for (Layer &l : m->L) {
        const int cw = l.in * l.out;
        segs.push_back({l.W, l.gW, l.mW, l.vW, l.Wb, cw, m->adam_blocks});
        m->adam_blocks += (cw + 255) / 256;
        segs.push_back({l.b, l.gb, l.mb, l.vb, nullptr, l.out, m->adam_blocks});
        m->adam_blocks += (l.out + 255) / 256;
    }
    m->nseg = (int)segs.size();
    MCK(cudaMalloc(&m->segs, sizeof(AdamSeg) * segs.size()));
    MCK(cudaMemcpy(m->segs, segs.data(), sizeof(AdamSeg) * segs.size(), cudaMemcpyHostToDevice));
    MCK(cudaMalloc(&m->loss, sizeof(float)));
    MCK(cudaMalloc(&m->step, sizeof(int)));
    MCK(cudaMemset(m->step, 0, sizeof(int)));
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

}  // namespace

extern "C" int vefem_mlp_create(int in_dim, int width, int out_dim, int hidden_layers,
                                uint64_t seed, int device, vefem_mlp **out)
{
    if (!out || in_dim <= 0 || width <= 0 || out_dim <= 0 || hidden_layers <= 0 || device < 0 ||
        (int64_t)in_dim * width > (1 << 28) || (int64_t)width * out_dim > (1 << 28))
        return mlp_fail(nullptr, VEFEM_ERR_ARG, "vefem_mlp_create: bad arguments");
    *out = nullptr;
    vefem_mlp *m = new vefem_mlp();
    m->device = device;
    m->in = in_dim;
    m->width = width;
    m->out = out_dim;
    m->hidden = hidden_layers;
    if (int rc = mlp_init(m, seed)) {
        vefem::set_global_error("vefem_mlp_create: " + m->err);
        vefem_mlp_destroy(m);
        return rc;
    }
    *out = m;
    return VEFEM_OK;
}

extern "C" int vefem_mlp_reset_optimizer(vefem_mlp *m)
{
    if (!m) return mlp_fail(nullptr, VEFEM_ERR_ARG, "NULL network");
    MCK(cudaSetDevice(m->device));
    for (Layer &l : m->L) {
        const size_t nw = (size_t)l.in * l.out;
        MCK(cudaMemsetAsync(l.mW, 0, sizeof(float) * nw, m->s));
        MCK(cudaMemsetAsync(l.vW, 0, sizeof(float) * nw, m->s));
        MCK(cudaMemsetAsync(l.mb, 0, sizeof(float) * l.out, m->s));
        MCK(cudaMemsetAsync(l.vb, 0, sizeof(float) * l.out, m->s));
    }
    MCK(cudaMemsetAsync(m->step, 0, sizeof(int), m->s));
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

extern "C" int64_t vefem_mlp_num_params(const vefem_mlp *m) { return m ? nparams(m) : -1; }

// parameters as one FP32 array: for each layer W [out][in] then b [out]
extern "C" int vefem_mlp_set_params(vefem_mlp *m, const float *p, int64_t n)
{
    if (!m || !p || n != nparams(m)) return mlp_fail(m, VEFEM_ERR_ARG, "parameter count");
    MCK(cudaSetDevice(m->device));
    int64_t o = 0;
    for (Layer &l : m->L) {
        const size_t nw = (size_t)l.in * l.out;
        MCK(cudaMemcpyAsync(l.W, p + o, sizeof(float) * nw, cudaMemcpyHostToDevice, m->s));
        o += nw;
        MCK(cudaMemcpyAsync(l.b, p + o, sizeof(float) * l.out, cudaMemcpyHostToDevice, m->s));
        o += l.out;
        k_to_bf16<<<(int)((nw + 255) / 256), 256, 0, m->s>>>((int)nw, l.W, l.Wb);
    }
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

extern "C" int vefem_mlp_get_params(const vefem_mlp *mc, float *p, int64_t n)
{
    vefem_mlp *m = const_cast<vefem_mlp *>(mc);
    if (!m || !p || n != nparams(m)) return mlp_fail(m, VEFEM_ERR_ARG, "parameter count");
    MCK(cudaSetDevice(m->device));
    int64_t o = 0;
    for (Layer &l : m->L) {
        const size_t nw = (size_t)l.in * l.out;
        MCK(cudaMemcpyAsync(p + o, l.W, sizeof(float) * nw, cudaMemcpyDeviceToHost, m->s));
        o += nw;
        MCK(cudaMemcpyAsync(p + o, l.b, sizeof(float) * l.out, cudaMemcpyDeviceToHost, m->s));
        o += l.out;
    }
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

extern "C" int vefem_mlp_forward(vefem_mlp *m, const float *X, int n, float *Y)
{
    if (!m || !X || !Y || n <= 0) return mlp_fail(m, VEFEM_ERR_ARG, "bad arguments");
    MCK(cudaSetDevice(m->device));
    if (int rc = ensure_rows(m, n)) return rc;
    MCK(cudaMemcpyAsync(m->X, X, sizeof(float) * n * m->in, cudaMemcpyHostToDevice, m->s));
    launch_forward(m, n, false, false, true);
    MCK(cudaGetLastError());
    MCK(cudaMemcpyAsync(Y, m->L.back().A, sizeof(float) * n * m->out, cudaMemcpyDeviceToHost, m->s));
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

// loss and the gradient w.r.t. all parameters (layout of vefem_mlp_get_params)
extern "C" int vefem_mlp_loss_grad(vefem_mlp *m, const float *X, const float *T, int n,
                                   float *loss, float *grad)
{
    if (!m || !X || !T || !loss || !grad || n <= 0) return mlp_fail(m, VEFEM_ERR_ARG, "bad arguments");
    MCK(cudaSetDevice(m->device));
    if (int rc = ensure_rows(m, n)) return rc;
    MCK(cudaMemcpyAsync(m->X, X, sizeof(float) * n * m->in, cudaMemcpyHostToDevice, m->s));
    MCK(cudaMemcpyAsync(m->T, T, sizeof(float) * n * m->out, cudaMemcpyHostToDevice, m->s));
    MCK(cudaMemsetAsync(m->loss, 0, sizeof(float), m->s));
    launch_forward(m, n, true, false, true);
    launch_backward(m, n, false, m->s2, nullptr);
    MCK(cudaGetLastError());
    int64_t o = 0;
    for (Layer &l : m->L) {
        const size_t nw = (size_t)l.in * l.out;
        MCK(cudaMemcpyAsync(grad + o, l.gW, sizeof(float) * nw, cudaMemcpyDeviceToHost, m->s));
        o += nw;
        MCK(cudaMemcpyAsync(grad + o, l.gb, sizeof(float) * l.out, cudaMemcpyDeviceToHost, m->s));
        o += l.out;
    }
    MCK(cudaMemcpyAsync(loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->s));
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

// iters full-batch Adam iterations on (X, T), replayed from CUDA graphs
extern "C" int vefem_mlp_train(vefem_mlp *m, const float *X, const float *T, int n, int iters,
                               float lr, float *final_loss)
{
    if (!m || !X || !T || n <= 0 || iters < 0) return mlp_fail(m, VEFEM_ERR_ARG, "bad arguments");
    MCK(cudaSetDevice(m->device));
    if (int rc = ensure_rows(m, n)) return rc;
    MCK(cudaMemcpyAsync(m->X, X, sizeof(float) * n * m->in, cudaMemcpyHostToDevice, m->s));
    MCK(cudaMemcpyAsync(m->T, T, sizeof(float) * n * m->out, cudaMemcpyHostToDevice, m->s));
    if (m->graph_n != n || m->graph_lr != lr) {
        drop_graphs(m);
        m->graph_n = n;
        m->graph_lr = lr;
    }
    for (int i = 0; i < iters;) {
        const int k = iters - i >= TRAIN_UNROLL ? 0 : 1;
        if (!m->graph[k]) MCK(capture_training(m, n, lr, k == 0 ? TRAIN_UNROLL : 1, &m->graph[k]));
        MCK(cudaGraphLaunch(m->graph[k], m->s));
        i += k == 0 ? TRAIN_UNROLL : 1;
    }
    if (final_loss) {
        MCK(cudaMemcpyAsync(final_loss, m->loss, sizeof(float), cudaMemcpyDeviceToHost, m->s));
    }
    MCK(cudaStreamSynchronize(m->s));
    return VEFEM_OK;
}

extern "C" int vefem_mlp_destroy(vefem_mlp *m)
{
    if (!m) return VEFEM_OK;
    cudaSetDevice(m->device);
    if (m->s) cudaStreamSynchronize(m->s);
    if (m->s2) cudaStreamSynchronize(m->s2);
    drop_graphs(m);
    for (Layer &l : m->L) {
        void *p[] = {l.W, l.b, l.Wb, l.mW, l.vW, l.mb, l.vb, l.gW, l.gb, l.Z, l.A, l.dA};
        for (void *q : p)
            if (q) cudaFree(q);
    }
    void *p[] = {m->X, m->T, m->loss, m->step, m->segs};
    for (void *q : p)
        if (q) cudaFree(q);
    if (m->fork) cudaEventDestroy(m->fork);
    if (m->join) cudaEventDestroy(m->join);
    if (m->s2) cudaStreamDestroy(m->s2);
    if (m->s) cudaStreamDestroy(m->s);
    delete m;
    return VEFEM_OK;
}

extern "C" const char *vefem_mlp_last_error(const vefem_mlp *m) { return m ? m->err.c_str() : ""; }
