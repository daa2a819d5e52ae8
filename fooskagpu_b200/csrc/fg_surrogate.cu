// Learned equilibrium surrogate: training (forward / backward / Adam on the GPU, FP32), batch
// prediction through the BF16 tensor-core forward the relaxation kernel uses, and the C ABI
// (fg_surrogate_*).  It has no counterpart in the reference, whose chemical relaxation is the
// per-cell Newton of DP/chemRlx.cu:4-267; the network only supplies that Newton's starting point.
//
// Training: inputs (rho, e, Y) and targets (p, T, alpha, Y_eq) are standardised with the
// statistics of the training set; loss = mean squared error over the 4 standardised outputs;
// parameters are FP32 with Adam.  Every reduction over samples (weight gradients, loss) sums
// fixed chunks in a fixed order, so training is deterministic for a given seed.
#include "../../include/fooskagpu.h"
#include "fg_sg_tc.cuh"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <string>
#include <vector>

namespace fg {
int set_error(int code, const std::string &msg);
}
static_assert(fg::SG_NPARAM == FG_SG_NPARAM, "parameter count of the C header");
static_assert(sizeof(fg::SurrogateNorm) == FG_SG_NNORM * sizeof(float), "normalisation record of the C header");

using namespace fg;

namespace {

struct Buf {
    void *p = nullptr;
    size_t bytes = 0;
    cudaError_t alloc(size_t b) {
        release();
        bytes = b;
        return cudaMalloc(&p, b ? b : 16);
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    ~Buf() { release(); }
    template <typename X> X *as() const { return static_cast<X *>(p); }
};

#define SG_TRY(expr)                                                                                  \
    do {                                                                                              \
        cudaError_t e_ = (expr);                                                                      \
        if (e_ != cudaSuccess)                                                                        \
            return fg::set_error(e_ == cudaErrorMemoryAllocation ? FG_ERR_NOMEM : FG_ERR_CUDA,        \
                                 std::string(#expr) + ": " + cudaGetErrorString(e_));                 \
    } while (0)

// ---- one training pass over a batch: forward, loss, backward and weight gradients in one kernel,
// then a reduction over its blocks with the Adam step.
//
// A block of 256 threads takes tiles of kTrainS samples (grid-stride), keeps the parameters and the
// tile's activations in shared memory, and accumulates its share of every weight gradient in registers
// over its tiles; the block's sums go to part[block][SG_NPARAM] once, at the end.  A thread computes
// 2 samples x 4 outputs of a layer (one 16-byte read of a weight row feeds 8 multiply-adds), 4 x 4 of a
// weight gradient.  Rows have a pitch of 68 values, so that 8 lanes reading 16 bytes of 8 consecutive rows
// hit distinct banks.  Up to 4096 samples (128 blocks, one on each of 128 SMs, 20 SMs idle) the time is
// that of one tile's chain of layers: 15.4 us for 64 samples, 15.9 for 512, 16.7 for 4096, 12.7 of the
// 74 TFLOP/s.  Where every block slot is taken it is bound by FP32 multiply-adds from shared memory (26 k
// per sample): 9,472 samples 25.8 us, 16,384 44.6, 131,072 274 us, 25 TFLOP/s.
// Summation order: a block's samples in order, then the blocks in a fixed order, so training is
// deterministic for a given batch size.
// Batch 4096: 16.7 us, and 3 us for the reduction, against 230 us for the 15 launches of one layer or one
// reduction each that it replaced; an epoch of 16 batches 4.44 -> 0.70 ms.
constexpr int kTrainS = 32, kTrainThreads = 256, kTrainPitch = SG_H + 4;
constexpr int kTrainMaxBlocks = 296;   // 2 resident blocks on each of 148 SMs
constexpr int kTrainRows = kTrainS * kTrainPitch;
// shared memory (values): W2, W3 with padded rows, W1, W4, biases; per layer the tile's activations
// and the derivative of its GELU (then its dZ); inputs, targets, output gradients
constexpr int TS_W2 = 0, TS_W3 = TS_W2 + SG_H * kTrainPitch, TS_W1 = TS_W3 + SG_H * kTrainPitch,
              TS_W4 = TS_W1 + SG_IN * SG_H, TS_B = TS_W4 + SG_H * SG_OUT, TS_A = TS_B + 3 * SG_H + SG_OUT,
              TS_D = TS_A + 3 * kTrainRows, TS_X = TS_D + 3 * kTrainRows, TS_Y = TS_X + kTrainS * 4,
              TS_G = TS_Y + kTrainS * SG_OUT, TS_RED = TS_G + kTrainS * SG_OUT, TS_END = TS_RED + 8;
static_assert(TS_A % 4 == 0 && TS_W4 % 4 == 0 && TS_X % 4 == 0, "16-byte aligned rows");

// GELU (tanh form) and its derivative: with u = c (z + a z^3), th = tanh(u),
//   gelu = z / 2 (1 + th),  gelu' = (1 + th) / 2 + z / 2 (1 - th^2) c (1 + 3 a z^2)
__device__ __forceinline__ float gelu_fd(float z, float &d) {
    const float th = tanhf(SG_GELU_C * fmaf(SG_GELU_A * z, z * z, z));
    d = 0.5f * (1.0f + th) + 0.5f * z * (1.0f - th * th) * SG_GELU_C * fmaf(3.0f * SG_GELU_A * z, z, 1.0f);
    return 0.5f * z * (1.0f + th);
}
__device__ __forceinline__ void fma4(float4 &c, float a, const float4 &w) {
    c.x = fmaf(a, w.x, c.x);
    c.y = fmaf(a, w.y, c.y);
    c.z = fmaf(a, w.z, c.z);
    c.w = fmaf(a, w.w, c.w);
}
__device__ __forceinline__ float dot4(float c, const float4 &a, const float4 &w) {
    return fmaf(a.w, w.w, fmaf(a.z, w.z, fmaf(a.y, w.y, fmaf(a.x, w.x, c))));
}
// store the GELU of a thread's 4 pre-activations of a sample and its derivative
__device__ __forceinline__ void train_act(float *A, float *D, int s, int n, const float4 &z) {
    float4 a, d;
    a.x = gelu_fd(z.x, d.x);
    a.y = gelu_fd(z.y, d.y);
    a.z = gelu_fd(z.z, d.z);
    a.w = gelu_fd(z.w, d.w);
    *reinterpret_cast<float4 *>(A + s * kTrainPitch + n) = a;
    *reinterpret_cast<float4 *>(D + s * kTrainPitch + n) = d;
}
// hidden layer: A = gelu(P W + b) for the thread's samples s0, s0 + 1 and outputs n .. n + 3
__device__ __forceinline__ void train_fwd(const float *W, const float *b, const float *P, float *A, float *D, int s0, int n) {
    float4 z0 = *reinterpret_cast<const float4 *>(b + n), z1 = z0;
#pragma unroll 4
    for (int k = 0; k < SG_H; k += 4) {
        const float4 p0 = *reinterpret_cast<const float4 *>(P + s0 * kTrainPitch + k);
        const float4 p1 = *reinterpret_cast<const float4 *>(P + (s0 + 1) * kTrainPitch + k);
        const float *w = W + k * kTrainPitch + n;
        float4 r = *reinterpret_cast<const float4 *>(w);
        fma4(z0, p0.x, r);
        fma4(z1, p1.x, r);
        r = *reinterpret_cast<const float4 *>(w + kTrainPitch);
        fma4(z0, p0.y, r);
        fma4(z1, p1.y, r);
        r = *reinterpret_cast<const float4 *>(w + 2 * kTrainPitch);
        fma4(z0, p0.z, r);
        fma4(z1, p1.z, r);
        r = *reinterpret_cast<const float4 *>(w + 3 * kTrainPitch);
        fma4(z0, p0.w, r);
        fma4(z1, p1.w, r);
    }
    train_act(A, D, s0, n, z0);
    train_act(A, D, s0 + 1, n, z1);
}
// backward data: D (derivative of the layer below, becomes its dZ) *= dZ W^T, for the thread's samples
// s0, s0 + 1 and inputs kk, kk + 16, kk + 32, kk + 48
__device__ __forceinline__ void train_bwd(const float *W, const float *dZ, float *D, int s0, int kk) {
    float c[2][4] = {};
#pragma unroll 4
    for (int n = 0; n < SG_H; n += 4) {
        const float4 d0 = *reinterpret_cast<const float4 *>(dZ + s0 * kTrainPitch + n);
        const float4 d1 = *reinterpret_cast<const float4 *>(dZ + (s0 + 1) * kTrainPitch + n);
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const float4 w = *reinterpret_cast<const float4 *>(W + (kk + 16 * j) * kTrainPitch + n);
            c[0][j] = dot4(c[0][j], d0, w);
            c[1][j] = dot4(c[1][j], d1, w);
        }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) D[(s0 + i) * kTrainPitch + kk + 16 * j] *= c[i][j];
}
// weight gradient of a hidden layer: g[i] += sum over the tile's samples of A[k0 + i] dZ[n .. n + 3];
// gb += the sums of dZ (the bias gradient, used by the threads of the first row group)
__device__ __forceinline__ void train_wgrad(const float *A, const float *dZ, int k0, int n, float4 *g, float4 &gb) {
#pragma unroll 4
    for (int s = 0; s < kTrainS; s++) {
        const float4 a = *reinterpret_cast<const float4 *>(A + s * kTrainPitch + k0);
        const float4 d = *reinterpret_cast<const float4 *>(dZ + s * kTrainPitch + n);
        fma4(g[0], a.x, d);
        fma4(g[1], a.y, d);
        fma4(g[2], a.z, d);
        fma4(g[3], a.w, d);
        if (k0 == 0) fma4(gb, 1.0f, d);
    }
}

// X [.][3], Y [.][4]: the batch's samples are rows perm[0 .. B) (rows 0 .. B without perm); scale =
// 1 / (4 B).  lossPart[block]: the block's sum of squared errors.
__global__ void __launch_bounds__(kTrainThreads, 2) k_sg_train(const float *__restrict__ P, const float *__restrict__ X,
                                                               const float *__restrict__ Y, const int32_t *__restrict__ perm,
                                                               int B, float scale, float *__restrict__ part,
                                                               float *__restrict__ lossPart) {
    extern __shared__ __align__(16) float sm[];
    const int t = threadIdx.x;
    for (int q = t; q < SG_H * SG_H; q += kTrainThreads) {
        const int o = (q / SG_H) * kTrainPitch + q % SG_H;
        sm[TS_W2 + o] = P[SG_OFF_W2 + q];
        sm[TS_W3 + o] = P[SG_OFF_W3 + q];
    }
    if (t < SG_IN * SG_H) sm[TS_W1 + t] = P[SG_OFF_W1 + t];
    sm[TS_W4 + t] = P[SG_OFF_W4 + t];
    if (t < SG_H) {
        sm[TS_B + t] = P[SG_OFF_B1 + t];
        sm[TS_B + SG_H + t] = P[SG_OFF_B2 + t];
        sm[TS_B + 2 * SG_H + t] = P[SG_OFF_B3 + t];
    }
    if (t < SG_OUT) sm[TS_B + 3 * SG_H + t] = P[SG_OFF_B4 + t];
    float *A1 = sm + TS_A, *A2 = A1 + kTrainRows, *A3 = A2 + kTrainRows;
    float *D1 = sm + TS_D, *D2 = D1 + kTrainRows, *D3 = D2 + kTrainRows;
    // the thread's 2 x 4 part of a layer (forward: outputs n ..; backward: inputs kk ..) and 4 x 4
    // part of a weight gradient (rows k0 .., columns n ..)
    const int kk = t & 15, n = 4 * kk, s0 = 2 * (t >> 4), k0 = 4 * (t >> 4);
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 g2[4] = {zero, zero, zero, zero}, g3[4] = {zero, zero, zero, zero}, b2 = zero, b3 = zero;
    float g1 = 0.f, g4 = 0.f, b4 = 0.f, loss = 0.f;
    for (int tile = blockIdx.x; tile * kTrainS < B; tile += gridDim.x) {
        __syncthreads();   // the parameters are there, the previous tile is done
        if (t < kTrainS * 4) {
            const int r = tile * kTrainS + (t >> 2), c = t & 3;
            const int row = r < B ? (perm ? perm[r] : r) : -1;
            // inputs with a 1 for the bias gradient of the first layer; a missing sample adds nothing
            sm[TS_X + t] = row >= 0 ? (c < SG_IN ? X[(size_t)row * SG_IN + c] : 1.0f) : 0.0f;
            sm[TS_Y + t] = row >= 0 ? Y[(size_t)row * SG_OUT + c] : 0.0f;
        }
        __syncthreads();
        {
            const float4 w0 = *reinterpret_cast<const float4 *>(sm + TS_W1 + n), bz = *reinterpret_cast<const float4 *>(sm + TS_B + n);
            const float4 w1 = *reinterpret_cast<const float4 *>(sm + TS_W1 + SG_H + n);
            const float4 w2 = *reinterpret_cast<const float4 *>(sm + TS_W1 + 2 * SG_H + n);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float4 x = *reinterpret_cast<const float4 *>(sm + TS_X + 4 * (s0 + i));
                float4 z = bz;
                fma4(z, x.x, w0);
                fma4(z, x.y, w1);
                fma4(z, x.z, w2);
                train_act(A1, D1, s0 + i, n, z);
            }
        }
        __syncthreads();
        train_fwd(sm + TS_W2, sm + TS_B + SG_H, A1, A2, D2, s0, n);
        __syncthreads();
        train_fwd(sm + TS_W3, sm + TS_B + 2 * SG_H, A2, A3, D3, s0, n);
        __syncthreads();
        {
            // output layer and loss: sample t / 8, output (t / 2) % 4, half of the inputs t % 2
            const int s = t >> 3, o = (t >> 1) & 3, h = (t & 1) * (SG_H / 2);
            float y = 0.f;
#pragma unroll 8
            for (int k = 0; k < SG_H / 2; k++) y = fmaf(A3[s * kTrainPitch + h + k], sm[TS_W4 + (h + k) * SG_OUT + o], y);
            y += __shfl_xor_sync(0xffffffffu, y, 1);
            if (!(t & 1)) {
                const bool on = tile * kTrainS + s < B;
                const float d = on ? y + sm[TS_B + 3 * SG_H + o] - sm[TS_Y + s * SG_OUT + o] : 0.0f;
                sm[TS_G + s * SG_OUT + o] = 2.f * d * scale;
                loss = fmaf(d, d, loss);
            }
        }
        __syncthreads();
        {
            // gradients of the output layer (one weight per thread) and dZ of the third
            const int k = t >> 2, o = t & 3;
            float b = 0.f;
#pragma unroll 8
            for (int s = 0; s < kTrainS; s++) {
                g4 = fmaf(A3[s * kTrainPitch + k], sm[TS_G + s * SG_OUT + o], g4);
                b += sm[TS_G + s * SG_OUT + o];
            }
            b4 += b;
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float4 d = *reinterpret_cast<const float4 *>(sm + TS_G + (s0 + i) * SG_OUT);
#pragma unroll
                for (int j = 0; j < 4; j++)
                    D3[(s0 + i) * kTrainPitch + kk + 16 * j] *=
                        dot4(0.f, d, *reinterpret_cast<const float4 *>(sm + TS_W4 + (kk + 16 * j) * SG_OUT));
            }
        }
        __syncthreads();
        train_bwd(sm + TS_W3, D3, D2, s0, kk);
        train_wgrad(A2, D3, k0, n, g3, b3);
        __syncthreads();
        train_bwd(sm + TS_W2, D2, D1, s0, kk);
        train_wgrad(A1, D2, k0, n, g2, b2);
        __syncthreads();
        {
            // first layer: weight row t / 64 (row 3: the bias) and column t % 64
            const int k = t >> 6, c = t & 63;
#pragma unroll 8
            for (int s = 0; s < kTrainS; s++) g1 = fmaf(sm[TS_X + 4 * s + k], D1[s * kTrainPitch + c], g1);
        }
    }
    float *out = part + (size_t)blockIdx.x * SG_NPARAM;
    out[t] = g1;   // W1 [3][64], then b1
#pragma unroll
    for (int i = 0; i < 4; i++) {
        *reinterpret_cast<float4 *>(out + SG_OFF_W2 + (k0 + i) * SG_H + n) = g2[i];
        *reinterpret_cast<float4 *>(out + SG_OFF_W3 + (k0 + i) * SG_H + n) = g3[i];
    }
    if (k0 == 0) {
        *reinterpret_cast<float4 *>(out + SG_OFF_B2 + n) = b2;
        *reinterpret_cast<float4 *>(out + SG_OFF_B3 + n) = b3;
    }
    out[SG_OFF_W4 + t] = g4;
    if (t < SG_OUT) out[SG_OFF_B4 + t] = b4;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
    if ((t & 31) == 0) sm[TS_RED + (t >> 5)] = loss;
    __syncthreads();
    if (t == 0) {
        float l = 0.f;
        for (int w = 0; w < kTrainThreads / 32; w++) l += sm[TS_RED + w];
        lossPart[blockIdx.x] = l;
    }
}
static_assert(SG_OFF_B1 == SG_IN * SG_H && SG_H * (SG_IN + 1) == kTrainThreads && SG_H * SG_OUT == kTrainThreads &&
                  (SG_H / 4) * (SG_H / 4) == kTrainThreads && kTrainS * SG_OUT * 2 == kTrainThreads,
              "thread maps of k_sg_train");
static_assert(SG_OFF_W2 % 4 == 0 && SG_OFF_B2 % 4 == 0 && SG_OFF_W3 % 4 == 0 && SG_OFF_B3 % 4 == 0 && SG_NPARAM % 4 == 0,
              "16-byte gradient stores");

struct AdamStep {
    float lr, b1, b2, eps, c1, c2;
};
// G = sum of the blocks' gradients; with kAdam the parameter update.  64 parameters per block of 256
// threads, each of 4 groups summing a quarter of the blocks: 2-3 us of dependent L2 reads instead of
// 9 with one thread per parameter.
constexpr int kReduceGroups = 4, kReduceParams = 64;
template <bool kAdam>
__global__ void __launch_bounds__(kReduceGroups *kReduceParams) k_sg_reduce(const float *__restrict__ part, int blocks,
                                                                           float *P, float *G, float *M, float *V, AdamStep s) {
    __shared__ float sh[kReduceGroups][kReduceParams];
    const int lane = threadIdx.x % kReduceParams, grp = threadIdx.x / kReduceParams;
    const int i = blockIdx.x * kReduceParams + lane;
    const int per = (blocks + kReduceGroups - 1) / kReduceGroups;
    const int lo = grp * per, hi = min(blocks, lo + per);
    float a = 0.f;
    if (i < SG_NPARAM) {
#pragma unroll 8
        for (int b = lo; b < hi; b++) a += part[(size_t)b * SG_NPARAM + i];
    }
    sh[grp][lane] = a;
    __syncthreads();
    if (grp || i >= SG_NPARAM) return;
    const float g = ((sh[0][lane] + sh[1][lane]) + sh[2][lane]) + sh[3][lane];
    G[i] = g;
    if (kAdam) {
        const float m = s.b1 * M[i] + (1.f - s.b1) * g;
        const float v = s.b2 * V[i] + (1.f - s.b2) * g * g;
        M[i] = m;
        V[i] = v;
        P[i] -= s.lr * (m / s.c1) / (sqrtf(v / s.c2) + s.eps);
    }
}

// packed BF16 weights of the tensor-core layers from the FP32 parameters: one thread per element of a
// layer's operand (N rows of K, K and N padded with zeros), in the canonical layout (tc_smem_off)
__global__ void k_sg_pack(const float *__restrict__ P, unsigned char *__restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= TC_WBYTES / 2) return;
    int wOff, K, N, rows, base;
    if (i < TC_W2 / 2) { wOff = SG_OFF_W1; K = SG_IN; N = SG_H; rows = 64; base = TC_W1; }
    else if (i < TC_W3 / 2) { wOff = SG_OFF_W2; K = SG_H; N = SG_H; rows = 64; base = TC_W2; }
    else if (i < TC_W4 / 2) { wOff = SG_OFF_W3; K = SG_H; N = SG_H; rows = 64; base = TC_W3; }
    else { wOff = SG_OFF_W4; K = SG_H; N = SG_OUT; rows = 16; base = TC_W4; }
    const int q = i - base / 2, n = q % rows, k = q / rows;
    const float w = (k < K && n < N) ? P[wOff + k * N + n] : 0.f;
    *reinterpret_cast<__nv_bfloat16 *>(out + base + tc_smem_off(n, k, rows)) = __float2bfloat16_rn(w);
}

// batch prediction input: raw samples X[n][3]
struct InPredict {
    const float *X;
    int n;
    __device__ int count() const { return n; }
    __device__ void features(int i, const SurrogateNorm &N, float (&z)[3]) const {
#pragma unroll
        for (int k = 0; k < 3; k++) z[k] = (X[(size_t)i * 3 + k] - N.xMean[k]) / N.xStd[k];
    }
};

// ---------------------------------------------------------------- host helpers
bool invert3(const double *a, double *inv) {
    const double det = a[0] * (a[4] * a[8] - a[5] * a[7]) - a[1] * (a[3] * a[8] - a[5] * a[6]) +
                       a[2] * (a[3] * a[7] - a[4] * a[6]);
    if (!(std::fabs(det) > 0)) return false;
    const double id = 1.0 / det;
    inv[0] = (a[4] * a[8] - a[5] * a[7]) * id;
    inv[1] = (a[2] * a[7] - a[1] * a[8]) * id;
    inv[2] = (a[1] * a[5] - a[2] * a[4]) * id;
    inv[3] = (a[5] * a[6] - a[3] * a[8]) * id;
    inv[4] = (a[0] * a[8] - a[2] * a[6]) * id;
    inv[5] = (a[2] * a[3] - a[0] * a[5]) * id;
    inv[6] = (a[3] * a[7] - a[4] * a[6]) * id;
    inv[7] = (a[1] * a[6] - a[0] * a[7]) * id;
    inv[8] = (a[0] * a[4] - a[1] * a[3]) * id;
    return true;
}

}  // namespace

struct fg_surrogate {
    int device = 0;
    Buf P, G, M, V, pack;           // parameters, gradient, Adam moments, packed BF16 fragments
    Buf X, Y;                       // standardised training data (n x 3, n x 4)
    Buf perm;
    int64_t n = 0;
    int64_t adamStep = 0;
    SurrogateNorm norm{};
    bool hasNorm = false;
    // batch work buffers (capacity cap rows)
    int cap = 0;
    Buf bx, by;           // batch of fg_surrogate_loss_grad
    Buf part, lossPart;   // per-block gradients and losses of a training pass

    int ensure_batch(int B) {
        if (B <= cap) return FG_OK;
        SG_TRY(bx.alloc((size_t)B * SG_IN * sizeof(float)));
        SG_TRY(by.alloc((size_t)B * SG_OUT * sizeof(float)));
        cap = B;
        return FG_OK;
    }
    // work buffers of a training pass and its kernel's shared memory (above 48 KB), once
    int ensure_train() {
        if (part.p && lossPart.p) return FG_OK;
        SG_TRY(cudaFuncSetAttribute(k_sg_train, cudaFuncAttributeMaxDynamicSharedMemorySize, TS_END * (int)sizeof(float)));
        SG_TRY(part.alloc((size_t)kTrainMaxBlocks * SG_NPARAM * sizeof(float)));
        SG_TRY(lossPart.alloc(kTrainMaxBlocks * sizeof(float)));
        return FG_OK;
    }

    int repack() {
        k_sg_pack<<<(TC_WBYTES / 2 + 255) / 256, 256>>>(P.as<float>(), pack.as<unsigned char>());
        SG_TRY(cudaGetLastError());
        SG_TRY(cudaStreamSynchronize(0));
        return FG_OK;
    }

    // forward, loss and backward over B samples (rows perm[0 .. B) of x / y, standardised); the
    // gradient goes into G, and with adam the parameters take the step
    int fwd_bwd(const float *x, const float *y, const int32_t *rows, int B, const AdamStep *adam, float *lossOut, cudaStream_t s) {
        const int rc = ensure_train();
        if (rc != FG_OK) return rc;
        const int blocks = std::min((B + kTrainS - 1) / kTrainS, kTrainMaxBlocks);
        k_sg_train<<<blocks, kTrainThreads, TS_END * sizeof(float), s>>>(P.as<float>(), x, y, rows, B, 1.0f / (float)(B * SG_OUT),
                                                                         part.as<float>(), lossPart.as<float>());
        const int rb = (SG_NPARAM + kReduceParams - 1) / kReduceParams, rt = kReduceGroups * kReduceParams;
        if (adam)
            k_sg_reduce<true><<<rb, rt, 0, s>>>(part.as<float>(), blocks, P.as<float>(), G.as<float>(), M.as<float>(),
                                                V.as<float>(), *adam);
        else
            k_sg_reduce<false><<<rb, rt, 0, s>>>(part.as<float>(), blocks, P.as<float>(), G.as<float>(), M.as<float>(),
                                                 V.as<float>(), AdamStep{});
        SG_TRY(cudaGetLastError());
        if (lossOut) {
            float lp[kTrainMaxBlocks];
            SG_TRY(cudaMemcpyAsync(lp, lossPart.p, blocks * sizeof(float), cudaMemcpyDeviceToHost, s));
            SG_TRY(cudaStreamSynchronize(s));
            double sum = 0;
            for (int i = 0; i < blocks; i++) sum += lp[i];
            *lossOut = (float)(sum / ((double)B * SG_OUT));
        }
        return FG_OK;
    }
};

namespace fg {
// device view of a surrogate for the relaxation kernel
int surrogate_view(const fg_surrogate *g, SurrogateDev *out) {
    if (!g || !g->hasNorm) return fg::set_error(FG_ERR_ARG, "surrogate has no training data statistics");
    out->pack = g->pack.as<unsigned char>();
    out->params = g->P.as<float>();
    out->norm = g->norm;
    out->enabled = 1;
    return FG_OK;
}
int surrogate_device(const fg_surrogate *g) { return g ? g->device : -1; }
}  // namespace fg

extern "C" {

int fg_surrogate_create(int32_t device, uint64_t seed, fg_surrogate **out) {
    if (!out) return fg::set_error(FG_ERR_ARG, "fg_surrogate_create: null argument");
    *out = nullptr;
    SG_TRY(cudaSetDevice(device));
    fg_surrogate *g = new fg_surrogate();
    g->device = device;
    int rc = FG_OK;
    auto fail = [&](int code) { delete g; return code; };
    if (cudaSuccess != g->P.alloc(SG_NPARAM * sizeof(float)) || cudaSuccess != g->G.alloc(SG_NPARAM * sizeof(float)) ||
        cudaSuccess != g->M.alloc(SG_NPARAM * sizeof(float)) || cudaSuccess != g->V.alloc(SG_NPARAM * sizeof(float)) ||
        cudaSuccess != g->pack.alloc(TC_WBYTES))
        return fail(fg::set_error(FG_ERR_NOMEM, "fg_surrogate_create: device allocation failed"));
    // He-style initialisation: W ~ N(0, 2 / fan_in), b = 0 (seeded, reproducible)
    std::vector<float> p(SG_NPARAM, 0.f);
    std::mt19937_64 rng(seed);
    auto init = [&](int off, int K, int N) {
        std::normal_distribution<double> nd(0.0, std::sqrt(2.0 / K));
        for (int i = 0; i < K * N; i++) p[off + i] = (float)nd(rng);
    };
    init(SG_OFF_W1, SG_IN, SG_H);
    init(SG_OFF_W2, SG_H, SG_H);
    init(SG_OFF_W3, SG_H, SG_H);
    init(SG_OFF_W4, SG_H, SG_OUT);
    if (cudaMemcpy(g->P.p, p.data(), SG_NPARAM * sizeof(float), cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(g->M.p, 0, SG_NPARAM * sizeof(float)) != cudaSuccess ||
        cudaMemset(g->V.p, 0, SG_NPARAM * sizeof(float)) != cudaSuccess ||
        cudaMemset(g->G.p, 0, SG_NPARAM * sizeof(float)) != cudaSuccess)
        return fail(fg::set_error(FG_ERR_CUDA, "fg_surrogate_create: initialisation copy failed"));
    rc = g->repack();
    if (rc != FG_OK) return fail(rc);
    *out = g;
    return FG_OK;
}

int fg_surrogate_destroy(fg_surrogate *g) {
    if (!g) return FG_OK;
    cudaSetDevice(g->device);
    delete g;
    return FG_OK;
}

int fg_surrogate_set_data(fg_surrogate *g, const float *X, const float *Y, int64_t n) {
    if (!g || !X || !Y) return fg::set_error(FG_ERR_ARG, "fg_surrogate_set_data: null argument");
    if (n < 16 || n > (int64_t)INT32_MAX) return fg::set_error(FG_ERR_ARG, "fg_surrogate_set_data: need 16 .. 2^31-1 samples");
    SG_TRY(cudaSetDevice(g->device));
    // statistics of the run's samples (FP64 accumulation)
    double mx[3] = {0, 0, 0}, my[4] = {0, 0, 0, 0}, sx[3] = {0, 0, 0}, sy[4] = {0, 0, 0, 0};
    for (int64_t i = 0; i < n; i++) {
        for (int k = 0; k < 3; k++) mx[k] += X[i * 3 + k];
        for (int k = 0; k < 4; k++) my[k] += Y[i * 4 + k];
    }
    for (int k = 0; k < 3; k++) mx[k] /= (double)n;
    for (int k = 0; k < 4; k++) my[k] /= (double)n;
    for (int64_t i = 0; i < n; i++) {
        for (int k = 0; k < 3; k++) sx[k] += (X[i * 3 + k] - mx[k]) * (X[i * 3 + k] - mx[k]);
        for (int k = 0; k < 4; k++) sy[k] += (Y[i * 4 + k] - my[k]) * (Y[i * 4 + k] - my[k]);
    }
    SurrogateNorm N{};
    for (int k = 0; k < 3; k++) {
        N.xMean[k] = (float)mx[k];
        N.xStd[k] = (float)std::max(std::sqrt(sx[k] / (double)n), 1e-30);
    }
    for (int k = 0; k < 4; k++) {
        N.yMean[k] = (float)my[k];
        N.yStd[k] = (float)std::max(std::sqrt(sy[k] / (double)n), 1e-30);
    }
    std::vector<float> xs((size_t)n * 3), ys((size_t)n * 4);
    double cov[9] = {0};
    for (int k = 0; k < 3; k++) {
        N.boxLo[k] = 1e30f;
        N.boxHi[k] = -1e30f;
    }
    for (int64_t i = 0; i < n; i++) {
        float z[3];
        for (int k = 0; k < 3; k++) {
            z[k] = (X[i * 3 + k] - N.xMean[k]) / N.xStd[k];
            xs[i * 3 + k] = z[k];
            N.boxLo[k] = std::min(N.boxLo[k], z[k]);
            N.boxHi[k] = std::max(N.boxHi[k], z[k]);
        }
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) cov[3 * a + b] += (double)z[a] * z[b];
        for (int k = 0; k < 4; k++) ys[i * 4 + k] = (Y[i * 4 + k] - N.yMean[k]) / N.yStd[k];
    }
    for (double &c : cov) c /= (double)n;
    double ci[9];
    if (!invert3(cov, ci)) return fg::set_error(FG_ERR_ARG, "fg_surrogate_set_data: degenerate input covariance");
    for (int k = 0; k < 9; k++) N.covInv[k] = (float)ci[k];
    double d2m = 0;
    for (int64_t i = 0; i < n; i++) {
        double d2 = 0;
        for (int a = 0; a < 3; a++)
            for (int b = 0; b < 3; b++) d2 += (double)xs[i * 3 + a] * N.covInv[3 * a + b] * xs[i * 3 + b];
        d2m = std::max(d2m, d2);
    }
    N.d2Max = (float)d2m;
    SG_TRY(g->X.alloc(xs.size() * sizeof(float)));
    SG_TRY(g->Y.alloc(ys.size() * sizeof(float)));
    SG_TRY(g->perm.alloc((size_t)n * sizeof(int32_t)));
    SG_TRY(cudaMemcpy(g->X.p, xs.data(), xs.size() * sizeof(float), cudaMemcpyHostToDevice));
    SG_TRY(cudaMemcpy(g->Y.p, ys.data(), ys.size() * sizeof(float), cudaMemcpyHostToDevice));
    g->n = n;
    g->norm = N;
    g->hasNorm = true;
    return FG_OK;
}

int fg_surrogate_train(fg_surrogate *g, int32_t epochs, int32_t batch, float lr, uint64_t seed, float *finalLoss) {
    if (!g) return fg::set_error(FG_ERR_ARG, "fg_surrogate_train: null argument");
    if (g->n == 0) return fg::set_error(FG_ERR_ARG, "fg_surrogate_train: no training data (fg_surrogate_set_data)");
    if (epochs < 0 || batch < 32 || batch > (1 << 20) || !(lr > 0))
        return fg::set_error(FG_ERR_ARG, "fg_surrogate_train: epochs >= 0, 32 <= batch <= 2^20, lr > 0");
    SG_TRY(cudaSetDevice(g->device));
    int rc = FG_OK;
    cudaStream_t s = 0;
    std::mt19937_64 rng(seed);
    std::vector<int32_t> perm((size_t)g->n);
    for (int64_t i = 0; i < g->n; i++) perm[i] = (int32_t)i;
    const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
    double epochLoss = 0;
    for (int ep = 0; ep < epochs; ep++) {
        std::shuffle(perm.begin(), perm.end(), rng);
        SG_TRY(cudaMemcpy(g->perm.p, perm.data(), perm.size() * sizeof(int32_t), cudaMemcpyHostToDevice));
        const int64_t nb = g->n / batch;   // full batches only
        double sum = 0;
        // cosine decay of the learning rate over the whole run
        for (int64_t b = 0; b < nb; b++) {
            const bool last = (b == nb - 1);
            float l = 0;
            g->adamStep++;
            const double prog = ((double)ep * nb + b) / std::max<double>(1.0, (double)epochs * nb);
            const float lrt = (float)(lr * 0.5 * (1.0 + std::cos(3.14159265358979 * prog)));
            const float c1 = 1.f - std::pow(b1, (float)g->adamStep), c2 = 1.f - std::pow(b2, (float)g->adamStep);
            const AdamStep adam{lrt, b1, b2, eps, c1, c2};
            rc = g->fwd_bwd(g->X.as<float>(), g->Y.as<float>(), g->perm.as<int32_t>() + b * batch, batch, &adam,
                            last ? &l : nullptr, s);
            if (rc != FG_OK) return rc;
            if (last) sum = l;
        }
        SG_TRY(cudaGetLastError());
        epochLoss = sum;
    }
    SG_TRY(cudaDeviceSynchronize());
    rc = g->repack();
    if (rc != FG_OK) return rc;
    if (finalLoss) *finalLoss = (float)epochLoss;
    return FG_OK;
}

int fg_surrogate_loss_grad(fg_surrogate *g, const float *X, const float *Y, int32_t n, float *loss, float *grad) {
    if (!g || !X || !Y || !grad) return fg::set_error(FG_ERR_ARG, "fg_surrogate_loss_grad: null argument");
    if (n < 1 || n > (1 << 20)) return fg::set_error(FG_ERR_ARG, "fg_surrogate_loss_grad: 1 <= n <= 2^20");
    SG_TRY(cudaSetDevice(g->device));
    int rc = g->ensure_batch(n);
    if (rc != FG_OK) return rc;
    SG_TRY(cudaMemcpy(g->bx.p, X, (size_t)n * SG_IN * sizeof(float), cudaMemcpyHostToDevice));
    SG_TRY(cudaMemcpy(g->by.p, Y, (size_t)n * SG_OUT * sizeof(float), cudaMemcpyHostToDevice));
    float l = 0;
    rc = g->fwd_bwd(g->bx.as<float>(), g->by.as<float>(), nullptr, n, nullptr, &l, 0);
    if (rc != FG_OK) return rc;
    SG_TRY(cudaMemcpy(grad, g->G.p, SG_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    if (loss) *loss = l;
    return FG_OK;
}

int fg_surrogate_get_params(fg_surrogate *g, float *params) {
    if (!g || !params) return fg::set_error(FG_ERR_ARG, "fg_surrogate_get_params: null argument");
    SG_TRY(cudaSetDevice(g->device));
    SG_TRY(cudaMemcpy(params, g->P.p, SG_NPARAM * sizeof(float), cudaMemcpyDeviceToHost));
    return FG_OK;
}

int fg_surrogate_set_params(fg_surrogate *g, const float *params) {
    if (!g || !params) return fg::set_error(FG_ERR_ARG, "fg_surrogate_set_params: null argument");
    SG_TRY(cudaSetDevice(g->device));
    SG_TRY(cudaMemcpy(g->P.p, params, SG_NPARAM * sizeof(float), cudaMemcpyHostToDevice));
    return g->repack();
}

int fg_surrogate_get_norm(fg_surrogate *g, float *norm) {
    if (!g || !norm) return fg::set_error(FG_ERR_ARG, "fg_surrogate_get_norm: null argument");
    if (!g->hasNorm) return fg::set_error(FG_ERR_ARG, "fg_surrogate_get_norm: no training data statistics");
    std::memcpy(norm, &g->norm, sizeof(SurrogateNorm));
    return FG_OK;
}

int fg_surrogate_set_norm(fg_surrogate *g, const float *norm) {
    if (!g || !norm) return fg::set_error(FG_ERR_ARG, "fg_surrogate_set_norm: null argument");
    std::memcpy(&g->norm, norm, sizeof(SurrogateNorm));
    g->hasNorm = true;
    return FG_OK;
}

int fg_surrogate_predict(fg_surrogate *g, const float *X, int32_t n, float *Y, int32_t *inHull) {
    if (!g || !X || !Y) return fg::set_error(FG_ERR_ARG, "fg_surrogate_predict: null argument");
    if (n < 1 || n > (1 << 24)) return fg::set_error(FG_ERR_ARG, "fg_surrogate_predict: 1 <= n <= 2^24");
    SG_TRY(cudaSetDevice(g->device));
    SurrogateDev S{};
    int rc = surrogate_view(g, &S);
    if (rc != FG_OK) return rc;
    Buf dx, dy, dh, de;
    SG_TRY(dx.alloc((size_t)n * 3 * sizeof(float)));
    SG_TRY(dy.alloc((size_t)n * 4 * sizeof(float)));
    SG_TRY(dh.alloc((size_t)n * sizeof(int32_t)));
    SG_TRY(de.alloc(sizeof(int32_t)));
    SG_TRY(cudaMemset(de.p, 0, sizeof(int32_t)));
    SG_TRY(cudaMemcpy(dx.p, X, (size_t)n * 3 * sizeof(float), cudaMemcpyHostToDevice));
    const int tiles = (n + TC_M - 1) / TC_M;
    k_sg_tc<InPredict><<<std::min(tiles, 148 * 4), 128, TC_SMEM>>>(S, S.pack, InPredict{dx.as<float>(), n},
                                                                   dy.as<float4>(), dh.as<int32_t>(), de.as<int32_t>());
    SG_TRY(cudaGetLastError());
    int32_t terr = 0;
    SG_TRY(cudaMemcpy(&terr, de.p, sizeof(int32_t), cudaMemcpyDeviceToHost));
    if (terr) return fg::set_error(FG_ERR_CUDA, "fg_surrogate_predict: tensor-core completion wait timed out");
    SG_TRY(cudaMemcpy(Y, dy.p, (size_t)n * 4 * sizeof(float), cudaMemcpyDeviceToHost));
    if (inHull) SG_TRY(cudaMemcpy(inHull, dh.p, (size_t)n * sizeof(int32_t), cudaMemcpyDeviceToHost));
    return FG_OK;
}

}  // extern "C"
