// Learned Krylov initial guess (sm_103a): a small per-dof MLP, its training kernels and the
// history/feature/prediction kernels around it. No counterpart in the reference: OpenCMP starts
// CG/GMRes from the previous step's solution (opencmp/models/base_model.py:925-937).
//
// Guess. From the last k solutions h_0 = u^n, h_1 = u^{n-1}, ... (k <= 6) every dof forms the
// backward differences D_j = nabla^j u^n (j = 1..k-1). The guess is
//     x = u^n + D_1 + ... + D_p  +  S_{k-1} * y(X),      X = [D_1 / S_1, ..., D_{k-1} / S_{k-1}],
// the degree-p Newton (backward-difference) extrapolation in time plus the network's correction,
// where S_j is the root mean square of D_j over the free dofs. Without the network (or before it
// is trusted) the guess is the extrapolation alone; with p = 0 it is OpenCMP's previous-step guess.
//
// Network: y = w3 . tanh(W2 tanh(W1 x + b1) + b2) + b3 + c . x, x in R^F (F <= 8), hidden width
// H = 16, FP32. It starts with zero output (w3, b3, c = 0), so an untrained network leaves the
// extrapolation unchanged.
//
// Training minimises the initial residual the guess would give the solve: for a stored step with
// target T = (u^{n+1} - base) / S_{k-1}, the error of the guess is e = S_{k-1} (y - T) and the loss
// |A e|^2 / |b|^2 over the free rows (ocmp_guess_residual_loss). Its gradient with respect to y is
// 2 S_{k-1} A^T A e / |b|^2, formed with A and its transpose (the pattern is structurally
// symmetric; A^T x gathers through a transpose-position map), and back-propagated through the
// network by ocmp_guess_backward. Gradients are deterministic: sums over rows run in two fixed-order
// stages (per-block partial sums in shared memory, then one pass over the blocks).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "ocmp_internal.h"
#include "ocmp_ff.cuh"
#include "ocmp_spmv.cuh"

namespace ocmp {
namespace {

constexpr int kH = 16;
constexpr int kMaxF = 8;
constexpr int kMaxK = 6;
constexpr int kRowsPerBlock = 256;
constexpr int kRedBlocks = 304;  // 2 x 152 SMs: fixed grid of the deterministic reductions

struct Layout {
    int F;
    int W1, b1, W2, b2, w3, b3, c, n;  // offsets into the flat parameter vector; c = linear skip
};
__host__ __device__ inline Layout layout(int F) {
    Layout L;
    L.F = F;
    L.W1 = 0;
    L.b1 = L.W1 + kH * F;
    L.W2 = L.b1 + kH;
    L.b2 = L.W2 + kH * kH;
    L.w3 = L.b2 + kH;
    L.b3 = L.w3 + kH;
    L.c = L.b3 + 1;
    L.n = L.c + F;
    return L;
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// true in every thread of the block that finishes last; resets the counter for the next launch
__device__ __forceinline__ bool last_block(unsigned* cnt) {
    __shared__ bool last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(cnt, 1u) == gridDim.x - 1;
    __syncthreads();
    if (last) {
        __threadfence();
        if (threadIdx.x == 0) *cnt = 0;
    }
    return last;
}

// forward of one row; h1, h2 returned for the backward pass. P is in shared memory, 16-byte aligned, and
// so are W2 and b2 in it. Loops over the features are unrolled to kMaxF so that x stays in registers.
__device__ __forceinline__ float mlp_row(const float* P, const Layout& L, const float* x, float* h1,
                                         float* h2) {
#pragma unroll
    for (int j = 0; j < kH; j++) {
        float a = P[L.b1 + j];
#pragma unroll
        for (int f = 0; f < kMaxF; f++)
            if (f < L.F) a = fmaf(P[L.W1 + j * L.F + f], x[f], a);
        h1[j] = tanhf(a);
    }
#pragma unroll
    for (int j = 0; j < kH; j++) {
        float a = P[L.b2 + j];
#pragma unroll
        for (int k = 0; k < kH; k += 4) {
            const float4 w = *reinterpret_cast<const float4*>(P + L.W2 + j * kH + k);
            a = fmaf(w.x, h1[k], a);
            a = fmaf(w.y, h1[k + 1], a);
            a = fmaf(w.z, h1[k + 2], a);
            a = fmaf(w.w, h1[k + 3], a);
        }
        h2[j] = tanhf(a);
    }
    float y = P[L.b3];
#pragma unroll
    for (int j = 0; j < kH; j++) y = fmaf(P[L.w3 + j], h2[j], y);
#pragma unroll
    for (int f = 0; f < kMaxF; f++)
        if (f < L.F) y = fmaf(P[L.c + f], x[f], y);
    return y;
}

// tanh on the special-function unit (one MUFU.TANH instruction; absolute error below 1e-3): the
// per-step prediction only; training and the forward/gradient kernels use tanhf
__device__ __forceinline__ float tanh_fast(float x) {
    float y;
    asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// the same forward with F known at compile time and tanh_fast (the per-step prediction kernel)
template <int F>
__device__ __forceinline__ float mlp_row_f(const float* __restrict__ P, const float (&x)[F]) {
    constexpr int W1 = 0, B1 = kH * F, W2 = B1 + kH, B2 = W2 + kH * kH, W3 = B2 + kH, B3 = W3 + kH, CC = B3 + 1;
    float h1[kH];
#pragma unroll
    for (int j = 0; j < kH; j++) {
        float a = P[B1 + j];
#pragma unroll
        for (int f = 0; f < F; f++) a = fmaf(P[W1 + j * F + f], x[f], a);
        h1[j] = tanh_fast(a);
    }
    float y = P[B3];
#pragma unroll
    for (int j = 0; j < kH; j++) {
        float a = P[B2 + j];
#pragma unroll
        for (int k = 0; k < kH; k++) a = fmaf(P[W2 + j * kH + k], h1[k], a);
        y = fmaf(P[W3 + j], tanh_fast(a), y);
    }
#pragma unroll
    for (int f = 0; f < F; f++) y = fmaf(P[CC + f], x[f], y);
    return y;
}

__global__ void __launch_bounds__(kRowsPerBlock) mlp_forward_kernel(int64_t rows, int F, const float* __restrict__ Pg,
                                                                    const float* __restrict__ X, float* __restrict__ Y) {
    extern __shared__ __align__(16) float P[];
    const Layout L = layout(F);
    for (int k = threadIdx.x; k < L.n; k += blockDim.x) P[k] = Pg[k];
    __syncthreads();
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= rows) return;
    float x[kMaxF], h1[kH], h2[kH];
#pragma unroll
    for (int f = 0; f < kMaxF; f++) x[f] = f < F ? X[r * F + f] : 0.f;
    Y[r] = mlp_row(P, L, x, h1, h2);
}

// Per row: forward and the gradient of the row's loss term with respect to y, either
//   mean squared error (T given): dy = 2 (y - t) / rows, loss term (y - t)^2 / rows, or
//   an upstream gradient (dY given): dy = dY[r], no loss;
// then the row's parameter gradients, outer products d2 x h1 (W2), d1 x x (W1), dy x h2 (w3), dy x x (c)
// and the sums of d2, d1, dy (the biases). A warp takes 32 rows at a time, a row per lane, and stages the
// six vectors in shared memory as one record per row; then its lanes turn from rows to parameters: a lane
// owns a 4 x 4 block of one of the outer products (at most 30 of them) and adds the 32 rows from two
// 16-byte reads each. The block keeps its sums in registers over all its rows and writes one partial
// gradient vector. Bound by the FP32 pipe and the shared-memory reads of the weights; a thread per
// parameter with two reads per product, a loss summed by one thread and a vector per 256 rows took 80 us
// at 185,193 rows and 68 more to add the 724 vectors, in an evaluation (forward, residual loss, backward)
// of 306 us that takes 173 now.
constexpr int kGradWarps = 8;
constexpr int kRecord = 4 * kH + kMaxF + 4;   // d2, h1, d1, h2, x, (dy, 0, 0, 0): lanes' records 48 bytes apart in the banks
constexpr int kGradBlocks = 2 * 152;          // as many partial vectors at most
static_assert(kRowsPerBlock == 32 * kGradWarps, "a row per thread");
static_assert(kRecord >= (kH * kMaxF + 2 * kH + kH * kH + kH + 1 + kMaxF + 31) / 32, "a warp's records hold its parameters");
__global__ void __launch_bounds__(kRowsPerBlock, 2) mlp_grad_partial_kernel(int64_t rows, int F,
                                                                         const float* __restrict__ Pg,
                                                                         const float* __restrict__ X,
                                                                         const float* __restrict__ T,
                                                                         const float* __restrict__ dY,
                                                                         float* __restrict__ Gpart,
                                                                         double* __restrict__ Lpart) {
    extern __shared__ __align__(16) float gsm[];
    __shared__ double sloss[kGradWarps];
    const Layout L = layout(F);
    float* P = gsm;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    float* rec = gsm + ((L.n + 3) & ~3) + w * (32 * kRecord);
    for (int k = tid; k < L.n; k += blockDim.x) P[k] = Pg[k];
    __syncthreads();
    constexpr int kD2 = 0, kH1 = kH, kD1 = 2 * kH, kH2 = 3 * kH, kX = 4 * kH, kDy = 4 * kH + kMaxF;
    // this lane's block of an outer product: quads a and b of the record
    const int fq = (F + 3) / 4;
    int a_off = kDy, b_off = kX;
    if (lane < 16) {
        a_off = kD2 + 4 * (lane >> 2);
        b_off = kH1 + 4 * (lane & 3);
    } else if (lane < 16 + 4 * fq) {
        a_off = kD1 + 4 * ((lane - 16) / fq);
        b_off = kX + 4 * ((lane - 16) % fq);
    } else if (lane < 20 + 4 * fq)
        b_off = kH2 + 4 * (lane - 16 - 4 * fq);
    else if (lane < 20 + 5 * fq)
        b_off = kX + 4 * (lane - 20 - 4 * fq);
    float acc[4][4] = {}, sum[4] = {};
    double loss = 0;
    for (int64_t c = blockIdx.x * (int64_t)kGradWarps + w; c * 32 < rows; c += (int64_t)gridDim.x * kGradWarps) {
        const int64_t r = c * 32 + lane;
        float x[kMaxF], h1[kH], h2[kH], d2[kH], d1[kH];
        float dy = 0.f;
        const int64_t rr = r < rows ? r : rows - 1;
#pragma unroll
        for (int f = 0; f < kMaxF; f++) x[f] = f < F ? X[rr * F + f] : 0.f;
        const float y = mlp_row(P, L, x, h1, h2);
        // the weights are read again below: kept in registers they would spill
        asm volatile("" ::: "memory");
        if (r < rows) {
            if (T) {
                const float e = y - T[r];
                dy = 2.f * e / (float)rows;
                loss += (double)e * (double)e;
            } else
                dy = dY[r];
        }
#pragma unroll
        for (int j = 0; j < kH; j++) d2[j] = dy * P[L.w3 + j] * (1.f - h2[j] * h2[j]);
#pragma unroll
        for (int k = 0; k < kH; k++) d1[k] = 0.f;
#pragma unroll
        for (int j = 0; j < kH; j++)
#pragma unroll
            for (int k = 0; k < kH; k += 4) {
                const float4 v = *reinterpret_cast<const float4*>(P + L.W2 + j * kH + k);
                d1[k] = fmaf(v.x, d2[j], d1[k]);
                d1[k + 1] = fmaf(v.y, d2[j], d1[k + 1]);
                d1[k + 2] = fmaf(v.z, d2[j], d1[k + 2]);
                d1[k + 3] = fmaf(v.w, d2[j], d1[k + 3]);
            }
        float4* q = reinterpret_cast<float4*>(rec + lane * kRecord);
#pragma unroll
        for (int k = 0; k < kH; k += 4) {
#pragma unroll
            for (int u = 0; u < 4; u++) d1[k + u] *= 1.f - h1[k + u] * h1[k + u];
            q[(kD2 + k) / 4] = make_float4(d2[k], d2[k + 1], d2[k + 2], d2[k + 3]);
            q[(kH1 + k) / 4] = make_float4(h1[k], h1[k + 1], h1[k + 2], h1[k + 3]);
            q[(kD1 + k) / 4] = make_float4(d1[k], d1[k + 1], d1[k + 2], d1[k + 3]);
            q[(kH2 + k) / 4] = make_float4(h2[k], h2[k + 1], h2[k + 2], h2[k + 3]);
        }
#pragma unroll
        for (int f = 0; f < kMaxF; f += 4) q[(kX + f) / 4] = make_float4(x[f], x[f + 1], x[f + 2], x[f + 3]);
        q[kDy / 4] = make_float4(dy, 0.f, 0.f, 0.f);
        __syncwarp();
#pragma unroll 4
        for (int t = 0; t < 32; t++) {
            const float4 a = *reinterpret_cast<const float4*>(rec + t * kRecord + a_off);
            const float4 b = *reinterpret_cast<const float4*>(rec + t * kRecord + b_off);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int u = 0; u < 4; u++) {
                sum[u] += av[u];
#pragma unroll
                for (int v = 0; v < 4; v++) acc[u][v] = fmaf(av[u], bv[v], acc[u][v]);
            }
        }
        __syncwarp();
    }
    // the warp's sums as a parameter vector over its records, then the block's
#pragma unroll
    for (int u = 0; u < 4; u++)
#pragma unroll
        for (int v = 0; v < 4; v++) {
            const float g = acc[u][v];
            if (lane < 16) rec[L.W2 + (a_off - kD2 + u) * kH + b_off - kH1 + v] = g;
            else if (lane < 16 + 4 * fq) {
                if (b_off - kX + v < F) rec[L.W1 + (a_off - kD1 + u) * F + b_off - kX + v] = g;
            } else if (u == 0 && lane < 20 + 4 * fq)
                rec[L.w3 + b_off - kH2 + v] = g;
            else if (u == 0 && lane < 20 + 5 * fq && b_off - kX + v < F)
                rec[L.c + b_off - kX + v] = g;
        }
#pragma unroll
    for (int u = 0; u < 4; u++) {
        if (lane < 16 && b_off == kH1) rec[L.b2 + a_off - kD2 + u] = sum[u];
        else if (lane >= 16 && lane < 16 + 4 * fq && b_off == kX) rec[L.b1 + a_off - kD1 + u] = sum[u];
    }
    if (lane == 16 + 4 * fq) rec[L.b3] = sum[0];
    if (T) {
        loss = warp_sum_d(loss);
        if (lane == 0) sloss[w] = loss / (double)rows;
    }
    __syncthreads();
    const float* first = gsm + ((L.n + 3) & ~3);
    for (int p = tid; p < L.n; p += blockDim.x) {
        float g = first[p];
#pragma unroll
        for (int v = 1; v < kGradWarps; v++) g += first[v * (32 * kRecord) + p];
        Gpart[(int64_t)blockIdx.x * L.n + p] = g;
    }
    if (tid == 0) {
        double ls = 0;
        if (T)
            for (int v = 0; v < kGradWarps; v++) ls += sloss[v];
        Lpart[blockIdx.x] = ls;
    }
}

// G[p] = sum over blocks of Gpart[b][p]; loss likewise (nl: 0 without one). 32 parameters per block, a
// warp per eighth of the vectors.
__global__ void __launch_bounds__(256) mlp_grad_reduce_kernel(int nblocks, int n, const float* __restrict__ Gpart,
                                                              float* __restrict__ G, const double* __restrict__ Lpart,
                                                              int nl, double* __restrict__ loss) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, p = blockIdx.x * 32 + lane;
    float acc = 0.f;
    if (p < n)
#pragma unroll 8
        for (int b = w; b < nblocks; b += 8) acc += Gpart[(int64_t)b * n + p];
    part[w][lane] = acc;
    __syncthreads();
    if (w == 0 && p < n) {
#pragma unroll
        for (int v = 1; v < 8; v++) acc += part[v][lane];
        G[p] = acc;
    }
    if (blockIdx.x == 0 && w == 1) {
        double s = 0;
        for (int q = lane; q < nl; q += 32) s += Lpart[q];
        if (nl) s = warp_sum_d(s);
        if (lane == 0) *loss = s;
    }
}

__global__ void adam_kernel(int n, float* __restrict__ P, const float* __restrict__ G, float* __restrict__ Mm,
                            float* __restrict__ Vv, float lr, float b1, float b2, float eps, float c1, float c2) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const float g = G[p];
    const float m = b1 * Mm[p] + (1.f - b1) * g;
    const float v = b2 * Vv[p] + (1.f - b2) * g * g;
    Mm[p] = m;
    Vv[p] = v;
    P[p] -= lr * (m / c1) / (sqrtf(v / c2) + eps);
}

// ---- the history as a backward-difference table in double-float ---------------------------------
// Row j of the table (n (hi, lo) float pairs, rows stored one after another) holds nabla^j u^n; row
// 0 is u^n itself. Every operation on it runs on the FP32 pipes (this part's FP64 rate is 1/58 of
// FP32): doubles are split into pairs with integer operations, differences and sums are TwoSum-exact
// float-pair arithmetic (about 48 significant bits), and only the final guess is widened to FP64.

__device__ __forceinline__ float2 tab_at(const float2* __restrict__ tab, int64_t n, int j, int64_t i) {
    return __ldg(tab + (int64_t)j * n + i);
}

// push u^{n+1}: row 0 <- u^{n+1}; row j <- (new row j-1) - (old row j-1) for 0 < j < min(m + 1, K).
// All old rows are loaded before any store, so the loads are in flight together.
template <int K>
__global__ void push_kernel(int64_t n, int m, float2* __restrict__ tab, const double* __restrict__ u) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 old[K];
#pragma unroll
    for (int j = 0; j < K; j++)
        if (j < m) old[j] = tab[(int64_t)j * n + i];
    float2 cur = split_d(u[i]);
    float2 nw[K];
#pragma unroll
    for (int j = 0; j < K; j++) {
        nw[j] = cur;
        if (j < m) cur = ff_addn(cur, old[j], true);
    }
    const int mn = m + 1 < K ? m + 1 : K;
#pragma unroll
    for (int j = 0; j < K; j++)
        if (j < mn) tab[(int64_t)j * n + i] = nw[j];
}

// S_j = sqrt(mean over free dofs of (row j)^2), j = 1..K-1 (from the high parts, floored at 1e-300),
// into sc[j-1]; as floats 1 / S_j and S_j into ((float*)(sc + 8))[j-1] and [8 + j-1]. One launch of
// kRedBlocks blocks, the last block summing the per-block partials in block order.
template <int K>
__global__ void __launch_bounds__(256) hist_scales_kernel(int64_t n, const float2* __restrict__ tab,
                                                          const uint8_t* __restrict__ freed,
                                                          double* __restrict__ part, unsigned* __restrict__ cnt,
                                                          double* __restrict__ sc) {
    constexpr int NQ = K;  // K-1 sums of squares + the free count
    float acc[NQ];
#pragma unroll
    for (int q = 0; q < NQ; q++) acc[q] = 0.f;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (freed && !freed[i]) continue;
#pragma unroll
        for (int j = 1; j < K; j++) {
            const float d = tab_at(tab, n, j, i).x;
            acc[j - 1] = fmaf(d, d, acc[j - 1]);
        }
        acc[K - 1] += 1.f;
    }
    __shared__ double sh[NQ][8];
#pragma unroll
    for (int q = 0; q < NQ; q++) {
        const double s = warp_sum_d((double)acc[q]);
        if ((threadIdx.x & 31) == 0) sh[q][threadIdx.x >> 5] = s;
    }
    __syncthreads();
    if (threadIdx.x < NQ) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[threadIdx.x][w];
        part[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
    }
    if (!last_block(cnt)) return;
    if (threadIdx.x < NQ) {
        double t = 0;
        for (unsigned b = 0; b < gridDim.x; b++) t += __ldcg(part + (int64_t)threadIdx.x * gridDim.x + b);
        sh[threadIdx.x][0] = t;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        const double nf = fmax(sh[K - 1][0], 1.0);
        float* fs = reinterpret_cast<float*>(sc + 8);
        for (int j = 1; j < K; j++) {
            const double S = fmax(sqrt(sh[j - 1][0] / nf), 1e-300);
            sc[j - 1] = S;
            fs[j - 1] = (float)(1.0 / S);
            fs[8 + j - 1] = (float)S;
        }
    }
}

// X[i] = [D_1 / S_1, ..., D_{K-1} / S_{K-1}] (FP32, F = K-1 per row); zero rows at constrained dofs
template <int K>
__global__ void features_kernel(int64_t n, const float2* __restrict__ tab, const uint8_t* __restrict__ freed,
                                const double* __restrict__ sc, float* __restrict__ X) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    constexpr int F = K - 1;
    const float* __restrict__ inv = reinterpret_cast<const float*>(sc + 8);
    const bool fr = freed == nullptr || freed[i];
#pragma unroll
    for (int j = 1; j < K; j++) X[i * F + j - 1] = fr ? tab_at(tab, n, j, i).x * inv[j - 1] : 0.f;
}

// x = u^n + D_1 + ... + D_base (+ S_{K-1} y(X) with the network) on free dofs, u^n elsewhere
template <int K, bool NET>
__global__ void __launch_bounds__(256) predict_kernel(int64_t n, const float2* __restrict__ tab,
                                                      const uint8_t* __restrict__ freed,
                                                      const double* __restrict__ sc, int base,
                                                      const float* __restrict__ Pg, int np,
                                                      double* __restrict__ x) {
    extern __shared__ float P[];
    if (NET) {
        for (int k = threadIdx.x; k < np; k += blockDim.x) P[k] = Pg[k];
        __syncthreads();
    }
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float2 D[K];
#pragma unroll
    for (int j = 0; j < K; j++) D[j] = tab_at(tab, n, j, i);
    if (freed && !freed[i]) {
        x[i] = ff_to_double(D[0].x, D[0].y);
        return;
    }
    float2 v = D[0];
#pragma unroll
    for (int j = 1; j < K; j++)
        if (j <= base) v = ff_addn(v, D[j], false);
    if constexpr (NET && K >= 2) {
        constexpr int F = K - 1;
        const float* __restrict__ fs = reinterpret_cast<const float*>(sc + 8);
        float xf[F];
#pragma unroll
        for (int j = 1; j <= F; j++) xf[j - 1] = D[j].x * fs[j - 1];
        v = ff_addn(v, make_float2(fs[8 + F - 1] * mlp_row_f<F>(P, xf), 0.f), false);
    }
    x[i] = ff_to_double(v.x, v.y);
}

// training target T_i = (u^{n+1}_i - u^n_i - D_1 - ... - D_base) / S_{K-1} (0 at constrained dofs)
template <int K>
__global__ void target_kernel(int64_t n, const float2* __restrict__ tab, const uint8_t* __restrict__ freed,
                              const double* __restrict__ sc, int base, const double* __restrict__ unext,
                              float* __restrict__ T) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (freed && !freed[i]) {
        T[i] = 0.f;
        return;
    }
    float2 d = split_d(unext[i]);
#pragma unroll
    for (int j = 0; j < K; j++)
        if (j <= base) d = ff_addn(d, tab_at(tab, n, j, i), true);
    const float* __restrict__ fs = reinterpret_cast<const float*>(sc + 8);
    T[i] = fmaxf(-1e6f, fminf(1e6f, __fadd_rn(d.x, d.y) * fs[K >= 2 ? K - 2 : 0]));
}

// e = S (Y - T) on free dofs, 0 elsewhere
__global__ void guess_error_kernel(int64_t n, const float* __restrict__ Y, const float* __restrict__ T,
                                   const double* __restrict__ scale, const uint8_t* __restrict__ freed,
                                   double* __restrict__ e) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    e[i] = (freed == nullptr || freed[i]) ? scale[0] * ((double)Y[i] - (double)T[i]) : 0.0;
}

// v := v on free rows, 0 elsewhere; out[0] = |v_free|^2, out[1] = |b_free|^2 (deterministic)
__global__ void __launch_bounds__(256) mask_norms_kernel(int64_t n, double* __restrict__ v,
                                                         const double* __restrict__ b,
                                                         const uint8_t* __restrict__ freed,
                                                         double* __restrict__ part, unsigned* __restrict__ cnt,
                                                         double* __restrict__ out) {
    double av = 0, ab = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        if (freed && !freed[i]) {
            v[i] = 0.0;
            continue;
        }
        const double vi = v[i], bi = b[i];
        av += vi * vi;
        ab += bi * bi;
    }
    __shared__ double sh[2][8];
    av = warp_sum_d(av);
    ab = warp_sum_d(ab);
    if ((threadIdx.x & 31) == 0) {
        sh[0][threadIdx.x >> 5] = av;
        sh[1][threadIdx.x >> 5] = ab;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        double t = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) t += sh[threadIdx.x][w];
        part[(int64_t)threadIdx.x * gridDim.x + blockIdx.x] = t;
    }
    if (!last_block(cnt)) return;
    // the blocks' partials: four warps per sum (one thread adding all 304 took 15 us)
    const int w = threadIdx.x >> 5, which = w >> 2;
    double t = 0;
    for (unsigned b2 = (threadIdx.x & 127); b2 < gridDim.x; b2 += 128) t += __ldcg(part + (int64_t)which * gridDim.x + b2);
    t = warp_sum_d(t);
    if ((threadIdx.x & 31) == 0) sh[which][w & 3] = t;
    __syncthreads();
    if (threadIdx.x < 2) out[threadIdx.x] = (sh[threadIdx.x][0] + sh[threadIdx.x][1]) + (sh[threadIdx.x][2] + sh[threadIdx.x][3]);
}

// dY_i = 2 wt S w_i / |b|^2 on free rows; loss = wt |A e|^2 / |b|^2 into nrm[2]
__global__ void guess_dy_kernel(int64_t n, const double* __restrict__ w, const double* __restrict__ scale,
                                const uint8_t* __restrict__ freed, double wt, double* __restrict__ nrm,
                                float* __restrict__ dY) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const double c = wt / (nrm[1] > 0 ? nrm[1] : 1.0);
    if (i == 0) nrm[2] = c * nrm[0];
    if (i >= n) return;
    dY[i] = (freed == nullptr || freed[i]) ? (float)(2.0 * c * scale[0] * w[i]) : 0.f;
}

// transpose positions of a structurally symmetric CSR pattern: tpos[k] = position of (col[k], row)
// in row col[k]; a missing mirror entry raises the flag
__global__ void tpos_kernel(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                            int32_t* __restrict__ tpos, int* __restrict__ bad) {
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (int32_t k = rp[r]; k < rp[r + 1]; k++) {
        const int32_t c = col[k];
        int32_t lo = rp[c], hi = rp[c + 1] - 1, at = -1;
        while (lo <= hi) {
            const int32_t mid = (lo + hi) >> 1;
            const int32_t v = col[mid];
            if (v == (int32_t)r) {
                at = mid;
                break;
            }
            if (v < (int32_t)r) lo = mid + 1;
            else hi = mid - 1;
        }
        tpos[k] = at < 0 ? k : at;
        if (at < 0) *bad = 1;
    }
}

// y = A^T x: row r gathers A[tpos[k]] x[col[k]] (the entries of column r), TPR lanes per row
template <int TPR>
__global__ void __launch_bounds__(256) spmv_t_kernel(int64_t n, const int32_t* __restrict__ rp,
                                                     const int32_t* __restrict__ col,
                                                     const int32_t* __restrict__ tpos, const double* __restrict__ A,
                                                     const double* __restrict__ x, double* __restrict__ y) {
    const int64_t r = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / TPR;
    const int lane = threadIdx.x % TPR;
    double acc = 0;
    if (r < n)
        for (int32_t k = rp[r] + lane; k < rp[r + 1]; k += TPR) acc += __ldg(A + __ldg(tpos + k)) * __ldg(x + __ldg(col + k));
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPR);
    if (r < n && lane == 0) y[r] = acc;
}

}  // namespace
}  // namespace ocmp

using namespace ocmp;

struct ocmp_guess_s {
    int F = 0;
    Layout L;
    float* P = nullptr;
    float* G = nullptr;
    float* M = nullptr;
    float* V = nullptr;
    float* Gpart = nullptr;
    double* Lpart = nullptr;
    double* loss = nullptr;
    int step = 0;
    double* spart = nullptr;  // reduction partials (kRedBlocks x up to kMaxK)
    unsigned* scnt = nullptr;
    double* nrm = nullptr;    // |A e|^2, |b|^2, loss
    double* vecs = nullptr;   // residual-loss workspace: e, A e, A^T A e (3 n-vectors)
    int64_t vec_n = 0;
};

static void guess_free(ocmp_guess_s* g) {
    void* ps[] = {g->P, g->G, g->M, g->V, g->Gpart, g->Lpart, g->loss, g->spart, g->scnt, g->nrm, g->vecs};
    for (void* p : ps) dfree(p);
}

static int ensure_parts(ocmp_guess_s* g) {
    if (g->Gpart && g->Lpart) return OCMP_OK;
    int st = dalloc(&g->Gpart, (size_t)kGradBlocks * g->L.n);
    if (!st) st = dalloc(&g->Lpart, (size_t)kGradBlocks);
    if (st) return st;
    return OCMP_OK;
}

static int ensure_vecs(ocmp_guess_s* g, int64_t n) {
    if (n <= g->vec_n) return OCMP_OK;
    dfree(g->vecs);
    g->vecs = nullptr;
    int st = dalloc(&g->vecs, (size_t)(3 * n));
    if (st) return st;
    g->vec_n = n;
    return OCMP_OK;
}

static int ensure_tpos(ocmp_space_s* s, cudaStream_t st) {
    if (s->d_tpos) return OCMP_OK;
    int* bad = nullptr;
    int rc = dalloc(&s->d_tpos, (size_t)s->nnz);
    if (!rc) rc = dalloc(&bad, 1);
    if (rc) {
        dfree(bad);
        return rc;
    }
    int hb = 0;
    OCMP_CUDA(cudaMemsetAsync(bad, 0, sizeof(int), st));
    OCMP_LAUNCH(tpos_kernel<<<(unsigned)((s->ndof + 255) / 256), 256, 0, st>>>(s->ndof, s->d_rowptr, s->d_col, s->d_tpos,
                                                                           bad));
    OCMP_CUDA(cudaMemcpyAsync(&hb, bad, sizeof(int), cudaMemcpyDeviceToHost, st));
    OCMP_CUDA(cudaStreamSynchronize(st));
    dfree(bad);
    if (hb) {
        dfree(s->d_tpos);
        s->d_tpos = nullptr;
        return fail(OCMP_ERR_UNSUPPORTED, "transpose product: the sparsity pattern is not structurally symmetric");
    }
    return OCMP_OK;
}

static int launch_spmv_t(ocmp_space_s* s, const double* A, const double* x, double* y, cudaStream_t st) {
    int rc = ensure_tpos(s, st);
    if (rc) return rc;
    const int64_t n = s->ndof;
    OCMP_LAUNCH(spmv_t_kernel<4><<<(unsigned)((n * 4 + 255) / 256), 256, 0, st>>>(n, s->d_rowptr, s->d_col, s->d_tpos, A, x,
                                                                              y));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

// dynamic shared memory of the gradient kernel
static size_t grad_smem(int F) { return sizeof(float) * (((layout(F).n + 3) & ~3) + kRowsPerBlock * kRecord); }

// K dispatch (history length 1..6) for a kernel template taking <int K>
#define OCMP_K_DISPATCH(k, ...)                           \
    switch (k) {                                          \
    case 1: { constexpr int KK = 1; __VA_ARGS__; } break;  \
    case 2: { constexpr int KK = 2; __VA_ARGS__; } break;  \
    case 3: { constexpr int KK = 3; __VA_ARGS__; } break;  \
    case 4: { constexpr int KK = 4; __VA_ARGS__; } break;  \
    case 5: { constexpr int KK = 5; __VA_ARGS__; } break;  \
    default: { constexpr int KK = 6; __VA_ARGS__; } break; \
    }

extern "C" {

int ocmp_guess_create(int32_t n_features, uint64_t seed, ocmp_guess_t* out) {
    if (!out || n_features < 1 || n_features > kMaxF) return fail(OCMP_ERR_ARG, "ocmp_guess_create: 1..8 features");
    auto* g = new ocmp_guess_s();
    g->F = n_features;
    g->L = layout(n_features);
    const int n = g->L.n;
    int st = smem_limit((const void*)mlp_grad_partial_kernel, grad_smem(kMaxF));
    if (!st) st = dalloc(&g->P, n);
    if (!st) st = dalloc(&g->G, n);
    if (!st) st = dalloc(&g->M, n);
    if (!st) st = dalloc(&g->V, n);
    if (!st) st = dalloc(&g->loss, 1);
    if (!st) st = dalloc(&g->spart, (size_t)kRedBlocks * kMaxK);
    if (!st) st = dalloc(&g->scnt, 1);
    if (!st) st = dalloc(&g->nrm, 4);
    if (st) {
        guess_free(g);
        delete g;
        return st;
    }
    // Xavier-uniform hidden weights from a 64-bit LCG seeded by `seed`; zero biases; zero output
    // layer and linear skip, so the untrained network adds nothing to the extrapolation
    std::vector<float> h(n, 0.f);
    uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
    auto rnd = [&]() {
        s = s * 6364136223846793005ull + 1442695040888963407ull;
        return (double)(s >> 11) * (1.0 / 9007199254740992.0);
    };
    const Layout& L = g->L;
    const double a1 = std::sqrt(6.0 / (n_features + kH)), a2 = std::sqrt(6.0 / (2 * kH));
    for (int k = 0; k < kH * n_features; k++) h[L.W1 + k] = (float)((2 * rnd() - 1) * a1);
    for (int k = 0; k < kH * kH; k++) h[L.W2 + k] = (float)((2 * rnd() - 1) * a2);
    std::vector<float> z(n, 0.f);
    if (cudaMemcpy(g->P, h.data(), sizeof(float) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(g->M, z.data(), sizeof(float) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemcpy(g->V, z.data(), sizeof(float) * n, cudaMemcpyHostToDevice) != cudaSuccess ||
        cudaMemset(g->scnt, 0, sizeof(unsigned)) != cudaSuccess) {
        guess_free(g);
        delete g;
        return fail(OCMP_ERR_CUDA, "ocmp_guess_create: upload failed");
    }
    *out = g;
    return OCMP_OK;
}

int ocmp_guess_destroy(ocmp_guess_t g) {
    if (!g) return OCMP_OK;
    guess_free(g);
    delete g;
    return OCMP_OK;
}

int ocmp_guess_nparams(ocmp_guess_t g) { return g ? g->L.n : -1; }

int ocmp_guess_params(ocmp_guess_t g, float* host, int32_t set) {
    if (!g || !host) return fail(OCMP_ERR_ARG, "ocmp_guess_params: null argument");
    if (set) {
        OCMP_CUDA(cudaMemcpy(g->P, host, sizeof(float) * g->L.n, cudaMemcpyHostToDevice));
        g->step = 0;
        OCMP_CUDA(cudaMemset(g->M, 0, sizeof(float) * g->L.n));
        OCMP_CUDA(cudaMemset(g->V, 0, sizeof(float) * g->L.n));
    } else {
        OCMP_CUDA(cudaMemcpy(host, g->P, sizeof(float) * g->L.n, cudaMemcpyDeviceToHost));
    }
    return OCMP_OK;
}

int ocmp_guess_forward(ocmp_guess_t g, const float* X, int64_t rows, float* Y, void* stream) {
    if (!g || !X || !Y || rows < 0) return fail(OCMP_ERR_ARG, "ocmp_guess_forward: bad argument");
    if (rows == 0) return OCMP_OK;
    OCMP_LAUNCH(mlp_forward_kernel<<<(unsigned)((rows + kRowsPerBlock - 1) / kRowsPerBlock), kRowsPerBlock,
                         sizeof(float) * g->L.n, (cudaStream_t)stream>>>(rows, g->F, g->P, X, Y));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

static int grad_launch(ocmp_guess_t g, const float* X, const float* T, const float* dY, int64_t rows,
                       cudaStream_t s) {
    int st = ensure_parts(g);
    if (st) return st;
    // two blocks fit on an SM; more blocks would only mean more partial vectors
    const int nb = (int)std::min<int64_t>((rows + kRowsPerBlock - 1) / kRowsPerBlock, kGradBlocks);
    const size_t smem = grad_smem(g->F);
    OCMP_LAUNCH(mlp_grad_partial_kernel<<<nb, kRowsPerBlock, smem, s>>>(rows, g->F, g->P, X, T, dY, g->Gpart, g->Lpart));
    OCMP_LAUNCH(mlp_grad_reduce_kernel<<<(g->L.n + 31) / 32, 256, 0, s>>>(nb, g->L.n, g->Gpart, g->G, g->Lpart, T ? nb : 0,
                                                                       g->loss));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_guess_loss_grad(ocmp_guess_t g, const float* X, const float* T, int64_t rows, double* loss_host,
                         float* grad_host, void* stream) {
    if (!g || !X || !T || rows <= 0) return fail(OCMP_ERR_ARG, "ocmp_guess_loss_grad: bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    int st = grad_launch(g, X, T, nullptr, rows, s);
    if (st) return st;
    if (loss_host) {
        OCMP_CUDA(cudaMemcpyAsync(loss_host, g->loss, sizeof(double), cudaMemcpyDeviceToHost, s));
        OCMP_CUDA(cudaStreamSynchronize(s));
    }
    if (grad_host) {
        OCMP_CUDA(cudaMemcpyAsync(grad_host, g->G, sizeof(float) * g->L.n, cudaMemcpyDeviceToHost, s));
        OCMP_CUDA(cudaStreamSynchronize(s));
    }
    return OCMP_OK;
}

int ocmp_guess_backward(ocmp_guess_t g, const float* X, const float* dY, int64_t rows, float* grad_host,
                        void* stream) {
    if (!g || !X || !dY || rows <= 0) return fail(OCMP_ERR_ARG, "ocmp_guess_backward: bad argument");
    cudaStream_t s = (cudaStream_t)stream;
    int st = grad_launch(g, X, nullptr, dY, rows, s);
    if (st) return st;
    if (grad_host) {
        OCMP_CUDA(cudaMemcpyAsync(grad_host, g->G, sizeof(float) * g->L.n, cudaMemcpyDeviceToHost, s));
        OCMP_CUDA(cudaStreamSynchronize(s));
    }
    return OCMP_OK;
}

int ocmp_guess_adam_step(ocmp_guess_t g, float lr, void* stream) {
    if (!g) return fail(OCMP_ERR_ARG, "ocmp_guess_adam_step: null argument");
    g->step++;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)g->step), c2 = 1.f - std::pow(b2, (float)g->step);
    OCMP_LAUNCH(adam_kernel<<<(g->L.n + 255) / 256, 256, 0, (cudaStream_t)stream>>>(g->L.n, g->P, g->G, g->M, g->V, lr, b1, b2,
                                                                        1e-8f, c1, c2));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_guess_push(int64_t n, int32_t k, int32_t m, float* tab, const double* u, void* stream) {
    if (!tab || !u || n < 0 || k < 1 || k > kMaxK || m < 0 || m > k)
        return fail(OCMP_ERR_ARG, "ocmp_guess_push: bad argument (table of 1..6 rows, 0 <= m <= k)");
    if (n == 0) return OCMP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    float2* T2 = reinterpret_cast<float2*>(tab);
    OCMP_K_DISPATCH(k, OCMP_LAUNCH(push_kernel<KK><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, m, T2, u)));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_guess_features(ocmp_guess_t g, int64_t n, int32_t k, const float* tab, const uint8_t* freed,
                        double* scales, float* X, void* stream) {
    if (!g || !tab || !scales || n < 0 || k < 2 || k > kMaxK)
        return fail(OCMP_ERR_ARG, "ocmp_guess_features: bad argument (table of 2..6 rows)");
    if (X && g->F != k - 1) return fail(OCMP_ERR_ARG, "ocmp_guess_features: the network takes F = k - 1 features");
    cudaStream_t st = (cudaStream_t)stream;
    const float2* T2 = reinterpret_cast<const float2*>(tab);
    OCMP_K_DISPATCH(k, OCMP_LAUNCH(hist_scales_kernel<KK><<<kRedBlocks, 256, 0, st>>>(n, T2, freed, g->spart, g->scnt, scales)));
    if (X && n > 0)
        OCMP_K_DISPATCH(k, OCMP_LAUNCH(features_kernel<KK><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, T2, freed, scales, X)));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_guess_predict(ocmp_guess_t g, int64_t n, int32_t k, const float* tab, const uint8_t* freed,
                       const double* scales, int32_t base_order, double* x, void* stream) {
    if (!x || !tab || n < 0 || k < 1 || k > kMaxK || base_order < 0 || base_order > k - 1)
        return fail(OCMP_ERR_ARG, "ocmp_guess_predict: bad argument (table of 1..6 rows, base order < k)");
    if (g && (k < 2 || !scales || g->F != k - 1))
        return fail(OCMP_ERR_ARG, "ocmp_guess_predict: the network needs k = F + 1 >= 2 and the history scales");
    if (n == 0) return OCMP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const float2* T2 = reinterpret_cast<const float2*>(tab);
    const unsigned nb = (unsigned)((n + 255) / 256);
    if (g) {
        OCMP_K_DISPATCH(k, OCMP_LAUNCH(predict_kernel<KK, true><<<nb, 256, sizeof(float) * g->L.n, st>>>(
                               n, T2, freed, scales, base_order, g->P, g->L.n, x)));
    } else {
        OCMP_K_DISPATCH(k, OCMP_LAUNCH(predict_kernel<KK, false><<<nb, 256, 0, st>>>(n, T2, freed, scales, base_order,
                                                                                nullptr, 0, x)));
    }
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_guess_target(int64_t n, int32_t k, const float* tab, const uint8_t* freed, const double* scales,
                      int32_t base_order, const double* unext, float* T, void* stream) {
    if (!unext || !T || !scales || !tab || n < 0 || k < 2 || k > kMaxK || base_order < 0 || base_order > k - 1)
        return fail(OCMP_ERR_ARG, "ocmp_guess_target: bad argument");
    if (n == 0) return OCMP_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const float2* T2 = reinterpret_cast<const float2*>(tab);
    OCMP_K_DISPATCH(k, OCMP_LAUNCH(target_kernel<KK><<<(unsigned)((n + 255) / 256), 256, 0, st>>>(n, T2, freed, scales,
                                                                                           base_order, unext, T)));
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_guess_residual_loss(ocmp_guess_t g, ocmp_matrix_t mat, const float* Y, const float* T, const double* scale,
                             const double* b, double weight, double* loss_host, float* dY, void* stream) {
    if (!g || !mat || !Y || !T || !scale || !b || !dY) return fail(OCMP_ERR_ARG, "ocmp_guess_residual_loss: null argument");
    if (mat->B != 1) return fail(OCMP_ERR_ARG, "ocmp_guess_residual_loss: batched matrix");
    ocmp_space_s* s = mat->space;
    const int64_t n = s->ndof;
    cudaStream_t st = (cudaStream_t)stream;
    int rc = ensure_vecs(g, n);
    if (!rc) rc = ensure_tpos(s, st);
    if (rc) return rc;
    double* e = g->vecs;
    double* v = g->vecs + n;
    double* w = g->vecs + 2 * n;
    const unsigned nb = (unsigned)((n + 255) / 256);
    OCMP_LAUNCH(guess_error_kernel<<<nb, 256, 0, st>>>(n, Y, T, scale, s->d_free, e));
    rc = launch_spmv64(s, mat->vals, e, v, st);
    if (rc) return rc;
    OCMP_LAUNCH(mask_norms_kernel<<<kRedBlocks, 256, 0, st>>>(n, v, b, s->d_free, g->spart, g->scnt, g->nrm));
    rc = launch_spmv_t(s, mat->vals, v, w, st);
    if (rc) return rc;
    OCMP_LAUNCH(guess_dy_kernel<<<nb, 256, 0, st>>>(n, w, scale, s->d_free, weight, g->nrm, dY));
    OCMP_CUDA(cudaGetLastError());
    if (loss_host) {
        OCMP_CUDA(cudaMemcpyAsync(loss_host, g->nrm + 2, sizeof(double), cudaMemcpyDeviceToHost, st));
        OCMP_CUDA(cudaStreamSynchronize(st));
    }
    return OCMP_OK;
}

int ocmp_spmv_transpose(ocmp_matrix_t mat, const double* x, double* y, void* stream) {
    if (!mat || !x || !y) return fail(OCMP_ERR_ARG, "ocmp_spmv_transpose: null argument");
    if (mat->B != 1) return fail(OCMP_ERR_ARG, "ocmp_spmv_transpose: batched matrix");
    return launch_spmv_t(mat->space, mat->vals, x, y, (cudaStream_t)stream);
}

}  // extern "C"
