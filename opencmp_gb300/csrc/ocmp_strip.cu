// Strip direct preconditioner of libopencmp_gpu.so (sm_103a): the GPU counterpart of the sparse
// direct solve in opencmp/models/base_model.py:906-922 (a.mat.Inverse(freedofs, 'pardiso' |
// 'umfpack'), then gfu += inv * (L - A gfu)), used as the preconditioner of FP64-refined GMRES.
//
// The dofs are cut into consecutive strips [s_k, s_k+1) chosen so that the matrix is block
// tridiagonal over them: strip k's rows reach no further than strip k+1 (greedy over the row
// bandwidth, or, when the pattern repeats with a period, uniform strips of that period: one row of
// elements of a structured mesh numbered row by row). Block elimination over the strips (the block Thomas algorithm) needs, per strip,
//     S_k = A_kk - A_k,k-1 S_{k-1}^-1 A_k-1,k,      G_k = S_k^-1,
// and a solve is a forward sweep y_k = G_k (b_k - A_k,k-1 y_k-1) and a backward sweep
// x_k = y_k - G_k A_k,k+1 x_k+1. Every G_k is kept explicitly (FP32, dense), so each sweep step is
// one dense matrix-vector product instead of two triangular solves; the sweeps of a
// preconditioner application are one launch (ocmp_sweeps.cuh).
//
// The elimination runs from both ends towards the middle strip (strip k of the second half takes
// k + 1's place for k - 1 above, and the middle strip is updated from both sides): two chains at once,
// half as long. "Previous" below is the neighbour farther from the middle, "next" the nearer one.
// Within a strip the dofs are ordered [N | I]: I = the dofs coupled to the previous strip (the
// only rows and columns the Schur update A_k,k-1 S_{k-1}^-1 A_k-1,k touches), N = the rest, each
// part padded to a multiple of 128 with decoupled unit rows. G_k is the block Gauss-Jordan inverse
// of S_k with 128 x 128 diagonal-tile pivots (each tile inverted with partial pivoting inside it):
// per tile one small inversion, one kernel for the panels and one rank-128 update of the whole strip, the
// dominant flops. Since the Schur update only adds to the II block, the N pivots can be eliminated
// before it:
//   phase 1 (side streams, all strips independent): fill S_k, eliminate its N tiles;
//   phase 2 (a stream per chain, strip after strip): S_k[I,I] -= A[I,J] G_k-1[J,J] A[J,I] (J = the
//     dofs of strip k-1 coupled to strip k; A[I,J] and A[J,I] hold a few entries per row, so the
//     update is two sparse-times-dense kernels over per-dof coupling lists), then eliminate the I
//     tiles.
// On a structured triangle mesh half of each strip's elements touch the previous row of elements,
// so phase 2, the sequential chains, does half of the pivot tiles.
// Newton-Schulz path, for a strip whose N dofs fall into independent groups of at most 32 (the
// elements of a row of DG elements that do not touch the previous row): phase 1 inverts the groups
// (a warp each) and forms the interface complement W0 = S_II - S_IN S_NN^-1 S_NI with one dense
// product; phase 2 subtracts the Schur update from W0 and inverts it by Newton-Schulz iteration
// started from the previous strip's interface inverse (two steps on a uniform DG mesh), then
// assembles G_k from the 2 x 2 block inverse with three dense products.
// The dense products are C = beta C0 + alpha A B^T with both operands K-contiguous: FP32 SIMT
// (sgemm_nt) or the tensor cores (tc_products, ocmp_tcgemm.cu).
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <cstring>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "ocmp_internal.h"
#include "ocmp_sweeps.cuh"

namespace ocmp {

constexpr int kNb = 128;   // Gauss-Jordan tile and padding granule
constexpr int kSide = 3;   // side streams of phase 1
constexpr int kAhead = 4;  // pairs of strips that the launches of phase 1 are ahead of phase 2

struct StripWork {
    float* P = nullptr;    // pivot-tile inverse, kNb x kNb, and its transpose
    float* Ck = nullptr;   // column panel, mp_max x kNb
    float* Rt = nullptr;   // row panel (transposed), mp_max x kNb
};

// One of the two chains of phase 2: its stream (at the highest priority so that the side streams'
// products never hold it back) and scratch.
struct StripChain {
    cudaStream_t stream = nullptr;
    StripWork work;
    float* T = nullptr;              // Schur update: G_prev[J, J] A[J, I] (nJ x nIp)
    // Newton-Schulz: buffers of an n x n matrix followed by its transpose; H: the last three interface
    // inverses, newest first, cur and nxt: the iterate and the next one (they change places)
    float* H[3] = {};
    int h_n[3] = {0, 0, 0};          // their padded sizes (0: none)
    float* cur = nullptr;
    float* nxt = nullptr;
    float* Rt = nullptr;             // the residual's transpose
    float* T1 = nullptr;
    float* Zt = nullptr;
    unsigned* rmax = nullptr;        // the residuals' norms
    unsigned* h_rmax = nullptr;      // pinned
    cudaEvent_t ev_read = nullptr;   // the residual's copy
    cudaEvent_t ev_done = nullptr;   // the chain's last strip
    // a strip in progress
    float rprev = 0.f;
    int it = 0;
};

struct Strip {
    int K = 0, mid = 0;              // strips, the middle one
    std::vector<int64_t> s;          // K + 1 strip boundaries
    std::vector<int> m, mp;          // strip sizes and padded sizes (nNp + nIp)
    std::vector<int> nN, nNp, nI, nJ;
    std::vector<int64_t> goff;       // offsets of G_k in d_G (floats)
    std::vector<int64_t> poff;       // offsets of strip k's permutation in d_perm
    std::vector<int64_t> ioff, joff; // offsets into d_I / d_J
    int mp_max = 0, nIp_max = 0, nJp_max = 0;
    int32_t* d_perm = nullptr;       // per strip position: local dof, -1 on padding
    int32_t* d_I = nullptr;          // I_k as positions in strip k's order (nNp + a)
    int32_t* d_J = nullptr;          // J_k as positions in strip k's order
    int32_t* jrow = nullptr;         // J_k as local dofs
    int32_t* d_pinv = nullptr;       // per dof: its position in its strip's order
    float* d_G = nullptr;            // the explicit strip inverses
    // per I dof (over all strips, indexed like d_I): its couplings to the previous strip's J, as
    // entries [cptr[i], cptr[i+1]) of (index b in J, CSR position of A[I_i, J_b], of A[J_b, I_i])
    int32_t* d_cptr = nullptr;
    int32_t* d_cb = nullptr;
    int32_t* d_crow = nullptr;
    int32_t* d_ccol = nullptr;
    int cmax = 0;                    // longest list
    int64_t coff2 = 0;               // the middle strip's lists to its second neighbour, as an offset into d_cptr
    StripWork work[kSide];           // of the side streams
    StripChain chain[2];             // the strips below the middle and the middle one; those above
    // the sweeps' steps and their coupling lists, whose values are refreshed by every factorisation, as
    // are the free rows' dofs
    SweepStep* d_steps = nullptr;
    uint32_t* d_blob = nullptr;
    uint2* d_words = nullptr;        // the sweeps' vector and results with their epochs
    SweepState* d_state = nullptr;
    SweepArgs sweep{};
    int sweep_grid = 1;
    size_t sweep_smem = 0;
    int32_t* d_prow = nullptr;       // per position (over all strips): its dof, -1 on padding
    int32_t* d_rdof = nullptr;       // per position: its dof if free, else -1
    int32_t* d_erow = nullptr;
    int32_t* d_epos = nullptr;       // per entry of the lists: its CSR position, -1 on padding
    int32_t* d_edst = nullptr;       // and its word of d_blob
    int64_t nell = 0, npos = 0;
    int* d_flag = nullptr;           // [0] pivot tiles that were singular or non-finite, [1] a tensor-core
                                     // product whose bounded wait gave up
    int64_t bytes = 0;
    int64_t schur_flops_pending = 0;
    cudaStream_t side[kSide] = {};
    cudaEvent_t ev_start = nullptr;
    std::vector<cudaEvent_t> ev_phase1;
    // statistics of the last factorisation
    bool timing = false;
    std::vector<cudaEvent_t> ev;
    size_t ev_used = 0;
    std::vector<int> ev_tag;            // per event pair: 0 product, 1 tile inversion, 2 panels
    double part_ms[3] = {0, 0, 0};
    cudaEvent_t fev[2] = {nullptr, nullptr};
    double factor_ms = 0, gemm_ms = 0, gemm_flops = 0, gemm_flops_pending = 0, gemm_bytes = 0, gemm_bytes_pending = 0;
    int singular = 0;
    int gemm_kind = 0;               // 0: FP32 SIMT, 1: tensor cores (3xTF32)
    // Newton-Schulz path (strips whose N dofs form small independent groups, e.g. the elements of a
    // row of DG elements that do not touch the previous row)
    std::vector<char> fast;          // per strip
    std::vector<int64_t> gofs;       // per strip: first group in d_gptr
    std::vector<int> ngrp;           // per strip: groups
    int32_t* d_gptr = nullptr;       // group offsets into d_gidx (concatenated per strip, each ends with its total)
    int32_t* d_gidx = nullptr;       // group members: positions in the strip's order (all in N)
    int32_t* d_gcomp = nullptr;      // per member: its component within the group (start << 8 | size)
    float* d_Yt[kSide] = {};         // phase 1 scratch per side stream: Y^T
    bool schulz = true;              // Newton-Schulz path on (off: block Gauss-Jordan throughout)
    int nfast = 0;
    int ns_iters = 0, ns_strips = 0, ns_fallbacks = 0;
};

namespace {

inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }
inline int pad(int64_t v) { return (int)((v + kNb - 1) / kNb * kNb); }

// ------------------------------------------------------------------ dense products (FP32 SIMT)
// C[M x N] = beta C0 + alpha A[M x K] B[N x K]^T (DenseProduct), row-major with leading dimensions;
// M, N multiples of 128, K a multiple of 16, rows 16-byte aligned. 256 threads, 128 x 128 tile,
// 8 x 8 outputs per thread, double-buffered K slices of 16.
constexpr int GB = 128, GK = 16;
__global__ void __launch_bounds__(256) sgemm_nt(const DenseProduct d) {
    const float* __restrict__ A = d.A;
    const float* __restrict__ B = d.B;
    const int M = d.M, N = d.N, K = d.K;
    const int64_t lda = d.lda, ldb = d.ldb;
    __shared__ __align__(16) float As[2][GK][GB + 4];
    __shared__ __align__(16) float Bs[2][GK][GB + 4];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t m0 = (int64_t)blockIdx.y * GB, n0 = (int64_t)blockIdx.x * GB;
    if (m0 >= M || n0 >= N) return;
    const int lr = tid >> 2, lk = (tid & 3) * 4;   // load: rows lr, lr + 64; k lk..lk+3
    float4 ra[2], rb[2];
    auto gload = [&](int k0) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            ra[q] = *reinterpret_cast<const float4*>(A + (m0 + lr + 64 * q) * lda + k0 + lk);
            rb[q] = *reinterpret_cast<const float4*>(B + (n0 + lr + 64 * q) * ldb + k0 + lk);
        }
    };
    auto sstore = [&](int buf) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int r = lr + 64 * q;
            As[buf][lk + 0][r] = ra[q].x;
            As[buf][lk + 1][r] = ra[q].y;
            As[buf][lk + 2][r] = ra[q].z;
            As[buf][lk + 3][r] = ra[q].w;
            Bs[buf][lk + 0][r] = rb[q].x;
            Bs[buf][lk + 1][r] = rb[q].y;
            Bs[buf][lk + 2][r] = rb[q].z;
            Bs[buf][lk + 3][r] = rb[q].w;
        }
    };
    float acc[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) acc[i][j] = 0.f;
    gload(0);
    sstore(0);
    __syncthreads();
    int buf = 0;
    for (int k0 = 0; k0 < K; k0 += GK) {
        const bool more = k0 + GK < K;
        if (more) gload(k0 + GK);
#pragma unroll
        for (int kk = 0; kk < GK; kk++) {
            const float4 a0 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4*>(&As[buf][kk][ty * 4 + 64]);
            const float4 b0 = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4]);
            const float4 b1 = *reinterpret_cast<const float4*>(&Bs[buf][kk][tx * 4 + 64]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
            const float b[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        if (more) sstore(buf ^ 1);
        __syncthreads();
        buf ^= 1;
    }
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int64_t r = m0 + (i < 4 ? ty * 4 + i : 64 + ty * 4 + i - 4);
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int64_t c = n0 + h * 64 + tx * 4;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            if (d.beta != 0.f)
                o = d.C0 ? *reinterpret_cast<const float4*>(d.C0 + r * d.ldc0 + c)
                         : make_float4(r == c ? 1.f : 0.f, r == c + 1 ? 1.f : 0.f, r == c + 2 ? 1.f : 0.f,
                                       r == c + 3 ? 1.f : 0.f);
            o.x = d.alpha * acc[i][h * 4 + 0] + d.beta * o.x;
            o.y = d.alpha * acc[i][h * 4 + 1] + d.beta * o.y;
            o.z = d.alpha * acc[i][h * 4 + 2] + d.beta * o.z;
            o.w = d.alpha * acc[i][h * 4 + 3] + d.beta * o.w;
            *reinterpret_cast<float4*>(d.C + r * d.ldc + c) = o;
        }
    }
}


// ------------------------------------------------------------------ strip assembly
// S (mp x mp, zeroed) <- the strip's diagonal block in the strip's [N | I] order; unit diagonal on
// constrained rows and on the padding. pinv: per dof its position in its strip's order.
__global__ void k_fill_strip(int mp, int64_t s0, const int32_t* __restrict__ perm, const int32_t* __restrict__ pinv,
                             const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                             const double* __restrict__ vals, const uint8_t* __restrict__ freed, int64_t s1,
                             float* __restrict__ S) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= mp) return;
    float* row = S + (int64_t)i * mp;
    const int ld = perm[i];
    if (ld < 0 || !freed[s0 + ld]) {
        row[i] = 1.f;
        return;
    }
    const int64_t r = s0 + ld;
    for (int32_t k = rp[r]; k < rp[r + 1]; k++) {
        const int64_t c = col[k];
        if (c >= s0 && c < s1 && freed[c]) row[pinv[c]] = (float)vals[k];
    }
}

// Schur update of strip k (rows and columns of its I block, I dofs at global s0 + Irow[i]) from the
// previous strip's inverse G (its J dofs at positions Jp, local dofs Jrow, strip start sp):
//   T[b, c] = sum_{(d, A[J_d, I_c]) in list(c)} G[J_b, J_d] A[J_d, I_c]           (k_schur_t)
//   S[I_a, I_c] -= sum_{(b, A[I_a, J_b]) in list(a)} A[I_a, J_b] T[b, c]           (k_schur_u)
// An entry counts only when both its row and its column dof are free (the constrained rows and
// columns of the strips are unit rows and columns).
constexpr int kSchurRows = 8;   // rows b of T per thread in k_schur_t
__global__ void __launch_bounds__(128) k_schur_t(int nI, int nJ, int nIp, int64_t s0, int64_t sp,
                                                 const int32_t* __restrict__ Irow, const int32_t* __restrict__ Jrow,
                                                 const int32_t* __restrict__ Jp, const int32_t* __restrict__ cptr,
                                                 const int32_t* __restrict__ cb, const int32_t* __restrict__ ccol,
                                                 const double* __restrict__ vals, const uint8_t* __restrict__ freed,
                                                 const float* __restrict__ G, int mpG, float* __restrict__ T) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, b0 = blockIdx.y * kSchurRows;
    if (c >= nIp) return;
    const float* grow[kSchurRows];
#pragma unroll
    for (int u = 0; u < kSchurRows; u++) grow[u] = G + (int64_t)Jp[min(b0 + u, nJ - 1)] * mpG;
    float acc[kSchurRows];
#pragma unroll
    for (int u = 0; u < kSchurRows; u++) acc[u] = 0.f;
    if (c < nI && freed[s0 + Irow[c]]) {
        for (int32_t e = cptr[c]; e < cptr[c + 1]; e++) {
            const int d = cb[e];
            const int32_t q = ccol[e];
            if (q < 0 || !freed[sp + Jrow[d]]) continue;
            const float v = (float)vals[q];
            const int jc = Jp[d];
#pragma unroll
            for (int u = 0; u < kSchurRows; u++) acc[u] = fmaf(grow[u][jc], v, acc[u]);
        }
    }
#pragma unroll
    for (int u = 0; u < kSchurRows; u++)
        if (b0 + u < nJ) T[(int64_t)(b0 + u) * nIp + c] = acc[u];
}

// four columns c per thread (T's rows are 16-byte aligned: nIp is a multiple of 128)
__global__ void __launch_bounds__(128) k_schur_u(int nI, int nIp, int nNp, int64_t s0, int64_t sp,
                                                 const int32_t* __restrict__ Irow, const int32_t* __restrict__ Jrow,
                                                 const int32_t* __restrict__ cptr, const int32_t* __restrict__ cb,
                                                 const int32_t* __restrict__ crow, const double* __restrict__ vals,
                                                 const uint8_t* __restrict__ freed, const float* __restrict__ T,
                                                 float* __restrict__ S, int mp) {
    const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x), a = blockIdx.y;
    if (c >= nI || !freed[s0 + Irow[a]]) return;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int32_t e = cptr[a]; e < cptr[a + 1]; e++) {
        const int b = cb[e];
        const int32_t q = crow[e];
        if (q < 0 || !freed[sp + Jrow[b]]) continue;
        const float v = (float)vals[q];
        const float4 t = *reinterpret_cast<const float4*>(T + (int64_t)b * nIp + c);
        acc.x = fmaf(v, t.x, acc.x);
        acc.y = fmaf(v, t.y, acc.y);
        acc.z = fmaf(v, t.z, acc.z);
        acc.w = fmaf(v, t.w, acc.w);
    }
    float* srow = S + (int64_t)(nNp + a) * mp + nNp + c;
    const float av[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
    for (int u = 0; u < 4; u++)
        if (c + u < nI) srow[u] -= av[u];
}

// ------------------------------------------------------------------ block Gauss-Jordan
// P <- inverse of the tile S[t0:t0+128, t0:t0+128], followed by its transpose, by Gauss-Jordan with
// partial pivoting inside the tile. The tile stays in registers, 8 x 8 per thread, a half warp per every
// 16th column, and rows are never moved: step k takes as pivot the largest |a_rk| (to 16 bits; the first
// of equals) over the rows not yet used, and the row and column permutation is applied when the result is
// written (P[step(r)][piv(c)] = M[r][c]). A step is a chain of latencies on one SM, so the chain is kept
// short: the half warp that holds column k publishes it in shared memory and finds the pivot by one
// integer reduction over keys that end in the row; one barrier; every half warp gets its part of the
// pivot row from its own lane by shuffles, while the reciprocal is computed; the update starts with the
// next pivot column, which is searched and published while the other warps update the rest. 286 us a tile
// with 16 x 1 entries per thread (bound by issue), 108 with the pivot's value, reciprocal and row found
// by the publishing half warp (800 of 1,600 clocks a step), 92 so. A zero or non-finite pivot is
// counted in *flag and replaced by a tiny value.
constexpr int kTileThreads = 256;
__global__ void __launch_bounds__(kTileThreads) k_tile_inv(const float* __restrict__ S, int mp, int t0,
                                                           float* __restrict__ P, int* __restrict__ flag) {
    __shared__ __align__(16) float colk[2][kNb];
    __shared__ int pk[2];
    __shared__ int piv[kNb];
    __shared__ int step[kNb];
    const int tid = threadIdx.x, tr = tid & 15, tc = tid >> 4;
    float v[8][8];
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
        for (int j = 0; j < 8; j++) v[i][j] = S[(int64_t)(t0 + tr * 8 + i) * mp + t0 + tc + 16 * j];
    unsigned open[8];       // all ones while this thread's row has not been a pivot
#pragma unroll
    for (int i = 0; i < 8; i++) open[i] = ~0u;
    // column k = tc + 16 kk and its pivot, by the half warp that holds it (own; the whole warp comes
    // along: a reduction over a part of a warp is slow); kk is a constant so that v stays in registers
    auto publish = [&](int k, bool own, auto col) {
        constexpr int kk = decltype(col)::value;
        const int b = k & 1;
        unsigned best = 0u;
#pragma unroll
        for (int i = 0; i < 8; i++)
            best = max(best, ((__float_as_uint(v[i][kk]) & 0x7fffff80u) | (0x80000000u + 127 - 8 * tr - i)) & open[i]);
        if (own)
#pragma unroll
            for (int i = 0; i < 8; i += 4)
                *reinterpret_cast<float4*>(&colk[b][tr * 8 + i]) =
                    make_float4(v[i][kk], v[i + 1][kk], v[i + 2][kk], v[i + 3][kk]);
        const unsigned top = __reduce_max_sync(0xffffffffu, own ? best : 0u);
        if (own && tr == 0) pk[b] = 127 - (int)(top & 127u);
    };
    // steps 16 kk .. 16 kk + 15
    auto eliminate = [&](auto col) {
        constexpr int kk = decltype(col)::value;
        if (tc < 2) publish(16 * kk, tc == 0, col);
#pragma unroll 1
        for (int t = 0; t < 16; t++) {
            const int b = t & 1;
            __syncthreads();
            const int p = pk[b];
            float pv = colk[b][p];
            const bool owner = tr == p >> 3;
            float cr[8], pr[8];
#pragma unroll
            for (int i = 0; i < 8; i += 4) {
                const float4 x = *reinterpret_cast<const float4*>(&colk[b][tr * 8 + i]);
                cr[i] = x.x, cr[i + 1] = x.y, cr[i + 2] = x.z, cr[i + 3] = x.w;
            }
            // column k becomes a column of the inverse: 1 in the pivot row before the scaling, 0 elsewhere
            const bool here = tc == t;
#pragma unroll
            for (int i = 0; i < 8; i++) v[i][kk] = here ? 0.f : v[i][kk];
            // the pivot row's update is 0 - (-1) times the scaled pivot row
            auto take = [&](auto row) {
                constexpr int i = decltype(row)::value;
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    pr[j] = v[i][j];
                    v[i][j] = owner ? 0.f : v[i][j];
                }
                cr[i] = owner ? -1.f : cr[i];
                open[i] = owner ? 0u : open[i];
            };
            if (p & 4) {
                if (p & 2) {
                    if (p & 1) take(std::integral_constant<int, 7>{});
                    else take(std::integral_constant<int, 6>{});
                } else {
                    if (p & 1) take(std::integral_constant<int, 5>{});
                    else take(std::integral_constant<int, 4>{});
                }
            } else {
                if (p & 2) {
                    if (p & 1) take(std::integral_constant<int, 3>{});
                    else take(std::integral_constant<int, 2>{});
                } else {
                    if (p & 1) take(std::integral_constant<int, 1>{});
                    else take(std::integral_constant<int, 0>{});
                }
            }
            if (!(fabsf(pv) > 0.f) || !isfinite(pv)) {
                if (tid == 0) atomicAdd(flag, 1);
                pv = 1e-30f;
            }
            const float d = 1.f / pv;
            if (tid == 0) {
                piv[16 * kk + t] = p;
                step[p] = 16 * kk + t;
            }
#pragma unroll
            for (int j = 0; j < 8; j++) pr[j] = __shfl_sync(0xffffffffu, pr[j], p >> 3, 16) * d;
            pr[kk] = here ? d : pr[kk];
#pragma unroll
            for (int i = 0; i < 8; i++) v[i][kk] -= cr[i] * pr[kk];
            if (tc >> 1 == (t + 1) >> 1) publish(16 * kk + t + 1, tc == t + 1, col);
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (j != kk) v[i][j] -= cr[i] * pr[j];
        }
    };
    eliminate(std::integral_constant<int, 0>{});
    eliminate(std::integral_constant<int, 1>{});
    eliminate(std::integral_constant<int, 2>{});
    eliminate(std::integral_constant<int, 3>{});
    eliminate(std::integral_constant<int, 4>{});
    eliminate(std::integral_constant<int, 5>{});
    eliminate(std::integral_constant<int, 6>{});
    eliminate(std::integral_constant<int, 7>{});
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int r = step[tr * 8 + i];
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const int c = piv[tc + 16 * j];
            P[r * kNb + c] = v[i][j];
            P[kNb * kNb + c * kNb + r] = v[i][j];
        }
    }
}

// The panels of a pivot tile, 16 columns and 16 rows per block. Columns c: R = P S[T, c] goes into the
// pivot rows S[T, c] and, transposed, into Rt. Rows i: Ck = S[i, T], S[i, T] = -Ck P. The rank-128 update
// S -= Ck Rt^T that follows leaves the pivot rows and columns alone because Ck is zero on the former and
// Rt on the latter; the tile itself becomes P. Both products have the form out[x][y] = sum_k M[k][y]
// V[k][x] with M = P^T or P in shared memory: four warps each, 4 x 4 outputs per lane, so that a product
// costs 1.25 shared-memory reads per 16 FMAs' issue slots. Two kernels (one of them after the update) with one or two
// reads per FMA and strided stores took 36 us each at 1,280; this one 5.
constexpr int kPanel = 16;
constexpr int kPanelSmem = (2 * kNb * kNb + 2 * kNb * kPanel) * (int)sizeof(float);
__global__ void __launch_bounds__(256) k_panels(float* __restrict__ S, int mp, int t0, const float* __restrict__ P,
                                                float* __restrict__ Rt, float* __restrict__ Ck) {
    extern __shared__ __align__(16) float sm[];
    float* Pt = sm;                        // [l][r]
    float* Ps = sm + kNb * kNb;            // [q][l]
    float* Sc = Ps + kNb * kNb;            // [l][16]: S[t0 + l, c0 + j]
    float* Cs = Sc + kNb * kPanel;         // [q][16]: S[c0 + i, t0 + q]
    const int tid = threadIdx.x, c0 = blockIdx.x * kPanel, lane = tid & 31, w = tid >> 5;
    const bool pivot = c0 >= t0 && c0 < t0 + kNb;
    for (int e = tid; e < kNb * kNb / 4; e += 256) {
        reinterpret_cast<float4*>(Ps)[e] = reinterpret_cast<const float4*>(P)[e];
        reinterpret_cast<float4*>(Pt)[e] = reinterpret_cast<const float4*>(P + kNb * kNb)[e];
    }
    for (int e = tid; e < kNb * kPanel / 4; e += 256) {
        const int l = e / (kPanel / 4), q = e % (kPanel / 4);
        reinterpret_cast<float4*>(Sc)[e] = *(reinterpret_cast<const float4*>(S + (int64_t)(t0 + l) * mp + c0) + q);
    }
    for (int e = tid; e < kNb * kPanel; e += 256) {
        const int i = e / kNb, q = e % kNb;
        const float x = pivot ? 0.f : S[(int64_t)(c0 + i) * mp + t0 + q];
        Cs[q * kPanel + i] = x;
        Ck[(int64_t)(c0 + i) * kNb + q] = x;
    }
    __syncthreads();
    const float* M = w < 4 ? Pt : Ps;
    const float* V = (w < 4 ? Sc : Cs) + 4 * (w & 3);
    float acc[4][4] = {};   // [x][y]
#pragma unroll 4
    for (int k = 0; k < kNb; k++) {
        const float4 m = *reinterpret_cast<const float4*>(M + k * kNb + 4 * lane);
        const float4 x = *reinterpret_cast<const float4*>(V + k * kPanel);
        const float xv[4] = {x.x, x.y, x.z, x.w}, mv[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
        for (int a = 0; a < 4; a++)
#pragma unroll
            for (int b = 0; b < 4; b++) acc[a][b] = fmaf(mv[b], xv[a], acc[a][b]);
    }
    const int x0 = c0 + 4 * (w & 3);
    if (w >= 4) {
        if (!pivot)
#pragma unroll
            for (int a = 0; a < 4; a++)
                *reinterpret_cast<float4*>(S + (int64_t)(x0 + a) * mp + t0 + 4 * lane) =
                    make_float4(-acc[a][0], -acc[a][1], -acc[a][2], -acc[a][3]);
        return;
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
        *reinterpret_cast<float4*>(Rt + (int64_t)(x0 + a) * kNb + 4 * lane) =
            pivot ? make_float4(0.f, 0.f, 0.f, 0.f) : make_float4(acc[a][0], acc[a][1], acc[a][2], acc[a][3]);
#pragma unroll
    for (int b = 0; b < 4; b++) {
        const int r = 4 * lane + b;
        *reinterpret_cast<float4*>(S + (int64_t)(t0 + r) * mp + x0) =
            pivot ? *reinterpret_cast<const float4*>(Ps + r * kNb + x0 - t0)
                  : make_float4(acc[0][b], acc[1][b], acc[2][b], acc[3][b]);
    }
}

// ------------------------------------------------------------------ Newton-Schulz path
// Inverse of each small group of N dofs (b <= 32 positions, packed from independent components),
// a warp per group, in place in the strip. Lane c owns column c of the group's block in shared
// memory; gcomp gives each position its component (start << 8 | size) within the group, and every
// component is eliminated on its own lanes at the same time: Gauss-Jordan with partial pivoting
// over the component's rows (each lane of a component scans them for the pivot, so all agree),
// rows never moved (as in k_tile_inv).
constexpr int kGroupWarps = 8;
__global__ void __launch_bounds__(32 * kGroupWarps) k_group_inv(float* __restrict__ S, int mp, const int32_t* __restrict__ gptr,
                                                                const int32_t* __restrict__ gidx,
                                                                const int32_t* __restrict__ gcomp, int ngroups,
                                                                int* __restrict__ flag) {
    __shared__ float tile[kGroupWarps][32][33];
    __shared__ float colk[kGroupWarps][32];
    __shared__ int pivs[kGroupWarps][32], steps[kGroupWarps][32];
    const int wl = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int grp = blockIdx.x * kGroupWarps + wl;
    if (grp >= ngroups) return;
    const int g0 = gptr[grp], b = gptr[grp + 1] - g0;
    const int32_t* g = gidx + g0;
    float(*t)[33] = tile[wl];
    const bool in = lane < b;
    const int cw = in ? gcomp[g0 + lane] : 0;
    const int cs = cw >> 8, cn = in ? (cw & 255) : 0;
    if (in) {
        const int myg = g[lane];
        for (int r = cs; r < cs + cn; r++) t[r][lane] = S[(int64_t)g[r] * mp + myg];
    }
    int maxn = cn;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) maxn = max(maxn, __shfl_xor_sync(0xffffffffu, maxn, off));
    __syncwarp();
    unsigned used = 0;
    for (int k = 0; k < maxn; k++) {
        const bool act = k < cn;
        const int pc = cs + k;
        int p = cs;
        float nk = 0.f;
        if (act) {
            float best = -1.f;
            for (int r = cs; r < cs + cn; r++) {
                if ((used >> r) & 1u) continue;
                float a = fabsf(t[r][pc]);
                if (!(a >= 0.f)) a = 0.f;
                if (a > best) {
                    best = a;
                    p = r;
                }
            }
            float pv = t[p][pc];
            if (!(fabsf(pv) > 0.f) || !isfinite(pv)) {
                if (lane == pc) atomicAdd(flag, 1);
                pv = 1e-30f;
            }
            nk = (lane == pc ? 1.f : t[p][lane]) / pv;
            colk[wl][lane] = t[lane][pc];   // row `lane` is in this component
        }
        __syncwarp();
        if (act) {
            for (int r = cs; r < cs + cn; r++)
                t[r][lane] = r == p ? nk : (lane == pc ? 0.f : t[r][lane]) - colk[wl][r] * nk;
            if (lane == pc) {
                pivs[wl][pc] = p;
                steps[wl][p] = pc;
            }
            used |= 1u << p;
        }
        __syncwarp();
    }
    if (in) {
        const int pcol = g[pivs[wl][lane]];
        for (int r = cs; r < cs + cn; r++) S[(int64_t)g[steps[wl][r]] * mp + pcol] = t[r][lane];
    }
}

// Y = X S_NI in place (rows of each group, columns of I): a block per group and 128 columns, a
// thread per column (X is zero between the group's components)
__global__ void __launch_bounds__(128) k_group_y(float* __restrict__ S, int mp, int nNp,
                                                 const int32_t* __restrict__ gptr, const int32_t* __restrict__ gidx) {
    __shared__ float X[32][33];
    __shared__ int gs[32];
    const int grp = blockIdx.x, tid = threadIdx.x;
    const int g0 = gptr[grp], b = gptr[grp + 1] - g0;
    if (tid < b) gs[tid] = gidx[g0 + tid];
    __syncthreads();
    for (int e = tid; e < b * b; e += 128) X[e / b][e % b] = S[(int64_t)gs[e / b] * mp + gs[e % b]];
    __syncthreads();
    const int c = nNp + blockIdx.y * 128 + tid;
    float sv[32];
#pragma unroll
    for (int q = 0; q < 32; q++) sv[q] = q < b ? S[(int64_t)gs[q < b ? q : 0] * mp + c] : 0.f;
    for (int r = 0; r < b; r++) {
        float acc = 0.f;
#pragma unroll
        for (int q = 0; q < 32; q++)
            if (q < b) acc = fmaf(X[r][q], sv[q], acc);
        S[(int64_t)gs[r] * mp + c] = acc;
    }
}

// S_IN <- Z = -S_IN X in place (rows i of I, the N columns of each group): a block per group and
// 128 rows, a thread per row, which reads its row's group entries before writing them
__global__ void __launch_bounds__(128) k_group_z(float* __restrict__ S, int mp, int nNp, int nIp,
                                                 const int32_t* __restrict__ gptr, const int32_t* __restrict__ gidx) {
    __shared__ float X[32][33];
    __shared__ int gs[32];
    const int grp = blockIdx.x, tid = threadIdx.x;
    const int g0 = gptr[grp], b = gptr[grp + 1] - g0;
    if (tid < b) gs[tid] = gidx[g0 + tid];
    __syncthreads();
    for (int e = tid; e < b * b; e += 128) X[e / b][e % b] = S[(int64_t)gs[e / b] * mp + gs[e % b]];
    __syncthreads();
    const int i = blockIdx.y * 128 + tid;
    if (i >= nIp) return;
    float* row = S + (int64_t)(nNp + i) * mp;
    float sv[32];
#pragma unroll
    for (int q = 0; q < 32; q++) sv[q] = q < b ? row[gs[q < b ? q : 0]] : 0.f;
    for (int r = 0; r < b; r++) {
        float acc = 0.f;
#pragma unroll
        for (int q = 0; q < 32; q++)
            if (q < b) acc = fmaf(sv[q], X[q][r], acc);
        row[gs[r]] = -acc;
    }
}

// dst (cols x rows, leading dimension ldd) = src^T (rows x cols, leading dimension lds); 32 x 32 tiles
__global__ void k_transpose(const float* __restrict__ src, int64_t lds, int rows, int cols, float* __restrict__ dst,
                            int64_t ldd) {
    __shared__ float tl[32][33];
    const int bx = blockIdx.x * 32, by = blockIdx.y * 32, tx = threadIdx.x, ty = threadIdx.y;
    for (int j = ty; j < 32; j += 8) {
        const int r = by + j, c = bx + tx;
        tl[j][tx] = (r < rows && c < cols) ? src[(int64_t)r * lds + c] : 0.f;
    }
    __syncthreads();
    for (int j = ty; j < 32; j += 8) {
        const int r = bx + j, c = by + tx;   // dst row = src column
        if (r < cols && c < rows) dst[(int64_t)r * ldd + c] = tl[tx][j];
    }
}

// dst = src (rows x cols, leading dimensions)
__global__ void k_copy2d(const float* __restrict__ src, int64_t lds, int rows, int cols, float* __restrict__ dst,
                         int64_t ldd) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= (int64_t)rows * cols) return;
    const int r = (int)(t / cols), c = (int)(t % cols);
    dst[(int64_t)r * ldd + c] = src[(int64_t)r * lds + c];
}

// the last blocks of a strip's inverse: S_NI = -T1 (nN x n), S_II = X (n x n)
__global__ void k_store_ni_ii(int nN, int n, int mp, const float4* __restrict__ T1, const float4* __restrict__ X,
                              float* __restrict__ S) {
    const int n4 = n / 4;
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const int r = (int)(t / n4), c = (int)(t % n4);
    if (r >= nN + n) return;
    float4 v = r < nN ? T1[t] : X[t - (int64_t)nN * n4];
    if (r < nN) v = make_float4(-v.x, -v.y, -v.z, -v.w);
    *(reinterpret_cast<float4*>(S + (int64_t)r * mp + nN) + c) = v;
}

// X0 = c1 H1 + c2 H2 + c3 H3 over n4 float4s (c3 = 0: H3 unused); clears the norms
__global__ void k_extrap(int64_t n4, const float4* __restrict__ h1, const float4* __restrict__ h2,
                         const float4* __restrict__ h3, float c1, float c2, float c3, float4* __restrict__ x,
                         unsigned* __restrict__ zero, int nzero) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < nzero) zero[t] = 0u;
    if (t >= n4) return;
    const float4 a = h1[t];
    const float4 b = h2 ? h2[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 c = h3 ? h3[t] : make_float4(0.f, 0.f, 0.f, 0.f);
    x[t] = make_float4(c1 * a.x + c2 * b.x + c3 * c.x, c1 * a.y + c2 * b.y + c3 * c.y, c1 * a.z + c2 * b.z + c3 * c.z,
                       c1 * a.w + c2 * b.w + c3 * c.w);
}

// *out = max over columns of sum |At[:, c]|, the infinity norm of A from its transpose (n x n;
// non-negative floats order like their bits, NaN above all): a block per 32 columns, a warp per eighth of
// the rows
__global__ void __launch_bounds__(256) k_infnorm_t(const float* __restrict__ At, int n, unsigned* __restrict__ out) {
    __shared__ float part[8][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, c = blockIdx.x * 32 + lane;
    float sm = 0.f;
#pragma unroll 16
    for (int r = w; r < n; r += 8) sm += fabsf(At[(int64_t)r * n + c]);
    part[w][lane] = sm;
    __syncthreads();
    if (w > 0) return;
#pragma unroll
    for (int v = 1; v < 8; v++) sm += part[v][lane];
    const unsigned top = __reduce_max_sync(0xffffffffu, sm == sm ? __float_as_uint(sm) : 0x7FFFFFFFu);
    if (lane == 0) atomicMax(out, top);
}

// ------------------------------------------------------------------ around the sweeps
template <class T>
__global__ void k_add_to(int64_t n, const T* __restrict__ z, double* __restrict__ x) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) x[i] += (double)z[i];
}

// the right-hand sides' values (0 where the row or the column is constrained) and the free rows' dofs
// of every strip, after an assembly
__global__ void k_list_refresh(int64_t nent, const int32_t* __restrict__ erow, const int32_t* __restrict__ epos,
                               const int32_t* __restrict__ col, const double* __restrict__ vals,
                               const uint8_t* __restrict__ freed, const int32_t* __restrict__ edst,
                               uint32_t* __restrict__ blob, int64_t npos,
                               const int32_t* __restrict__ prow, int32_t* __restrict__ rdof) {
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t < nent) {
        const int32_t q = epos[t];
        blob[edst[t]] = __float_as_uint(q >= 0 && freed[erow[t]] && freed[col[q]] ? (float)vals[q] : 0.f);
    }
    if (t < npos) {
        const int32_t d = prow[t];
        rdof[t] = (d >= 0 && freed[d]) ? d : -1;
    }
}

// ------------------------------------------------------------------ host helpers
void strip_free(Strip* p) {
    void* ps[] = {p->d_perm, p->d_I, p->d_J, p->jrow, p->d_pinv, p->d_G, p->d_cptr, p->d_cb, p->d_crow, p->d_ccol, p->d_flag};
    for (void* q : ps) dfree(q);
    for (auto& w : p->work) {
        dfree(w.P);
        dfree(w.Ck);
        dfree(w.Rt);
    }
    void* qs2[] = {p->d_prow, p->d_rdof, p->d_erow, p->d_epos, p->d_edst, p->d_steps, p->d_blob, p->d_words, p->d_state};
    for (void* q : qs2) dfree(q);
    void* qs[] = {p->d_gptr, p->d_gidx, p->d_gcomp};
    for (void* q : qs) dfree(q);
    for (auto& c : p->chain) {
        void* cs[] = {c.work.P, c.work.Ck, c.work.Rt, c.T, c.cur, c.nxt, c.Rt, c.H[0], c.H[1], c.H[2], c.T1, c.Zt, c.rmax};
        for (void* q : cs) dfree(q);
        if (c.h_rmax) cudaFreeHost(c.h_rmax);
        if (c.ev_read) cudaEventDestroy(c.ev_read);
        if (c.ev_done) cudaEventDestroy(c.ev_done);
        if (c.stream) cudaStreamDestroy(c.stream);
    }
    for (float* q : p->d_Yt) dfree(q);
    for (cudaEvent_t e : p->ev) cudaEventDestroy(e);
    for (cudaEvent_t e : p->ev_phase1) cudaEventDestroy(e);
    for (cudaEvent_t e : p->fev)
        if (e) cudaEventDestroy(e);
    if (p->ev_start) cudaEventDestroy(p->ev_start);
    for (cudaStream_t q : p->side)
        if (q) cudaStreamDestroy(q);
}

// timing of the factorisation's kernels by class (ocmp_solver_strip_timing): an event pair around
// each launch on its stream
int tbegin(Strip* p, cudaStream_t st) {
    if (!p->timing) return OCMP_OK;
    while (p->ev.size() < p->ev_used + 2) {
        cudaEvent_t e;
        OCMP_CUDA(cudaEventCreate(&e));
        p->ev.push_back(e);
    }
    OCMP_CUDA(cudaEventRecord(p->ev[p->ev_used], st));
    return OCMP_OK;
}
int tend(Strip* p, cudaStream_t st, int tag) {
    if (!p->timing) return OCMP_OK;
    OCMP_CUDA(cudaEventRecord(p->ev[p->ev_used + 1], st));
    p->ev_used += 2;
    p->ev_tag.push_back(tag);
    return OCMP_OK;
}

int products(Strip* p, const DenseProduct* d, int count, cudaStream_t st) {
    for (int q = 0; q < count; q++)
        if (d[q].M % GB || d[q].N % GB || d[q].K % 32 || d[q].M <= 0 || d[q].N <= 0 || d[q].K <= 0)
            return fail(OCMP_ERR_ARG, "strip gemm: sizes must be multiples of the tile");
    const bool t = p->timing;
    if (t && tbegin(p, st)) return OCMP_ERR_CUDA;
    if (p->gemm_kind == 1) {
        const int r = tc_products(d, count, p->d_flag + 1, st);
        if (r) return r;
    } else
        for (int q = 0; q < count; q++)
            OCMP_LAUNCH(sgemm_nt<<<dim3(d[q].N / GB, d[q].M / GB), 256, 0, st>>>(d[q]));
    if (t && tend(p, st, 0)) return OCMP_ERR_CUDA;
    for (int q = 0; q < count; q++) {
        p->gemm_flops_pending += 2.0 * d[q].M * d[q].N * (double)d[q].K;
        // operands read once, C written (and C0 read when beta != 0): the product's algorithmic bytes
        p->gemm_bytes_pending += 4.0 * ((double)d[q].M * d[q].K + (double)d[q].N * d[q].K +
                                        (d[q].beta != 0.f ? 2.0 : 1.0) * d[q].M * (double)d[q].N);
    }
    return OCMP_OK;
}
// C = beta C + alpha A B^T
int gemm(Strip* p, int M, int N, int K, const float* A, int64_t lda, const float* B, int64_t ldb, float* C, int64_t ldc,
         float alpha, float beta, cudaStream_t st) {
    const DenseProduct d{M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, C, ldc};
    return products(p, &d, 1, st);
}

// Gauss-Jordan over the pivot tiles [t_begin, t_end) of S (mp x mp) on stream st with workspace w
int gj_tiles(Strip* p, float* S, int mp, int t_begin, int t_end, const StripWork& w, cudaStream_t st) {
    for (int t0 = t_begin; t0 < t_end; t0 += kNb) {
        int r = tbegin(p, st);
        OCMP_LAUNCH(k_tile_inv<<<1, kTileThreads, 0, st>>>(S, mp, t0, w.P, p->d_flag));
        if (!r) r = tend(p, st, 1);
        if (!r) r = tbegin(p, st);
        OCMP_LAUNCH(k_panels<<<mp / kPanel, 256, kPanelSmem, st>>>(S, mp, t0, w.P, w.Rt, w.Ck));
        if (!r) r = tend(p, st, 2);
        if (!r) r = gemm(p, mp, mp, kNb, w.Ck, kNb, w.Rt, kNb, S, mp, -1.f, 1.f, st);
        if (r) return r;
    }
    return OCMP_OK;
}

int transpose(const float* src, int64_t lds, int rows, int cols, float* dst, int64_t ldd, cudaStream_t st) {
    const dim3 g(nblk(cols, 32), nblk(rows, 32)), b(32, 8);
    OCMP_LAUNCH(k_transpose<<<g, b, 0, st>>>(src, lds, rows, cols, dst, ldd));
    return OCMP_OK;
}
int copy2d(const float* src, int64_t lds, int rows, int cols, float* dst, int64_t ldd, cudaStream_t st) {
    OCMP_LAUNCH(k_copy2d<<<nblk((int64_t)rows * cols, 256), 256, 0, st>>>(src, lds, rows, cols, dst, ldd));
    return OCMP_OK;
}

// Phase 1 of a strip whose N block is block diagonal (groups of at most 32 positions): X = S_NN^-1
// group by group, S_NI <- Y = X S_NI, S_II <- W0 = S_II - S_IN Y (one dense product), S_IN <- Z =
// -S_IN X. The strip then holds [[X, Y], [Z, W0]].
int phase1_groups(Strip* p, int k, float* S, int q, cudaStream_t ss) {
    const int mp = p->mp[k], nNp = p->nNp[k], nIp = mp - nNp, ng = p->ngrp[k];
    const int32_t* gp = p->d_gptr + p->gofs[k];
    int r = tbegin(p, ss);
    OCMP_LAUNCH(k_group_inv<<<nblk(ng, kGroupWarps), 32 * kGroupWarps, 0, ss>>>(S, mp, gp, p->d_gidx, p->d_gcomp, ng,
                                                                              p->d_flag));
    if (!r) r = tend(p, ss, 1);
    OCMP_LAUNCH(k_group_y<<<dim3(ng, nIp / 128), 128, 0, ss>>>(S, mp, nNp, gp, p->d_gidx));
    if (!r) r = transpose(S + nNp, mp, nNp, nIp, p->d_Yt[q], nNp, ss);
    if (!r) r = gemm(p, nIp, nIp, nNp, S + (int64_t)nNp * mp, mp, p->d_Yt[q], nNp, S + (int64_t)nNp * mp + nNp, mp, -1.f,
                     1.f, ss);
    if (r) return r;
    OCMP_LAUNCH(k_group_z<<<dim3(ng, nblk(nIp, 128)), 128, 0, ss>>>(S, mp, nNp, nIp, gp, p->d_gidx));
    return OCMP_OK;
}

// Inverse of the interface Schur complement W = S_II (n x n, leading dimension mp) into the chain's
// buffer `cur` (its transpose in Xt). Newton-Schulz X <- X + X R, R = I - W X, started from the previous
// strips' interface inverses extrapolated along the strips (quadratic from three, linear from two, the
// last one alone; the interface complements of the strips of a row-by-row structured mesh vary smoothly
// from row to row). The step squares R, so with rho = ||R||_inf read back after each product:
// rho <= kSchulzTol: X is taken; rho^2 <= kSchulzTol: one more step is taken unchecked; a step that does
// not reduce rho (or a non-finite rho, or kSchulzMax steps) falls back to block Gauss-Jordan on a copy
// of W, as does a strip without a previous inverse of its size. The host drives both chains: while it
// waits for one's rho, the other's kernels run.
constexpr float kSchulzTol = 1e-5f;
constexpr int kSchulzMax = 8;

// The transpose of the current iterate's residual, R^T = I - X^T W^T, and its norm, on the way to the host.
// Working with both X and X^T, and with R^T alone, every product has its operands in place: no
// transposes and no copies on the chain.
int schulz_residual(Strip* p, StripChain& c, const float* W, int mp, int n) {
    cudaStream_t cs = c.stream;
    const float* Xt = c.cur + (int64_t)n * n;
    const DenseProduct d{n, n, n, Xt, n, W, mp, c.Rt, n, -1.f, 1.f, nullptr, 0};
    const int r = products(p, &d, 1, cs);
    if (r) return r;
    unsigned* at = c.rmax + c.it;
    OCMP_LAUNCH(k_infnorm_t<<<n / 32, 256, 0, cs>>>(c.Rt, n, at));
    OCMP_CUDA(cudaMemcpyAsync(c.h_rmax, at, sizeof(unsigned), cudaMemcpyDeviceToHost, cs));
    OCMP_CUDA(cudaEventRecord(c.ev_read, cs));
    return OCMP_OK;
}

// start of an interface inversion: *pending when a residual is on its way
int schulz_begin(Strip* p, StripChain& c, const float* W, int mp, int n, bool* pending) {
    c.rprev = INFINITY;
    c.it = 0;
    *pending = false;
    int hist = 0;
    while (hist < 3 && c.h_n[hist] == n) hist++;
    if (!p->schulz || hist == 0) return OCMP_OK;
    const int64_t n4 = (int64_t)n * n / 2;   // with the transpose
    const float co[3][3] = {{1.f, 0.f, 0.f}, {2.f, -1.f, 0.f}, {3.f, -3.f, 1.f}};
    const float* cc = co[hist - 1];
    OCMP_LAUNCH(k_extrap<<<nblk(n4, 256), 256, 0, c.stream>>>(
        n4, reinterpret_cast<const float4*>(c.H[0]), hist > 1 ? reinterpret_cast<const float4*>(c.H[1]) : nullptr,
        hist > 2 ? reinterpret_cast<const float4*>(c.H[2]) : nullptr, cc[0], cc[1], cc[2],
        reinterpret_cast<float4*>(c.cur), c.rmax, kSchulzMax));
    *pending = true;
    return schulz_residual(p, c, W, mp, n);
}

// the residual is there: done (*pending false; *ok whether the iterate is taken) or one more step
int schulz_step(Strip* p, StripChain& c, const float* W, int mp, int n, bool* pending, bool* ok) {
    OCMP_CUDA(cudaEventSynchronize(c.ev_read));
    float rho;
    std::memcpy(&rho, c.h_rmax, sizeof(float));
    *pending = false;
    *ok = false;
    if (!std::isfinite(rho) || rho >= c.rprev) return OCMP_OK;
    if (rho <= kSchulzTol) {
        *ok = true;
        return OCMP_OK;
    }
    c.rprev = rho;
    // X + X R and its transpose
    const int64_t nn = (int64_t)n * n;
    const DenseProduct d[2] = {{n, n, n, c.cur, n, c.Rt, n, c.nxt, n, 1.f, 1.f, c.cur, n},
                               {n, n, n, c.Rt, n, c.cur, n, c.nxt + nn, n, 1.f, 1.f, c.cur + nn, n}};
    const int r = products(p, d, 2, c.stream);
    if (r) return r;
    std::swap(c.cur, c.nxt);
    p->ns_iters++;
    if (rho * rho <= kSchulzTol) {
        *ok = true;
        return OCMP_OK;
    }
    if (++c.it >= kSchulzMax) return OCMP_OK;
    *pending = true;
    return schulz_residual(p, c, W, mp, n);
}

// End of an interface inversion: the fallback. In the history (schulz_keep) the end strip's inverse (step 0 of the chain)
// starts the second strip's iteration (spectral radius 0.9, eight steps at 96 x 96 DG P2), but it lacks a
// Schur update and would spoil the extrapolation (2 X_1 - X_0 for the third: 0.87, against 0.05 for X_1).
int schulz_end(Strip* p, StripChain& c, const float* W, int mp, int n, bool started, bool ok) {
    cudaStream_t cs = c.stream;
    if (ok) p->ns_strips++;
    else if (started) p->ns_fallbacks++;
    if (!ok) {
        int r = copy2d(W, mp, n, n, c.cur, n, cs);
        if (!r) r = gj_tiles(p, c.cur, n, 0, n, c.work, cs);
        if (!r) r = transpose(c.cur, n, n, n, c.cur + (int64_t)n * n, n, cs);
        if (r) return r;
    }
    return OCMP_OK;
}

// the new inverse joins the history, the oldest one's buffer becomes the next iterate's
void schulz_keep(StripChain& c, int n, int step) {
    float* h = c.H[2];
    c.H[2] = c.H[1];
    c.H[1] = c.H[0];
    c.H[0] = c.cur;
    c.cur = h;
    c.h_n[2] = step == 1 ? 0 : c.h_n[1];
    c.h_n[1] = step == 1 ? 0 : c.h_n[0];
    c.h_n[0] = n;
}

// Phase 2 of a block-diagonal-N strip after the Schur update: with X_I = W^-1 (W = S_II),
//   G_II = X_I, G_IN = X_I Z, G_NI = -T, G_NN = X - T Z, T = Y X_I.
// Z^T is in Zt: it is made while the host waits for the first residual.
int phase2_assemble(Strip* p, StripChain& c, int k, float* S) {
    cudaStream_t cs = c.stream;
    const int mp = p->mp[k], nNp = p->nNp[k], n = mp - nNp;
    const float* Xt = c.cur + (int64_t)n * n;
    const DenseProduct d[2] = {
        {nNp, n, n, S + nNp, mp, Xt, n, c.T1, n, 1.f, 0.f, nullptr, 0},
        {n, nNp, n, c.cur, n, c.Zt, n, S + (int64_t)nNp * mp, mp, 1.f, 0.f, nullptr, 0}};
    int r = products(p, d, 2, cs);
    if (!r) r = gemm(p, nNp, nNp, n, c.T1, n, c.Zt, n, S, mp, -1.f, 1.f, cs);
    if (r) return r;
    OCMP_LAUNCH(k_store_ni_ii<<<nblk((int64_t)mp * (n / 4), 256), 256, 0, cs>>>(
        nNp, n, mp, reinterpret_cast<const float4*>(c.T1), reinterpret_cast<const float4*>(c.cur), S));
    return OCMP_OK;
}

// S_k[I, I] -= A[I, J] G_prev[J, J] A[J, I], the couplings given by the lists at offset lists
int schur_update(Strip* p, StripChain& c, int k, int prev, int64_t lists, const ocmp_space_s* s, const double* vals,
                 float* S) {
    if (p->nI[k] == 0 || p->nJ[prev] == 0) return OCMP_OK;
    const int nI = p->nI[k], nJ = p->nJ[prev], nIp = pad(nI);
    const int64_t s0 = p->s[k], sp = p->s[prev];
    const int32_t* Irow = p->d_I + p->ioff[k];
    const int32_t* Jrow = p->jrow + p->joff[prev];
    const int32_t* cp = p->d_cptr + lists;
    OCMP_LAUNCH(k_schur_t<<<dim3(nblk(nIp, 128), nblk(nJ, kSchurRows)), 128, 0, c.stream>>>(
        nI, nJ, nIp, s0, sp, Irow, Jrow, p->d_J + p->joff[prev], cp, p->d_cb, p->d_ccol, vals, s->d_free,
        p->d_G + p->goff[prev], p->mp[prev], c.T));
    OCMP_LAUNCH(k_schur_u<<<dim3(nblk(nI, 4 * 128), nI), 128, 0, c.stream>>>(nI, nIp, p->nNp[k], s0, sp, Irow, Jrow, cp,
                                                                           p->d_cb, p->d_crow, vals, s->d_free, c.T, S,
                                                                           p->mp[k]));
    return OCMP_OK;
}

// Phase 2 of up to one strip of each chain (-1: none), the chains' step-th, after their Schur updates:
// the I pivots, the two chains' Newton-Schulz iterations in turns.
int phase2(Strip* p, const int (&ks)[2], int step) {
    bool pending[2] = {false, false}, started[2] = {false, false}, ok[2] = {false, false}, fast[2] = {false, false};
    auto S = [&](int q) { return p->d_G + p->goff[ks[q]]; };
    auto W = [&](int q) { return S(q) + (int64_t)p->nNp[ks[q]] * p->mp[ks[q]] + p->nNp[ks[q]]; };
    auto n = [&](int q) { return p->mp[ks[q]] - p->nNp[ks[q]]; };
    auto finish = [&](int q) {
        int r = schulz_end(p, p->chain[q], W(q), p->mp[ks[q]], n(q), started[q], ok[q]);
        if (!r) r = phase2_assemble(p, p->chain[q], ks[q], S(q));
        schulz_keep(p->chain[q], n(q), step);
        return r;
    };
    for (int q = 0; q < 2; q++) {
        const int k = ks[q];
        if (k < 0) continue;
        StripChain& c = p->chain[q];
        fast[q] = p->schulz && p->fast[k];
        if (!p->fast[k])
            for (int& h : c.h_n) h = 0;
        int r = fast[q] ? schulz_begin(p, c, W(q), p->mp[k], n(q), &pending[q])
                        : gj_tiles(p, S(q), p->mp[k], p->nNp[k], p->mp[k], c.work, c.stream);
        started[q] = pending[q];
        const int nNp = p->nNp[k];
        if (!r && fast[q]) r = transpose(S(q) + (int64_t)nNp * p->mp[k], p->mp[k], n(q), nNp, c.Zt, n(q), c.stream);
        if (!r && fast[q] && !pending[q]) r = finish(q);
        if (r) return r;
    }
    while (pending[0] || pending[1])
        for (int q = 0; q < 2; q++) {
            if (!pending[q]) continue;
            int r = schulz_step(p, p->chain[q], W(q), p->mp[ks[q]], n(q), &pending[q], &ok[q]);
            if (!r && !pending[q]) r = finish(q);
            if (r) return r;
        }
    return OCMP_OK;
}

}  // namespace

int strip_create(const ocmp_space_s* s, Strip** out) {
    *out = nullptr;
    const int64_t n = s->ndof;
    if (n <= 0) return fail(OCMP_ERR_ARG, "strip preconditioner: empty space");
    const std::vector<int64_t>& rp = s->rowptr;
    const std::vector<int32_t>& col = s->col;
    std::vector<int64_t> mx(n), mn(n);
    for (int64_t r = 0; r < n; r++) {
        int64_t a = r, b = r;
        for (int64_t k = rp[r]; k < rp[r + 1]; k++) {
            a = std::min<int64_t>(a, col[k]);
            b = std::max<int64_t>(b, col[k]);
        }
        mn[r] = a;
        mx[r] = b;
    }
    auto* p = new Strip();
    p->s.push_back(0);
    while (p->s.back() < n) {
        int64_t nxt;
        if (p->s.size() == 1) nxt = mx[0] + 1;
        else {
            nxt = 0;
            for (int64_t r = p->s[p->s.size() - 2]; r < p->s.back(); r++) nxt = std::max(nxt, mx[r] + 1);
        }
        nxt = std::min<int64_t>(n, std::max<int64_t>(nxt, p->s.back() + 1));
        p->s.push_back(nxt);
    }
    // uniform strips when the pattern repeats with a period w (a structured mesh numbered row by
    // row of elements): strips of exactly w dofs, each one row, make neighbouring strips' Schur
    // complements alike (the Newton-Schulz start relies on it) where the greedy strips drift
    // against the rows. w: the smallest width from half to twice the greedy one for which the
    // rows of a sample match the rows w further on (same column offsets) and the uniform strips
    // are block tridiagonal.
    if (p->s.size() > 4) {
        std::vector<int64_t> wd;
        for (size_t q = 2; q + 1 < p->s.size(); q++) wd.push_back(p->s[q] - p->s[q - 1]);
        std::nth_element(wd.begin(), wd.begin() + wd.size() / 2, wd.end());
        const int64_t wg = wd[wd.size() / 2];
        auto same = [&](int64_t r, int64_t w) {
            const int64_t r2 = r + w;
            if (rp[r + 1] - rp[r] != rp[r2 + 1] - rp[r2]) return false;
            for (int64_t e = 0; e < rp[r + 1] - rp[r]; e++)
                if ((int64_t)col[rp[r2] + e] - r2 != (int64_t)col[rp[r] + e] - r) return false;
            return true;
        };
        auto valid = [&](int64_t w) {
            for (int64_t r = 0; r < n; r++) {
                const int64_t k = r / w;
                if (mn[r] < (k - 1) * w || mx[r] >= (k + 2) * w) return false;
            }
            return true;
        };
        constexpr int kSample = 64;
        for (int64_t w = std::max<int64_t>(1, wg / 2); w <= 2 * wg && 3 * w <= n; w++) {
            int hits = 0;
            for (int q = 0; q < kSample; q++) {
                const int64_t r = (n - w - 1) * (2 * q + 1) / (2 * kSample);
                hits += same(r, w);
            }
            if (hits * 8 < kSample * 7 || !valid(w)) continue;
            std::vector<int64_t> u;
            for (int64_t b = 0; b < n; b += w) u.push_back(b);
            u.push_back(n);
            p->s.swap(u);
            break;
        }
    }
    // consecutive strips merge (the block-tridiagonal structure survives) until a strip holds at
    // least kMergeMin dofs: narrow bands (a P1 Laplacian's band is one row of vertices) would
    // otherwise give many small strips, whose sweeps are launch-bound
    {
        constexpr int64_t kMergeMin = 1024, kMergeMax = 4096;
        std::vector<int64_t> merged{0};
        size_t q = 1;
        while (q < p->s.size()) {
            int64_t end = p->s[q++];
            while (q < p->s.size() && end - merged.back() < kMergeMin && p->s[q] - merged.back() <= kMergeMax)
                end = p->s[q++];
            merged.push_back(end);
        }
        p->s.swap(merged);
    }
    p->K = (int)p->s.size() - 1;
    const int K = p->K;
    // every row must reach only its own and the neighbouring strips
    {
        int64_t k = 0;
        for (int64_t r = 0; r < n; r++) {
            while (r >= p->s[k + 1]) k++;
            const int64_t lo = k > 0 ? p->s[k - 1] : 0, hi = k + 2 <= K ? p->s[k + 2] : n;
            if (mn[r] < lo || mx[r] >= hi) {
                delete p;
                return fail(OCMP_ERR_UNSUPPORTED, "strip preconditioner: the pattern is not block tridiagonal over "
                                                  "its bandwidth strips (structurally unsymmetric)");
            }
        }
    }
    // interface sets: I_k = dofs of strip k coupled to its previous strip (by their row or their
    // column), the middle strip's to both neighbours; J_k = those coupled to its next strip
    const int mid = p->mid = K / 2;
    auto next_of = [&](int k) { return k < mid ? k + 1 : k - 1; };
    p->m.resize(K);
    p->nN.resize(K);
    p->nNp.resize(K);
    p->nI.assign(K, 0);
    p->nJ.assign(K, 0);
    std::vector<std::vector<char>> inI(K), inJ(K);
    for (int k = 0; k < K; k++) {
        p->m[k] = (int)(p->s[k + 1] - p->s[k]);
        inI[k].assign(p->m[k], 0);
        inJ[k].assign(p->m[k], 0);
    }
    for (int k = 0; k < K; k++) {
        const int64_t s0 = p->s[k], s1 = p->s[k + 1];
        for (int64_t r = s0; r < s1; r++)
            for (int64_t q = rp[r]; q < rp[r + 1]; q++) {
                const int64_t c = col[q];
                if (c >= s0 && c < s1) continue;
                const int o = c < s0 ? k - 1 : k + 1;
                const bool outer = k != mid && next_of(k) == o;   // k is farther from the middle than o
                (outer ? inJ : inI)[k][r - s0] = 1;
                (outer ? inI : inJ)[o][c - p->s[o]] = 1;
            }
    }
    // the end strips have no previous one and may take any I: where the dofs coupled to the next strip
    // form independent groups of at most 32 (a row of DG elements), the others, which makes them strips
    // of the Newton-Schulz path like the rest (their I block then costs half the pivot tiles and starts
    // the next strip's iteration)
    for (const int k : {0, K - 1}) {
        if (K == 1 || k == mid) continue;
        const int64_t s0 = p->s[k], s1 = p->s[k + 1];
        std::vector<int> par(p->m[k]), count(p->m[k], 0);
        std::iota(par.begin(), par.end(), 0);
        auto find = [&](int a) {
            while (par[a] != a) a = par[a] = par[par[a]];
            return a;
        };
        for (int i = 0; i < p->m[k]; i++)
            if (inJ[k][i])
                for (int64_t e = rp[s0 + i]; e < rp[s0 + i + 1]; e++)
                    if (col[e] >= s0 && col[e] < s1 && inJ[k][col[e] - s0]) par[find(i)] = find((int)(col[e] - s0));
        int largest = 0, nJ = 0;
        for (int i = 0; i < p->m[k]; i++)
            if (inJ[k][i]) {
                nJ++;
                largest = std::max(largest, ++count[find(i)]);
            }
        if (largest == 0 || largest > 32 || nJ == p->m[k]) continue;
        for (int i = 0; i < p->m[k]; i++) inI[k][i] = !inJ[k][i];
    }
    p->mp.resize(K);
    p->goff.resize(K + 1);
    p->poff.resize(K + 1);
    p->ioff.assign(K + 1, 0);
    p->joff.assign(K + 1, 0);
    std::vector<int32_t> perm, pinv(n, -1), Ipos, Jpos, Iinv(n, -1), Jinv(n, -1);
    int64_t total = 0;
    for (int k = 0; k < K; k++) {
        const int m = p->m[k];
        const int64_t s0 = p->s[k];
        std::vector<int32_t> Nl, Il;
        for (int i = 0; i < m; i++) (inI[k][i] ? Il : Nl).push_back(i);
        p->nN[k] = (int)Nl.size();
        p->nNp[k] = pad(p->nN[k]);
        p->nI[k] = (int)Il.size();
        p->mp[k] = p->nNp[k] + pad(p->nI[k]);
        p->goff[k] = total;
        total += (int64_t)p->mp[k] * p->mp[k];
        p->poff[k] = (int64_t)perm.size();
        p->mp_max = std::max(p->mp_max, p->mp[k]);
        std::vector<int32_t> pm(p->mp[k], -1);
        for (int q = 0; q < p->nN[k]; q++) pm[q] = Nl[q];
        for (int q = 0; q < p->nI[k]; q++) pm[p->nNp[k] + q] = Il[q];
        for (int q = 0; q < p->mp[k]; q++)
            if (pm[q] >= 0) pinv[s0 + pm[q]] = q;
        perm.insert(perm.end(), pm.begin(), pm.end());
        p->ioff[k] = (int64_t)Ipos.size();
        for (int q = 0; q < p->nI[k]; q++) {
            Iinv[s0 + Il[q]] = q;
            Ipos.push_back(Il[q]);         // local dofs (fill_iface); their positions are nNp + q
        }
        p->joff[k] = (int64_t)Jpos.size();
        for (int i = 0; i < m; i++)
            if (inJ[k][i]) {
                Jinv[s0 + i] = p->nJ[k]++;
                Jpos.push_back(i);
            }
        p->nIp_max = std::max(p->nIp_max, pad(p->nI[k]));
        p->nJp_max = std::max(p->nJp_max, pad(p->nJ[k]));
    }
    p->goff[K] = total;
    p->poff[K] = (int64_t)perm.size();
    p->ioff[K] = (int64_t)Ipos.size();
    p->joff[K] = (int64_t)Jpos.size();
    if (p->mp_max > 16384) {
        const int mm = p->mp_max;
        delete p;
        return fail(OCMP_ERR_UNSUPPORTED, "strip preconditioner: a strip of " + std::to_string(mm) +
                                              " dofs exceeds the 16384-dof limit (number the dofs so the matrix is banded)");
    }
    // J_k as positions in strip k's order (the Schur update gathers G_k[J, J]); the local dofs stay in
    // Jrow for the interface fill
    std::vector<int32_t> Jp(Jpos.size());
    for (int k = 0; k < K; k++)
        for (int64_t q = p->joff[k]; q < p->joff[k + 1]; q++) Jp[q] = pinv[p->s[k] + Jpos[q]];
    // strips whose N positions split into independent groups of at most 32 (union-find over the
    // pattern inside the strip, constrained dofs included, so the groups hold for any constraints),
    // packed greedily into warps' worth; the padding of N joins as single positions
    p->fast.assign(K, 0);
    p->gofs.assign(K + 1, 0);
    p->ngrp.assign(K, 0);
    std::vector<int32_t> gptr{0}, gidx, gcomp;
    for (int k = 0; k < K; k++) {
        p->gofs[k] = (int64_t)gptr.size() - 1;
        const int nN = p->nN[k];
        if (nN == 0 || p->nI[k] == 0) continue;
        const int64_t s0 = p->s[k], s1 = p->s[k + 1];
        std::vector<int> par(nN);
        std::iota(par.begin(), par.end(), 0);
        auto find = [&](int a) {
            while (par[a] != a) a = par[a] = par[par[a]];
            return a;
        };
        for (int q = 0; q < nN; q++) {
            const int64_t r = s0 + perm[p->poff[k] + q];
            for (int64_t e = rp[r]; e < rp[r + 1]; e++) {
                const int64_t c = col[e];
                if (c < s0 || c >= s1) continue;
                const int pc = pinv[c];
                if (pc < nN) {
                    const int a = find(q), b = find(pc);
                    if (a != b) par[std::max(a, b)] = std::min(a, b);
                }
            }
        }
        std::vector<std::vector<int32_t>> comp(nN);
        bool small = true;
        for (int q = 0; q < nN && small; q++) {
            auto& c = comp[find(q)];
            c.push_back(q);
            small = c.size() <= 32;
        }
        if (!small) continue;
        for (int q = nN; q < p->nNp[k]; q++) comp.push_back({q});
        const size_t g0 = gptr.size();
        int fill = 0;
        for (const auto& c : comp) {
            if (c.empty()) continue;
            if (fill + (int)c.size() > 32) {
                gptr.push_back((int32_t)gidx.size());
                fill = 0;
            }
            gidx.insert(gidx.end(), c.begin(), c.end());
            for (size_t e = 0; e < c.size(); e++) gcomp.push_back((fill << 8) | (int32_t)c.size());
            fill += (int)c.size();
        }
        gptr.push_back((int32_t)gidx.size());
        p->ngrp[k] = (int)(gptr.size() - g0);
        p->fast[k] = 1;
        p->nfast++;
    }
    p->gofs[K] = (int64_t)gptr.size() - 1;
    std::vector<int32_t> lo_ptr(n + 1, 0), hi_ptr(n + 1, 0), lo_pos, hi_pos;
    for (int k = 0; k < K; k++) {
        const int64_t s0 = p->s[k], s1 = p->s[k + 1];
        for (int64_t r = s0; r < s1; r++) {
            for (int64_t q = rp[r]; q < rp[r + 1]; q++) {
                if (col[q] >= s0 && col[q] < s1) continue;
                const bool next = k != mid && (col[q] >= s1) == (k < mid);
                (next ? hi_pos : lo_pos).push_back((int32_t)q);
            }
            lo_ptr[r + 1] = (int32_t)lo_pos.size();
            hi_ptr[r + 1] = (int32_t)hi_pos.size();
        }
    }
    // coupling lists of the I dofs to the previous strip's J dofs (the Schur update's sparse factors):
    // one list per I dof in the order of d_I; the middle strip's to the strip below it, and at the end
    // those to the strip above
    std::vector<int32_t> cptr{0}, cb, crow, ccol;
    auto couple = [&](int k, int prev) {
        std::vector<std::vector<std::array<int32_t, 3>>> lists(p->nI[k]);
        if (prev >= 0 && prev < K) {
            const int64_t s0 = p->s[k], s1 = p->s[k + 1], sp = p->s[prev], sq = p->s[prev + 1];
            auto entry = [&](int a, int32_t b) -> std::array<int32_t, 3>& {
                for (auto& e : lists[a])
                    if (e[0] == b) return e;
                lists[a].push_back({b, -1, -1});
                return lists[a].back();
            };
            for (int a = 0; a < p->nI[k]; a++) {
                const int64_t r = s0 + Ipos[p->ioff[k] + a];
                for (int64_t q = rp[r]; q < rp[r + 1]; q++)
                    if (col[q] >= sp && col[q] < sq) entry(a, Jinv[col[q]])[1] = (int32_t)q;
            }
            for (int64_t d = sp; d < sq; d++)
                for (int64_t q = rp[d]; q < rp[d + 1]; q++)
                    if (col[q] >= s0 && col[q] < s1) entry(Iinv[col[q]], Jinv[d])[2] = (int32_t)q;
        }
        for (auto& l : lists) {
            std::sort(l.begin(), l.end());
            for (auto& e : l) {
                cb.push_back(e[0]);
                crow.push_back(e[1]);
                ccol.push_back(e[2]);
            }
            cptr.push_back((int32_t)cb.size());
            p->cmax = std::max(p->cmax, (int)l.size());
        }
    };
    for (int k = 0; k < K; k++) couple(k, k <= mid ? k - 1 : k + 1);
    p->coff2 = (int64_t)cptr.size() - 1;
    couple(mid, mid + 1);
    // interface sizes of the strips that take the Newton-Schulz path; the second chain only where there
    // are strips above the middle
    int ns_max = 0;
    for (int k = 0; k < K; k++)
        if (p->fast[k]) ns_max = std::max(ns_max, p->mp[k] - p->nNp[k]);
    const int chains = mid + 1 < K ? 2 : 1;
    const int64_t fast_floats = p->nfast ? (int64_t)chains * (11 * (int64_t)ns_max * ns_max + 2 * (int64_t)p->mp_max * ns_max) +
                                                (int64_t)kSide * p->mp_max * ns_max
                                          : 0;
    const int64_t need = total * 4 + (int64_t)chains * p->nJp_max * p->nIp_max * 4 +
                         (int64_t)(kSide + chains) * (2 * (int64_t)p->mp_max * kNb + 2 * kNb * kNb) * 4 + fast_floats * 4;
    size_t fr = 0, tot = 0;
    cudaMemGetInfo(&fr, &tot);
    if ((size_t)need > fr) {
        delete p;
        return fail(OCMP_ERR_NOMEM, "strip preconditioner: the strip inverses need " + std::to_string(need >> 20) +
                                        " MiB of device memory");
    }
    int st = OCMP_OK;
    auto U = [&](auto** d, const auto& h) {
        if (!st) st = upload(d, h.data(), h.size());
    };
    U(&p->d_perm, perm);
    U(&p->d_pinv, pinv);
    U(&p->d_I, Ipos);
    U(&p->d_J, Jp);
    p->bytes = total * 4 + (int64_t)(perm.size() + Ipos.size() + Jp.size() + n) * 4;
    auto A = [&](auto** d, size_t cnt) {
        if (!st) st = dalloc(d, cnt);
    };
    A(&p->d_G, (size_t)total);
    U(&p->d_cptr, cptr);
    U(&p->d_cb, cb);
    U(&p->d_crow, crow);
    U(&p->d_ccol, ccol);
    p->bytes += (int64_t)(cptr.size() + 3 * cb.size()) * 4;
    auto work = [&](StripWork& w) {
        A(&w.P, 2 * (size_t)kNb * kNb);
        A(&w.Ck, (size_t)p->mp_max * kNb);
        A(&w.Rt, (size_t)p->mp_max * kNb);
    };
    for (auto& w : p->work) work(w);
    for (int q = 0; q < chains; q++) {
        work(p->chain[q].work);
        A(&p->chain[q].T, (size_t)std::max<int64_t>(1, (int64_t)p->nJp_max * p->nIp_max));
    }
    A(&p->d_flag, 2);
    {
        int dev = 0, sms = 1;
        if (!st && (cudaGetDevice(&dev) != cudaSuccess ||
                    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess))
            st = fail(OCMP_ERR_CUDA, "strip preconditioner: device attributes");
        // a block per SM, but no more than leaves each a few rows
        p->sweep_grid = std::max(1, std::min(sms, p->mp_max / kSweepMinRows));
        std::vector<SweepStep> steps;
        std::vector<int32_t> prow, erow, epos, edst;
        std::vector<uint32_t> blob;
        for (int k = 0; k < K; k++)
            for (int q = 0; q < p->mp[k]; q++) {
                const int32_t ld = perm[p->poff[k] + q];
                prow.push_back(ld < 0 ? -1 : (int32_t)(p->s[k] + ld));
            }
        // strip k as a step of the forward (mode 0) or backward sweep
        std::vector<int32_t> at(n);
        auto step = [&](int k, int mode, int gs) {
            const std::vector<int32_t>& ptr = mode == 0 ? lo_ptr : hi_ptr;
            const std::vector<int32_t>& pos = mode == 0 ? lo_pos : hi_pos;
            SweepStep t{};
            t.G = p->d_G + p->goff[k];
            t.p0 = (int32_t)p->poff[k];
            t.mp = p->mp[k];
            t.gs = gs;
            t.m = p->m[k];
            t.nN = p->nN[k];
            t.gap = p->nNp[k] - p->nN[k];
            t.per = sweep_rows(t.m, gs);
            std::vector<int32_t> cols, list;
            for (int q = 0; q < t.mp; q++) {
                const int32_t r = prow[t.p0 + q];
                if (r < 0 || ptr[r] == ptr[r + 1]) continue;
                list.push_back(q);
                t.len = std::max(t.len, ptr[r + 1] - ptr[r]);
                for (int32_t e = ptr[r]; e < ptr[r + 1]; e++) cols.push_back(col[pos[e]]);
            }
            std::sort(cols.begin(), cols.end());
            cols.erase(std::unique(cols.begin(), cols.end()), cols.end());
            t.cnt = (int32_t)list.size();
            t.nj = (int32_t)cols.size();
            const SweepLists li = sweep_lists(t.cnt, t.len, t.nj);
            t.blob = (int64_t)blob.size();
            t.words = li.words;
            blob.resize(blob.size() + li.words, 0u);
            uint32_t* b = blob.data() + t.blob;
            uint16_t* idx = reinterpret_cast<uint16_t*>(b + li.idx);
            for (int q = 0; q < t.nj; q++) {
                at[cols[q]] = q;
                b[li.jd + q] = (uint32_t)cols[q];
            }
            for (int c = 0; c < t.cnt; c++) {
                const int32_t r = prow[t.p0 + list[c]];
                reinterpret_cast<uint16_t*>(b + li.cq)[c] = (uint16_t)list[c];
                for (int e = 0; e < t.len; e++) {
                    const int32_t cp = ptr[r] + e < ptr[r + 1] ? pos[ptr[r] + e] : -1;
                    idx[e * t.cnt + c] = (uint16_t)(cp >= 0 ? at[col[cp]] : 0xffff);
                    erow.push_back(r);
                    epos.push_back(cp);
                    edst.push_back((int32_t)(t.blob + e * t.cnt + c));
                }
            }
            steps.push_back(t);
        };
        // forward from both ends to the middle strip, backward from it; the strips of a pair on one half
        // of the blocks each
        const int half = p->sweep_grid / 2;
        auto pair = [&](int k0, int k1, int mode) {
            if (half > 0 && k0 >= 0 && k1 >= 0) {
                step(k0, mode, half);
                step(k1, mode, p->sweep_grid - half);
                return;
            }
            for (const int k : {k0, k1})
                if (k >= 0) {
                    step(k, mode, p->sweep_grid);
                    steps.push_back(SweepStep{});
                }
        };
        const int up = K - 1 - mid;   // strips above the middle; below it are as many or one more
        for (int t = mid - 1; t >= 0; t--) pair(mid - 1 - t, t < up ? mid + 1 + t : -1, 0);
        pair(mid, -1, 0);
        const int nfwd = (int)steps.size() / 2;
        for (int t = 0; t < mid; t++) pair(mid - 1 - t, t < up ? mid + 1 + t : -1, 1);
        SweepArgs& a = p->sweep;
        a.nsteps = (int)steps.size() / 2;
        a.nfwd = nfwd;
        int most = 1;   // floats of a step's rows and lists in a block
        for (const SweepStep& t : steps) {
            a.rows = std::max(a.rows, t.per);
            a.mp_max = std::max(a.mp_max, t.mp);
            a.nj_max = std::max(a.nj_max, t.nj);
        }
        // the lists are staged when they take no more than a third of the ring
        const size_t fixed = sweep_fixed_smem(a.mp_max, a.nj_max, a.rows);
        const int room = fixed < kSweepSmem ? (int)((kSweepSmem - fixed) / sizeof(float)) & ~31 : 0;
        for (SweepStep& t : steps) {
            if (t.words > room / 3) t.words = 0;
            most = std::max(most, t.words + t.per * t.mp);
        }
        a.stages = std::max(1, std::min({kSweepStages, room / most, a.nsteps}));
        a.stage = std::min(most, room);
        p->sweep_smem = fixed + sizeof(float) * (size_t)a.stages * a.stage;
        if (!st && (blob.size() > (size_t)INT32_MAX || a.nj_max >= 0xffff || p->sweep_smem > kSweepSmem))
            st = fail(OCMP_ERR_UNSUPPORTED, "strip preconditioner: the couplings between the strips are too large");
        for (SweepStep& t : steps) {
            if (t.gs == 0) continue;
            t.ns = std::min(t.per, (a.stage - t.words) / t.mp);
            const int groups = (t.ns + 7) / 8 + (t.per - t.ns + 7) / 8;
            while (t.lwg < 4 && groups << (t.lwg + 1) <= kSweepWarps) t.lwg++;
        }
        if (!st && a.rows > kSweepThreads) st = fail(OCMP_ERR_UNSUPPORTED, "strip preconditioner: too few SMs");
        p->nell = (int64_t)epos.size();
        p->npos = (int64_t)prow.size();
        U(&p->d_steps, steps);
        U(&p->d_blob, blob);
        U(&p->d_prow, prow);
        U(&p->d_erow, erow);
        U(&p->d_epos, epos);
        U(&p->d_edst, edst);
        A(&p->d_rdof, prow.size());
        A(&p->d_words, 3 * (size_t)n);
        A(&p->d_state, 1);
        p->bytes += (int64_t)(prow.size() * 2 + epos.size() * 3 + blob.size() + 6 * n) * 4 +
                    (int64_t)(steps.size() * sizeof(SweepStep));
        a.steps = p->d_steps;
        a.prow = p->d_prow;
        a.rdof = p->d_rdof;
        a.blob = p->d_blob;
        a.b = p->d_words;
        a.y = p->d_words + n;
        a.x = p->d_words + 2 * n;
        a.n = n;
        a.state = p->d_state;
        if (!st) st = strip_reset(p, nullptr);
    }
    if (p->nfast) {
        const size_t i2 = (size_t)ns_max * ns_max, mi = (size_t)p->mp_max * ns_max;
        U(&p->d_gptr, gptr);
        U(&p->d_gidx, gidx);
        U(&p->d_gcomp, gcomp);
        for (int q = 0; q < chains; q++) {
            StripChain& c = p->chain[q];
            A(&c.cur, 2 * i2);
            A(&c.nxt, 2 * i2);
            for (float*& h : c.H) A(&h, 2 * i2);
            A(&c.Rt, i2);
            A(&c.T1, mi);
            A(&c.Zt, mi);
            A(&c.rmax, kSchulzMax);
            if (!st && cudaMallocHost((void**)&c.h_rmax, sizeof(unsigned)) != cudaSuccess)
                st = fail(OCMP_ERR_NOMEM, "strip preconditioner: pinned flag");
        }
        for (float*& y : p->d_Yt) A(&y, mi);
        p->bytes += (int64_t)(gptr.size() + 2 * gidx.size()) * 4;
    }
    U(&p->jrow, Jpos);
    p->bytes += (int64_t)Jpos.size() * 4;
    // every buffer a kernel of the factorisation or the sweeps dereferences must exist
    if (!st) {
        std::vector<const void*> need_ptr{p->d_perm, p->d_pinv, p->d_G, p->d_cptr, p->d_flag, p->d_prow, p->d_rdof,
                                          p->d_steps, p->d_words, p->d_state, p->work[0].P, p->work[0].Ck, p->work[0].Rt};
        for (int q = 0; q < chains; q++) {
            const StripChain& c = p->chain[q];
            need_ptr.insert(need_ptr.end(), {c.T, c.work.P, c.work.Ck, c.work.Rt});
            if (p->nfast)
                need_ptr.insert(need_ptr.end(), {c.cur, c.nxt, c.Rt, c.H[0], c.H[1], c.H[2], c.T1, c.Zt, c.rmax, c.h_rmax});
        }
        if (p->nfast)
            need_ptr.insert(need_ptr.end(), {p->d_gptr, p->d_gidx, p->d_gcomp, p->d_Yt[0], p->d_Yt[1], p->d_Yt[2]});
        bool ok = std::all_of(need_ptr.begin(), need_ptr.end(), [](const void* q) { return q != nullptr; });
        if (p->nell) ok = ok && p->d_blob && p->d_erow && p->d_epos && p->d_edst;
        if (!ok) st = fail(OCMP_ERR_NOMEM, "strip preconditioner: a work buffer was not allocated");
    }
    if (!st && (cudaEventCreateWithFlags(&p->fev[0], cudaEventDefault) != cudaSuccess ||
                cudaEventCreateWithFlags(&p->fev[1], cudaEventDefault) != cudaSuccess ||
                cudaEventCreateWithFlags(&p->ev_start, cudaEventDisableTiming) != cudaSuccess))
        st = fail(OCMP_ERR_CUDA, "cudaEventCreate");
    for (int q = 0; q < kSide && !st; q++)
        if (cudaStreamCreateWithFlags(&p->side[q], cudaStreamNonBlocking) != cudaSuccess)
            st = fail(OCMP_ERR_CUDA, "cudaStreamCreateWithFlags");
    if (!st) {
        int lo = 0, hi = 0;
        if (cudaDeviceGetStreamPriorityRange(&lo, &hi) != cudaSuccess)
            st = fail(OCMP_ERR_CUDA, "strip preconditioner: stream priorities");
        for (int q = 0; q < chains && !st; q++)
            if (cudaStreamCreateWithPriority(&p->chain[q].stream, cudaStreamNonBlocking, hi) != cudaSuccess ||
                cudaEventCreateWithFlags(&p->chain[q].ev_read, cudaEventDisableTiming) != cudaSuccess ||
                cudaEventCreateWithFlags(&p->chain[q].ev_done, cudaEventDisableTiming) != cudaSuccess)
                st = fail(OCMP_ERR_CUDA, "strip preconditioner: chain stream");
    }
    p->ev_phase1.assign(K, nullptr);
    for (int k = 0; k < K && !st; k++)
        if (cudaEventCreateWithFlags(&p->ev_phase1[k], cudaEventDisableTiming) != cudaSuccess)
            st = fail(OCMP_ERR_CUDA, "cudaEventCreate");
    if (!st) {
        if (cudaFuncSetAttribute(k_panels, cudaFuncAttributeMaxDynamicSharedMemorySize, kPanelSmem) != cudaSuccess ||
            cudaFuncSetAttribute(k_sweeps<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSweepSmem) != cudaSuccess ||
            cudaFuncSetAttribute(k_sweeps<float>, cudaFuncAttributeMaxDynamicSharedMemorySize, kSweepSmem) != cudaSuccess)
            st = fail(OCMP_ERR_CUDA, "strip preconditioner: shared-memory attribute");
    }
    if (st) {
        strip_free(p);
        delete p;
        return st;
    }
    *out = p;
    return OCMP_OK;
}

void strip_destroy(Strip* p) {
    if (!p) return;
    strip_free(p);
    delete p;
}

int strip_factor(Strip* p, const ocmp_space_s* s, const double* vals, cudaStream_t st) {
    const int K = p->K;
    p->ev_used = 0;
    p->ev_tag.clear();
    p->gemm_flops_pending = 0;
    p->gemm_bytes_pending = 0;
    p->ns_iters = p->ns_strips = p->ns_fallbacks = 0;
    for (auto& c : p->chain)
        for (int& h : c.h_n) h = 0;
    OCMP_CUDA(cudaEventRecord(p->fev[0], st));
    OCMP_CUDA(cudaMemsetAsync(p->d_flag, 0, 2 * sizeof(int), st));
    {
        const int64_t nt = std::max(p->nell, p->npos);
        OCMP_LAUNCH(k_list_refresh<<<nblk(nt, 256), 256, 0, st>>>(p->nell, p->d_erow, p->d_epos, s->d_col, vals, s->d_free,
                                                                 p->d_edst, p->d_blob, p->npos, p->d_prow, p->d_rdof));
    }
    OCMP_CUDA(cudaEventRecord(p->ev_start, st));
    for (int q = 0; q < kSide; q++) OCMP_CUDA(cudaStreamWaitEvent(p->side[q], p->ev_start, 0));
    const int mid = p->mid, chains = mid + 1 < K ? 2 : 1;
    for (int q = 0; q < chains; q++) OCMP_CUDA(cudaStreamWaitEvent(p->chain[q].stream, p->ev_start, 0));
    // phase 1: fill every strip and eliminate its N pivots, strips spread over the side streams in the
    // order in which phase 2 takes them
    std::vector<int> order;
    for (int t = 0; t < mid; t++) {
        order.push_back(t);
        if (K - 1 - t > mid) order.push_back(K - 1 - t);
    }
    order.push_back(mid);
    auto phase1 = [&](int o) {
        const int k = order[o], q = o % kSide;
        cudaStream_t ss = p->side[q];
        const int mp = p->mp[k];
        float* S = p->d_G + p->goff[k];
        OCMP_CUDA(cudaMemsetAsync(S, 0, sizeof(float) * (size_t)mp * mp, ss));
        OCMP_LAUNCH(k_fill_strip<<<nblk(mp, 128), 128, 0, ss>>>(mp, p->s[k], p->d_perm + p->poff[k], p->d_pinv, s->d_rowptr,
                                                               s->d_col, vals, s->d_free, p->s[k + 1], S));
        const int r = p->schulz && p->fast[k] ? phase1_groups(p, k, S, q, ss)
                                              : gj_tiles(p, S, mp, 0, p->nNp[k], p->work[q], ss);
        if (r) return r;
        OCMP_CUDA(cudaEventRecord(p->ev_phase1[k], ss));
        return (int)OCMP_OK;
    };
    // a few pairs ahead of phase 2, which then does not wait for the host to have launched all of phase 1
    int issued = 0;
    // phase 2: the two chains side by side, then the middle strip on the first
    for (int t = 0; t <= mid; t++) {
        const int ks[2] = {t, t < mid && K - 1 - t > mid ? K - 1 - t : -1};
        for (; issued < K && issued < 2 * (t + kAhead); issued++)
            if (const int r = phase1(issued)) return r;
        for (int q = 0; q < 2; q++) {
            const int k = ks[q];
            if (k < 0) continue;
            StripChain& c = p->chain[q];
            float* S = p->d_G + p->goff[k];
            OCMP_CUDA(cudaStreamWaitEvent(c.stream, p->ev_phase1[k], 0));
            int r = OCMP_OK;
            const int prev = q == 0 ? k - 1 : k + 1;
            if (prev >= 0 && prev < K) r = schur_update(p, c, k, prev, p->ioff[k], s, vals, S);
            if (!r && k == mid && mid + 1 < K) {
                OCMP_CUDA(cudaEventRecord(p->chain[1].ev_done, p->chain[1].stream));
                OCMP_CUDA(cudaStreamWaitEvent(c.stream, p->chain[1].ev_done, 0));
                r = schur_update(p, c, k, mid + 1, p->coff2, s, vals, S);
            }
            if (r) return r;
        }
        if (const int r = phase2(p, ks, t)) return r;
    }
    OCMP_CUDA(cudaGetLastError());
    OCMP_CUDA(cudaEventRecord(p->chain[0].ev_done, p->chain[0].stream));
    OCMP_CUDA(cudaStreamWaitEvent(st, p->chain[0].ev_done, 0));
    OCMP_CUDA(cudaEventRecord(p->fev[1], st));
    int flags[2] = {0, 0};
    OCMP_CUDA(cudaMemcpyAsync(flags, p->d_flag, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
    OCMP_CUDA(cudaStreamSynchronize(st));
    float ms = 0;
    OCMP_CUDA(cudaEventElapsedTime(&ms, p->fev[0], p->fev[1]));
    p->factor_ms = ms;
    p->singular = flags[0];
    if (flags[1]) return fail(OCMP_TIMEOUT, "strip preconditioner: a tensor-core product gave up a bounded wait");
    p->gemm_flops = p->gemm_flops_pending;
    p->gemm_bytes = p->gemm_bytes_pending;
    p->gemm_ms = 0;
    for (double& x : p->part_ms) x = 0;
    for (size_t q = 0; q + 1 < p->ev_used; q += 2) {
        float e = 0;
        OCMP_CUDA(cudaEventElapsedTime(&e, p->ev[q], p->ev[q + 1]));
        p->part_ms[p->ev_tag[q / 2]] += e;
    }
    p->gemm_ms = p->part_ms[0];
    if (flags[0]) return fail(OCMP_BREAKDOWN, "strip preconditioner: " + std::to_string(flags[0]) +
                                                  " zero or non-finite pivots in the strip factorisation");
    return OCMP_OK;
}

template <class T>
int strip_apply(Strip* p, const T* v, const double* scale, int j, T* z, const int* flags, int* err, cudaStream_t st) {
    SweepArgs a = p->sweep;
    a.err = err;
    void* kp[] = {&a, &v, &scale, &j, &z, &flags};
    OCMP_LAUNCH(OCMP_CUDA(cudaLaunchCooperativeKernel((const void*)k_sweeps<T>, dim3(p->sweep_grid), dim3(kSweepThreads),
                                                      kp, p->sweep_smem, st)));
    return OCMP_OK;
}
template int strip_apply<double>(Strip*, const double*, const double*, int, double*, const int*, int*, cudaStream_t);
template int strip_apply<float>(Strip*, const float*, const double*, int, float*, const int*, int*, cudaStream_t);

// no word of an earlier launch may carry a later epoch: the results are cleared with the count
int strip_reset(Strip* p, cudaStream_t st) {
    OCMP_CUDA(cudaMemsetAsync(p->d_state, 0, sizeof(SweepState), st));
    OCMP_CUDA(cudaMemsetAsync(p->d_words, 0, sizeof(uint2) * 3 * (size_t)p->s.back(), st));
    return OCMP_OK;
}

// a test: a wait of the next application runs out
int strip_starve(Strip* p) {
    const int on = 1;
    OCMP_CUDA(cudaMemcpy(&p->d_state->starve, &on, sizeof(int), cudaMemcpyHostToDevice));
    return OCMP_OK;
}

template <class T>
int strip_add(int64_t n, const T* z, double* x, cudaStream_t st) {
    OCMP_LAUNCH(k_add_to<T><<<nblk(n, 256), 256, 0, st>>>(n, z, x));
    return OCMP_OK;
}
template int strip_add<double>(int64_t, const double*, double*, cudaStream_t);
template int strip_add<float>(int64_t, const float*, double*, cudaStream_t);

void strip_stats(const Strip* p, ocmp_strip_stats_t* o) {
    o->nstrips = p->K;
    o->max_strip = p->mp_max;
    o->bytes = p->bytes;
    o->factor_ms = p->factor_ms;
    o->gemm_ms = p->gemm_ms;
    o->gemm_flops = p->gemm_flops;
    o->gemm_bytes = p->gemm_bytes;
    o->singular_tiles = p->singular;
    o->gemm_kind = p->gemm_kind;
    o->tile_ms = p->part_ms[1];
    o->panel_ms = p->part_ms[2];
    o->fast_strips = p->schulz ? p->nfast : 0;
    o->schulz_strips = p->ns_strips;
    o->schulz_iterations = p->ns_iters;
    o->schulz_fallbacks = p->ns_fallbacks;
}

void strip_set_timing(Strip* p, bool on) { p->timing = on; }
void strip_set_gemm(Strip* p, int kind) { p->gemm_kind = kind; }
void strip_set_schulz(Strip* p, bool on) { p->schulz = on; }

}  // namespace ocmp

using namespace ocmp;

extern "C" int ocmp_dense_gemm_nt(int32_t kind, int32_t M, int32_t N, int32_t K, const float* A, int64_t lda,
                                  const float* B, int64_t ldb, float* C, int64_t ldc, float alpha, float beta,
                                  void* stream) {
    if (!A || !B || !C) return fail(OCMP_ERR_ARG, "ocmp_dense_gemm_nt: null argument");
    if (kind != 0 && kind != 1) return fail(OCMP_ERR_ARG, "ocmp_dense_gemm_nt: kind is 0 (SIMT) or 1 (tensor cores)");
    if (lda < K || ldb < K || ldc < N) return fail(OCMP_ERR_ARG, "ocmp_dense_gemm_nt: leading dimension too small");
    cudaStream_t st = (cudaStream_t)stream;
    if (kind == 0) {
        if (M <= 0 || N <= 0 || K <= 0 || M % GB || N % GB || K % GK || (lda | ldb | ldc) & 3)
            return fail(OCMP_ERR_ARG, "ocmp_dense_gemm_nt: M, N must be multiples of 128, K of 16");
        const dim3 g(N / GB, M / GB);
        OCMP_LAUNCH(sgemm_nt<<<g, 256, 0, st>>>(DenseProduct{M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, C, ldc}));
        OCMP_CUDA(cudaGetLastError());
        return OCMP_OK;
    }
    int* err = nullptr;
    OCMP_CUDA(cudaMallocAsync((void**)&err, sizeof(int), st));
    OCMP_CUDA(cudaMemsetAsync(err, 0, sizeof(int), st));
    int r = tc_gemm_nt(M, N, K, A, lda, B, ldb, C, ldc, alpha, beta, err, st);
    int h = 0;
    if (!r && cudaMemcpyAsync(&h, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess)
        r = fail(OCMP_ERR_CUDA, "ocmp_dense_gemm_nt: flag copy");
    cudaFreeAsync(err, st);
    if (!r) OCMP_CUDA(cudaStreamSynchronize(st));
    if (!r && h) r = fail(OCMP_TIMEOUT, "ocmp_dense_gemm_nt: a bounded wait of the tensor-core product gave up");
    return r;
}
