// Krylov solvers of libopencmp_gpu.so (sm_103a): the GPU counterpart of the linear solve in
// opencmp/models/base_model.py:886-947 (solvers.CG with the 'local' = point-Jacobi preconditioner
// restricted to free dofs, solvers.GMRes with freedofs). This file holds the handles, the
// preconditioners' set-up and the launches; the iterations are the persistent kernels of
// ocmp_cg.cuh and ocmp_gmres.cuh, a whole solve in one cooperative launch (the preconditioners that
// are kernels of their own, strip and Cahouet-Chabard, one launch per phase). Every sum runs in a
// fixed order, so results are bit-reproducible run to run.
//
// Precision: OCMP_FP64 runs everything in FP64. OCMP_MIXED runs an outer FP64 iterative
// refinement (r = b - A x with the FP64 matrix, x += correction) around an inner GMRES/CG whose
// matrix values, vectors and preconditioner are FP32; dot products are sums of FP32 products in float
// pairs or FP64; the Hessenberg matrix and rotations stay FP64.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <mutex>
#include <string>
#include <type_traits>

#include "ocmp_internal.h"
#include "ocmp_spmv.cuh"
#include "ocmp_cg.cuh"
#include "ocmp_gmres.cuh"

// Cahouet-Chabard block preconditioner of a Taylor-Hood saddle-point system [u | p]
// (OCMP_PRE_CAHOUET_CHABARD): velocity point Jacobi, and on the pressure block
// z_p = -(alpha S^-1 r_p + beta M_p,diag^-1 r_p) / tc^2 with S = L_p + delta M_p solved exactly by the
// strip direct factorisation of the pressure operator.
struct CCPre {
    ocmp::Strip* strip = nullptr;
    ocmp_matrix_s* pop = nullptr;   // the pressure operator S (pressure space)
    int64_t nu = 0, np = 0;         // velocity dofs (all components) and pressure dofs
    double alpha = 1, beta = 0, tc = 1;
    double* vdinv = nullptr;        // nu
    double* mpinv = nullptr;        // np
    double* zp64 = nullptr;         // np: pressure-solve vector
    float* zp32 = nullptr;
};

struct ocmp_solver_s {
    ocmp_matrix_s* mat = nullptr;
    ocmp_space_s* s = nullptr;
    ocmp_solve_params_t prm{};
    int64_t n = 0;
    int m = 0;                  // GMRES restart
    // FP64 path
    double* dinv = nullptr;     // Jacobi (0 on constrained rows)
    double* udiag = nullptr;    // caller's inverse diagonal (OCMP_PRE_USER)
    bool udiag_set = false;
    double* Binv = nullptr;     // block Jacobi (L2 element blocks)
    ocmp::Strip* strip = nullptr;  // strip direct preconditioner (OCMP_PRE_STRIP)
    bool strip_ready = false;       // factorised by ocmp_solver_update since the last failure
    CCPre* cc = nullptr;           // Cahouet-Chabard data (OCMP_PRE_CAHOUET_CHABARD), once set
    double* V = nullptr;        // (m+1) x n
    double* w = nullptr;
    double* z = nullptr;
    double* r = nullptr;
    double* p = nullptr;
    // FP32 inner path (OCMP_MIXED)
    float* dinv32 = nullptr;
    float* Binv32 = nullptr;
    float* V32 = nullptr;
    float* w32 = nullptr;
    float* z32 = nullptr;
    float* r32 = nullptr;
    float* p32 = nullptr;
    float* d32 = nullptr;       // inner correction
    double* pb = nullptr;       // second search direction (CG)
    float* p32b = nullptr;
    ocmp::CgState* dcg = nullptr;    // CG: results and exchange slots
    ocmp::CgState* hcg = nullptr;    // pinned: the results and the head of the slots
    // GMRES
    double* small = nullptr;    // per system: R, rotations, scales (kept between the launches of phases)
    ocmp::GmResult* gout = nullptr;  // per system: what the host reads
    ocmp::GmResult* hout = nullptr;  // pinned; behind the systems' results two slots for the phases' checks
    cudaEvent_t ev_check[2] = {nullptr, nullptr};
    ocmp::GmTeams* teams = nullptr;  // the blocks' teams
    double* As64 = nullptr;     // A D^-1 (Jacobi folded) or A, FP64 Krylov matrix (owned)
    float* As32 = nullptr;      // same in FP32 (OCMP_MIXED)
    const double* K64 = nullptr;  // Krylov matrix in use: As64, or the matrix's own scaled values
    const float* K32 = nullptr;
    bool borrow = false;        // Jacobi-scaled values and D^-1 come from the assembly
    int B = 1;                  // systems in the batch (matrix instances)
    int u64 = 4;                // GMRES: entries in flight per lane of the FP64 products
    // optional timing of the Krylov products (ocmp_solver_spmv_timing)
    bool time_spmv = false;
    unsigned long long* tlog = nullptr;   // per product: complement of the start, and end (global timer, ns)
    // the FP32 Krylov matrix is the assembly's SELL-32 copy (OCMP_MAT_SELL32, borrowed)
    bool sell = false;
    int last_iters = 0;         // iterations of the last GMRES solve (adaptive host checks)
    int64_t spmv_launches = 0;
    double spmv_ms = 0;
};

// A group of GMRES solvers whose instances (every system of every member, members of different
// sizes and patterns) are solved in one launch.
struct ocmp_group_s {
    std::vector<ocmp_solver_s*> members;
    std::vector<int> first;          // per member: its first instance
    int ninst = 0, m = 0, maxit = 0;
    bool mixed = false;
    std::vector<ocmp::GmInst> h_inst;
    ocmp::GmTeams* teams = nullptr;
    ocmp::GmResult* gout = nullptr;
    ocmp::GmResult* hout = nullptr;  // pinned
};

namespace ocmp {
namespace {

constexpr int kThreads = 256;
inline unsigned nblk(int64_t n, int t) { return (unsigned)((n + t - 1) / t); }

template <class T>
__global__ void jacobi_setup(int64_t n, const int32_t* __restrict__ diag, const double* __restrict__ vals,
                             const uint8_t* __restrict__ freed, T* __restrict__ dinv) {
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    double d = vals[diag[i]];
    dinv[i] = (T)((freed[i] && d != 0.0) ? 1.0 / d : 0.0);
}

// block-Jacobi inverse of each element block (L2 spaces), Gauss-Jordan with partial pivoting, FP64
template <int L>
__global__ void block_jacobi_setup(int64_t ne, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                                   const double* __restrict__ vals, double* __restrict__ Binv,
                                   float* __restrict__ Binv32) {
    int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= ne) return;
    double A[L][2 * L];
    for (int i = 0; i < L; i++) {
        const int64_t r = e * L + i;
        const int32_t a = rp[r], b = rp[r + 1];
        for (int j = 0; j < L; j++) {
            A[i][j] = 0;
            A[i][L + j] = (i == j) ? 1.0 : 0.0;
        }
        for (int32_t k = a; k < b; k++) {
            const int32_t c = col[k];
            if (c >= e * L && c < (e + 1) * L) A[i][c - e * L] = vals[k];
        }
    }
    for (int c = 0; c < L; c++) {
        int pr = c;
        for (int i = c + 1; i < L; i++)
            if (fabs(A[i][c]) > fabs(A[pr][c])) pr = i;
        if (pr != c)
            for (int j = 0; j < 2 * L; j++) {
                double t = A[c][j];
                A[c][j] = A[pr][j];
                A[pr][j] = t;
            }
        const double d = A[c][c];
        const double id = d != 0.0 ? 1.0 / d : 0.0;
        for (int j = 0; j < 2 * L; j++) A[c][j] *= id;
        for (int i = 0; i < L; i++)
            if (i != c) {
                const double mm = A[i][c];
                for (int j = 0; j < 2 * L; j++) A[i][j] -= mm * A[c][j];
            }
    }
    for (int i = 0; i < L; i++)
        for (int j = 0; j < L; j++) {
            Binv[(e * L + i) * L + j] = A[i][L + j];
            if (Binv32) Binv32[(e * L + i) * L + j] = (float)A[i][L + j];
        }
}

// Blocks of the current device's SMs a team may have.
int team_blocks(int* out) {
    int dev = 0, sms = 0;
    OCMP_CUDA(cudaGetDevice(&dev));
    OCMP_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    *out = std::max(1, std::min(sms, kTeamMaxBlocks));
    return OCMP_OK;
}

template <class T>
int cg_launch(const void* k, CgArgs<T>& a, int grid, int threads, size_t smem, cudaStream_t st) {
    void* kp[] = {&a};
    OCMP_LAUNCH(OCMP_CUDA(cudaLaunchCooperativeKernel(k, dim3(grid), dim3(threads), kp, smem, st)));
    return OCMP_OK;
}

// The whole CG solve in one cooperative launch. Resident form: a system of few rows and entries is one
// block's (its exchanges are __syncthreads); above, the slices of 32 rows are dealt to the SMs. One block
// against many (us an iteration): FP64 6.7 and 10.8 at 289 rows of 3,073 entries, 8.4 and 8.4 at 625 of
// 4,177, 9.2 and 9.9 at 625 of 6,817, 10.7 and 9.6 at 961 of 10,591; FP32 5.7 and 8.8, 5.8 and 7.2, 6.4 and
// 8.6, 6.5 and 8.0.
constexpr int64_t kCgOneBlockRows = 1024, kCgOneBlockNnz = 8192;
constexpr int64_t kCgFuseNnz = 4900;   // entries per block whose second FMA costs the barrier's 2,450 clocks
constexpr size_t kCgSmem = 200 * 1024;

template <class T>
int cg_smem_limit() {
    return smem_limit((const void*)cg_res_kernel<T>, kCgSmem);
}

template <class T>
int cg_solve(const CgArgs<T>& args, const ocmp_space_s* s, bool two_p, cudaStream_t st, CgState* out) {
    CgArgs<T> a = args;
    constexpr bool D = sizeof(T) == 8;
    int sms = 1;
    if (const int r = team_blocks(&sms)) return r;
    const int64_t slices = (a.n + 31) / 32;
    int r = -1;
    if (a.n <= (int64_t)sms * kCgRowsRes) {
        const int grid = a.n <= kCgOneBlockRows && s->nnz <= kCgOneBlockNnz ? 1 : (int)std::min<int64_t>(sms, slices);
        const int per = (int)((slices + grid - 1) / grid);   // slices of a block
        int64_t cap = 0;
        for (int b = 0; b < grid; b++) {
            int64_t c = 0;
            for (int64_t q = b; q < slices; q += grid) c += s->slice_width[q];
            cap = std::max(cap, 32 * c);
        }
        const size_t smem = (size_t)cap * (sizeof(T) + 4) + (grid == 1 ? 2 * kCgRowsRes * sizeof(T) : 0);
        a.cap = (int)cap;
        a.fuse = grid > 1 && two_p && (!D || cap <= kCgFuseNnz);
        const int threads = 32 * std::max(4, std::min(kCgThreadsRes / 32, per));
        if (per <= kCgSlicesRes && smem <= kCgSmem)
            r = cg_launch((const void*)cg_res_kernel<T>, a, grid, threads, smem, st);
    }
    if (r < 0) {
        // few lanes per row where the FP64 pipe bounds the product
        const double avg = (double)s->nnz / (double)s->ndof;
        const int tpr = avg <= 14 ? (D ? 2 : 4) : avg <= 40 ? (D ? 4 : 8) : (D ? 8 : 16);
        const int rt = kCgThreadsStream / tpr;
        const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(sms, (a.n + rt - 1) / rt));
        const void* k = tpr == 2   ? (const void*)cg_stream_kernel<double, 2>
                        : tpr == 4 ? (const void*)cg_stream_kernel<T, 4>
                        : tpr == 8 ? (const void*)cg_stream_kernel<T, 8>
                                   : (const void*)cg_stream_kernel<float, 16>;
        r = cg_launch(k, a, grid, kCgThreadsStream, 0, st);
    }
    if (r) return r;
    OCMP_CUDA(cudaMemcpyAsync(out, a.state, kCgReadBytes, cudaMemcpyDeviceToHost, st));
    OCMP_CUDA(cudaStreamSynchronize(st));
    if (out->t.abort) {
        OCMP_CUDA(cudaMemsetAsync(a.state, 0, sizeof(CgState), st));
        return fail(OCMP_TIMEOUT, "CG: a block gave up waiting for the others");
    }
    return OCMP_OK;
}

// A_s = A D^-1 (Jacobi) or A, cast to T
template <class T>
__global__ void gm_scale_matrix(int64_t n, const int32_t* __restrict__ rp, const int32_t* __restrict__ col,
                                const double* __restrict__ A, const double* __restrict__ dinv64, T* __restrict__ As,
                                int64_t nnz) {
    A += blockIdx.y * nnz;
    As += blockIdx.y * nnz;
    if (dinv64) dinv64 += blockIdx.y * n;
    const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (int32_t k = rp[r]; k < rp[r + 1]; k++) {
        const double d = dinv64 ? dinv64[col[k]] : 1.0;
        As[k] = (T)(A[k] * d);
    }
}

__global__ void gm_cast(int64_t n, const double* __restrict__ a, float* __restrict__ b) {
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) b[i] = (float)a[i];
}

// Cahouet-Chabard after the pressure solve zp = S^-1 (sc v_p): z_u = sc D_u^-1 v_u,
// z_p = -(alpha zp + beta M^-1 (sc v_p)) / tc^2; z may be v
template <class T>
__global__ void cc_combine(int64_t nu, int64_t np, const T* v, const double* __restrict__ scale, int j,
                           const double* __restrict__ vdinv, const double* __restrict__ mpinv,
                           const T* __restrict__ zp, T* z, double alpha, double beta, double tc,
                           const int* __restrict__ flags) {
    if (flags && flags[F_CONV]) return;
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= nu + np) return;
    const double sv = (scale ? scale[j] : 1.0) * (i < nu ? vdinv[i] : 1.0) * (double)v[i];
    z[i] = (T)(i < nu ? sv : -(alpha * (double)zp[i - nu] + beta * mpinv[i - nu] * sv) / (tc * tc));
}

template <class T>
int cc_apply(CCPre* cc, const T* v, const double* scale, int j, T* z, const int* flags, int* err, cudaStream_t st) {
    T* zp = nullptr;
    if constexpr (std::is_same<T, float>::value) zp = cc->zp32;
    else zp = cc->zp64;
    const int r = strip_apply<T>(cc->strip, v + cc->nu, scale, j, zp, flags, err, st);
    if (r) return r;
    OCMP_LAUNCH(cc_combine<T><<<nblk(cc->nu + cc->np, kThreads), kThreads, 0, st>>>(
        cc->nu, cc->np, v, scale, j, cc->vdinv, cc->mpinv, zp, z, cc->alpha, cc->beta, cc->tc, flags));
    return OCMP_OK;
}

// Lanes per row of a Krylov product: the autotuned choice, or the row length's; of an FP64 product half
// of that (bound by the FP64 pipe, on which a shuffle-reduction step costs as much as a product). The
// autotuned choice is an FP64 product's already, so rows of more than 16 entries are not left a single lane
// by it. Halved against as tuned (us an iteration): P2 triangles (11.5 entries) 56.4 and 60.8, P1 tetrahedra
// 40.7 and 41.6; P3 triangles (17) 50.5 and 44.3, DG P2 triangles (24) 121 and 106, P2 tetrahedra at
// 2,146,689 rows 485 and 438.
int gm_lanes(const ocmp_space_s* s, bool fp64) {
    const int t = row_cfg(s).tpr;
    if (fp64 && s->tuned_tpr > 0 && s->nnz > 16 * s->ndof) return t;
    return fp64 ? std::max(1, t / 2) : t;
}

// Entries in flight per lane of an FP64 solve's products: 8, unless that pads the rows (an entry past a
// row's end takes its turn on the FP64 pipe) by over 4% more than 4 does, the longest row of each slice of
// 32 counted. Per iteration: P2 tetrahedra (3% more) 30.9 -> 30.3 us at 79,507 rows, 391 -> 367 at 1,771,561;
// P3 tetrahedra (2%) 245 -> 213 at 753,571; but DG P2 triangles, rows of 24 (33%), 28.2 -> 29.8 at 62,208 and
// P3 triangles (5%) 183 -> 185 at 811,801.
int gm_unroll(const ocmp_space_s* s) {
    const int lanes = gm_lanes(s, true);
    int64_t pad4 = 0, pad8 = 0;
    for (const int w : s->slice_width) {
        pad4 += (w + 4 * lanes - 1) / (4 * lanes) * 4;
        pad8 += (w + 8 * lanes - 1) / (8 * lanes) * 8;
    }
    return 25 * pad8 <= 26 * pad4 ? 8 : 4;
}

template <class T>
GmInst gm_inst(const ocmp_solver_s* sv, int q, const double* b, double* x, int tile) {
    const ocmp_space_s* s = sv->s;
    constexpr bool D = sizeof(T) == 8;
    const int64_t n = sv->n, m = sv->m;
    const int pre = sv->prm.precond;
    const bool diag = pre == OCMP_PRE_JACOBI || pre == OCMP_PRE_USER;
    GmInst d{};
    d.n = n;
    d.ld = gm_ld<T>(n);
    d.rp = s->d_rowptr;
    d.col = s->d_col;
    d.freed = s->d_free;
    d.lift_ptr = s->d_lift_ptr;
    d.lift_pos = s->d_lift_pos;
    d.A64 = sv->mat->vals + q * s->nnz;
    if constexpr (D) {
        d.K = sv->K64 + q * s->nnz;
        d.dinv = diag ? sv->dinv + q * n : nullptr;
        d.Binv = sv->Binv;
        d.V = sv->V + q * (m + 1) * d.ld;
        d.z = sv->z;
    } else {
        d.K = sv->K32 + q * s->nnz;
        d.dinv = diag ? sv->dinv32 + q * n : nullptr;
        d.Binv = sv->Binv32;
        d.V = sv->V32 + q * (m + 1) * d.ld;
        d.z = sv->z32;
        if (sv->sell) {
            d.soff = s->d_sell_off;
            d.scol = s->d_sell_col;
        }
    }
    d.b = b;
    d.x = x;
    d.small = sv->small + (size_t)q * gm_small_doubles(sv->m);
    d.out = sv->gout + q;
    d.tol = sv->prm.tol;
    d.inner = D ? 0.0 : (sv->prm.inner_tol > 0 ? sv->prm.inner_tol : 1e-4);
    d.maxit = sv->prm.maxit;
    d.L = s->nloc;
    // whole elements in a tile when they are preconditioned as blocks (3, 6 or 10 rows)
    d.TR = d.Binv ? (d.L == 10 ? 160 : 96) : tile;
    d.tpr = gm_lanes(s, D);
    d.rtpr = gm_lanes(s, true);
    d.u64 = sv->u64;
    return d;
}

// One block up to these rows: its exchanges are __syncthreads, but one SM does all the arithmetic. One block
// against many (us an iteration): FP64 11.7 and 14.5 at 169 rows, 13.6 and 14.1 at 289, 15.0 and 14.1 at 441,
// 17.3 and 14.1 at 529; FP32 13.9 and 17.6 at 289, 16.9 and 17.1 at 1,024, 20.5 and 15.5 at 1,681.
constexpr int64_t kGmOneBlock64 = 512, kGmOneBlock32 = 1024;

void gm_teams_free(GmTeams* t) {
    if (!t) return;
    void* ps[] = {t->state, t->part, t->map, t->qinst, t->queue, t->inst};
    for (void* p : ps) dfree(p);
    delete t;
}

constexpr size_t kGmSmem = 160 * 1024;   // the rest is left to L1, which the gathers live on
constexpr int kGmMaxRestart = 128;
template <class T>
constexpr size_t kGmLargestTables = std::max(GmCfg<T, kGmThreads<T>>::smem(kGmMaxRestart),
                                             GmCfg<T, kGmSmallThreads>::smem(kGmMaxRestart));
static_assert(kGmLargestTables<double> <= kGmSmem && kGmLargestTables<float> <= kGmSmem, "the largest restart's tables");

template <class T>
int gm_smem_limit() {
    int r = smem_limit((const void*)gm_kernel<T, kGmThreads<T>>, kGmSmem);
    if (!r) r = smem_limit(gm_small_kernel<T>(), kGmSmem);
    return r ? r : smem_limit(gm_many_kernel<T>(), kGmSmem);
}

// dynamic shared memory of a launch: the tables and, where there is room, the rows' pointers
template <class T, int NT>
size_t gm_smem(const GmTeams* t, int m, bool pointers, int* slices) {
    const size_t base = GmCfg<T, NT>::smem(m);
    *slices = pointers && base < kGmSmem ? (int)std::min<int64_t>(t->max_slices, (kGmSmem - base) / (33 * 4)) : 0;
    return base + (size_t)*slices * 33 * 4;
}

template <class T>
int gm_launch(GmArgs& a, const GmTeams* t, cudaStream_t st) {
    void* kp[] = {&a};
    if (t->small) {
        const size_t smem = gm_smem<T, kGmSmallThreads>(t, a.m, true, &a.rp_slices);
        OCMP_LAUNCH(OCMP_CUDA(cudaLaunchKernel(gm_small_kernel<T>(), dim3(t->grid), dim3(kGmSmallThreads), kp, smem, st)));
        return OCMP_OK;
    }
    const size_t smem = gm_smem<T, kGmThreads<T>>(t, a.m, a.mode == GM_FULL, &a.rp_slices);
    const void* k = t->nteam ? gm_many_kernel<T>() : (const void*)gm_kernel<T, kGmThreads<T>>;
    OCMP_LAUNCH(OCMP_CUDA(cudaLaunchCooperativeKernel(k, dim3(t->grid), dim3(kGmThreads<T>), kp, smem, st)));
    return OCMP_OK;
}

// A queue of more systems than SMs, each of up to so many rows, is taken by blocks of 128 threads where at
// least so many fit an SM: such a solve is a chain of latencies, and a block per SM ran one at a time (slower
// than a launch per operation over all systems where they are tiny). Whole solves, one block per SM against
// these (ms): 5,000 systems of 81 rows FP64 9.1 -> 4.8, FP32 11.1 -> 3.5 (a launch per operation: 11.4, 9.7);
// 20,000 of 9 rows 7.2 -> 4.5 and 11.2 -> 4.8 (5.5, 6.8); 500 of 1,089 rows 11.1 -> 9.7 and 6.0 -> 4.5; but at
// restart 60 in FP64, where two fit, 1,500 of 1,089 rows 30.1 -> 42.4.
constexpr int64_t kGmSmallRows = 1024;
constexpr int kGmSmallBlocks = 3;

template <class T>
int gm_small_blocks(const GmTeams* t, int m, int* per_sm) {
    int slices = 0;
    const size_t smem = gm_smem<T, kGmSmallThreads>(t, m, true, &slices);
    OCMP_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, gm_small_kernel<T>(), kGmSmallThreads, smem));
    return OCMP_OK;
}

// Shares in proportion leave a large system of a large batch to a block or two, and since the numbers of
// iterations differ the last ones end long after the rest: more than kGmTeamRows rows to a block of any
// system, and teams of as many blocks as the largest needs to get below take the systems one after another
// instead (those of kGmTeamMinRows rows a block and more; the others follow, one per block). 512 systems of
// 289 to 148,225 rows, 91 to 1,815 iterations: 2.36 -> 0.80 s (1.67 with a launch per operation over all).
constexpr int64_t kGmTeamRows = 20480, kGmTeamMinRows = 2048;

int gm_teams_create(const std::vector<GmInst>& inst, const std::vector<int64_t>& nnz, int m, bool fp64, GmTeams** out) {
    int sms = 1;
    if (const int r = team_blocks(&sms)) return r;
    auto* t = new GmTeams();
    const int N = (int)inst.size();
    std::vector<int4> map;
    std::vector<int> qinst, blocks(N, 1);   // blocks: of each system
    t->nteams = 1;
    if (N == 1) {
        const int64_t n = inst[0].n;
        t->grid = n <= (fp64 ? kGmOneBlock64 : kGmOneBlock32)
                      ? 1 : (int)std::min<int64_t>(sms, (n + inst[0].TR - 1) / inst[0].TR);
        t->tile.push_back(!fp64 && n >= kGmVecRows * t->grid ? 128 : 32);
        blocks[0] = t->grid;
    } else {
        t->grid = sms;
        std::vector<double> cost(N);
        double total = 0;
        for (int k = 0; k < N; k++) total += cost[k] = (double)nnz[k] + (double)inst[k].n * m;
        std::vector<int> ord(N);
        for (int k = 0; k < N; k++) ord[k] = k;
        std::stable_sort(ord.begin(), ord.end(), [&](int a, int b) { return cost[a] > cost[b]; });
        t->nteams = 0;
        for (int k = 0; k < N; k++) t->tile.push_back(!fp64 && inst[k].n >= kGmVecRows ? 128 : 32);
        auto team = [&](int k, int s) {
            blocks[k] = s;
            t->tile[k] = !fp64 && inst[k].n >= kGmVecRows * s ? 128 : 32;
        };
        for (int k : ord) {
            const int64_t most = std::max<int64_t>(1, (inst[k].n + 63) / 64);
            const int s = (int)std::min<int64_t>(most, (int64_t)(cost[k] * sms / total));
            if (s < 2 || (int)map.size() + s > sms) {
                qinst.push_back(k);
                continue;
            }
            for (int r = 0; r < s; r++) map.push_back(make_int4(t->nteams, r, s, k));
            team(k, s);
            t->nteams++;
        }
        int64_t rows = 0, crowded = 0;
        for (int k = 0; k < N; k++) {
            rows = std::max(rows, inst[k].n);
            crowded = std::max(crowded, inst[k].n / blocks[k]);
        }
        if (crowded > kGmTeamRows) {
            const int need = (int)std::min<int64_t>(sms, (rows + kGmTeamRows - 1) / kGmTeamRows);
            t->nteams = sms / need;
            const int s = sms / t->nteams;
            map.clear();
            qinst.clear();
            for (int q = 0; q < t->nteams; q++)
                for (int r = 0; r < s; r++) map.push_back(make_int4(q, r, s, -2));
            for (int k : ord) {
                team(k, inst[k].n >= s * kGmTeamMinRows ? s : 1);
                if (blocks[k] == s) qinst.push_back(k);
            }
            t->nteam = (int)qinst.size();
            for (int k : ord)
                if (blocks[k] != s) qinst.push_back(k);
        }
        while ((int)map.size() < sms) map.push_back(make_int4(0, 0, 1, -1));
        t->nqueue = (int)qinst.size() - t->nteam;
        if (qinst.empty()) qinst.push_back(0);
    }
    for (int k = 0; k < N; k++) {
        const int64_t tr = std::max(t->tile[k], inst[k].TR);
        t->max_slices = std::max(t->max_slices, ((inst[k].n + tr - 1) / tr + blocks[k] - 1) / blocks[k] * (tr / 32));
    }
    int st = OCMP_OK;
    int64_t rows = 0;
    for (const GmInst& d : inst) rows = std::max(rows, d.n);
    if (N > sms && t->nteams == 0 && rows <= kGmSmallRows) {
        int per_sm = 0;
        st = fp64 ? gm_small_blocks<double>(t, m, &per_sm) : gm_small_blocks<float>(t, m, &per_sm);
        t->small = per_sm >= kGmSmallBlocks;
        if (t->small) t->grid = std::min(N, sms * per_sm);
    }
    if (!st) st = dalloc(&t->state, (size_t)std::max(1, t->nteams));
    if (!st) st = dalloc(&t->part, (size_t)(m + 2) * t->grid);
    if (!st && N > 1) {
        if (!t->small) st = upload(&t->map, map.data(), map.size());
        if (!st) st = upload(&t->qinst, qinst.data(), qinst.size());
        if (!st) st = dalloc(&t->queue, 2);
        if (!st) st = dalloc(&t->inst, (size_t)N);
    }
    if (!st && cudaMemset(t->state, 0, sizeof(TeamState) * std::max(1, t->nteams)) != cudaSuccess)
        st = fail(OCMP_ERR_CUDA, "cudaMemset");
    if (st) {
        gm_teams_free(t);
        return st;
    }
    *out = t;
    return OCMP_OK;
}

GmArgs gm_args(const GmTeams* t, int m) {
    GmArgs a{};
    a.map = t->map;
    a.queue_inst = t->qinst;
    a.queue = t->queue;
    a.nteam = t->nteam;
    a.nqueue = t->nqueue;
    a.teams = t->state;
    a.part = t->part;
    a.list = t->inst;
    a.m = m;
    return a;
}

// the results, and whether a block gave up waiting
int gm_read(const GmTeams* t, GmResult* out, GmResult* dev, int count, cudaStream_t st) {
    OCMP_CUDA(cudaMemcpyAsync(out, dev, sizeof(GmResult) * count, cudaMemcpyDeviceToHost, st));
    OCMP_CUDA(cudaStreamSynchronize(st));
    for (int q = 0; q < count; q++)
        if (out[q].gaveup) {
            OCMP_CUDA(cudaMemsetAsync(t->state, 0, sizeof(TeamState) * std::max(1, t->nteams), st));
            OCMP_CUDA(cudaMemsetAsync(dev, 0, sizeof(GmResult) * count, st));
            return fail(OCMP_TIMEOUT, "GMRES: a block gave up waiting for the others");
        }
    return OCMP_OK;
}

constexpr int kTimedProducts = 4096;

// product times of the last solve (ocmp_solver_spmv_timing)
int gm_collect_times(ocmp_solver_s* sv, cudaStream_t st) {
    if (!sv->time_spmv) return OCMP_OK;
    std::vector<unsigned long long> t(2 * kTimedProducts);
    OCMP_CUDA(cudaMemcpyAsync(t.data(), sv->tlog, sizeof(unsigned long long) * t.size(), cudaMemcpyDeviceToHost, st));
    OCMP_CUDA(cudaStreamSynchronize(st));
    for (int k = 0; k < kTimedProducts; k++)
        if (t[2 * k + 1]) {   // (a product shorter than the timer's step takes 0)
            sv->spmv_ms += 1e-6 * (double)(t[2 * k + 1] - ~t[2 * k]);
            sv->spmv_launches++;
        }
    return OCMP_OK;
}

// Solves of all B systems of the solver's matrix, one launch.
template <class T>
int gm_full(ocmp_solver_s* sv, const double* b, double* x, cudaStream_t st) {
    GmArgs a = gm_args(sv->teams, sv->m);
    a.mode = GM_FULL;
    std::vector<GmInst> inst;
    if (sv->B == 1) {
        a.one = gm_inst<T>(sv, 0, b, x, sv->teams->tile[0]);
        if (sv->time_spmv) {
            OCMP_CUDA(cudaMemsetAsync(sv->tlog, 0, sizeof(unsigned long long) * 2 * kTimedProducts, st));
            a.tlog = sv->tlog;
            a.tcap = kTimedProducts;
        }
    } else {
        for (int q = 0; q < sv->B; q++) inst.push_back(gm_inst<T>(sv, q, b + q * sv->n, x + q * sv->n,
                                                                      sv->teams->tile[q]));
        OCMP_CUDA(cudaMemcpyAsync(sv->teams->inst, inst.data(), sizeof(GmInst) * inst.size(), cudaMemcpyHostToDevice, st));
        OCMP_CUDA(cudaMemsetAsync(sv->teams->queue, 0, 2 * sizeof(int), st));
    }
    int r = gm_launch<T>(a, sv->teams, st);
    if (!r) r = gm_read(sv->teams, sv->hout, sv->gout, sv->B, st);
    if (!r) r = gm_collect_times(sv, st);
    return r;
}

// A solve whose preconditioner runs in kernels of its own: a launch per phase, the host reading the
// convergence flags every check_every iterations (launches queued past convergence return at once). The
// flags of an iteration are looked at when the next one is queued, so that the GPU does not wait for the
// host between them (10 us of 135 at 148,739 dofs); the one queued in vain returns at once.
template <class T>
int gm_phases(ocmp_solver_s* sv, const double* b, double* x, cudaStream_t st, int* cycles) {
    const int m = sv->m, maxit = sv->prm.maxit;
    GmArgs a = gm_args(sv->teams, m);
    a.one = gm_inst<T>(sv, 0, b, x, sv->teams->tile[0]);
    T* V = (T*)a.one.V;
    T* z = (T*)a.one.z;
    int* flags = sv->gout->flags;
    double* scale = sv->small + m * (m + 1) / 2 + 3 * m + 2;
    const GmResult* H = sv->hout;
    auto read = [&]() {
        const int r = gm_read(sv->teams, sv->hout, sv->gout, 1, st);
        if (r == OCMP_TIMEOUT) strip_reset(sv->strip ? sv->strip : sv->cc->strip, st);
        return r;
    };
    auto launch = [&](int mode, int j) {
        a.mode = mode;
        a.j = j;
        return gm_launch<T>(a, sv->teams, st);
    };
    auto apply = [&](const T* v, const double* sc, int j, const int* fl) {
        return sv->strip ? strip_apply<T>(sv->strip, v, sc, j, z, fl, &sv->gout->gaveup, st)
                         : cc_apply<T>(sv->cc, v, sc, j, z, fl, &sv->gout->gaveup, st);
    };
    if (sv->time_spmv) OCMP_CUDA(cudaMemsetAsync(sv->tlog, 0, sizeof(unsigned long long) * 2 * kTimedProducts, st));
    int r = launch(GM_FIRST, 0);
    if (!r) r = read();
    if (r) return r;
    int it = 0, cyc = 0;
    const bool adaptive = sv->prm.check_every < 0;
    int next_check = std::max(1, sv->last_iters - 1);
    while (!H->flags[F_OUTER] && !H->flags[F_NONFIN] && it < maxit) {
        int pending = -1;   // the slot of a check on its way
        for (int j = 0; j < m; j++) {
            if ((r = apply(V + (int64_t)j * a.one.ld, scale, j, flags))) return r;
            if (sv->time_spmv && it < kTimedProducts) {
                a.tlog = sv->tlog + 2 * it;
                a.tcap = 1;
            } else
                a.tlog = nullptr;
            if ((r = launch(GM_ITER, j))) return r;
            if (++it >= maxit) break;
            // fixed interval, or (check_every < 0) the first check one iteration before the
            // previous solve's count and then after every iteration
            const bool check = adaptive ? it >= next_check : ((j + 1) % std::max(1, sv->prm.check_every)) == 0;
            const int before = pending;
            pending = -1;
            if (check) {
                pending = it & 1;
                next_check = it + 1;
                OCMP_CUDA(cudaMemcpyAsync(&sv->hout[1 + pending], sv->gout, sizeof(GmResult), cudaMemcpyDeviceToHost, st));
                OCMP_CUDA(cudaEventRecord(sv->ev_check[pending], st));
            }
            if (before >= 0) {
                OCMP_CUDA(cudaEventSynchronize(sv->ev_check[before]));
                const GmResult& R = sv->hout[1 + before];
                if (R.gaveup) break;   // found again, and cleared, by the read below
                if (R.flags[F_CONV]) {
                    it--;
                    break;
                }
            }
        }
        a.tlog = nullptr;
        if ((r = launch(GM_COMBINE, 0))) return r;
        if ((r = apply(z, nullptr, 0, nullptr))) return r;
        if ((r = strip_add<T>(sv->n, z, x, st))) return r;
        if ((r = launch(GM_START, 0))) return r;
        cyc++;
        if ((r = read())) return r;
    }
    sv->last_iters = H->flags[F_ITERS];
    *cycles = cyc;
    return gm_collect_times(sv, st);
}

// the status of a finished solve
int gm_status(const GmResult& r, double tol) {
    if ((r.bits & GM_NONFIN) || !std::isfinite(r.res) || !std::isfinite(r.res0)) return OCMP_ERR_NONFINITE;
    if (r.res > tol) return r.bits & GM_BREAK ? OCMP_BREAKDOWN : OCMP_NOT_CONVERGED;
    return OCMP_OK;
}

}  // namespace
}  // namespace ocmp

using namespace ocmp;

static void free_solver(ocmp_solver_s* sv) {
    void* ps[] = {sv->udiag, sv->dinv, sv->Binv, sv->V,   sv->w,    sv->z,    sv->r,    sv->p,    sv->dinv32, sv->Binv32,
                  sv->V32,   sv->w32,  sv->z32,  sv->r32, sv->p32,  sv->d32,  sv->pb,   sv->p32b, sv->dcg,    sv->small,
                  sv->gout,  sv->As64, sv->As32, sv->tlog};
    for (void* q : ps) dfree(q);
    gm_teams_free(sv->teams);
    if (sv->strip) strip_destroy(sv->strip);
    if (sv->cc) {
        if (sv->cc->strip) strip_destroy(sv->cc->strip);
        dfree(sv->cc->vdinv);
        dfree(sv->cc->mpinv);
        dfree(sv->cc->zp64);
        dfree(sv->cc->zp32);
        delete sv->cc;
    }
    if (sv->hout) cudaFreeHost(sv->hout);
    for (cudaEvent_t e : sv->ev_check)
        if (e) cudaEventDestroy(e);
    if (sv->hcg) cudaFreeHost(sv->hcg);
}

extern "C" {

int ocmp_solver_create(ocmp_matrix_t mat, const ocmp_solve_params_t* prm, ocmp_solver_t* out) {
    if (!mat || !prm || !out) return fail(OCMP_ERR_ARG, "ocmp_solver_create: null argument");
    if (prm->method != OCMP_CG && prm->method != OCMP_GMRES) return fail(OCMP_ERR_ARG, "ocmp_solver_create: method");
    if (prm->precond < OCMP_PRE_NONE || prm->precond > OCMP_PRE_CAHOUET_CHABARD)
        return fail(OCMP_ERR_ARG, "ocmp_solver_create: precond");
    if (prm->precision == OCMP_MIXED && prm->method == OCMP_CG && !mat->vals32)
        return fail(OCMP_ERR_ARG, "ocmp_solver_create: mixed-precision CG needs a matrix created with OCMP_MAT_FP32");
    if (prm->method == OCMP_CG && prm->precond != OCMP_PRE_JACOBI && prm->precond != OCMP_PRE_USER)
        return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solver_create: CG is built with a diagonal preconditioner");
    ocmp_space_s* s = mat->space;
    if (prm->precond == OCMP_PRE_BLOCK_JACOBI && (s->kind != OCMP_L2 || (s->nloc != 3 && s->nloc != 6 && s->nloc != 10)))
        return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solver_create: block Jacobi is built for L2 element blocks");
    if ((prm->precond == OCMP_PRE_STRIP || prm->precond == OCMP_PRE_CAHOUET_CHABARD) &&
        (prm->method != OCMP_GMRES || mat->B != 1))
        return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solver_create: the strip and Cahouet-Chabard preconditioners are built "
                                          "for GMRES on one matrix");
    auto* sv = new ocmp_solver_s();
    sv->mat = mat;
    sv->s = s;
    sv->prm = *prm;
    if (sv->prm.check_every == 0) sv->prm.check_every = 8;
    // a strip-preconditioned iteration costs two full sweeps: read the flags after every one
    if (prm->precond == OCMP_PRE_STRIP) sv->prm.check_every = 1;
    const int64_t n = sv->n = s->ndof;
    const int NB = sv->B = mat->B;
    if (NB > 1 && (prm->method != OCMP_GMRES || prm->precond == OCMP_PRE_BLOCK_JACOBI)) {
        delete sv;
        return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solver_create: batches are solved with GMRES + point Jacobi");
    }
    sv->m = std::max(1, std::min(kGmMaxRestart, prm->restart > 0 ? prm->restart : 30));
    const int m = sv->m;
    const bool gm = prm->method == OCMP_GMRES, mixed = prm->precision == OCMP_MIXED;
    const bool blk = prm->precond == OCMP_PRE_BLOCK_JACOBI;
    int st = gm ? (mixed ? gm_smem_limit<float>() : gm_smem_limit<double>())
                : (mixed ? cg_smem_limit<float>() : cg_smem_limit<double>());
    auto A = [&](auto** p, size_t cnt) {
        if (!st) st = dalloc(p, cnt);
    };
    A(&sv->dinv, (size_t)n * NB);
    if (prm->precond == OCMP_PRE_USER) A(&sv->udiag, (size_t)n * NB);
    A(&sv->z, n);
    if (!gm) {
        A(&sv->w, n);
        A(&sv->r, n);
    }
    if (!mixed) {
        if (gm) A(&sv->V, (size_t)(m + 1) * gm_ld<double>(n) * NB);
        else {
            A(&sv->p, n);
            A(&sv->pb, n);
        }
    }
    if (blk) A(&sv->Binv, (size_t)s->mesh->ne * s->nloc * s->nloc);
    if (prm->precond == OCMP_PRE_STRIP || prm->precond == OCMP_PRE_CAHOUET_CHABARD)
        for (cudaEvent_t& e : sv->ev_check)
            if (!st && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess)
                st = fail(OCMP_ERR_CUDA, "ocmp_solver_create: event");
    if (!st && prm->precond == OCMP_PRE_STRIP) st = strip_create(s, &sv->strip);
    if (mixed) {
        A(&sv->dinv32, (size_t)n * NB);
        A(&sv->z32, n);
        if (gm) A(&sv->V32, (size_t)(m + 1) * gm_ld<float>(n) * NB);
        else {
            A(&sv->w32, n);
            A(&sv->d32, n);
            A(&sv->r32, n);
            A(&sv->p32, n);
            A(&sv->p32b, n);
        }
        if (blk) A(&sv->Binv32, (size_t)s->mesh->ne * s->nloc * s->nloc);
    }
    if (!gm) {
        A(&sv->dcg, 1);
        if (!st && cudaMemset(sv->dcg, 0, sizeof(CgState)) != cudaSuccess) st = fail(OCMP_ERR_CUDA, "cudaMemset");
        if (!st && cudaMallocHost((void**)&sv->hcg, kCgReadBytes) != cudaSuccess)
            st = fail(OCMP_ERR_NOMEM, "cudaMallocHost");
    }
    if (gm) {
        A(&sv->small, (size_t)gm_small_doubles(m) * NB);
        A(&sv->gout, (size_t)NB);
        // the basis is read past n (its stride is padded)
        if (!st && cudaMemset(mixed ? (void*)sv->V32 : (void*)sv->V, 0,
                              (mixed ? sizeof(float) * gm_ld<float>(n) : sizeof(double) * gm_ld<double>(n)) *
                                  (size_t)(m + 1) * NB) != cudaSuccess)
            st = fail(OCMP_ERR_CUDA, "cudaMemset");
        if (!st && cudaMemset(sv->gout, 0, sizeof(GmResult) * NB) != cudaSuccess) st = fail(OCMP_ERR_CUDA, "cudaMemset");
        if (!st && cudaMallocHost((void**)&sv->hout, sizeof(GmResult) * (NB + 2)) != cudaSuccess)
            st = fail(OCMP_ERR_NOMEM, "cudaMallocHost");
    }
    sv->borrow = gm && prm->precond == OCMP_PRE_JACOBI && mat->dinv &&
                 (mixed ? mat->svals32 != nullptr : mat->svals64 != nullptr);
    if (gm && !sv->borrow) {
        if (mixed) A(&sv->As32, (size_t)s->nnz * NB);
        else A(&sv->As64, (size_t)s->nnz * NB);
    }
    sv->K64 = sv->borrow ? mat->svals64 : sv->As64;
    sv->K32 = sv->borrow ? mat->svals32 : sv->As32;
    sv->sell = sv->borrow && mixed && (mat->flags & OCMP_MAT_SELL32) && s->d_sell_off != nullptr;
    if (gm && !mixed) sv->u64 = gm_unroll(s);
    if (gm && !st) {
        std::vector<GmInst> inst;
        for (int q = 0; q < NB; q++) inst.push_back(mixed ? gm_inst<float>(sv, q, nullptr, nullptr, 32)
                                                          : gm_inst<double>(sv, q, nullptr, nullptr, 32));
        st = gm_teams_create(inst, std::vector<int64_t>(NB, s->nnz), m, !mixed, &sv->teams);
    }
    if (st) {
        free_solver(sv);
        delete sv;
        return st;
    }
    // USER: after ocmp_solver_set_diag; STRIP: after the matrix is assembled (OpenCMP builds its
    // preconditioners before the first assembly and updates them after every one)
    if (prm->precond != OCMP_PRE_USER && prm->precond != OCMP_PRE_STRIP) st = ocmp_solver_update(sv, nullptr);
    if (st) {
        free_solver(sv);
        delete sv;
        return st;
    }
    OCMP_CUDA(cudaDeviceSynchronize());
    *out = sv;
    return OCMP_OK;
}

int ocmp_solver_destroy(ocmp_solver_t sv) {
    if (!sv) return OCMP_OK;
    free_solver(sv);
    delete sv;
    return OCMP_OK;
}

int ocmp_solver_update(ocmp_solver_t sv, void* stream) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_solver_update: null solver");
    cudaStream_t st = (cudaStream_t)stream;
    ocmp_space_s* s = sv->s;
    const int64_t n = sv->n;
    const int NB = sv->B;
    if (sv->prm.precond == OCMP_PRE_USER) {
        if (!sv->udiag_set) return fail(OCMP_ERR_ARG, "ocmp_solver_update: set the diagonal with ocmp_solver_set_diag");
        OCMP_CUDA(cudaMemcpyAsync(sv->dinv, sv->udiag, sizeof(double) * n * NB, cudaMemcpyDeviceToDevice, st));
        if (sv->dinv32) OCMP_LAUNCH(gm_cast<<<nblk(n * NB, kThreads), kThreads, 0, st>>>(n * NB, sv->dinv, sv->dinv32));
    } else if (sv->borrow) {
        // the assembly's D^-1 scaled the Krylov matrix: use the same one for x = D^-1 y
        OCMP_CUDA(cudaMemcpyAsync(sv->dinv, sv->mat->dinv, sizeof(double) * n * NB, cudaMemcpyDeviceToDevice, st));
        if (sv->dinv32) OCMP_LAUNCH(gm_cast<<<nblk(n * NB, kThreads), kThreads, 0, st>>>(n * NB, sv->mat->dinv, sv->dinv32));
    } else {
        for (int q = 0; q < NB; q++) {
            OCMP_LAUNCH(jacobi_setup<double><<<nblk(n, kThreads), kThreads, 0, st>>>(n, s->d_diag, sv->mat->vals + q * s->nnz,
                                                                        s->d_free, sv->dinv + q * n));
            if (sv->dinv32)
                OCMP_LAUNCH(jacobi_setup<float><<<nblk(n, kThreads), kThreads, 0, st>>>(n, s->d_diag, sv->mat->vals + q * s->nnz,
                                                                           s->d_free, sv->dinv32 + q * n));
        }
    }
    if (sv->Binv) {
        const int64_t ne = s->mesh->ne;
        switch (s->nloc) {
        case 3: OCMP_LAUNCH(block_jacobi_setup<3><<<nblk(ne, 128), 128, 0, st>>>(ne, s->d_rowptr, s->d_col, sv->mat->vals, sv->Binv, sv->Binv32)); break;
        case 6: OCMP_LAUNCH(block_jacobi_setup<6><<<nblk(ne, 128), 128, 0, st>>>(ne, s->d_rowptr, s->d_col, sv->mat->vals, sv->Binv, sv->Binv32)); break;
        case 10: OCMP_LAUNCH(block_jacobi_setup<10><<<nblk(ne, 128), 128, 0, st>>>(ne, s->d_rowptr, s->d_col, sv->mat->vals, sv->Binv, sv->Binv32)); break;
        default: break;
        }
    }
    if (sv->strip) {
        sv->strip_ready = false;
        const int r = strip_factor(sv->strip, s, sv->mat->vals, st);
        if (r) return r;
        sv->strip_ready = true;
    }
    if (sv->As64 || sv->As32) {
        const double* d = sv->prm.precond == OCMP_PRE_JACOBI || sv->prm.precond == OCMP_PRE_USER ? sv->dinv : nullptr;
        const dim3 g(nblk(n, kThreads), NB);
        if (sv->As64)
            OCMP_LAUNCH(gm_scale_matrix<double><<<g, kThreads, 0, st>>>(n, s->d_rowptr, s->d_col, sv->mat->vals, d, sv->As64, s->nnz));
        if (sv->As32)
            OCMP_LAUNCH(gm_scale_matrix<float><<<g, kThreads, 0, st>>>(n, s->d_rowptr, s->d_col, sv->mat->vals, d, sv->As32, s->nnz));
    }
    OCMP_CUDA(cudaGetLastError());
    return OCMP_OK;
}

int ocmp_solver_set_diag(ocmp_solver_t sv, const double* dinv, void* stream) {
    if (!sv || !dinv) return fail(OCMP_ERR_ARG, "ocmp_solver_set_diag: null argument");
    if (sv->prm.precond != OCMP_PRE_USER) return fail(OCMP_ERR_ARG, "ocmp_solver_set_diag: solver not created with OCMP_PRE_USER");
    OCMP_CUDA(cudaMemcpyAsync(sv->udiag, dinv, sizeof(double) * sv->n * sv->B, cudaMemcpyDeviceToDevice,
                              (cudaStream_t)stream));
    sv->udiag_set = true;
    return OCMP_OK;
}

int ocmp_solver_spmv_timing(ocmp_solver_t sv, int32_t on) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_solver_spmv_timing: null solver");
    sv->time_spmv = on != 0;
    sv->spmv_launches = 0;
    sv->spmv_ms = 0;
    if (on && !sv->tlog) return dalloc(&sv->tlog, 2 * kTimedProducts);
    return OCMP_OK;
}

int ocmp_solver_spmv_stats(ocmp_solver_t sv, int64_t* launches, double* total_ms) {
    if (!sv || !launches || !total_ms) return fail(OCMP_ERR_ARG, "ocmp_solver_spmv_stats: null argument");
    *launches = sv->spmv_launches;
    *total_ms = sv->spmv_ms;
    return OCMP_OK;
}

int ocmp_solver_set_graph(ocmp_solver_t sv, int32_t on) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_solver_set_graph: null solver");
    if (on && sv->prm.method != OCMP_GMRES)
        return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solver_set_graph: graphs are built for GMRES");
    if (on && (sv->strip || sv->prm.precond == OCMP_PRE_CAHOUET_CHABARD))
        return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solver_set_graph: the strip preconditioners run without graphs");
    return OCMP_OK;
}

int ocmp_solver_set_cahouet_chabard(ocmp_solver_t sv, ocmp_matrix_t pop, const double* vdinv, const double* mpinv,
                                    int64_t nu, double alpha, double beta, double tc, int32_t refactor,
                                    void* stream) {
    if (!sv || !pop || !vdinv || !mpinv) return fail(OCMP_ERR_ARG, "ocmp_solver_set_cahouet_chabard: null argument");
    if (sv->prm.precond != OCMP_PRE_CAHOUET_CHABARD)
        return fail(OCMP_ERR_ARG, "ocmp_solver_set_cahouet_chabard: solver not created with OCMP_PRE_CAHOUET_CHABARD");
    const int64_t np = pop->space->ndof;
    if (nu < 0 || nu + np != sv->n || pop->B != 1)
        return fail(OCMP_ERR_ARG, "ocmp_solver_set_cahouet_chabard: velocity + pressure dofs must make the system");
    if (!(tc != 0.0)) return fail(OCMP_ERR_ARG, "ocmp_solver_set_cahouet_chabard: tc must not be zero");
    cudaStream_t st = (cudaStream_t)stream;
    CCPre* cc = sv->cc;
    if (cc && cc->pop != pop) {
        if (cc->strip) strip_destroy(cc->strip);
        cc->strip = nullptr;
        cc->pop = pop;
        refactor = 1;
    }
    if (!cc) {
        cc = new CCPre();
        cc->pop = pop;
        cc->np = np;
        int r = dalloc(&cc->vdinv, (size_t)std::max<int64_t>(nu, 1));
        if (!r) r = dalloc(&cc->mpinv, (size_t)np);
        if (!r) r = dalloc(&cc->zp64, (size_t)np);
        if (!r) r = dalloc(&cc->zp32, (size_t)np);
        if (r) {
            dfree(cc->vdinv);
            dfree(cc->mpinv);
            dfree(cc->zp64);
            delete cc;
            return r;
        }
        sv->cc = cc;
        refactor = 1;
    }
    cc->nu = nu;
    cc->np = np;
    cc->alpha = alpha;
    cc->beta = beta;
    cc->tc = tc;
    if (nu) OCMP_CUDA(cudaMemcpyAsync(cc->vdinv, vdinv, sizeof(double) * nu, cudaMemcpyDeviceToDevice, st));
    OCMP_CUDA(cudaMemcpyAsync(cc->mpinv, mpinv, sizeof(double) * np, cudaMemcpyDeviceToDevice, st));
    if (!cc->strip) {
        const int r = strip_create(pop->space, &cc->strip);
        if (r) return r;
    }
    if (refactor) {
        const int r = strip_factor(cc->strip, pop->space, pop->vals, st);
        if (r) return r;
    }
    return OCMP_OK;
}

int ocmp_solver_strip_stats(ocmp_solver_t sv, ocmp_strip_stats_t* out) {
    if (!sv || !out) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_stats: null argument");
    if (!sv->strip) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_stats: solver not created with OCMP_PRE_STRIP");
    strip_stats(sv->strip, out);
    return OCMP_OK;
}

int ocmp_solver_strip_timing(ocmp_solver_t sv, int32_t on) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_timing: null solver");
    if (!sv->strip) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_timing: solver not created with OCMP_PRE_STRIP");
    strip_set_timing(sv->strip, on != 0);
    return OCMP_OK;
}

int ocmp_solver_strip_gemm(ocmp_solver_t sv, int32_t kind) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_gemm: null solver");
    if (!sv->strip) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_gemm: solver not created with OCMP_PRE_STRIP");
    if (kind != 0 && kind != 1) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_gemm: kind is 0 (SIMT) or 1 (tensor cores)");
    strip_set_gemm(sv->strip, kind);
    return OCMP_OK;
}

int ocmp_solver_strip_schulz(ocmp_solver_t sv, int32_t on) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_schulz: null solver");
    if (!sv->strip) return fail(OCMP_ERR_ARG, "ocmp_solver_strip_schulz: solver not created with OCMP_PRE_STRIP");
    strip_set_schulz(sv->strip, on != 0);
    return OCMP_OK;
}

// A test's entry, not part of the interface: in the next solve a wait of one block for another (which 0),
// or of the strip's sweeps (1), runs out.
int ocmp_test_starve(ocmp_solver_t sv, int32_t which) {
    if (!sv) return fail(OCMP_ERR_ARG, "ocmp_test_starve: null solver");
    if (which == 1) {
        Strip* p = sv->strip ? sv->strip : sv->cc ? sv->cc->strip : nullptr;
        return p ? strip_starve(p) : fail(OCMP_ERR_ARG, "ocmp_test_starve: no strip");
    }
    const int on = 1;
    TeamState* t = sv->dcg ? &sv->dcg->t : sv->teams->state;
    for (int k = 0; k < (sv->dcg ? 1 : std::max(1, sv->teams->nteams)); k++)
        OCMP_CUDA(cudaMemcpy(&t[k].starve, &on, sizeof(int), cudaMemcpyHostToDevice));
    return OCMP_OK;
}

// Batched GMRES solve of all B systems of the solver's matrix: b and x hold B vectors of ndof.
int ocmp_solve_batch(ocmp_solver_t sv, const double* b, double* x, void* stream, ocmp_solve_info_t* infos) {
    if (!sv || !b || !x) return fail(OCMP_ERR_ARG, "ocmp_solve_batch: null argument");
    if (sv->prm.method != OCMP_GMRES) return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solve_batch: GMRES only");
    const int NB = sv->B;
    const ocmp_solve_params_t& P = sv->prm;
    const int st = P.precision == OCMP_MIXED ? gm_full<float>(sv, b, x, (cudaStream_t)stream)
                                             : gm_full<double>(sv, b, x, (cudaStream_t)stream);
    if (st) return st;
    int worst = OCMP_OK;
    for (int q = 0; q < NB; q++) {
        const GmResult& R = sv->hout[q];
        const int status = gm_status(R, P.tol);
        if (infos) {
            infos[q].status = status;
            infos[q].iterations = R.iters;
            infos[q].outer_iterations = R.cycles;
            infos[q].relres0 = R.res0;
            infos[q].relres = R.res;
        }
        if (status != OCMP_OK && worst == OCMP_OK) worst = status;
    }
    if (worst != OCMP_OK) set_error("ocmp_solve_batch: at least one system did not reach the tolerance");
    return worst;
}

int ocmp_solve(ocmp_solver_t sv, const double* b, double* x, void* stream, ocmp_solve_info_t* info) {
    if (!sv || !b || !x) return fail(OCMP_ERR_ARG, "ocmp_solve: null argument");
    cudaStream_t cst = (cudaStream_t)stream;
    const int64_t n = sv->n;
    const ocmp_solve_params_t& P = sv->prm;
    const bool gm = P.method == OCMP_GMRES, mixed = P.precision == OCMP_MIXED;
    int st = OCMP_OK;
    int iters = 0, outer = 0;
    bool nonfin = false, brk = false;
    double relres0 = 0, relres = 0;
    if (gm) {
        if (sv->B != 1) return fail(OCMP_ERR_ARG, "ocmp_solve: batched matrix, use ocmp_solve_batch");
        if (sv->strip && !sv->strip_ready)
            return fail(OCMP_ERR_ARG, "ocmp_solve: the strip preconditioner is not factorised (call ocmp_solver_update "
                                      "after assembling the matrix)");
        if (P.precond == OCMP_PRE_CAHOUET_CHABARD && !sv->cc)
            return fail(OCMP_ERR_ARG, "ocmp_solve: set the Cahouet-Chabard data (ocmp_solver_set_cahouet_chabard)");
        const GmResult& R = *sv->hout;
        if (sv->strip || sv->cc) {
            st = mixed ? gm_phases<float>(sv, b, x, cst, &outer) : gm_phases<double>(sv, b, x, cst, &outer);
            if (st) return st;
            iters = R.flags[F_ITERS];
            nonfin = R.flags[F_NONFIN] != 0;
            brk = R.flags[F_BREAK] != 0;
        } else {
            st = mixed ? gm_full<float>(sv, b, x, cst) : gm_full<double>(sv, b, x, cst);
            if (st) return st;
            iters = R.iters;
            outer = R.cycles;
            nonfin = (R.bits & GM_NONFIN) != 0;
            brk = (R.bits & GM_BREAK) != 0;
        }
        relres0 = R.res0;
        relres = R.res;
        nonfin = nonfin || !std::isfinite(relres0);
    } else {
        if (mixed) {
            CgArgs<float> a{n, sv->s->d_rowptr, sv->s->d_col, sv->mat->vals, sv->mat->vals32, sv->s->d_free, sv->s->d_lift_ptr,
                            sv->s->d_lift_pos, sv->dinv32, b, x, sv->r, sv->r32, sv->z32, sv->p32, sv->p32b, sv->w32, sv->d32,
                            sv->dcg, P.tol, P.inner_tol > 0 ? P.inner_tol : 1e-4, kTargetMargin, P.maxit, 0};
            st = cg_solve(a, sv->s, true, cst, sv->hcg);
        } else {
            CgArgs<double> a{n, sv->s->d_rowptr, sv->s->d_col, sv->mat->vals, sv->mat->vals, sv->s->d_free, sv->s->d_lift_ptr,
                             sv->s->d_lift_pos, sv->dinv, b, x, sv->r, sv->r, sv->z, sv->p, sv->pb, sv->w, nullptr,
                             sv->dcg, P.tol, 0.0, kTargetMargin, P.maxit, 0};
            st = cg_solve(a, sv->s, true, cst, sv->hcg);
        }
        if (st) return st;
        const CgResult& R = sv->hcg->r;
        relres0 = R.res0;
        relres = R.res;
        iters = R.iters;
        outer = R.outer;
        nonfin = (R.bits & CG_NONFIN) != 0;
        brk = (R.bits & CG_BREAK) != 0;
    }
    int status = OCMP_OK;
    if (nonfin || !std::isfinite(relres)) status = OCMP_ERR_NONFINITE;
    else if (relres > P.tol) status = brk ? OCMP_BREAKDOWN : OCMP_NOT_CONVERGED;
    if (info) {
        info->status = status;
        info->iterations = iters;
        info->outer_iterations = outer;
        info->relres0 = relres0;
        info->relres = relres;
    }
    if (status == OCMP_ERR_NONFINITE) set_error("ocmp_solve: non-finite value in the right-hand side or iteration");
    else if (status == OCMP_NOT_CONVERGED) set_error("ocmp_solve: iteration cap reached before the tolerance");
    else if (status == OCMP_BREAKDOWN) set_error("ocmp_solve: Krylov breakdown");
    return status;
}


int ocmp_group_create(const ocmp_solver_t* solvers, int32_t count, ocmp_group_t* out) {
    if (!solvers || count <= 0 || !out) return fail(OCMP_ERR_ARG, "ocmp_group_create: no solvers");
    *out = nullptr;
    auto* g = new ocmp_group_s();
    std::vector<int64_t> nnz;
    for (int i = 0; i < count; i++) {
        ocmp_solver_s* sv = solvers[i];
        const ocmp_solve_params_t& P = sv ? sv->prm : ocmp_solve_params_t{};
        const char* why = nullptr;
        if (!sv) why = "null solver";
        else if (P.method != OCMP_GMRES) why = "members must be GMRES solvers";
        else if (P.precond != OCMP_PRE_JACOBI && P.precond != OCMP_PRE_USER && P.precond != OCMP_PRE_NONE)
            why = "members must use point Jacobi (or no) preconditioning";
        else if (sv->sell) why = "members' FP32 Krylov matrices must be in CSR order (no OCMP_MAT_SELL32)";
        else if (i > 0 && (sv->m != g->m || (P.precision == OCMP_MIXED) != g->mixed || P.maxit != g->maxit))
            why = "members must share the restart, the precision and the iteration cap";
        if (why) {
            delete g;
            return fail(OCMP_ERR_UNSUPPORTED, std::string("ocmp_group_create: ") + why);
        }
        if (i == 0) {
            g->m = sv->m;
            g->mixed = P.precision == OCMP_MIXED;
            g->maxit = P.maxit;
        }
        g->members.push_back(sv);
        g->first.push_back(g->ninst);
        for (int q = 0; q < sv->B; q++) {
            g->h_inst.push_back(g->mixed ? gm_inst<float>(sv, q, nullptr, nullptr, 32) : gm_inst<double>(sv, q, nullptr, nullptr, 32));
            nnz.push_back(sv->s->nnz);
            g->ninst++;
        }
    }
    int st = gm_teams_create(g->h_inst, nnz, g->m, !g->mixed, &g->teams);
    if (!st) st = dalloc(&g->gout, (size_t)g->ninst);
    if (!st && cudaMemset(g->gout, 0, sizeof(GmResult) * g->ninst) != cudaSuccess) st = fail(OCMP_ERR_CUDA, "cudaMemset");
    if (!st && cudaMallocHost((void**)&g->hout, sizeof(GmResult) * g->ninst) != cudaSuccess)
        st = fail(OCMP_ERR_NOMEM, "ocmp_group_create: pinned results");
    if (st) {
        ocmp_group_destroy(g);
        return st;
    }
    *out = g;
    return OCMP_OK;
}

int ocmp_group_destroy(ocmp_group_t g) {
    if (!g) return OCMP_OK;
    gm_teams_free(g->teams);
    dfree(g->gout);
    if (g->hout) cudaFreeHost(g->hout);
    delete g;
    return OCMP_OK;
}

int ocmp_group_solve(ocmp_group_t g, const double* const* b, double* const* x, void* stream, ocmp_solve_info_t* infos) {
    if (!g || !b || !x) return fail(OCMP_ERR_ARG, "ocmp_group_solve: null argument");
    cudaStream_t st = (cudaStream_t)stream;
    for (size_t i = 0; i < g->members.size(); i++) {
        ocmp_solver_s* sv = g->members[i];
        if (!b[i] || !x[i]) return fail(OCMP_ERR_ARG, "ocmp_group_solve: null right-hand side or solution");
        for (int q = 0; q < sv->B; q++) {
            GmInst& d = g->h_inst[g->first[i] + q];
            const int tile = g->teams->tile[g->first[i] + q];
            d = g->mixed ? gm_inst<float>(sv, q, b[i] + q * sv->n, x[i] + q * sv->n, tile)
                         : gm_inst<double>(sv, q, b[i] + q * sv->n, x[i] + q * sv->n, tile);
            d.out = g->gout + g->first[i] + q;
        }
    }
    GmArgs a = gm_args(g->teams, g->m);
    a.mode = GM_FULL;
    if (g->ninst == 1) a.one = g->h_inst[0];
    else {
        OCMP_CUDA(cudaMemcpyAsync(g->teams->inst, g->h_inst.data(), sizeof(GmInst) * g->ninst, cudaMemcpyHostToDevice, st));
        OCMP_CUDA(cudaMemsetAsync(g->teams->queue, 0, 2 * sizeof(int), st));
    }
    int r = g->mixed ? gm_launch<float>(a, g->teams, st) : gm_launch<double>(a, g->teams, st);
    if (!r) r = gm_read(g->teams, g->hout, g->gout, g->ninst, st);
    if (r) return r;
    int worst = OCMP_OK;
    for (size_t i = 0; i < g->members.size(); i++)
        for (int q = 0; q < g->members[i]->B; q++) {
            const int k = g->first[i] + q;
            const GmResult& R = g->hout[k];
            const int status = gm_status(R, g->members[i]->prm.tol);
            if (infos) {
                infos[k].status = status;
                infos[k].iterations = R.iters;
                infos[k].outer_iterations = R.cycles;
                infos[k].relres0 = R.res0;
                infos[k].relres = R.res;
            }
            if (status != OCMP_OK && worst == OCMP_OK) worst = status;
        }
    if (worst != OCMP_OK) set_error("ocmp_group_solve: at least one system did not reach the tolerance");
    return worst;
}

}  // extern "C"

// ---------------------------------------------------------------------------------------------
// Allocation-free CG. Some callers cannot call cudaMalloc at the moment they need a solve: hosts
// whose device memory belongs to another allocator's fixed pool (cudaMalloc would take memory that
// pool has already claimed, or fail), and loops that cannot take the implicit device-wide
// synchronisation of cudaFree. ocmp_solve_cg_noalloc serves them: it runs the
// same FP64 Jacobi-preconditioned CG as ocmp_solve with method OCMP_CG, but its workspace (the
// vectors, the blocks' exchange slots and the results) lives in the file-scope device array below,
// which the CUDA driver allocates once per device when this library is loaded and keeps until exit.
// The caller passes only the assembled matrix, the right-hand side and the initial guess/result.
namespace {

constexpr int64_t kNoAllocMaxN = OCMP_NOALLOC_MAX_NDOF;      // 1,048,576 dofs
constexpr int64_t kNoAllocState = int64_t(1) << 17;          // exchange slots and results (1 MiB)
constexpr int64_t kNoAllocDoubles = 5 * kNoAllocMaxN + kNoAllocState;  // 41 MiB

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocDoubles];

std::mutex g_noalloc_mu;
double* g_noalloc_ptr[128] = {};

// Device address of the scratch array for the current device. Host code must not use the array's
// name as a pointer (it names a host-side shadow); cudaGetSymbolAddress gives the device address.
// Done once per device, under a lock, with that device current.
int noalloc_scratch(double** scratch) {
    int dev = 0;
    OCMP_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 128) return fail(OCMP_ERR_ARG, "ocmp_solve_cg_noalloc: device index out of range");
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    if (!g_noalloc_ptr[dev]) {
        double* p = nullptr;
        cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_scratch);
        if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
        g_noalloc_ptr[dev] = p;
    }
    *scratch = g_noalloc_ptr[dev];
    return OCMP_OK;
}

}  // namespace

extern "C" int ocmp_solve_cg_noalloc(ocmp_matrix_t mat, const double* b, double* x, double tol, int32_t maxit,
                                     void* stream, ocmp_solve_info_t* info) {
    if (!mat || !b || !x) return fail(OCMP_ERR_ARG, "ocmp_solve_cg_noalloc: null argument");
    if (mat->B != 1) return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solve_cg_noalloc: batched matrices are not supported");
    {
        // the solve waits for its result on the host (device-to-host copy, stream synchronisation); on a
        // stream under capture those calls would invalidate the caller's capture
        cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
        OCMP_CUDA(cudaStreamIsCapturing((cudaStream_t)stream, &cs));
        if (cs != cudaStreamCaptureStatusNone)
            return fail(OCMP_ERR_UNSUPPORTED, "ocmp_solve_cg_noalloc: the stream is being captured; the solve "
                                              "synchronises with the host and cannot run under capture");
    }
    ocmp_space_s* s = mat->space;
    const int64_t n = s->ndof;
    if (n > kNoAllocMaxN)
        return fail(OCMP_ERR_ARG, "ocmp_solve_cg_noalloc: " + std::to_string(n) + " dofs exceed the " +
                                      std::to_string(kNoAllocMaxN) + "-dof limit of its static workspace");
    double* scr = nullptr;
    int st = noalloc_scratch(&scr);
    if (!st) st = cg_smem_limit<double>();
    if (st) return st;
    // the second search direction fits beside the other five vectors in every system of the resident form
    cudaStream_t cst = (cudaStream_t)stream;
    double *dinv = scr, *r = scr + n, *z = scr + 2 * n, *p = scr + 3 * n, *w = scr + 4 * n, *pb = scr + 5 * n;
    const bool two = 6 * n <= 5 * kNoAllocMaxN;
    // results and exchange slots follow the vectors; the workspace keeps the previous call's contents
    auto* state = reinterpret_cast<CgState*>(scr + 5 * kNoAllocMaxN);
    static_assert(sizeof(CgState) <= kNoAllocState * sizeof(double), "state of the CG");
    OCMP_CUDA(cudaMemsetAsync(state, 0, sizeof(CgState), cst));
    OCMP_LAUNCH(jacobi_setup<double><<<nblk(n, kThreads), kThreads, 0, cst>>>(n, s->d_diag, mat->vals, s->d_free, dinv));
    OCMP_CUDA(cudaGetLastError());
    CgArgs<double> a{n, s->d_rowptr, s->d_col, mat->vals, mat->vals, s->d_free, s->d_lift_ptr, s->d_lift_pos, dinv, b, x,
                     r, r, z, p, two ? pb : p, w, nullptr, state, tol, 0.0, kTargetMargin, maxit, 0};
    CgState H;
    st = cg_solve(a, s, two, cst, &H);
    if (st) return st;
    const CgResult& R = H.r;
    const double relres0 = R.res0, relres = R.res;
    const int iters = R.iters;
    const bool nonfin = (R.bits & CG_NONFIN) != 0, brk = (R.bits & CG_BREAK) != 0;
    int status = OCMP_OK;
    if (nonfin || !std::isfinite(relres)) status = OCMP_ERR_NONFINITE;
    else if (relres > tol) status = brk ? OCMP_BREAKDOWN : OCMP_NOT_CONVERGED;
    if (info) {
        info->status = status;
        info->iterations = iters;
        info->outer_iterations = 0;
        info->relres0 = relres0;
        info->relres = relres;
    }
    if (status != OCMP_OK) set_error("ocmp_solve_cg_noalloc: did not reach the tolerance (status " +
                                     std::to_string(status) + ")");
    return status;
}
