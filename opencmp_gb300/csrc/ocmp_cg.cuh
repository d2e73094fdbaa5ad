// Jacobi-preconditioned CG in one launch (sm_103a): the whole solve of ocmp_solve with OCMP_CG, FP64 or
// FP32 inner iteration with FP64 refinement, by one team of blocks (ocmp_team.cuh).
//
// A block owns every size-th tile of kCgThreads / TPR rows (interleaved, so that the long vertex rows
// and the short edge rows of a higher-order space spread over the blocks). One iteration is
//   q = A p on the owned rows, p . q                        barrier
//   x += alpha p, r -= alpha q, z = D^-1 r, r . z, |r|^2    barrier
//   p = z + beta p                                          barrier
// What bounds it: the barriers (about 1.3 us each among 152 blocks) up to about 10^5 rows, then the
// FP64 pipe or L2. Systems of few entries per block therefore save the third barrier: the product
// gathers z and the previous p and forms p = z + beta p at every use (FUSEP), one more FMA and load per
// matrix entry; the line is where that costs as much as the barrier.
#pragma once

#include "ocmp_internal.h"
#include "ocmp_team.cuh"

namespace ocmp {

constexpr int kCgThreads = 512;

enum { CG_NONFIN = 1, CG_BREAK = 2 };
// What the host reads after a solve, in one copy.
struct CgResult {
    double res0, res;
    int iters, outer, bits, pad;
    TeamState team;
};

// sqrt of a sum of squares; NaN and infinity pass through
__device__ __forceinline__ double cg_norm(double s) { return s < 0 ? 0.0 : sqrt(s); }

template <class T>
struct CgArgs {
    int64_t n;
    const int32_t *rp, *col;
    const double* A;        // FP64 values: residuals (and the iteration, T = double)
    const T* K;             // values the iteration multiplies with
    const uint8_t* freed;
    const int32_t *lift_ptr, *lift_pos;
    const T* dinv;
    const double* b;
    double* x;
    double* r64;            // FP64 residual (T = float); unused for T = double
    T *r, *z, *p0, *p1, *q;
    T* d;                   // inner correction (T = float)
    double* part;           // 6 x team size
    CgResult* out;
    double tol, inner_tol, margin;
    int maxit, fusep;
};

template <class T, int TPR>
__global__ void __launch_bounds__(kCgThreads, 1) cg_solve_kernel(CgArgs<T> a) {
    constexpr int RT = kCgThreads / TPR;
    constexpr int U = 4;
    constexpr bool MIX = sizeof(T) == 4;
    __shared__ T shv[2][kCgThreads];
    __shared__ double shd[2][kCgThreads];
    __shared__ double sum[2];
    __shared__ double s_alpha, s_beta;
    __shared__ int s_stop, s_nonfin, s_brk;
    const int tid = threadIdx.x, lane = tid % TPR, wid = tid >> 5, l32 = tid & 31;
    Team tm{&a.out->team, (int)blockIdx.x, (int)gridDim.x, 0u};
    const int64_t n = a.n, step = (int64_t)tm.size * RT;
    const int64_t first = (int64_t)tm.rank * RT;
    // partials of the residual, of p . q and of the update: a buffer is written again only after
    // another barrier than the one its last values were read behind
    double *partR = a.part, *partA = partR + 2 * tm.size, *partB = partA + 2 * tm.size;

    // the owned rows as one list, for the row-per-thread phases
    const int64_t tiles = (n + RT - 1) / RT;
    const int nown = first < n ? (int)((tiles - tm.rank + tm.size - 1) / tm.size) * RT : 0;
    auto row = [&](int li) { return ((int64_t)(li / RT) * tm.size + tm.rank) * RT + li % RT; };
    const int vcnt = min(kCgThreads, nown);   // threads that hold a value in them
    const int scnt = min(RT, nown);           // and in the products

    // this block's partials of nv values held per thread in sh[v][0 .. cnt)
    auto publish = [&](auto* s0, auto* s1, int nv, int cnt, double* part) {
        __syncthreads();
        if (wid < nv) {
            const double v = team_row_sum(wid == 0 ? s0 : s1, cnt, l32);
            if (l32 == 0) part[wid * tm.size + tm.rank] = v;
        }
    };
    // r = (b - A x)_free into r64 / r; sum[0] = |r|^2 and, with lift, sum[1] = |(b - A x_D)_free|^2
    auto residual = [&](double* rout, bool lift) -> bool {
        double acc = 0, accd = 0;
        for (int64_t t0 = first; t0 < n; t0 += step) {
            const int64_t r = t0 + tid / TPR;
            int32_t k0 = 0, k1 = 0;
            if (r < n) {
                k0 = __ldg(a.rp + r);
                k1 = __ldg(a.rp + r + 1);
            }
            const double ax = team_row_dot<double, double, TPR, U>(k0, k1, a.col, a.A, a.x, lane);
            if (r < n && lane == 0) {
                const bool fr = a.freed[r] != 0;
                const double v = fr ? a.b[r] - ax : 0.0;
                if (rout) rout[r] = v;
                acc += v * v;
                if (lift && fr) {
                    double s = 0;
                    for (int32_t q = a.lift_ptr[r]; q < a.lift_ptr[r + 1]; q++) {
                        const int32_t k = a.lift_pos[q];
                        s += a.A[k] * a.x[a.col[k]];
                    }
                    const double vd = a.b[r] - s;
                    accd += vd * vd;
                }
            }
        }
        if (lane == 0) {
            shd[0][tid / TPR] = acc;
            shd[1][tid / TPR] = accd;
        }
        publish(&shd[0][0], &shd[1][0], 2, scnt, partR);
        if (!team_sync(tm)) return false;
        team_sums(partR, tm.size, 2, sum);
        __syncthreads();
        return true;
    };

    double* r64 = MIX ? a.r64 : (double*)a.r;
    if (!residual(r64, true)) return;
    const double nbs = cg_norm(sum[1]), nb = nbs > 0 ? nbs : 1.0;
    double beta_n = cg_norm(sum[0]);
    const double res0 = beta_n / nb;
    double res = res0;
    int iters = 0, outer = 0;
    bool nonfin = !isfinite(res0), brk = false;
    bool run = !nonfin && res0 > a.tol;
    while (run && iters < a.maxit) {
        // start of an (inner) iteration: r (scaled for FP32), z = D^-1 r, p
        const double inb = MIX ? 1.0 : nb;
        const double itol = MIX ? fmax(a.inner_tol, a.margin * a.tol * nb / beta_n) : a.tol;
        const double inv = MIX ? (beta_n > 0 ? 1.0 / beta_n : 0.0) : 1.0;
        const int itmax = a.maxit - iters;
        T rz_p = 0, rr_p = 0;
        for (int li = tid; li < nown; li += kCgThreads) {
            const int64_t i = row(li);
            if (i >= n) continue;
            const T ri = MIX ? (T)(r64[i] * inv) : (T)r64[i];
            const T zi = a.dinv[i] * ri;
            if (MIX) {
                a.r[i] = ri;
                a.d[i] = (T)0;
            }
            a.z[i] = zi;
            a.p0[i] = a.fusep ? (T)0 : zi;
            rz_p += ri * zi;
            rr_p += ri * ri;
        }
        shv[0][tid] = rz_p;
        shv[1][tid] = rr_p;
        publish(&shv[0][0], &shv[1][0], 2, vcnt, partB);
        if (!team_sync(tm)) return;
        team_sums(partB, tm.size, 2, sum);
        __syncthreads();
        double rz = sum[0];
        const double rs = sqrt(fmax(sum[1], 0.0)) / inb;
        bool stop = !(rs > itol);       // NaN stops too
        bool in_nonfin = !isfinite(rs);
        int it = 0;
        T *pc = a.p0, *pn = a.p1;       // FUSEP: previous p, this p; else p in place
        double beta = 0;
        while (!stop && it < itmax) {
            // q = A p and p . q
            T pq = 0;
            const T bt = (T)beta;
            for (int64_t t0 = first; t0 < n; t0 += step) {
                const int64_t r = t0 + tid / TPR;
                int32_t k0 = 0, k1 = 0;
                if (r < n) {
                    k0 = __ldg(a.rp + r);
                    k1 = __ldg(a.rp + r + 1);
                }
                T qv, pv = 0;
                if (a.fusep) {
                    T acc = 0;
                    for (int32_t base = k0 + lane; base < k1; base += U * TPR) {
                        int32_t c[U];
                        T v[U];
#pragma unroll
                        for (int u = 0; u < U; u++) {
                            const int32_t k = base + u * TPR;
                            c[u] = k < k1 ? __ldg(a.col + k) : -1;
                            v[u] = k < k1 ? __ldg(a.K + k) : (T)0;
                        }
#pragma unroll
                        for (int u = 0; u < U; u++)
                            if (c[u] >= 0) acc += v[u] * (a.z[c[u]] + bt * pc[c[u]]);
                    }
#pragma unroll
                    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPR);
                    qv = acc;
                    if (r < n && lane == 0) {
                        pv = a.z[r] + bt * pc[r];
                        pn[r] = pv;
                    }
                } else {
                    qv = team_row_dot<T, T, TPR, U>(k0, k1, a.col, a.K, pc, lane);
                    if (r < n && lane == 0) pv = pc[r];
                }
                if (r < n && lane == 0) {
                    qv = a.freed[r] ? qv : (T)0;
                    a.q[r] = qv;
                    pq += pv * qv;
                }
            }
            if (lane == 0) shv[0][tid / TPR] = pq;
            publish(&shv[0][0], &shv[0][0], 1, scnt, partA);
            if (!team_sync(tm)) return;
            team_sums(partA, tm.size, 1, sum);
            if (tid == 0) {
                const double v = sum[0];
                s_stop = s_nonfin = s_brk = 0;
                if (v == 0.0 || !isfinite(v)) {
                    s_stop = 1;
                    if (v == 0.0) s_brk = 1;
                    else s_nonfin = 1;
                    s_alpha = 0;
                } else
                    s_alpha = rz / v;
            }
            __syncthreads();
            if (s_stop) {
                stop = true;
                if (s_nonfin) in_nonfin = true;
                if (s_brk && !MIX) brk = true;
                break;
            }
            // x += alpha p, r -= alpha q, z, r . z, |r|^2
            const T alpha = (T)s_alpha;
            const T* pu = a.fusep ? pn : pc;
            rz_p = rr_p = 0;
            for (int li = tid; li < nown; li += kCgThreads) {
                const int64_t i = row(li);
                if (i >= n) continue;
                const T pi = pu[i];
                if (MIX) a.d[i] += alpha * pi;
                else a.x[i] += (double)(alpha * pi);
                const T ri = a.r[i] - alpha * a.q[i];
                a.r[i] = ri;
                const T zi = a.dinv[i] * ri;
                a.z[i] = zi;
                rz_p += ri * zi;
                rr_p += ri * ri;
            }
            shv[0][tid] = rz_p;
            shv[1][tid] = rr_p;
            publish(&shv[0][0], &shv[1][0], 2, vcnt, partB);
            if (!team_sync(tm)) return;
            team_sums(partB, tm.size, 2, sum);
            __syncthreads();
            if (tid == 0) {
                const double rs1 = sqrt(fmax(sum[1], 0.0)) / inb;
                s_beta = rz != 0.0 ? sum[0] / rz : 0.0;
                s_nonfin = !isfinite(rs1);
                s_stop = !(rs1 > itol);
            }
            __syncthreads();
            rz = sum[0];
            beta = s_beta;
            it++;
            if (s_stop) {
                stop = true;
                if (s_nonfin) in_nonfin = true;
                break;
            }
            if (a.fusep) {
                T* t = pc;
                pc = pn;
                pn = t;
            } else {
                const T b2 = (T)beta;
                for (int li = tid; li < nown; li += kCgThreads) {
                    const int64_t i = row(li);
                    if (i < n) pc[i] = a.z[i] + b2 * pc[i];
                }
                if (!team_sync(tm)) return;
            }
        }
        if (in_nonfin) nonfin = true;
        if (!MIX) {
            iters = it;
            run = false;
        } else {
            iters += max(it, 1);
            outer++;
            if (in_nonfin) break;
            for (int li = tid; li < nown; li += kCgThreads) {
                const int64_t i = row(li);
                if (i < n) a.x[i] += beta_n * (double)a.d[i];
            }
            if (!team_sync(tm)) return;
            if (!residual(r64, false)) return;
            beta_n = cg_norm(sum[0]);
            res = beta_n / nb;
            if (!isfinite(beta_n)) {
                nonfin = true;
                break;
            }
            run = !(res <= a.tol);
        }
    }
    if (!MIX && iters > 0) {
        // the recurrence's residual drifts from the true one: measure the returned x
        if (!residual(nullptr, false)) return;
        res = cg_norm(sum[0]) / nb;
    }
    if (tm.rank == 0 && tid == 0) {
        a.out->res0 = res0;
        a.out->res = res;
        a.out->iters = iters;
        a.out->outer = outer;
        a.out->bits = (nonfin ? CG_NONFIN : 0) | (brk ? CG_BREAK : 0);
    }
    team_leave(tm);
}

}  // namespace ocmp
