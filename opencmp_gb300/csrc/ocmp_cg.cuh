// Jacobi-preconditioned CG in one launch (sm_103a): the whole solve of ocmp_solve with OCMP_CG, FP64 or
// FP32 inner iteration with FP64 refinement, by one team of blocks (ocmp_team.cuh). One iteration is
//   q = A p on the owned rows, p . q                        exchange
//   x += alpha p, r -= alpha q, z = D^-1 r, r . z, |r|^2    exchange
//   p = z + beta p                                          barrier
// Two forms:
//  - resident (cg_res_kernel), systems of up to 1024 rows a block whose matrix entries fit the blocks'
//    shared memory (31 MB over the chip): a thread owns a row (two in the largest), its vector entries
//    stay in registers and its matrix row in shared memory for the whole solve, in slices of 32 rows
//    (entry j of the slice's rows side by side). Only z and p, which other blocks gather, go through
//    global memory. A warp-wide FP64 instruction takes 64 clocks whatever its lanes do, so a lane per
//    row, with no shuffle reduction, is the cheapest product. While a block's share of it costs less
//    than the barrier's 2,450 clocks the barrier is saved (fuse): the product gathers z and the
//    previous p and forms z + beta p at every use, one more FMA and load per entry. Bound by the
//    latency of the exchanges. A launch per operation (seven an iteration) took 47 us an iteration at
//    289 rows and 38 us at 16,641 (2D, P2, FP64); one launch takes 5.9 and 10.4.
//  - streaming (cg_stream_kernel), larger systems: bound by L2 or HBM and, in FP64, by the FP64 pipe,
//    so a row takes few lanes. Tiles of rows are dealt to the blocks in turn, so that the long vertex
//    rows and the short edge rows of a higher-order space spread over them.
#pragma once

#include "ocmp_internal.h"
#include "ocmp_team.cuh"

namespace ocmp {

constexpr int kCgThreadsRes = 512, kCgThreadsStream = 1024;
constexpr int kCgRowsPerThread = 2;                                // resident form
constexpr int kCgRowsRes = kCgRowsPerThread * kCgThreadsRes;
constexpr int kCgSlicesRes = kCgRowsRes / 32;

enum { CG_NONFIN = 1, CG_BREAK = 2 };
// FP32: p . A p of up to so many times sum |p_i| |a_ij| |p_j| may be rounding alone (an entry's and a
// product's). More negative curvature than that is the matrix's own and stepped along. From 1 to 64 times
// 2^-24 the solves of the nearly singular Neumann pressure operator stop where they should; at 4 and above
// P1 triangles on 200 x 200 with one negative eigenvalue (-div grad - 30) diverge, at 64 those on 100 x 100.
constexpr double kCgUnresolved = 2.0 / 16777216;
// What the host reads after a solve.
struct CgResult {
    double res0, res;
    int iters, outer, bits, pad;
};
struct CgState {
    CgResult r;
    TeamState t;            // its head (the abort flag) travels with the result
};
constexpr size_t kCgReadBytes = sizeof(CgResult) + 16;

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
    double* r64;            // FP64 residual
    T *r, *z, *p0, *p1, *q; // r (= r64 when T is double) and q: streaming form; p1: resident form
    T* d;                   // inner correction (T = float, streaming form)
    CgState* state;
    double tol, inner_tol, margin;
    int maxit;
    int cap, fuse;          // resident form: matrix entries of the largest block's slices
};

// sqrt of a sum of squares; NaN and infinity pass through
__device__ __forceinline__ double cg_norm(double s) { return s < 0 ? 0.0 : sqrt(s); }
__device__ __forceinline__ double cg_wide(double v) { return v; }
__device__ __forceinline__ double cg_wide(float v) { return f2d(v); }

// A thread's sum of products over many rows: FP64, or pairs of FP32. In FP32 alone, 60 equal products a
// thread made p . A p ten units too large; pairs cost 2.4% of an iteration at 753,571 rows (89.0 -> 91.1 us).
template <class T>
struct CgSum {
    double s = 0;
    __device__ __forceinline__ void add(double a, double b) { s += a * b; }
    __device__ __forceinline__ double value() const { return s; }
};
template <>
struct CgSum<float> {
    float h = 0.f, l = 0.f;
    __device__ __forceinline__ void add(float a, float b) {
        ff_mac(h, l, a, b);
        ff_norm(h, l);
    }
    __device__ __forceinline__ double value() const { return ff_wide(h, l); }
};

// The row's share of |b - A x|^2 (free rows) and, with lift, of |b - A x_D|^2
template <class T>
__device__ __forceinline__ void cg_resid_row(const CgArgs<T>& a, int64_t r, double ax, bool lift, double* out, double* acc) {
    const bool fr = a.freed[r] != 0;
    const double v = fr ? a.b[r] - ax : 0.0;
    if (out) *out = v;
    acc[0] += v * v;
    if (lift && fr) {
        double s = 0;
        for (int32_t q = a.lift_ptr[r]; q < a.lift_ptr[r + 1]; q++) {
            const int32_t k = a.lift_pos[q];
            s += a.A[k] * a.x[a.col[k]];
        }
        const double vd = a.b[r] - s;
        acc[1] += vd * vd;
    }
}

// The quantities of one (inner) iteration's end: thresholds in |r|^2, so that no square root is on the path
struct CgOuter {
    double nb, beta_n, res0, res;
    int iters, outer;
    bool nonfin, brk, run;
};
__device__ __forceinline__ void cg_begin(CgOuter& o, const double* sum, double tol) {
    const double nbs = cg_norm(sum[1]);
    o.nb = nbs > 0 ? nbs : 1.0;
    o.beta_n = cg_norm(sum[0]);
    o.res = o.res0 = o.beta_n / o.nb;
    o.iters = o.outer = 0;
    o.nonfin = !isfinite(o.res0);
    o.brk = false;
    o.run = !o.nonfin && o.res0 > tol;
}
template <bool MIX>
__device__ __forceinline__ void cg_end(CgOuter& o, const double* sum, double tol) {
    o.beta_n = cg_norm(sum[0]);
    o.res = o.beta_n / o.nb;
    if (MIX) {
        if (!isfinite(o.beta_n)) o.nonfin = true;
        o.run = o.run && !o.nonfin && !(o.res <= tol);
    }
}
template <class T>
__device__ __forceinline__ void cg_report(const CgArgs<T>& a, const Team& tm, const CgOuter& o) {
    if (tm.rank == 0 && threadIdx.x == 0) {
        a.state->r.res0 = o.res0;
        a.state->r.res = o.res;
        a.state->r.iters = o.iters;
        a.state->r.outer = o.outer;
        a.state->r.bits = (o.nonfin ? CG_NONFIN : 0) | (o.brk ? CG_BREAK : 0);
    }
    team_leave(tm);
}

template <class T>
__global__ void __launch_bounds__(kCgThreadsRes, 1) cg_res_kernel(CgArgs<T> a) {
    constexpr int RPT = kCgRowsPerThread, U = 12;   // U: gathers in flight (a P2 edge row is one batch)
    constexpr bool MIX = sizeof(T) == 4;
    extern __shared__ double cg_smem[];
    __shared__ int soff[kCgSlicesRes + 1];
    __shared__ double s_scal;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
    Team tm = team_join(&a.state->t, (int)blockIdx.x, (int)gridDim.x);
    const int64_t n = a.n;
    const int slices = (int)((n + 31) / 32);
    const int own = slices > tm.rank ? (slices - tm.rank + tm.size - 1) / tm.size : 0;   // this block's slices
    const int live = min((int)blockDim.x, own * 32);

    // slice q of the block is its warp q % nw's, and the thread's row k = q / nw
    int64_t row[RPT];
    bool in[RPT], fr[RPT];
    int len[RPT];
#pragma unroll
    for (int k = 0; k < RPT; k++) {
        const int q = w + k * nw;
        row[k] = ((int64_t)tm.rank + (int64_t)q * tm.size) * 32 + lane;
        in[k] = q < own && row[k] < n;
        fr[k] = in[k] && a.freed[row[k]] != 0;
        len[k] = in[k] ? a.rp[row[k] + 1] - a.rp[row[k]] : 0;
        const int wd = __reduce_max_sync(0xffffffffu, len[k]);
        if (lane == 0 && q < own) soff[q + 1] = wd * 32;
    }
    if (tid == 0) soff[0] = 0;
    __syncthreads();
    if (tid == 0)
        for (int q = 0; q < own; q++) soff[q + 1] += soff[q];
    __syncthreads();
    T* sval = reinterpret_cast<T*>(cg_smem);
    int32_t* scol = reinterpret_cast<int32_t*>(sval + a.cap);
    T *gz = a.z, *pc = a.p0, *pn = a.p1;
    if (tm.size == 1) {   // nobody else gathers: the gathered vectors in shared memory too
        gz = reinterpret_cast<T*>(cg_smem) + a.cap + a.cap / (int)(sizeof(T) / 4);
        pc = gz + kCgRowsRes;
        pn = pc;
    }
    T dv[RPT];
#pragma unroll
    for (int k = 0; k < RPT; k++) {
        dv[k] = in[k] ? a.dinv[row[k]] : (T)0;
        const int32_t k0 = in[k] ? a.rp[row[k]] : 0, o = w + k * nw < own ? soff[w + k * nw] + lane : 0;
        for (int j = 0; j < len[k]; j++) {
            sval[o + j * 32] = a.K[k0 + j];
            scol[o + j * 32] = a.col[k0 + j];
        }
    }

    auto residual = [&](bool lift, double* out) -> bool {
        double acc[2] = {0, 0};
#pragma unroll
        for (int k = 0; k < RPT; k++)
            if (in[k]) {
                const double ax = team_row_dot<double, double, 1, 4>(a.rp[row[k]], a.rp[row[k] + 1], a.col, a.A, a.x, 0);
                cg_resid_row(a, row[k], ax, lift, a.r64 + row[k], acc);
            }
        return team_reduce<2>(tm, acc, out, live);
    };

    double sum[2], part[2];
    CgOuter o;
    if (!residual(true, sum)) return;
    cg_begin(o, sum, a.tol);
    while (o.run && o.iters < a.maxit) {
        // start of an (inner) iteration: r (scaled for FP32), z = D^-1 r
        const double itol = MIX ? fmax(a.inner_tol, a.margin * a.tol * o.nb / o.beta_n) : a.tol;
        const double inv = MIX ? (o.beta_n > 0 ? 1.0 / o.beta_n : 0.0) : 1.0;
        const double stop1 = itol * (MIX ? 1.0 : o.nb), stop2 = stop1 * stop1;
        const int itmax = a.maxit - o.iters;
        T rv[RPT], zv[RPT], pv[RPT], xv[RPT];
        T rz_p = 0, rr_p = 0;
#pragma unroll
        for (int k = 0; k < RPT; k++) {
            rv[k] = zv[k] = pv[k] = xv[k] = (T)0;
            if (!in[k]) continue;
            rv[k] = MIX ? (T)(a.r64[row[k]] * inv) : (T)a.r64[row[k]];
            zv[k] = dv[k] * rv[k];
            if (a.fuse) {
                gz[row[k]] = zv[k];
                pc[row[k]] = (T)0;
            }
            rz_p += rv[k] * zv[k];
            rr_p += rv[k] * rv[k];
        }
        part[0] = cg_wide(rz_p);
        part[1] = cg_wide(rr_p);
        if (!team_reduce<2>(tm, part, sum, live)) return;
        double rz = sum[0], beta = 0;
        bool stop = !(sum[1] > stop2);       // NaN stops too
        bool in_nonfin = !isfinite(sum[1]);
        int it = 0;
        while (!stop && it < itmax) {
            // p, q = A p, p . q
            const T bt = (T)beta;
#pragma unroll
            for (int k = 0; k < RPT; k++)
                if (in[k]) {
                    pv[k] = zv[k] + bt * pv[k];
                    (a.fuse ? pn : pc)[row[k]] = pv[k];
                }
            if (!a.fuse && !team_barrier(tm)) return;
            T qv[RPT], pq = 0;
            double pq2 = 0;   // FP32: the second row's product is added in FP64
#pragma unroll
            for (int k = 0; k < RPT; k++) {
                T acc0 = 0, acc1 = 0;
                const int base = w + k * nw < own ? soff[w + k * nw] + lane : 0;
                for (int j0 = 0; j0 < len[k]; j0 += U) {
                    T g[U], g2[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const int32_t c = j0 + u < len[k] ? scol[base + (j0 + u) * 32] : -1;
                        if (a.fuse) g2[u] = c >= 0 ? gz[c] : (T)0;
                        g[u] = c >= 0 ? pc[c] : (T)0;
                    }
#pragma unroll
                    for (int u = 0; u < U; u++)
                        if (j0 + u < len[k]) {
                            const T v = a.fuse ? g2[u] + bt * g[u] : g[u];
                            (u & 1 ? acc1 : acc0) += sval[base + (j0 + u) * 32] * v;
                        }
                }
                qv[k] = fr[k] ? acc0 + acc1 : (T)0;
                if (!MIX) pq += pv[k] * qv[k];
                else if (k == 0) pq2 = cg_wide(pv[k] * qv[k]);
                else if (in[k]) pq2 += cg_wide(pv[k] * qv[k]);
            }
            part[0] = MIX ? pq2 : cg_wide(pq);
            if (!team_reduce<1>(tm, part, sum, live)) return;
            const double pap = sum[0];
            if (pap == 0.0 || !isfinite(pap)) {
                if (pap != 0.0) in_nonfin = true;
                else if (!MIX) o.brk = true;
                break;
            }
            // a step against the descent direction that rounding explains: a mode that the FP32 values do
            // not resolve. What was reached is kept, and refined from its true residual.
            if (MIX && pap * rz <= 0) {
                const T* p = a.fuse ? pn : pc;   // everyone's is there since the last exchange
                part[0] = 0;
#pragma unroll 1
                for (int k = 0; k < RPT; k++) {
                    T s = 0;
                    const int base = w + k * nw < own ? soff[w + k * nw] + lane : 0;
                    for (int j = 0; j < len[k]; j++) s += fabs(sval[base + j * 32] * p[scol[base + j * 32]]);
                    if (fr[k]) part[0] += cg_wide(fabs(pv[k]) * s);
                }
                if (!team_reduce<1>(tm, part, sum, live)) return;
                if (!(fabs(pap) > kCgUnresolved * sum[0])) break;
            }
            if (tid == 0) s_scal = rz / pap;
            __syncthreads();
            // x += alpha p, r -= alpha q, z, r . z, |r|^2
            const T alpha = (T)s_scal;
            rz_p = rr_p = 0;
#pragma unroll
            for (int k = 0; k < RPT; k++)
                if (in[k]) {
                    xv[k] += alpha * pv[k];
                    rv[k] -= alpha * qv[k];
                    zv[k] = dv[k] * rv[k];
                    if (a.fuse) gz[row[k]] = zv[k];
                    rz_p += rv[k] * zv[k];
                    rr_p += rv[k] * rv[k];
                }
            part[0] = cg_wide(rz_p);
            part[1] = cg_wide(rr_p);
            if (!team_reduce<2>(tm, part, sum, live)) return;
            it++;
            if (!(sum[1] > stop2)) {
                if (!isfinite(sum[1])) in_nonfin = true;
                break;
            }
            if (tid == 0) s_scal = rz != 0.0 ? sum[0] / rz : 0.0;
            __syncthreads();
            rz = sum[0];
            beta = s_scal;
            if (a.fuse) {
                T* t = pc;
                pc = pn;
                pn = t;
            }
        }
        if (in_nonfin) o.nonfin = true;
        o.iters += MIX ? max(it, 1) : it;
        if (MIX && it == 0) o.run = false;   // no step could be taken
        if (MIX) o.outer++;
        else o.run = false;
        if (MIX && in_nonfin) break;
#pragma unroll
        for (int k = 0; k < RPT; k++)
            if (in[k]) a.x[row[k]] += MIX ? o.beta_n * (double)xv[k] : (double)xv[k];
        // the true residual of the returned x (the recurrence's drifts from it)
        if (!team_barrier(tm)) return;
        if (!residual(false, sum)) return;
        cg_end<MIX>(o, sum, a.tol);
    }
    cg_report(a, tm, o);
}

template <class T, int TPR>
__global__ void __launch_bounds__(kCgThreadsStream, 1) cg_stream_kernel(CgArgs<T> a) {
    constexpr int NT = kCgThreadsStream, RT = NT / TPR, U = 4;
    constexpr bool MIX = sizeof(T) == 4;
    __shared__ double s_scal;
    const int tid = threadIdx.x, lane = tid % TPR;
    Team tm = team_join(&a.state->t, (int)blockIdx.x, (int)gridDim.x);
    const int64_t n = a.n, step = (int64_t)tm.size * RT, first = (int64_t)tm.rank * RT;
    // the owned rows as one list, for the row-per-thread phases
    const int64_t tiles = (n + RT - 1) / RT;
    const int nown = first < n ? (int)((tiles - tm.rank + tm.size - 1) / tm.size) * RT : 0;
    auto each = [&](auto fn) {
        for (int li = tid; li < nown; li += NT) {
            const int64_t i = ((int64_t)(li / RT) * tm.size + tm.rank) * RT + li % RT;
            if (i < n) fn(i);
        }
    };
    const int live = min(NT, nown);
    // fn(r, A_r . x) on lane 0 of each owned row
    auto rows = [&](const auto* val, const auto* x, auto fn) {
        using TV = std::remove_cv_t<std::remove_reference_t<decltype(*x)>>;
        for (int64_t t0 = first; t0 < n; t0 += step) {
            const int64_t r = t0 + tid / TPR;
            int32_t k0 = 0, k1 = 0;
            if (r < n) {
                k0 = __ldg(a.rp + r);
                k1 = __ldg(a.rp + r + 1);
            }
            const TV v = team_row_dot<TV, TV, TPR, U>(k0, k1, a.col, val, x, lane);
            if (r < n && lane == 0) fn(r, v);
        }
    };
    auto residual = [&](bool lift, double* out) -> bool {
        double acc[2] = {0, 0};
        rows(a.A, (const double*)a.x, [&](int64_t r, double ax) { cg_resid_row(a, r, ax, lift, a.r64 + r, acc); });
        return team_reduce<2>(tm, acc, out, NT);
    };

    double sum[2], part[2];
    CgOuter o;
    if (!residual(true, sum)) return;
    cg_begin(o, sum, a.tol);
    while (o.run && o.iters < a.maxit) {
        // start of an (inner) iteration: r (scaled for FP32), z = D^-1 r, p
        const double itol = MIX ? fmax(a.inner_tol, a.margin * a.tol * o.nb / o.beta_n) : a.tol;
        const double inv = MIX ? (o.beta_n > 0 ? 1.0 / o.beta_n : 0.0) : 1.0;
        const double stop1 = itol * (MIX ? 1.0 : o.nb), stop2 = stop1 * stop1;
        const int itmax = a.maxit - o.iters;
        CgSum<T> rz_p, rr_p;
        each([&](int64_t i) {
            const T ri = MIX ? (T)(a.r64[i] * inv) : (T)a.r64[i], zi = a.dinv[i] * ri;
            if (MIX) {
                a.r[i] = ri;
                a.d[i] = (T)0;
            }
            a.p0[i] = zi;
            rz_p.add(ri, zi);
            rr_p.add(ri, ri);
        });
        part[0] = rz_p.value();
        part[1] = rr_p.value();
        if (!team_reduce<2>(tm, part, sum, live)) return;
        double rz = sum[0];
        bool stop = !(sum[1] > stop2);       // NaN stops too
        bool in_nonfin = !isfinite(sum[1]);
        int it = 0;
        while (!stop && it < itmax) {
            // q = A p, p . q
            CgSum<T> pq;
            rows(a.K, (const T*)a.p0, [&](int64_t r, T v) {
                const T qv = a.freed[r] ? v : (T)0;
                a.q[r] = qv;
                pq.add(a.p0[r], qv);
            });
            part[0] = pq.value();
            if (!team_reduce<1>(tm, part, sum, NT)) return;
            const double pap = sum[0];
            if (pap == 0.0 || !isfinite(pap)) {
                if (pap != 0.0) in_nonfin = true;
                else if (!MIX) o.brk = true;
                break;
            }
            // a step against the descent direction that rounding explains: a mode that the FP32 values do
            // not resolve. What was reached is kept, and refined from its true residual.
            if (MIX && pap * rz <= 0) {
                CgSum<T> s;
                each([&](int64_t r) {
                    T v = 0;
                    for (int32_t k = a.rp[r]; k < a.rp[r + 1]; k++) v += fabs(a.K[k] * a.p0[a.col[k]]);
                    if (a.freed[r]) s.add(fabs(a.p0[r]), v);
                });
                part[0] = s.value();
                if (!team_reduce<1>(tm, part, sum, live)) return;
                if (!(fabs(pap) > kCgUnresolved * sum[0])) break;
            }
            if (tid == 0) s_scal = rz / pap;
            __syncthreads();
            // x += alpha p, r -= alpha q, z, r . z, |r|^2
            const T alpha = (T)s_scal;
            rz_p = rr_p = CgSum<T>();
            each([&](int64_t i) {
                const T pi = a.p0[i];
                if (MIX) a.d[i] += alpha * pi;
                else a.x[i] += (double)(alpha * pi);
                const T ri = a.r[i] - alpha * a.q[i];
                a.r[i] = ri;
                const T zi = a.dinv[i] * ri;
                a.z[i] = zi;
                rz_p.add(ri, zi);
                rr_p.add(ri, ri);
            });
            part[0] = rz_p.value();
            part[1] = rr_p.value();
            if (!team_reduce<2>(tm, part, sum, live)) return;
            it++;
            if (!(sum[1] > stop2)) {
                if (!isfinite(sum[1])) in_nonfin = true;
                break;
            }
            if (tid == 0) s_scal = rz != 0.0 ? sum[0] / rz : 0.0;
            __syncthreads();
            rz = sum[0];
            const T beta = (T)s_scal;
            each([&](int64_t i) { a.p0[i] = a.z[i] + beta * a.p0[i]; });
            if (!team_barrier(tm)) return;
        }
        if (in_nonfin) o.nonfin = true;
        o.iters += MIX ? max(it, 1) : it;
        if (MIX && it == 0) o.run = false;   // no step could be taken
        if (MIX) {
            o.outer++;
            if (in_nonfin) break;
            each([&](int64_t i) { a.x[i] += o.beta_n * (double)a.d[i]; });
            if (!team_barrier(tm)) return;
        } else
            o.run = false;
        // the true residual of the returned x (the recurrence's drifts from it)
        if (!residual(false, sum)) return;
        cg_end<MIX>(o, sum, a.tol);
    }
    cg_report(a, tm, o);
}

}  // namespace ocmp
