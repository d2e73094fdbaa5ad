// Fused GMRES(m), right-preconditioned, in one launch (sm_103a): whole solves by teams of blocks
// (ocmp_team.cuh), one system on every SM or many uneven systems side by side.
//
// The Krylov matrix is A D^-1 (point Jacobi folded into the values), A with an explicit block-Jacobi
// application, or A behind a preconditioner applied by other kernels (strip, Cahouet-Chabard: then one
// launch per phase). The basis is kept unnormalised, v_k = scale[k] V[k], so no pass normalises. Rows
// are dealt to the blocks in tiles of TR, and a block's rows stay its own in every phase, so an
// iteration needs two exchanges only:
//   w = A_s v_j and, over the same rows, V_k . w (k <= j) and |w|^2        exchange
//   w -= sum_k h_k v_k (beside it one warp rotates the Hessenberg column)
//   and |w|^2                                                              exchange
// then every block makes the same Givens step on its own copy of the small state: no block waits for
// another's scalar work. A second Gram-Schmidt pass runs when the first cancelled nearly all of |w|.
// Sums run in a fixed order: bit-reproducible.
//
// What bounds it. FP32: HBM or L2 (matrix and basis). FP64: the FP64 pipe, 64 clocks for a warp
// instruction in each quarter of an SM, so the row products take few lanes, the dot products keep
// eight accumulators in each of 128 threads' rows, and sums over threads go through shared memory with
// every lane adding (a butterfly wastes 31 of 32 additions). Below about 10^4 rows: the exchanges,
// 2,430 clocks each. Five launches per iteration with two-stage reductions in each took 54 us an
// iteration at 79,507 rows (P2 tetrahedra, FP64, basis of 15) and 33 us at 1,156; one launch takes 29
// (product 10.4 from the first block's start to the last one's end, bound by its gathers; dots 4.6,
// orthogonalisation 4.3) and 13. From 1.8 M rows on in FP64, where the basis streams from HBM, a launch per
// operation was faster with its 64 warps per SM: 349 against 362 us at 1,771,561 rows, 512 against 559 at
// 2,803,221.
#pragma once

#include <type_traits>

#include "ocmp_internal.h"
#include "ocmp_team.cuh"

namespace ocmp {

constexpr double kTargetMargin = 0.9;  // a GMRES cycle stops at kTargetMargin x the outer tolerance
// Classical Gram-Schmidt, repeated only when |w| lost more than 99.9% of its length to the projection
// (|w_new|^2 < 1e-6 |w|^2); the mass-dominated systems here lose far less per step.
constexpr double kReorth = 1e-6;

// device flags of a solve in phases (its preconditioner's kernels return at once when F_CONV is set)
enum { F_CONV = 0, F_BREAK, F_NONFIN, F_JDONE, F_ITERS, F_OUTER, F_NFLAG = 8 };
enum { GM_NONFIN = 1, GM_BREAK = 2 };
// phases: GM_FULL a whole solve; for the preconditioners applied by other kernels: GM_FIRST / GM_START
// the residual and the start of a cycle, GM_ITER iteration j, GM_COMBINE z = sum_k y_k v_k
enum { GM_FULL = 0, GM_FIRST, GM_START, GM_ITER, GM_COMBINE };

// What the host reads after a solve (flags: the phases' device flags). gaveup is set by any block whose wait
// ran out and cleared by the host alone, so that no result of a block that had passed hides it.
struct GmResult {
    double res0, res;
    int iters, cycles, bits, gaveup;
    int flags[F_NFLAG];
};

// One system.
struct GmInst {
    int64_t n, ld;
    const int32_t *rp, *col;
    const uint8_t* freed;
    const int32_t *lift_ptr, *lift_pos;
    const double* A64;      // FP64 matrix values (residuals)
    const void* K;          // T: Krylov matrix values
    const void* dinv;       // T: D^-1 of the final update, or null
    const void* Binv;       // T: block-Jacobi inverses (L x L per element), or null
    void* V;                // T: basis, m + 1 vectors at a stride of ld, zero past n
    void* z;                // T: preconditioned vector (block Jacobi, phases)
    const int32_t *soff, *scol;   // SELL-32 layout of K, or null
    const double* b;
    double* x;
    double* small;          // R (packed columns), cos, sin, g, scale: kept between the launches of phases
    GmResult* out;
    double tol, inner;
    int maxit, L, TR, tpr, rtpr;  // rows per tile; lanes per row of the Krylov product and of the FP64 one
    int u64, pad;           // entries in flight per lane of an FP64 solve's products
};

struct GmArgs {
    GmInst one;
    const GmInst* list;     // null: `one`
    const int4* map;        // per block: team, rank, size, instance (-1: none, -2: the team takes them from the
                            // teams' queue); null: one team, or (with a queue) none
    const int* queue_inst;  // instances of the teams' queue, then those of single blocks, largest first
    int* queue;             // next of either: single blocks', teams'
    int nteam, nqueue;
    TeamState* teams;
    double* part;           // (m + 2) x blocks
    unsigned long long* tlog;   // product timing: complement of the start, and end per product, or null
    int tcap, m, mode, j;
    int rp_slices;          // slices of 32 rows whose row pointers fit the blocks' shared memory
};

// The blocks of a launch as teams: one team of all of them for one system; for several, each system
// gets blocks in proportion to its work (two or more: a team of its own) and the systems of less than
// two blocks' work form a queue that the remaining blocks, and later the teams' blocks, empty one
// system per block, largest first. Where that would leave too many rows to a block, teams of one size
// empty a queue of the larger systems first.
struct GmTeams {
    int grid = 0, nteam = 0, nqueue = 0, nteams = 0;
    bool small = false;          // queue only, blocks of kGmSmallThreads
    std::vector<int> tile;       // per system: rows per tile
    int64_t max_slices = 0;      // slices of 32 rows of the largest block
    TeamState* state = nullptr;
    double* part = nullptr;
    int4* map = nullptr;         // null: one team
    int* qinst = nullptr;
    int* queue = nullptr;
    GmInst* inst = nullptr;      // device descriptors (several systems)
};

// FP32 systems of this many rows a block have tiles of 128 rows (16-byte loads of the basis). Against 32 rows
// (us an iteration): 17.9 and 18.0 at 255 rows a block, 19.7 and 20.6 at 512, 37.3 and 41.1 at 1,807.
constexpr int64_t kGmVecRows = 512;

// Stride of the basis vectors: whole tiles of 128 rows where they are read in 16-byte loads; elsewhere 16
// values (64 or 128 bytes), since the vectors of a batch of tiny systems would be mostly padding (9 rows,
// restart 30, FP64: 36 KB a system, and 9 KB so; a stride of n without alignment before took 11).
template <class T>
__host__ __device__ constexpr int64_t gm_ld(int64_t n) {
    const int64_t pad = sizeof(T) == 4 && n >= kGmVecRows ? 128 : 16;
    return (n + pad - 1) / pad * pad;
}

__host__ __device__ constexpr int gm_small_doubles(int m) { return m * (m + 1) / 2 + 4 * m + 8; }

// Threads of a block: one block per SM, or kGmSmallThreads where several blocks of an SM each solve systems of
// few rows.
template <class T>
constexpr int kGmThreads = sizeof(T) == 8 ? 512 : 1024;
constexpr int kGmSmallThreads = 128;

template <class T, int NT_>
struct GmCfg {
    static constexpr int NT = NT_;
    static constexpr int DT = 128;                         // FP64: threads holding a dot product's partials
    static constexpr int rows(int m) { return m + 8 < 64 ? m + 8 : 64; }   // values in that table at a time
    static constexpr int ES = sizeof(T) == 8 ? DT + 8 : NT / 32 + 1;   // stride of their shared table
    static constexpr size_t smem(int m) { return ((size_t)gm_small_doubles(m) + 3 * (m + 2) + (size_t)rows(m) * ES) * 8; }
};

__device__ __forceinline__ unsigned long long gm_time() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// dst[k] = sum_i get(k, i), i < E, for k < nv: eight lanes per value, ten entries of each in flight
template <class Get, class Put>
__device__ __forceinline__ void gm_sum_rows(int nv, int E, Get get, Put put) {
    constexpr int F = 10;
    const int lane = threadIdx.x & 31;
    for (int q0 = threadIdx.x & ~31; q0 < nv * 8; q0 += blockDim.x) {
        const int q = q0 + lane, k = min(q >> 3, nv - 1), p = q & 7;
        double s = 0;
        for (int i0 = p; i0 < E; i0 += 8 * F) {
            double v[F];
#pragma unroll
            for (int f = 0; f < F; f++) v[f] = i0 + 8 * f < E ? get(k, i0 + 8 * f) : 0.0;
            double s2 = 0;
#pragma unroll
            for (int f = 0; f < F; f += 2)
                if (i0 - p + 8 * f < E) {
                    s += v[f];
                    s2 += v[f + 1];
                }
            s += s2;
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (p == 0 && (q >> 3) < nv) put(k, s);
    }
}

// One halving step of a warp's sums of 2 HALF values per lane (float pairs): lanes OFF apart exchange
// half of their values and keep the sums of the other half.
template <int HALF, int OFF, int N>
__device__ __forceinline__ void gm_halve(float (&h)[N], float (&l)[N], int lane) {
    const bool up = (lane & OFF) != 0;
#pragma unroll
    for (int u = 0; u < HALF; u++) {
        const float sh = up ? h[u] : h[u + HALF], sl = up ? l[u] : l[u + HALF];
        float kh = up ? h[u + HALF] : h[u], kl = up ? l[u + HALF] : l[u];
        const float oh = __shfl_xor_sync(0xffffffffu, sh, OFF), ol = __shfl_xor_sync(0xffffffffu, sl, OFF);
        ff_add(kh, kl, oh, ol);
        h[u] = kh;
        l[u] = kl;
    }
}

// A block's work on one system of its team.
template <class T, int NT_>
struct GmRun {
    using C = GmCfg<T, NT_>;
    static constexpr int NT = C::NT, NW = NT / 32, DT = C::DT, ES = C::ES;
    static constexpr bool D = sizeof(T) == 8;
    const GmArgs& a;
    const GmInst& d;
    Team& tm;
    double *R, *cs, *sn, *g, *scale, *hraw, *hcol, *dsum, *tab, *part;   // all but part in shared memory
    T* V;
    int64_t n, ld;
    int32_t* srp;           // the owned rows' pointers, 33 per slice, or null
    int nsl, TS, w, lane;   // the block's slices of 32 rows, slices per tile
    int live;               // threads with a row
    unsigned products = 0;

    __device__ __forceinline__ GmRun(const GmArgs& a_, const GmInst& d_, Team& t_, double* sm, double* pt)
        : a(a_), d(d_), tm(t_), part(pt) {
        const int m = a.m;
        R = sm;
        cs = R + m * (m + 1) / 2;
        sn = cs + m;
        g = sn + m;
        scale = g + m + 2;
        hraw = R + gm_small_doubles(m);
        hcol = hraw + m + 2;
        dsum = hcol + m + 2;
        tab = dsum + m + 2;
        srp = reinterpret_cast<int32_t*>(tab + C::rows(m) * ES);
        V = (T*)d.V;
        n = d.n;
        ld = d.ld;
        TS = d.TR / 32;
        const int64_t tiles = (n + d.TR - 1) / d.TR;
        nsl = tiles > tm.rank ? (int)((tiles - tm.rank + tm.size - 1) / tm.size) * TS : 0;
        w = threadIdx.x >> 5;
        lane = threadIdx.x & 31;
        live = min(NT, nsl * 32);
        // a product starts with its rows' pointers, a third of the chain of loads of a short row
        if (a.mode == GM_FULL && nsl <= a.rp_slices) {
            for (int s = w; s < nsl; s += NW) {
                const int64_t r = slice(s) + lane;
                srp[s * 33 + lane] = d.rp[min(r, n)];
                if (lane == 0) srp[s * 33 + 32] = d.rp[min(r + 32, n)];
            }
            __syncthreads();
        } else
            srp = nullptr;
    }
    __device__ __forceinline__ int64_t slice(int s) const {   // first row of the block's slice s
        return ((int64_t)(s / TS) * tm.size + tm.rank) * d.TR + (s % TS) * 32;
    }
    template <class F>
    __device__ __forceinline__ void rows(int first, int stride, F fn) const {   // a row per lane
        for (int s = first; s < nsl; s += stride) {
            const int64_t r = slice(s) + lane;
            if (r < n) fn(r);
        }
    }
    template <class F>
    __device__ __forceinline__ void tiles4(int first, int stride, F fn) const {   // tiles of 128: four rows per lane
        for (int s = 4 * first; s < nsl; s += 4 * stride) fn(slice(s) + 4 * lane);
    }
    // fn(row, A_row . x) on one lane of each row, TPR lanes per row
    template <int TPR, int U, class TM, class F>
    __device__ __forceinline__ void products_of(const TM* val, const TM* x, F fn) const {
        for (int q = w; q < nsl * TPR; q += NW) {
            const int i = (q % TPR) * (32 / TPR) + lane / TPR;
            const int64_t r = slice(q / TPR) + i;
            int32_t k0 = 0, k1 = 0;
            if (srp) {
                k0 = srp[q / TPR * 33 + i];
                k1 = srp[q / TPR * 33 + i + 1];
            } else if (r < n) {
                k0 = __ldg(d.rp + r);
                k1 = __ldg(d.rp + r + 1);
            }
            const TM v = team_row_dot<TM, TM, TPR, U>(k0, k1, d.col, val, x, lane % TPR);
            if (r < n && lane % TPR == 0) fn(r, v);
        }
    }
    template <int U, class TM, class F>
    __device__ __forceinline__ void products_lanes(int tpr, const TM* val, const TM* x, F fn) const {
        if (tpr == 1) products_of<1, U>(val, x, fn);
        else if (tpr == 2) products_of<2, U>(val, x, fn);
        else if (tpr == 4) products_of<4, U>(val, x, fn);
        else if (tpr == 8) products_of<8, U>(val, x, fn);
        else products_of<16, U>(val, x, fn);
    }
    template <class TM, class F>
    __device__ __forceinline__ void products_by(int tpr, const TM* val, const TM* x, F fn) const {
        // entries in flight per lane, as the threads' registers allow
        if constexpr (D) {
            if (d.u64 == 8) products_lanes<8>(tpr, val, x, fn);
            else products_lanes<4>(tpr, val, x, fn);
        } else
            products_lanes<sizeof(TM) == 4 ? 8 : 4>(tpr, val, x, fn);
    }

    // z = B^-1 v (or x += B^-1 v) over the owned elements (their rows are the block's own)
    template <int L>
    __device__ __forceinline__ void block_apply_of(const T* v, T* z, double* x) const {
        const T* B = (const T*)d.Binv;
        rows(w, NW, [&](int64_t r) {
            const int64_t e0 = r / L * L;
            T b[L], y[L];
#pragma unroll
            for (int k = 0; k < L; k++) {
                b[k] = __ldg(B + r * L + k);
                y[k] = v[e0 + k];
            }
            T acc = 0;
#pragma unroll
            for (int k = 0; k < L; k++) acc += b[k] * y[k];
            if (x) x[r] += (double)acc;
            else z[r] = acc;
        });
    }
    __device__ __forceinline__ void block_apply(const T* v, T* z, double* x) const {
        if (d.L == 3) block_apply_of<3>(v, z, x);
        else if (d.L == 6) block_apply_of<6>(v, z, x);
        else block_apply_of<10>(v, z, x);
    }

    // r = (b - A x)_free -> V_0; out[0] = |r|^2 and, with lift, out[1] = |(b - A x_D)_free|^2
    __device__ __forceinline__ bool residual(bool lift, double* out) {
        double acc[2] = {0, 0};
        products_by<double>(d.rtpr, d.A64, d.x, [&](int64_t r, double ax) {
            const bool fr = d.freed[r] != 0;
            const double v = fr ? d.b[r] - ax : 0.0;
            V[r] = (T)v;
            acc[0] += v * v;
            if (lift && fr) {
                double s = 0;
                for (int32_t q = d.lift_ptr[r]; q < d.lift_ptr[r + 1]; q++) {
                    const int32_t k = d.lift_pos[q];
                    s += d.A64[k] * d.x[d.col[k]];
                }
                const double vd = d.b[r] - s;
                acc[1] += vd * vd;
            }
        });
        if (d.Binv) {
            __syncthreads();
            block_apply(V, (T*)d.z, nullptr);
        }
        return team_reduce<2, NT>(tm, acc, out, NT);
    }

    // V_{j+1} = sc (K xin)_free
    __device__ __forceinline__ void product(int j, bool basis) {
        unsigned long long* tl = nullptr;
        if (a.tlog && products < (unsigned)a.tcap) {
            tl = a.tlog + 2 * products;
            if (threadIdx.x == 0) atomicMax(tl, ~gm_time());   // the first block's start
        }
        products++;
        const T* xin = basis ? V + (int64_t)j * ld : (const T*)d.z;
        const T sc = basis || d.Binv ? (T)scale[j] : (T)1;
        T* __restrict__ out = V + (int64_t)(j + 1) * ld;
        bool done = false;
        if constexpr (!D) {
            if (d.soff) {
                // a warp per slice, a lane per row, 16-byte loads of columns and values
                for (int s = w; s < nsl; s += NW) {
                    const int64_t r0 = slice(s), sl = r0 / 32;
                    if (r0 >= n) continue;
                    const int32_t o0 = __ldg(d.soff + sl), wd = (__ldg(d.soff + sl + 1) - o0) >> 7;   // chunks of 4
                    const int4* Cc = reinterpret_cast<const int4*>(d.scol + o0) + lane;
                    const float4* A = reinterpret_cast<const float4*>((const float*)d.K + o0) + lane;
                    float acc0 = 0.f, acc1 = 0.f;
                    int c = 0;
                    for (; c + 1 < wd; c += 2) {
                        const int4 c0 = __ldg(Cc + c * 32), c1 = __ldg(Cc + (c + 1) * 32);
                        const float4 a0 = __ldg(A + c * 32), a1 = __ldg(A + (c + 1) * 32);
                        acc0 = fmaf(a0.x, xin[c0.x], acc0);
                        acc1 = fmaf(a1.x, xin[c1.x], acc1);
                        acc0 = fmaf(a0.y, xin[c0.y], acc0);
                        acc1 = fmaf(a1.y, xin[c1.y], acc1);
                        acc0 = fmaf(a0.z, xin[c0.z], acc0);
                        acc1 = fmaf(a1.z, xin[c1.z], acc1);
                        acc0 = fmaf(a0.w, xin[c0.w], acc0);
                        acc1 = fmaf(a1.w, xin[c1.w], acc1);
                    }
                    if (c < wd) {
                        const int4 c0 = __ldg(Cc + c * 32);
                        const float4 a0 = __ldg(A + c * 32);
                        acc0 = fmaf(a0.x, xin[c0.x], acc0);
                        acc0 = fmaf(a0.y, xin[c0.y], acc0);
                        acc0 = fmaf(a0.z, xin[c0.z], acc0);
                        acc0 = fmaf(a0.w, xin[c0.w], acc0);
                    }
                    const int64_t r = r0 + lane;
                    if (r < n) out[r] = d.freed[r] ? (acc0 + acc1) * sc : 0.f;
                }
                done = true;
            }
        }
        if (!done)
            products_by<T>(d.tpr, (const T*)d.K, xin, [&](int64_t r, T v) { out[r] = d.freed[r] ? v * sc : (T)0; });
        if (tl) {
            __syncthreads();
            if (threadIdx.x == 0) atomicMax(tl + 1, gm_time());
        }
        __syncthreads();
    }

    // tab[k][wg] = V_k . w over the rows of warp wg of gw, for k in [k0, k0 + 8) or [k0, k0 + 4): float pairs
    // over the rows and through the lanes. One FP32 chain per lane, up to 111 products at 2.1 M rows, is three
    // times less exact there than the 14 products and FP64 lanes of a reduction spread over the chip: error
    // over |v||w| of random vectors 1.4e-10 against 5.8e-11 (and 1.0e-9 of both at 1,000 rows). The pairs' is
    // 1.3e-11 (6.2e-10); they cost nothing at 2.1 M rows (178.7 -> 176.6 us an iteration) and up to 3% of it
    // below 10^5 (21.7 -> 22.2 us at 79,507), 6% with element blocks, whose rows are read one at a time (49.3 ->
    // 52.2 at 307,200).
    __device__ __forceinline__ void lanes_to_tab(float h, float l, int k, int nv, int wg) {
#pragma unroll
        for (int off = 2; off > 0; off >>= 1) {
            const float oh = __shfl_xor_sync(0xffffffffu, h, off), ol = __shfl_xor_sync(0xffffffffu, l, off);
            ff_add(h, l, oh, ol);
        }
        if ((lane & 3) == 0 && k < nv) tab[k * ES + wg] = ff_wide(h, l);
    }
    __device__ __forceinline__ void dots8(const float* Vb, const float* W, int k0, int nv, int wg, int gw) {
        float h[8] = {0, 0, 0, 0, 0, 0, 0, 0}, l[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        for (int s = wg, c = 1; s < nsl; s += gw, c++) {
            const int64_t at = slice(s) + lane, r = min(at, n - 1);   // (a tile's rows may reach past n)
            const float wr = at < n ? W[r] : 0.f;
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; u++) v[u] = Vb[(int64_t)min(k0 + u, nv - 1) * ld + r];
#pragma unroll
            for (int u = 0; u < 8; u++) ff_mac(h[u], l[u], v[u], wr);
            if ((c & 7) == 0)
#pragma unroll
                for (int u = 0; u < 8; u++) ff_norm(h[u], l[u]);
        }
        gm_halve<4, 16>(h, l, lane);
        gm_halve<2, 8>(h, l, lane);
        gm_halve<1, 4>(h, l, lane);
        lanes_to_tab(h[0], l[0], k0 + ((lane & 16) ? 4 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 1 : 0), nv, wg);
    }
    __device__ __forceinline__ void dots4(const float* Vb, const float* W, int k0, int nv, int wg, int gw) {
        float h[4] = {0, 0, 0, 0}, l[4] = {0, 0, 0, 0};
        for (int s = 4 * wg, c = 1; s < nsl; s += 4 * gw, c++) {
            const int64_t r = slice(s) + 4 * lane;
            const float4 wr = *reinterpret_cast<const float4*>(W + r);
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; u++)
                v[u] = *reinterpret_cast<const float4*>(Vb + (int64_t)min(k0 + u, nv - 1) * ld + r);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                ff_mac(h[u], l[u], v[u].x, wr.x);
                ff_mac(h[u], l[u], v[u].y, wr.y);
                ff_mac(h[u], l[u], v[u].z, wr.z);
                ff_mac(h[u], l[u], v[u].w, wr.w);
            }
            if ((c & 7) == 0)
#pragma unroll
                for (int u = 0; u < 4; u++) ff_norm(h[u], l[u]);
        }
        gm_halve<2, 16>(h, l, lane);
        gm_halve<1, 8>(h, l, lane);
        {
            const float oh = __shfl_xor_sync(0xffffffffu, h[0], 4), ol = __shfl_xor_sync(0xffffffffu, l[0], 4);
            ff_add(h[0], l[0], oh, ol);
        }
        lanes_to_tab(h[0], l[0], (lane & 4) ? nv : k0 + ((lane & 16) ? 2 : 0) + ((lane & 8) ? 1 : 0), nv, wg);
    }

    // dsum[k] = V_k . w for k < nv (w = V_{j+1}; value j + 1 is |w|^2), over the team
    __device__ __forceinline__ bool dots(int j, int nv) {
        const T* W = V + (int64_t)(j + 1) * ld;
        for (int kb = 0; kb < nv; kb += 64) {
            const int nb = min(nv - kb, 64);
            const T* Vb = V + (int64_t)kb * ld;
            int E;
            if constexpr (D) {
                // groups of four warps (one per quarter of the SM) take eight values at a time
                const int grp = w >> 2, first = (w + grp) & 3;
                E = min(DT, max(32, nsl * 32));
                for (int k0 = grp * 8; k0 < nb; k0 += 2 * NW) {
                    double acc[8] = {};
                    // (loads past the last value repeat it: a branch around each would leave one in flight)
                    rows(first, 4, [&](int64_t r) {
                        const double wr = W[r];
                        double v[8];
#pragma unroll
                        for (int u = 0; u < 8; u++) v[u] = Vb[(int64_t)min(k0 + u, nb - 1) * ld + r];
#pragma unroll
                        for (int u = 0; u < 8; u++) acc[u] += v[u] * wr;
                    });
                    if (first * 32 < E)
#pragma unroll
                        for (int u = 0; u < 8; u++)
                            if (k0 + u < nb) tab[(k0 + u) * ES + first * 32 + lane] = acc[u];
                }
            } else {
                // four values of four rows per lane in tiles of 128 rows (a row at a time left the loads of L2
                // and HBM at 2.5 TB/s), eight of a row elsewhere; as many groups of warps as there are such
                // sets of values, at least four warps each (a warp's sum over its lanes costs as much as 40
                // rows)
                const bool vec = TS == 4;
                const int per = vec ? 4 : 8, sets = (nb + per - 1) / per;
                int gw = NW;
                while (gw > 4 && NW / gw < sets) gw >>= 1;
                E = min(gw, max(1, vec ? nsl / 4 : nsl));
                if (w % gw < E) {
                    if (vec)
                        for (int k0 = w / gw * 4; k0 < nb; k0 += NW / gw * 4) dots4(Vb, W, k0, nb, w % gw, gw);
                    else
                        for (int k0 = w / gw * 8; k0 < nb; k0 += NW / gw * 8) dots8(Vb, W, k0, nb, w % gw, gw);
                }
            }
            __syncthreads();
            gm_sum_rows(nb, E, [&](int k, int i) { return tab[k * ES + i]; },
                        [&](int k, double s) {
                            if (tm.size == 1) dsum[kb + k] = s;
                            else part[(int64_t)(kb + k) * tm.size + tm.rank] = s;
                        });
            if (kb + 64 < nv) __syncthreads();
        }
        if (tm.size > 1) {
            if (!team_barrier(tm)) return false;
            gm_sum_rows(nv, tm.size, [&](int k, int i) { return __ldcg(part + (int64_t)k * tm.size + i); },
                        [&](int k, double s) { dsum[k] = s; });
        }
        __syncthreads();
        return true;
    }

    // w -= sum_k h_k v_k over the owned rows, |w|^2 over the team; the last warp meanwhile rotates the
    // column hraw into hcol (all but its last rotation)
    __device__ __forceinline__ bool orthogonalise(int j, double* hn2) {
        T* W = V + (int64_t)(j + 1) * ld;
        double acc[1] = {0};
        float fh = 0.f, fl = 0.f;
        if (w == NW - 1) {
            // the two products that do not wait for the chain first, a lane per rotation; then the chain, one
            // FMA and one shuffle per rotation: lane 0 the rotated entry, lane 1 the one carried on
            double* carry = dsum;   // the sums are done with
            for (int k = lane; k < j; k += 32) {
                const double hi = hraw[k + 1];
                hcol[k] = sn[k] * hi;
                carry[k] = cs[k] * hi;
            }
            __syncwarp();
            double h = hraw[0];
#pragma unroll 4
            for (int k = 0; k < j; k++) {
                const double c = lane == 1 ? -sn[k] : cs[k], pre = lane == 1 ? carry[k] : hcol[k];
                const double v = fma(c, h, pre);
                if (lane == 0) hcol[k] = v;
                h = __shfl_sync(0xffffffffu, v, 1);
            }
            if (lane == 0) hcol[j] = h;
        } else {
            const double* coef = tab;   // the partial sums are done with
            T ah = 0, al = 0;
            bool done = false;
            if constexpr (!D) {
                if (TS == 4) {
                    tiles4(w, NW - 1, [&](int64_t r) {
                        float4 x = *reinterpret_cast<const float4*>(W + r);
                        for (int k = 0; k <= j; k += 4) {
                            float4 v[4];
#pragma unroll
                            for (int u = 0; u < 4; u++)
                                v[u] = *reinterpret_cast<const float4*>(V + (int64_t)min(k + u, j) * ld + r);
#pragma unroll
                            for (int u = 0; u < 4; u++) {
                                const float c = -((const float*)coef)[k + u];
                                x.x = fmaf(c, v[u].x, x.x);
                                x.y = fmaf(c, v[u].y, x.y);
                                x.z = fmaf(c, v[u].z, x.z);
                                x.w = fmaf(c, v[u].w, x.w);
                            }
                        }
                        // the padding past n stays zero whatever the coefficients (a NaN there would outlive
                        // the solve: nothing else writes it)
                        if (r + 3 >= n) {
                            if (r >= n) x.x = 0.f;
                            if (r + 1 >= n) x.y = 0.f;
                            if (r + 2 >= n) x.z = 0.f;
                            x.w = 0.f;
                        }
                        *reinterpret_cast<float4*>(W + r) = x;
                        ff_mac(ah, al, x.x, x.x);
                        ff_mac(ah, al, x.y, x.y);
                        ff_mac(ah, al, x.z, x.z);
                        ff_mac(ah, al, x.w, x.w);
                        ff_norm(ah, al);
                    });
                    done = true;
                }
            }
            if (!done) rows(w, NW - 1, [&](int64_t r) {
                T w0 = W[r], w1 = 0;
                for (int k = 0; k <= j; k += 8) {   // (coefficients past j are 0)
                    T v[8];
#pragma unroll
                    for (int u = 0; u < 8; u++) v[u] = V[(int64_t)min(k + u, j) * ld + r];
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        (u & 1 ? w1 : w0) -= ((const T*)coef)[k + u] * v[u];
                }
                w0 += w1;
                W[r] = w0;
                if constexpr (D) ah += w0 * w0;
                else {
                    ff_mac(ah, al, w0, w0);
                    ff_norm(ah, al);
                }
            });
            if constexpr (D) acc[0] = ah;
            else fh = ah, fl = al;
        }
        if (d.Binv) {
            __syncthreads();
            block_apply(W, (T*)d.z, nullptr);
        }
        if constexpr (D) return team_reduce<1, NT>(tm, acc, hn2, live);
        else return team_reduce_ff<NT>(tm, fh, fl, hn2);
    }

    // Residual and start of a cycle; false when the team gave up. Sets `beta`, `nb`, `res`.
    double nb, beta, res, target;
    __device__ __forceinline__ bool begin(bool first) {
        double s[2];
        if (!residual(first, s)) return false;
        beta = isfinite(s[0]) ? sqrt(fmax(s[0], 0.0)) : (double)NAN;
        if (first) {
            const double b = isfinite(s[1]) ? sqrt(fmax(s[1], 0.0)) : (double)NAN;
            nb = (b > 0 || !isfinite(b)) ? b : 1.0;
        }
        res = beta / nb;
        // stop the cycle at the outer tolerance (with a margin: the cycle's residual estimate is accurate
        // to far below it, and the FP64 residual of the result is checked after the cycle), or at the
        // inner reduction for mixed precision
        target = fmax(kTargetMargin * d.tol * nb, d.inner * beta);
        if (threadIdx.x == 0) {
            g[0] = beta;
            scale[0] = beta > 0 ? 1.0 / beta : 0.0;
        }
        __syncthreads();
        return true;
    }

    // One iteration: 0 go on, 1 the cycle ends, 2 the team gave up. bits: GM_NONFIN, GM_BREAK; jd: columns
    int *s_end, *s_bits;
    __device__ __forceinline__ int iteration(int j, bool basis, int* bits, int* jd) {
        const int m = a.m;
        product(j, basis);
        double nw2 = 0, hn2 = 0;
        for (int pass = 1; pass <= 2; pass++) {
            if (!dots(j, pass == 1 ? j + 2 : j + 1)) return 2;
            if (pass == 1) nw2 = dsum[j + 1];
            for (int k = threadIdx.x; k < (j | 7) + 1; k += NT) {
                const double h = k <= j ? dsum[k] * scale[k] : 0.0;
                if (k <= j) hraw[k] = pass == 1 ? h : hraw[k] + h;
                ((T*)tab)[k] = (T)(k <= j ? h * scale[k] : 0.0);
            }
            __syncthreads();
            if (!orthogonalise(j, &hn2)) return 2;
            if (!(hn2 < kReorth * nw2)) break;   // (NaN ends here and is found below)
        }
        if (threadIdx.x == 0) {
            // the last rotation, the residual estimate and the next basis vector's scale
            const double q2 = isfinite(hn2) ? fmax(hn2, 0.0) : (double)NAN;
            const double ri = q2 > 0 ? rsqrt(q2) : 0.0, hn = q2 > 0 ? q2 * ri : q2;
            const double h = hcol[j], d2 = h * h + q2;
            int e = 0, bt = 0;
            if (!isfinite(d2)) {
                bt = GM_NONFIN;   // column j is dropped
                e = 1;
            } else if (d2 == 0.0) {
                bt = GM_BREAK;
                e = 1;
            } else {
                const double rd = rsqrt(d2), c = h * rd, s = hn * rd;
                cs[j] = c;
                sn[j] = s;
                R[j * (j + 1) / 2 + j] = d2 * rd;
                const double gj = g[j];
                g[j] = c * gj;
                g[j + 1] = -s * gj;
                scale[j + 1] = ri;
                e = fabs(s * gj) <= target || hn == 0.0 || j + 1 >= m ? 1 : 0;
            }
            *s_end = e;
            *s_bits = bt;
        } else if (w == 1)
            for (int k = lane; k < j; k += 32) R[j * (j + 1) / 2 + k] = hcol[k];
        __syncthreads();
        const int e = *s_end, bt = *s_bits;
        *bits |= bt;
        if (!bt) *jd = j + 1;
        __syncthreads();
        return e;
    }

    // u = sum_k y_k v_k with R y = g over the completed columns; x += D^-1 u, or B^-1 u, or z = u
    __device__ __forceinline__ void combine(int jd, bool to_z) {
        T* z = (T*)d.z;
        if (jd == 0) {
            if (to_z) rows(w, NW, [&](int64_t r) { z[r] = (T)0; });
            return;
        }
        T* cf = (T*)tab;
        if (w == 0) {
            // back substitution, a warp per column: y in hraw, the reciprocal pivots in hcol
            for (int k = lane; k < jd; k += 32) {
                hraw[k] = g[k];
                hcol[k] = 1.0 / R[k * (k + 1) / 2 + k];
            }
            __syncwarp();
            for (int k = jd - 1; k >= 0; k--) {
                const double y = hraw[k] * hcol[k];
                const double* col = R + k * (k + 1) / 2;
                for (int l = lane; l < k; l += 32) hraw[l] -= col[l] * y;
                if (lane == 0) cf[k] = (T)(y * scale[k]);
                __syncwarp();
            }
            for (int k = jd + lane; k < (jd + 7) / 8 * 8; k += 32) cf[k] = (T)0;
        }
        __syncthreads();
        const T* dinv = (const T*)d.dinv;
        const bool blk = d.Binv != nullptr && !to_z;
        if constexpr (!D) {
            if (TS == 4 && !blk) {
                tiles4(w, NW, [&](int64_t r) {
                    float acc[4] = {};
                    for (int k = 0; k < jd; k += 4) {
                        float4 v[4];
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            v[u] = *reinterpret_cast<const float4*>(V + (int64_t)min(k + u, jd - 1) * ld + r);
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const float c = cf[k + u];
                            acc[0] = fmaf(c, v[u].x, acc[0]);
                            acc[1] = fmaf(c, v[u].y, acc[1]);
                            acc[2] = fmaf(c, v[u].z, acc[2]);
                            acc[3] = fmaf(c, v[u].w, acc[3]);
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (r + u < n) {
                            if (to_z) z[r + u] = acc[u];
                            else d.x[r + u] += (double)(dinv ? dinv[r + u] * acc[u] : acc[u]);
                        }
                });
                return;
            }
        }
        rows(w, NW, [&](int64_t r) {
            T acc = 0, acc1 = 0;
            for (int k = 0; k < jd; k += 8) {
                T v[8];
#pragma unroll
                for (int u = 0; u < 8; u++) v[u] = V[(int64_t)min(k + u, jd - 1) * ld + r];
#pragma unroll
                for (int u = 0; u < 8; u++) (u & 1 ? acc1 : acc) += cf[k + u] * v[u];
            }
            acc += acc1;
            if (to_z || blk) z[r] = acc;
            else d.x[r] += (double)(dinv ? dinv[r] * acc : acc);
        });
        if (blk) {
            __syncthreads();
            block_apply(z, nullptr, d.x);
        }
    }

    // the whole solve
    __device__ __forceinline__ bool solve() {
        int iters = 0, cycles = 0, bits = 0;
        if (!begin(true)) return false;
        const double res0 = res;
        if (!isfinite(beta)) bits |= GM_NONFIN;
        while (!(bits & GM_NONFIN) && !(res <= d.tol) && iters < d.maxit) {
            int jd = 0;
            for (int j = 0; j < a.m; j++) {
                const int e = iteration(j, d.Binv == nullptr, &bits, &jd);
                if (e == 2) return false;
                iters++;
                if (e || iters >= d.maxit) break;
            }
            combine(jd, false);
            if (!team_barrier(tm)) return false;
            if (!begin(false)) return false;
            if (!isfinite(beta)) bits |= GM_NONFIN;
            cycles++;
        }
        if (tm.rank == 0 && threadIdx.x == 0) {
            d.out->res0 = res0;
            d.out->res = res;
            d.out->iters = iters;
            d.out->cycles = cycles;
            d.out->bits = bits;
        }
        return true;
    }

    // a phase of a solve whose preconditioner runs in other kernels; the small state travels in d.small
    __device__ __forceinline__ bool phase() {
        int* fl = d.out->flags;
        const int m = a.m;
        double *sg = d.small + m * (m + 1) / 2, *st = d.small + gm_small_doubles(m) - 4;   // cs, sn, g, scale; nb, target
        if (a.mode == GM_FIRST || a.mode == GM_START) {
            if (a.mode == GM_START) {
                if (fl[F_OUTER]) return true;
                nb = st[0];
            }
            if (!begin(a.mode == GM_FIRST)) return false;
            if (tm.rank == 0 && threadIdx.x == 0) {
                st[0] = nb;
                st[1] = target;
                sg[2 * m] = g[0];
                sg[3 * m + 2] = scale[0];
                const bool bad = !isfinite(beta), done = bad || res <= d.tol;
                fl[F_JDONE] = 0;
                fl[F_CONV] = fl[F_OUTER] = done;
                if (a.mode == GM_FIRST) {
                    d.out->res0 = res;
                    fl[F_BREAK] = fl[F_NONFIN] = fl[F_ITERS] = 0;
                }
                if (bad) fl[F_NONFIN] = 1;
                d.out->res = res;
            }
            return true;
        }
        if (a.mode == GM_ITER) {
            if (fl[F_CONV]) return true;
            const int j = a.j;
            for (int k = threadIdx.x; k <= j; k += NT) {
                if (k < j) {
                    cs[k] = sg[k];
                    sn[k] = sg[m + k];
                }
                scale[k] = sg[3 * m + 2 + k];
            }
            if (threadIdx.x == 0) g[j] = sg[2 * m + j];
            target = st[1];
            __syncthreads();
            int bits = 0, jd = j;
            const int e = iteration(j, false, &bits, &jd);
            if (e == 2) return false;
            if (tm.rank == 0) {
                // (every block has read the flags: the iteration's exchanges are behind it)
                for (int k = threadIdx.x; k <= j; k += NT) d.small[j * (j + 1) / 2 + k] = R[j * (j + 1) / 2 + k];
                if (threadIdx.x == 0) {
                    sg[j] = cs[j];
                    sg[m + j] = sn[j];
                    sg[2 * m + j] = g[j];
                    sg[2 * m + j + 1] = g[j + 1];
                    sg[3 * m + 2 + j + 1] = scale[j + 1];
                    fl[F_JDONE] = jd;
                    fl[F_ITERS]++;
                    if (bits & GM_NONFIN) fl[F_NONFIN] = 1;
                    if (bits & GM_BREAK) fl[F_BREAK] = 1;
                    if (e) fl[F_CONV] = 1;
                }
            }
            return true;
        }
        const int jd = fl[F_JDONE];
        for (int k = threadIdx.x; k < jd * (jd + 1) / 2; k += NT) R[k] = d.small[k];
        for (int k = threadIdx.x; k < jd; k += NT) {
            g[k] = sg[2 * m + k];
            scale[k] = sg[3 * m + 2 + k];
        }
        __syncthreads();
        combine(jd, true);
        return true;
    }
};

// MANY: teams that take systems from their queue
template <class T, int NT, bool MANY = false>
__global__ void __launch_bounds__(NT, NT == kGmSmallThreads ? 4 : 1) gm_kernel(const __grid_constant__ GmArgs a) {
    extern __shared__ double gm_smem[];
    __shared__ int s_end, s_bits, s_next;
    __shared__ GmInst s_inst;
    auto fetch = [&](int i) {   // the system's descriptor: read on every access otherwise
        const int* src = reinterpret_cast<const int*>(a.list ? a.list + i : &a.one);
        for (int k = threadIdx.x; k < (int)(sizeof(GmInst) / 4); k += blockDim.x) reinterpret_cast<int*>(&s_inst)[k] = src[k];
        __syncthreads();
    };
    int4 at = make_int4(0, (int)blockIdx.x, (int)gridDim.x, 0);   // team, rank, size, instance
    if (a.map) at = a.map[blockIdx.x];
    else if (a.queue) at.w = -1;
    if constexpr (MANY) {
        if (at.w == -2) {
            Team tm = team_join(a.teams + at.x, at.y, at.z);
            double* part = a.part + (int64_t)(blockIdx.x - at.y) * (a.m + 2);
            while (true) {
                if (at.y == 0 && threadIdx.x == 0) a.teams[at.x].next = atomicAdd(a.queue + 1, 1);
                if (!team_barrier(tm)) {
                    if (threadIdx.x == 0) atomicExch(&a.list[0].out->gaveup, 1);
                    return;
                }
                const int q = __ldcg(&a.teams[at.x].next);
                if (q >= a.nteam) break;
                fetch(a.queue_inst[q]);
                GmRun<T, NT> run(a, s_inst, tm, gm_smem, part);
                run.s_end = &s_end;
                run.s_bits = &s_bits;
                if (!run.solve()) {
                    if (threadIdx.x == 0) atomicExch(&run.d.out->gaveup, 1);
                    return;
                }
                __syncthreads();   // the descriptor is read to the end of the solve
            }
            team_leave(tm);
        }
    } else if (at.w >= 0) {
        fetch(at.w);
        Team tm = team_join(a.teams + at.x, at.y, at.z);
        GmRun<T, NT> run(a, s_inst, tm, gm_smem, a.part + (int64_t)(a.map ? blockIdx.x - at.y : 0) * (a.m + 2));
        run.s_end = &s_end;
        run.s_bits = &s_bits;
        if (!(a.mode == GM_FULL ? run.solve() : run.phase())) {
            if (threadIdx.x == 0) atomicExch(&run.d.out->gaveup, 1);
            return;
        }
        team_leave(tm);
    }
    if (!a.queue) return;
    // then the blocks by themselves: the systems too small for a team, largest first
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) s_next = atomicAdd(a.queue, 1);
        __syncthreads();
        const int q = s_next;
        if (q >= a.nqueue) return;
        fetch(a.queue_inst[a.nteam + q]);
        Team tm = team_join(nullptr, 0, 1);
        GmRun<T, NT> run(a, s_inst, tm, gm_smem, nullptr);
        run.s_end = &s_end;
        run.s_bits = &s_bits;
        run.solve();
    }
}

// The kernels for queues of systems of few rows and for teams with a queue (translation units of their own).
template <class T>
const void* gm_small_kernel();
template <class T>
const void* gm_many_kernel();

}  // namespace ocmp
