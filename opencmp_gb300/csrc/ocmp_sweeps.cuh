// The block elimination's two sweeps over the strips as one cooperative launch: forward
// y_k = G_k (b_k - A_k,p y_p), p the neighbour farther from the middle strip (both, for that one),
// backward x_k = y_k - G_k A_k,q x_q, q the nearer one: from both ends to the middle and back, one step
// per pair of strips and sweep, each a dense matrix-vector product whose right-hand side needs the step
// before. Half of the blocks take either strip of a pair.
//
// What bounds a step is the way from one block's result to the next step's right-hand side, not the
// bytes: a strip of 1,152 dofs holds 5.3 MB, 1.2 us of L2 or 0.8 us of HBM, and none of them depends on
// the step before. So
//  - each block owns the same rows of a strip in both sweeps and fetches them, with the step's coupling
//    lists, by bulk copies into a ring of shared-memory stages, up to four steps ahead;
//  - there is no barrier between the blocks: a result is stored as one 8-byte word with the launch's
//    epoch, and every block polls just the interface dofs that it needs, into shared memory. A barrier
//    costs the stores' acknowledgement, the counter and the reload, 5,500 clocks with the gather;
//  - every block makes the whole right-hand side for itself (a few entries per dof of the interface)
//    instead of paying a second exchange. The vector is scaled and rounded once, each block its share (an
//    FP64 instruction takes its pipe for 64 clocks), and read as such words as well;
//  - the few loads of a step that go to registers are issued one or two steps ahead.
//
// Measured (us per preconditioner application): 16,641 pressure dofs in 17 strips 226 -> 85 in one launch
// -> 49 from both ends; 110,592 in 96 strips 1,430 -> 690 -> 314 (one stage, a padded strip's rows) -> 290
// (two, its real rows in one or two copies) -> 279 (an entry's loads not waiting for another's); before, two
// launches per strip and sweep, replayed from a graph. A step is 5,000 clocks: 1,500 until the polled results are there, 1,500 for the product, the rest the gather,
// the stores and the block's own barriers.
#pragma once

#include "ocmp_mbar.cuh"
#include "ocmp_team.cuh"

namespace ocmp {

constexpr int kSweepWarps = 16;
constexpr int kSweepThreads = 32 * kSweepWarps;
constexpr int kSweepStages = 4;
constexpr int kSweepValues = 3;              // values of the vector held in registers per thread
constexpr int kSweepAhead = 8;               // descriptors are loaded so many steps ahead
constexpr int kSweepSmem = 227 * 1024 - 2048;
constexpr int kSweepMinRows = 4;             // rows of a block of the largest strip, at least
constexpr long long kSweepWaitCycles = 8000000000LL;

// One strip in one sweep. Its lists couple positions to the strip before: jd, the dofs that the step
// polls; cq, the list's positions; per position len entries, entry-major, of an index into jd (0xffff on
// padding) and a value (0 where a dof is constrained).
struct SweepStep {
    const float* G;
    int64_t blob;               // the lists, in words: values, jd, then 16-bit indices and positions
    int32_t words, p0;          // their words (a multiple of 32; 0: read in place); the strip's first position
    int32_t mp, cnt, len, nj;
    int32_t per, ns, lwg, gs;   // rows of a block, of which staged; log2 of the warps per group of 8 rows; blocks
    int32_t m, nN, gap, pad;    // rows without the padding: row r is position r, from nN on r + gap
};
__device__ __forceinline__ int sweep_position(const SweepStep& s, int r) { return r < s.nN ? r : r + s.gap; }

// `left` blocks are done with this launch; the last one counts the epoch on. starve (a test): the first
// block of the next launch keeps its share of the vector to itself.
struct SweepState {
    unsigned epoch, left;
    int abort, starve;   // side by side: a wait gets the address of the first
};

struct SweepArgs {
    const SweepStep* steps;   // two per step: the first group's strip and the second's (gs 0: none)
    int nsteps, nfwd;         // the last forward step's result is final
    const int32_t* prow;      // per position: its dof, -1 on padding
    const int32_t* rdof;      // the same, -1 also on constrained dofs
    const uint32_t* blob;
    uint2* b;                 // per dof, each with the epoch: the vector, the forward results, the final ones
    uint2* y;
    uint2* x;
    SweepState* state;
    int* err;                 // set when a wait gave up
    int64_t n;
    int stages, stage;        // the ring: stages of so many floats
    int rows;                 // largest number of rows of a block
    int mp_max, nj_max;
};

struct SweepLists {
    int32_t jd, idx, cq, words;   // offsets in words; the values come first
};
__host__ __device__ __forceinline__ SweepLists sweep_lists(int cnt, int len, int nj) {
    SweepLists l;
    l.jd = cnt * len;
    l.idx = l.jd + nj;
    l.cq = l.idx + (cnt * len + 1) / 2;
    l.words = (l.cq + (cnt + 1) / 2 + 31) & ~31;
    return l;
}

inline size_t sweep_fixed_smem(int mp_max, int nj_max, int rows) {
    return sizeof(float) * ((size_t)mp_max + (nj_max + 31) / 32 * 32 + (size_t)rows * kSweepWarps) + 8 * kSweepStages;
}

// rows of a strip that a block of a group of gs takes
inline int sweep_rows(int m, int gs) { return (m + gs - 1) / gs; }

// Rows against r, up to 8: a warp takes every wg-th group of 128 columns. In global memory the rows from
// the split-th on lie gap rows further.
template <bool SM>
__device__ __forceinline__ void sweep_rows8(const float* g, int mp, int nrow, int split, int gap, const float4* r,
                                            int part, int lwg, int lane, float acc[8]) {
    const int nq = mp >> 2;
    for (int q = part * 32 + lane; q < nq; q += 32 << lwg) {
        const float4 b = r[q];
#pragma unroll
        for (int h = 0; h < 8; h += 4) {
            float4 a[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int64_t at = SM || h + u < split ? h + u : h + u + gap;
                const float4* p = reinterpret_cast<const float4*>(g + at * mp) + q;
                a[u] = h + u >= nrow ? make_float4(0.f, 0.f, 0.f, 0.f) : SM ? *p : __ldcs(p);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                acc[h + u] = fmaf(a[u].x, b.x, acc[h + u]);
                acc[h + u] = fmaf(a[u].y, b.y, acc[h + u]);
                acc[h + u] = fmaf(a[u].z, b.z, acc[h + u]);
                acc[h + u] = fmaf(a[u].w, b.w, acc[h + u]);
            }
        }
    }
}

// The word of a dof once it carries the epoch; false when the wait gave up.
__device__ __forceinline__ bool sweep_poll(const uint2* p, unsigned epoch, volatile int* abort, float* out) {
    long long t0 = 0;
    for (unsigned spin = 1;; spin++) {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
        if ((unsigned)(v >> 32) == epoch) {
            *out = __uint_as_float((unsigned)v);
            return true;
        }
        if (spin & 63u) continue;
        if (*abort) return false;
        if (t0 == 0) t0 = clock64();
        else if (clock64() - t0 > (abort[1] ? kStarvedCycles : kSweepWaitCycles)) return false;
    }
}
__device__ __forceinline__ void sweep_put(uint2* p, float v, unsigned epoch) {
    const unsigned long long w = ((unsigned long long)epoch << 32) | __float_as_uint(v);
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"(w) : "memory");
}

template <class T>
__global__ void __launch_bounds__(kSweepThreads, 1)
    k_sweeps(const SweepArgs a, const T* v, const double* scale, int j, T* z, const int* flags) {
    extern __shared__ __align__(128) float sweep_smem[];
    __shared__ SweepStep desc[2 * kSweepAhead];
    if (flags && flags[0]) return;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    float* ring = sweep_smem;
    float* rs = ring + (int64_t)a.stages * a.stage;
    float* part = rs + a.mp_max;
    float* js = part + a.rows * kSweepWarps;
    const uint32_t full = saddr(js + (a.nj_max + 31) / 32 * 32);
    const int size = gridDim.x, half = size >> 1, block = blockIdx.x;
    // this block's strip of a step: the second group's, where there is one
    auto source = [&](int t) {
        const SweepStep* s = a.steps + 2 * (int64_t)t;
        return s + (block >= half && __ldg(&s[1].gs) > 0);
    };
    if (tid < kSweepAhead && tid < a.nsteps) desc[tid] = *source(tid);
    if (tid == 0) {
        for (int i = 0; i < a.stages; i++) mbar_init(full + 8 * i, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const unsigned epoch = *(volatile unsigned*)&a.state->epoch + 1u;
    volatile int* abort = &a.state->abort;
    __syncthreads();
    auto at = [&](int t) -> const SweepStep& { return desc[t & (2 * kSweepAhead - 1)]; };
    auto rows_of = [&](const SweepStep& s, int* r0) {
        *r0 = min(s.m, (s.gs == size || block < half ? block : block - half) * s.per);
        return min(s.per, s.m - *r0);
    };
    // the copies of a step into its stage
    auto fetch = [&](int t, int i) {
        const SweepStep& s = at(t);
        int r0;
        const int mp = s.mp, nr = min(rows_of(s, &r0), s.ns), words = s.words;
        const uint32_t dst = saddr(ring + (int64_t)i * a.stage), row = dst + words * 4;
        mbar_expect_tx(full + 8 * i, (uint32_t)(nr * mp + words) * 4);
        if (words) bulk_load(dst, a.blob + s.blob, words * 4, full + 8 * i);
        // the rows are contiguous but for the padding between the two parts of the strip
        const int n0 = max(0, min(nr, s.nN - r0)), n1 = nr - n0;
        if (n0 > 0) bulk_load(row, s.G + (int64_t)r0 * mp, n0 * mp * 4, full + 8 * i);
        if (n1 > 0) bulk_load(row + n0 * mp * 4, s.G + (int64_t)(r0 + n0 + s.gap) * mp, n1 * mp * 4, full + 8 * i);
    };
    constexpr int kFetcher = kSweepThreads - 1, kLoader = kSweepThreads - 64;
    if (tid == kFetcher)
        for (int t = 0; t < min(a.stages, a.nsteps); t++) fetch(t, t);
    {
        const double sc = scale ? scale[j] : 1.0;
        const int64_t n = block == 0 && abort[1] ? 0 : a.n;
        for (int64_t q = block * (int64_t)kSweepThreads + tid; q < n; q += (int64_t)size * kSweepThreads)
            sweep_put(a.b + q, scale ? (float)(T)((double)v[q] * sc) : (float)v[q], epoch);
    }

    // the dofs of this thread's positions of a step (-1 also where the vector has no part), their values
    int32_t vd[kSweepValues];
    unsigned long long vx[kSweepValues];
    auto load_dofs = [&](int t) {
#pragma unroll
        for (int u = 0; u < kSweepValues; u++) {
            const int q = tid + u * kSweepThreads;
            vd[u] = t < a.nfwd && q < at(t).mp ? __ldg(a.rdof + at(t).p0 + q) : -1;
        }
    };
    auto load_values = [&]() {
#pragma unroll
        for (int u = 0; u < kSweepValues; u++)
            if (vd[u] >= 0)
                asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(vx[u]) : "l"(a.b + vd[u]) : "memory");
    };
    // `from`: the dofs that the values were loaded for
    auto put_values = [&](int t, const int32_t* from) {
        const SweepStep& s = at(t);
        bool got = true;
#pragma unroll
        for (int u = 0; u < kSweepValues; u++) {
            const int q = tid + u * kSweepThreads;
            float x = 0.f;
            if (from[u] >= 0) {
                x = __uint_as_float((unsigned)vx[u]);
                if ((unsigned)(vx[u] >> 32) != epoch) got = got && sweep_poll(a.b + from[u], epoch, abort, &x);
            }
            if (q < s.mp) rs[q] = x;
        }
        for (int q = tid + kSweepValues * kSweepThreads; q < s.mp; q += kSweepThreads) {
            const int32_t d = t < a.nfwd ? __ldg(a.rdof + s.p0 + q) : -1;
            float x = 0.f;
            if (d >= 0) got = got && sweep_poll(a.b + d, epoch, abort, &x);
            rs[q] = x;
        }
        return got;
    };
    // the dof whose result this thread stores
    auto load_row = [&](int t) {
        int r0;
        const int nr = rows_of(at(t), &r0);
        return tid < nr ? __ldg(a.prow + at(t).p0 + sweep_position(at(t), r0 + tid)) : -1;
    };

    load_dofs(0);
    load_values();
    bool ok = put_values(0, vd);
    int32_t dof = load_row(0), dof1 = -1;
    if (a.nsteps > 1) {
        load_dofs(1);
        dof1 = load_row(1);
    }
    float own = 0.f;
    int fetched = min(a.stages, a.nsteps);
    for (int t = 0, i = 0, ph = 0; t < a.nsteps; t++) {
        const SweepStep& s = at(t);
        const int mode = t < a.nfwd ? 0 : 1, mp = s.mp, cnt = s.cnt, len = s.len, nj = s.nj;
        const bool more = t + 1 < a.nsteps, load = t + kSweepAhead < a.nsteps && tid >= kLoader &&
                                                  tid < kLoader + (int)(sizeof(SweepStep) / 4);
        int r0;
        const int nr = rows_of(s, &r0);
        const float* stage = ring + i * a.stage;
        const SweepLists li = sweep_lists(cnt, len, nj);
        const uint32_t* list = s.words ? reinterpret_cast<const uint32_t*>(stage) : a.blob + s.blob;
        // what nothing waits for before the end of this step: a descriptor, the next step's values,
        // this thread's own result of the forward sweep
        int32_t word = 0, was[kSweepValues];
        if (load) word = __ldg(reinterpret_cast<const int32_t*>(source(t + kSweepAhead)) + tid - kLoader);
        if (more) load_values();
#pragma unroll
        for (int u = 0; u < kSweepValues; u++) was[u] = vd[u];
        const float own1 = more && t + 1 >= a.nfwd && dof1 >= 0 ? __uint_as_float(a.y[dof1].x) : 0.f;
        if (ok) ok = mbar_wait(full + 8 * i, ph, abort);
        if (nr > 0) {
            const uint2* src = mode == 0 ? a.y : a.x;
            for (int q = tid; q < nj && ok; q += kSweepThreads)
                ok = sweep_poll(src + (int32_t)list[li.jd + q], epoch, abort, js + q);
        }
        ok = __syncthreads_and(ok);
        if (!ok) break;
        // r: minus (forward) or plus (backward) the couplings to the strip before; an entry's loads do not
        // wait for another's
        auto couple = [&](const uint32_t* l) {
            const float* val = reinterpret_cast<const float*>(l);
            const uint16_t* idx = reinterpret_cast<const uint16_t*>(l + li.idx);
            const uint16_t* cq = reinterpret_cast<const uint16_t*>(l + li.cq);
            for (int c = tid; c < cnt; c += kSweepThreads) {
                float acc = 0.f;
#pragma unroll 6
                for (int e = 0; e < len; e++) {
                    const int k = idx[e * cnt + c];
                    const float v0 = val[e * cnt + c], g = js[k == 0xffff ? 0 : k];
                    acc = k == 0xffff ? acc : fmaf(v0, g, acc);
                }
                float* r = rs + cq[c];
                *r = mode == 0 ? *r - acc : acc;
            }
        };
        if (nr > 0) {
            if (s.words) couple(reinterpret_cast<const uint32_t*>(stage));
            else couple(a.blob + s.blob);
        }
        int32_t dof2 = -1;
        if (t + 2 < a.nsteps) {
            load_dofs(t + 2);
            dof2 = load_row(t + 2);
        }
        __syncthreads();
        // the product: groups of 8 rows, first those in shared memory, then what did not fit
        const int ns = min(nr, s.ns), g1 = (ns + 7) >> 3, ng = g1 + ((nr - ns + 7) >> 3), lwg = s.lwg;
        const int wg = 1 << lwg, slots = kSweepWarps >> lwg, pt = w & (wg - 1);
        for (int gr = w >> lwg; gr < ng; gr += slots) {
            const int row = gr < g1 ? 8 * gr : ns + 8 * (gr - g1), nrow = min(8, (gr < g1 ? ns : nr) - row);
            float acc[8] = {};
            if (gr < g1)
                sweep_rows8<true>(stage + s.words + row * mp, mp, nrow, s.nN, 0, reinterpret_cast<const float4*>(rs), pt, lwg,
                                  lane, acc);
            else
                sweep_rows8<false>(s.G + (int64_t)(r0 + row) * mp, mp, nrow, s.nN - r0 - row, s.gap,
                                   reinterpret_cast<const float4*>(rs), pt, lwg, lane, acc);
            // 8 sums over 32 lanes: halve the values three times, then two plain steps
#pragma unroll
            for (int o = 16, h = 4; h > 0; o >>= 1, h >>= 1)
#pragma unroll
                for (int u = 0; u < h; u++) {
                    const bool up = lane & o;
                    const float give = up ? acc[u] : acc[u + h], keep = up ? acc[u + h] : acc[u];
                    acc[u] = keep + __shfl_xor_sync(0xffffffffu, give, o);
                }
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 2);
            acc[0] += __shfl_xor_sync(0xffffffffu, acc[0], 1);
            const int u = (lane >> 4 & 1) * 4 + (lane >> 3 & 1) * 2 + (lane >> 2 & 1);
            if ((lane & 3) == 0 && u < nrow) part[(row + u) * kSweepWarps + pt] = acc[0];
        }
        __syncthreads();
        if (dof >= 0) {
            float acc = 0.f;
            for (int q = 0; q < wg; q++) acc += part[tid * kSweepWarps + q];
            if (mode == 1) acc = own - acc;
            sweep_put((t >= a.nfwd - 1 ? a.x : a.y) + dof, acc, epoch);
            if (t >= a.nfwd - 1) z[dof] = (T)acc;
        }
        if (tid == kFetcher && fetched < a.nsteps) fetch(fetched++, i);
        if (load) reinterpret_cast<int32_t*>(&desc[(t + kSweepAhead) & (2 * kSweepAhead - 1)])[tid - kLoader] = word;
        if (more) ok = put_values(t + 1, was);
        dof = dof1;
        dof1 = dof2;
        own = own1;
        if (++i == a.stages) {
            i = 0;
            ph ^= 1;
        }
    }
    if (!ok) {
        if (tid == 0) {
            atomicExch(&a.state->abort, 1);
            if (a.err) atomicExch(a.err, 1);
        }
        // the copies in flight: the last one of each stage
        if (tid == kFetcher)
            for (int q = max(0, fetched - a.stages); q < fetched; q++) {
                const long long t0 = clock64();
                while (!mbar_try(full + 8 * (q % a.stages), (q / a.stages) & 1) && clock64() - t0 < kWaitCycles) {
                }
            }
        return;
    }
    if (tid == 0) {
        __threadfence();
        if (atomicAdd(&a.state->left, 1u) == (unsigned)size - 1u) {
            a.state->left = 0;
            a.state->epoch = epoch;
        }
    }
}

}  // namespace ocmp
