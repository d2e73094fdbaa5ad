// Building blocks of the persistent Krylov kernels (sm_103a): a solve runs in one cooperative launch
// by a team of co-resident blocks, one per SM at most, that exchange their partial sums through
// global memory.
//
// What bounds such a solve is latency, measured on this part (clocks at 2.07 GHz):
//  - a warp-wide FP64 instruction takes its SM quarter's pipe for 64 clocks, however few lanes are
//    active, so a butterfly of five additions costs 600, and 1,800 when 16 warps do it. team_list_sum
//    adds as integers instead: the values are aligned to the largest exponent, cut into three limbs
//    and added by redux.sync (hardware integer reductions), 380 clocks for 32 values and 570 when 16
//    warps do it. At least 69 bits below the largest value are kept and the total is rounded once, so
//    the sum is at least as exact as any order of FP64 additions, and does not depend on the order;
//  - a barrier on one counter in global memory takes 2,430 clocks among 152 blocks (2,250 among 16),
//    where polling every block's own slot took 7,500: the polls hold up the stores they wait for.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ocmp_ff.cuh"

namespace ocmp {

// A poll gives up after about four seconds of SM clock; no phase between two exchanges takes longer
// than a few milliseconds.
constexpr long long kTeamWaitCycles = 8000000000LL;
constexpr long long kStarvedCycles = 1000000LL;   // of a wait that a test lets run out
constexpr int kTeamMaxBlocks = 160;   // one block per SM of this part
constexpr int kTeamMaxValues = 2;     // values of one exchange
constexpr int kTeamMaxThreads = 1024;

// Device state of a team: arrivals at the barrier (never reset: a launch starts from the count its
// predecessor left), the blocks that have left, the flag of a poll that gave up, and the blocks'
// partial sums (exchanges alternate between two sets: a set is written again only after another
// exchange, which no block passes before all have read it). Zeroed at creation, and by the host after a
// wait that gave up. starve (a test): the next launch waits for one arrival too many.
struct TeamState {
    unsigned arrive, left;
    int abort;
    unsigned start;
    int starve, next;   // next: the system that a team takes from its queue
    double part[2][kTeamMaxValues][kTeamMaxBlocks];
};

struct Team {
    TeamState* s;
    int rank, size;
    unsigned goal;   // the count that ends the next barrier, less `size`
    int set;
};

__device__ __forceinline__ Team team_join(TeamState* s, int rank, int size) {
    return Team{s, rank, size, size > 1 ? *(volatile unsigned*)&s->start + (*(volatile int*)&s->starve ? 1u : 0u) : 0u, 0};
}

// Sum of cnt <= 32 CAP doubles, entry i read by get(i), by one warp; every lane returns it.
template <int CAP, class Get>
__device__ __forceinline__ double team_list_sum(int cnt, int lane, Get get) {
    static_assert(CAP >= 1 && CAP <= 8, "entries per lane");
    // a limb's sum over 32 CAP entries must stay below 2^31
    constexpr int HB = CAP == 1 ? 5 : CAP <= 2 ? 6 : CAP <= 4 ? 7 : 8;
    constexpr int B = 31 - HB, W = 3 * B;   // limb bits, bits kept (69 to 78)
    const unsigned full = 0xffffffffu;
    double v[CAP];
    unsigned em = 1u;
#pragma unroll
    for (int k = 0; k < CAP; k++) {
        const int i = lane + 32 * k;
        v[k] = i < cnt ? get(i) : 0.0;
        em = max(em, ((unsigned)__double2hiint(v[k]) >> 20) & 0x7ffu);
    }
    em = __reduce_max_sync(full, em);
    double out;
    bool plain = em == 0x7ffu;   // an infinity or a NaN
    if (!plain) {
        int d2 = 0, d1 = 0, d0 = 0;
#pragma unroll
        for (int k = 0; k < CAP; k++) {
            const unsigned hi = (unsigned)__double2hiint(v[k]), lo = (unsigned)__double2loint(v[k]);
            const unsigned e = (hi >> 20) & 0x7ffu;
            const unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | lo;
            const unsigned s = em - max(1u, e);
            // m 2^(W - 53) >> s as W bits: the top 64 in h, W - 64 more from l
            const unsigned long long a = m << 11;
            const unsigned long long h = s < 64u ? a >> s : 0ull;
            const unsigned long long l = s == 0u ? 0ull : s < 64u ? a << (64u - s) : s < 128u ? a >> (s - 64u) : 0ull;
            constexpr unsigned MB = (1u << B) - 1u;
            int x2 = (int)(h >> (64 - B)), x1 = (int)((unsigned)(h >> (64 - 2 * B)) & MB),
                x0 = (int)((((unsigned)h << (W - 64)) | (unsigned)(l >> (128 - W))) & MB);
            if (hi & 0x80000000u) {
                x2 = -x2;
                x1 = -x1;
                x0 = -x0;
            }
            d2 += x2;
            d1 += x1;
            d0 += x0;
        }
        const int s2 = __reduce_add_sync(full, d2), s1 = __reduce_add_sync(full, d1), s0 = __reduce_add_sync(full, d0);
        // (s2 2^B + s1) 2^B + s0, in units of 2^(em - 1022 - W)
        const int c = s0 >> B;
        long long q = ((long long)s2 << B) + s1 + c;
        unsigned r = (unsigned)(s0 - (c << B));
        const bool neg = q < 0;
        if (neg) {
            q = -q - (r ? 1 : 0);
            r = r ? (1u << B) - r : 0u;
        }
        unsigned long long x;
        int ex = (int)em - 1022 - W + 63 + 1023;   // biased exponent of the result
        if (q) {
            const int z = __clzll(q);
            x = (unsigned long long)q << z;
            x |= z >= B ? (unsigned long long)r << (z - B) : (unsigned long long)(r >> (B - z));
            ex += B - z;
        } else {
            const int z = __clzll((long long)r);
            x = r ? (unsigned long long)r << z : 0ull;
            ex -= z;
        }
        if (x == 0ull) out = 0.0;
        else if (ex >= 1 && ex <= 2045) {
            const unsigned long long y = (x >> 11) + ((x >> 10) & 1ull);
            out = __longlong_as_double((long long)(((unsigned long long)neg << 63) | (((unsigned long long)(ex - 1) << 52) + y)));
        } else
            plain = true;   // near the ends of the range
    }
    if (plain) {
        out = 0.0;
#pragma unroll
        for (int k = 0; k < CAP; k++) out += v[k];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) out += __shfl_xor_sync(full, out, o);
    }
    return out;
}

// Barrier over the team's blocks: writes before it are visible to every thread of the team after it
// (plain loads included, but not loads through the read-only path). False in every thread when a poll
// gave up; the kernel then returns.
__device__ __forceinline__ bool team_barrier(Team& t) {
    if (t.size == 1) {
        __syncthreads();
        return true;
    }
    __shared__ int team_ok;
    t.goal += (unsigned)t.size;
    __syncthreads();
    if (threadIdx.x == 0) {
        // release and acquire on the counter itself: 2,430 clocks, a fence on either side 2,800
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&t.s->arrive) : "memory");
        int ok = 1;
        long long t0 = 0;
        for (unsigned spin = 1;; spin++) {
            unsigned v;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(&t.s->arrive) : "memory");
            if ((int)(v - t.goal) >= 0) break;
            if (spin & 63u) continue;
            if (*(volatile int*)&t.s->abort) ok = 0;
            else if (t0 == 0) t0 = clock64();
            else if (clock64() - t0 > (*(volatile int*)&t.s->starve ? kStarvedCycles : kTeamWaitCycles)) {
                atomicExch(&t.s->abort, 1);
                ok = 0;
            }
            if (!ok) break;
        }
        team_ok = ok;
    }
    __syncthreads();
    return team_ok != 0;
}

// Exchange of NV values: every thread passes its contributions and gets the team's sums; it is a
// barrier as well. Only the first `live` threads' contributions are looked at. Four warps (one per
// quarter of the SM) add the block's values per lane in FP64, then sum their lanes; 16 warps summing
// theirs at once took 2,000 clocks.
template <int NV, int NT = kTeamMaxThreads>   // NT: threads of the block, at most
__device__ __forceinline__ bool team_reduce(Team& t, const double* v, double* out, int live) {
    static_assert(NV >= 1 && NV <= kTeamMaxValues, "values of an exchange");
    __shared__ double val[NV][NT > 128 ? NT : 1];
    __shared__ double wsum[NV][4];
    __shared__ double res[NV];
    const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
    if (NT > 128 && live > 128) {
        if (tid < live)
#pragma unroll
            for (int i = 0; i < NV; i++) val[i][tid] = v[i];
        __syncthreads();
    }
    if (w < 4) {
#pragma unroll
        for (int i = 0; i < NV; i++) {
            double x = 0;
            if (NT > 128 && live > 128) {
                x = val[i][tid];
                for (int q = tid + 128; q < live; q += 128) x += val[i][q];
            } else if (tid < live)
                x = v[i];
            const double s = w * 32 < live ? team_list_sum<1>(32, lane, [&](int) { return x; }) : 0.0;
            if (lane == 0) wsum[i][w] = s;
        }
    }
    __syncthreads();
    if (w < NV && lane == 0) {
        double s = wsum[w][0];
        for (int q = 1; q < 4 && q * 32 < live; q++) s += wsum[w][q];
        if (t.size == 1) res[w] = s;
        else t.s->part[t.set][w][t.rank] = s;
    }
    if (!team_barrier(t)) return false;
    if (t.size > 1) {
        if (w < NV) {
            const double* p = t.s->part[t.set][w];
            auto get = [&](int i) { return __ldcg(p + i); };
            const double s = t.size <= 32   ? team_list_sum<1>(t.size, lane, get)
                             : t.size <= 64 ? team_list_sum<2>(t.size, lane, get)
                                            : team_list_sum<5>(t.size, lane, get);
            if (lane == 0) res[w] = s;
        }
        t.set ^= 1;
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < NV; i++) out[i] = res[i];
    return true;
}

// The same for one value held as float pairs: summed over the warps' lanes as pairs (48 bits).
template <int NT = kTeamMaxThreads>
__device__ __forceinline__ bool team_reduce_ff(Team& t, float h, float l, double* out) {
    __shared__ double wv[32];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
        ff_add(h, l, oh, ol);
    }
    if (lane == 0) wv[w] = ff_wide(h, l);
    __syncthreads();
    double s = 0;
    if (w == 0) s = team_list_sum<1>(nw, lane, [&](int i) { return wv[i]; });
    double v[1] = {lane == 0 ? s : 0.0};
    return team_reduce<1, NT>(t, v, out, 1);
}

// After its last exchange every block leaves; the last one writes down where the count stands.
__device__ __forceinline__ void team_leave(const Team& t) {
    if (t.size == 1 || threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&t.s->left, 1u) == (unsigned)t.size - 1) {
        t.s->left = 0;
        t.s->start = t.goal;
    }
}

// Row product with x gathered at the columns: x is written during the launch, so it must not go through
// the read-only path. Two accumulators: the FP64 latency, not the loads, is the chain.
template <class TM, class TV, int TPR, int U>
__device__ __forceinline__ TV team_row_dot(int32_t a, int32_t b, const int32_t* __restrict__ col,
                                           const TM* __restrict__ val, const TV* x, int lane) {
    TV acc0 = 0, acc1 = 0;
    for (int32_t base = a + lane; base < b; base += U * TPR) {
        int32_t c[U];
        TM v[U];
        TV g[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int32_t k = base + u * TPR;
            c[u] = k < b ? __ldg(col + k) : -1;
            v[u] = k < b ? __ldg(val + k) : (TM)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++) g[u] = c[u] >= 0 ? x[c[u]] : (TV)0;
#pragma unroll
        for (int u = 0; u < U; u++) (u & 1 ? acc1 : acc0) += (TV)v[u] * g[u];
    }
    TV acc = acc0 + acc1;
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPR);
    return acc;
}

}  // namespace ocmp
