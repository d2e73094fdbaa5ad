// Building blocks of the persistent Krylov kernels (sm_103a): a solve runs in one cooperative launch
// by a team of co-resident blocks that meet at barriers in global memory, one block per SM.
//
// What a launch per operation costs on this part, and a barrier inside one launch does not: on a
// 289-dof system a CG iteration of seven launches took 47 us, all of it launch gaps and kernel
// start-up; a barrier among 152 blocks takes about 1.3 us, a block of its own pays a __syncthreads.
//
// FP64 additions are as scarce as FP64 multiplications here (about two lanes per clock and SM: a
// warp-wide DADD holds the pipe for 16 clocks), so a block reduces through shared memory with one
// warp per value instead of a butterfly in every warp; FP32 contributions are summed as (hi, lo)
// float pairs on the FP32 pipes.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "ocmp_ff.cuh"

namespace ocmp {

// A wait at a barrier gives up after about four seconds of SM clock; no phase between two barriers
// takes longer than a few milliseconds.
constexpr long long kTeamWaitCycles = 8000000000LL;

// Device state of a team's barrier: arrivals, blocks that have left, and the flag of a wait that
// gave up. Zeroed at creation; the last block to leave puts it back to zero.
struct TeamState {
    unsigned arrive, left;
    int abort, pad;
};

struct Team {
    TeamState* s;
    int rank, size;
    unsigned goal;   // arrivals the next barrier waits for, less `size`
};

__device__ __forceinline__ unsigned team_load(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Barrier over the team's blocks: writes before it are visible to every thread of the team after it
// (plain loads included, but not loads through the read-only path). False in every thread when a
// wait gave up; the kernel then returns.
__device__ __forceinline__ bool team_sync(Team& t) {
    if (t.size == 1) {
        __syncthreads();
        return true;
    }
    __shared__ int team_ok;
    t.goal += (unsigned)t.size;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(&t.s->arrive) : "memory");
        int ok = 1;
        const long long t0 = clock64();
        for (unsigned spin = 1; (int)(team_load(&t.s->arrive) - t.goal) < 0; spin++) {
            if (spin & 63u) continue;
            if (*(volatile int*)&t.s->abort) ok = 0;
            else if (clock64() - t0 > kTeamWaitCycles) {
                atomicExch(&t.s->abort, 1);
                ok = 0;
            }
            if (!ok) break;
        }
        __threadfence();
        team_ok = ok;
    }
    __syncthreads();
    return team_ok != 0;
}

// After its last barrier every block leaves; the last one resets the counters for the next launch.
__device__ __forceinline__ void team_leave(const Team& t) {
    if (t.size == 1 || threadIdx.x != 0) return;
    __threadfence();
    if (atomicAdd(&t.s->left, 1u) == (unsigned)t.size - 1) {
        t.s->arrive = 0;
        t.s->left = 0;
    }
}

__device__ __forceinline__ double team_warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Sum of the first cnt entries of sh by one warp; every lane returns it. FP32 entries are summed as
// float pairs (about 48 bits).
__device__ __forceinline__ double team_row_sum(const double* sh, int cnt, int lane) {
    double a = 0, b = 0;
    int i = lane;
    for (; i + 32 < cnt; i += 64) {
        a += sh[i];
        b += sh[i + 32];
    }
    if (i < cnt) a += sh[i];
    return team_warp_sum(a + b);
}
__device__ __forceinline__ double team_row_sum(const float* sh, int cnt, int lane) {
    float h = 0.f, l = 0.f;
    for (int i = lane; i < cnt; i += 32) ff_add(h, l, sh[i], 0.f);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float oh = __shfl_xor_sync(0xffffffffu, h, o), ol = __shfl_xor_sync(0xffffffffu, l, o);
        ff_add(h, l, oh, ol);
    }
    return (double)h + (double)l;
}

// The team's sums of nv values from its blocks' partials (part[v * size + rank]), after the barrier:
// warp v of the block, in rank order per lane, so every block gets the same bits. out in shared memory.
__device__ __forceinline__ void team_sums(const double* part, int size, int nv, double* out) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
    for (int v = w; v < nv; v += nw) {
        double a = 0;
        for (int b = lane; b < size; b += 32) a += __ldcg(part + (int64_t)v * size + b);
        a = team_warp_sum(a);
        if (lane == 0) out[v] = a;
    }
}

// x gathered at c: x is written during the launch, so it must not go through the read-only path
template <class TM, class TV, int TPR, int U>
__device__ __forceinline__ TV team_row_dot(int32_t a, int32_t b, const int32_t* __restrict__ col,
                                           const TM* __restrict__ val, const TV* x, int lane) {
    TV acc = 0;
    for (int32_t base = a + lane; base < b; base += U * TPR) {
        int32_t c[U];
        TM v[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int32_t k = base + u * TPR;
            c[u] = k < b ? __ldg(col + k) : -1;
            v[u] = k < b ? __ldg(val + k) : (TM)0;
        }
#pragma unroll
        for (int u = 0; u < U; u++)
            if (c[u] >= 0) acc += (TV)v[u] * x[c[u]];
    }
#pragma unroll
    for (int o = TPR / 2; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o, TPR);
    return acc;
}

}  // namespace ocmp
