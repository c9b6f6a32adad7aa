// Bounded grid-wide waits and block sums shared by the persistent field
// solvers (k_sor_fast.cu, k_poisson.cu).
#pragma once

#include <cuda_runtime.h>

namespace hv {

// default bounds of the device-side waits (hv_fast_options.sor_wait_limit
// replaces both): polls of a grid barrier or a neighbour's phase counter before
// the wait gives up (~1 s), and polls of one tagged mirror entry
constexpr long long kDefaultSpin = 1ll << 24;
constexpr long long kDefaultPoll = 1ll << 22;

__device__ __forceinline__ unsigned ld_relaxed(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void st_release(unsigned *p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_acq_rel() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ int ld_volatile(const int *p) { return *(const volatile int *)p; }

// Grid barrier for co-resident blocks; false when a wait timed out or another
// block reported an error.
static __device__ bool grid_barrier(unsigned *bar, int nblocks, int *err, long long max_spin) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        unsigned gen = ld_relaxed(bar + 1);
        fence_acq_rel();
        unsigned arrived = atomicAdd(bar, 1u) + 1u;
        if (arrived == (unsigned)nblocks) {
            atomicExch(bar, 0u);
            st_release(bar + 1, gen + 1u);
        } else {
            long long spin = 0;
            while (ld_relaxed(bar + 1) == gen) {
                if (++spin > max_spin || ld_volatile(err)) {
                    atomicExch(err, 1);
                    ok = 0;
                    break;
                }
            }
        }
        fence_acq_rel();
    }
    __syncthreads();
    return ok;
}

// The same with half the round trips: one counter that only grows.  Each block
// adds one (a release) and polls for the sum of all; `target` is the count that
// ends the barrier, advanced by every call.  bar[1] holds the count at which
// the launch before ended: every block takes it as its first target's base
// (epoch_base) before its first barrier, and block 0 leaves the final count
// there after the last one (epoch_end).  A solve that gave up leaves the words
// inconsistent; the host zeroes them before the next run.
// Per barrier on 126 blocks: 2.1 us against 3.1.
__device__ __forceinline__ unsigned epoch_base(const unsigned *bar) { return ld_relaxed(bar + 1); }
__device__ __forceinline__ void epoch_end(unsigned *bar, unsigned target) { bar[1] = target; }
static __device__ bool epoch_barrier(unsigned *bar, unsigned &target, int nblocks, int *err, long long max_spin) {
    __shared__ int ok;
    target += (unsigned)nblocks;
    __syncthreads();
    if (threadIdx.x == 0) {
        int good = 1;
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
        long long spin = 0;
        while ((int)(ld_relaxed(bar) - target) < 0) {
            if (++spin > max_spin || ((spin & 15) == 0 && ld_volatile(err))) {
                atomicExch(err, 1);
                good = 0;
                break;
            }
        }
        fence_acq_rel();
        ok = good;
    }
    __syncthreads();
    return ok;
}

// Deterministic block sum of two doubles (fixed shuffle tree, fixed warp order)
// for blocks of whole warps, at most 32; the result is valid in thread 0.
static __device__ void block_sum2(double &u, double &v) {
    __shared__ double su[32], sv[32];
    for (int o = 16; o > 0; o >>= 1) {
        u += __shfl_xor_sync(0xffffffffu, u, o);
        v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) {
        su[w] = u;
        sv[w] = v;
    }
    __syncthreads();
    if (w == 0) {
        const int nw = blockDim.x >> 5;
        u = l < nw ? su[l] : 0.0;
        v = l < nw ? sv[l] : 0.0;
        for (int o = 16; o > 0; o >>= 1) {
            u += __shfl_xor_sync(0xffffffffu, u, o);
            v += __shfl_xor_sync(0xffffffffu, v, o);
        }
    }
}

}  // namespace hv
