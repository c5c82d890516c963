// gg_grid.cuh -- helpers of the cooperative (persistent) kernels: the global
// timer and a bounded grid barrier.
//
// The barrier is the persistent kernels' only wait.  It is bounded by a
// %globaltimer deadline; a CTA that gives up sets DEV_ERR_TIMEOUT in *err and
// returns false, and every CTA leaves at its next barrier, so the host gets
// GG_ERR_TIMEOUT and the context stays usable.  Co-residency of all CTAs is
// guaranteed by the cooperative launch, so in normal operation the deadline
// is never reached.
//
// A CTA decides as one whether it goes on: its first thread reads the error
// word, once, and the barrier that releases the others hands them what it saw
// (read by every thread, an error set meanwhile by another CTA would send some
// threads of a warp out and let the others on into its shuffles).
#pragma once
#include "gg_internal.cuh"

namespace gg {
namespace grid {

__device__ __forceinline__ unsigned long long globaltimer() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

struct Barrier {
    unsigned int count;
    unsigned int gen;
    unsigned int err;
};

__device__ __forceinline__ bool sync(Barrier *b, unsigned long long timeout_ns) {
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        volatile unsigned int *genp = &b->gen;
        const unsigned int gen = *genp;
        if (atomicAdd(&b->count, 1u) == gridDim.x - 1) {
            atomicExch(&b->count, 0u);
            __threadfence();
            atomicAdd(&b->gen, 1u);
        } else {
            const unsigned long long t0 = globaltimer();
            while (*genp == gen) {
                if (globaltimer() - t0 > timeout_ns) {
                    atomicOr(&b->err, DEV_ERR_TIMEOUT);
                    break;
                }
                if (*(volatile unsigned int *)&b->err) break;
                __nanosleep(64);
            }
        }
        __threadfence();
        ok = *(volatile unsigned int *)&b->err == 0;
    }
    return __syncthreads_and(ok);
}

// Barrier on one counter of arrivals that only grows: the e-th barrier is
// over when e * gridDim.x CTAs have arrived, so the waiting CTAs see the last
// arrival itself (the two-word barrier above adds a reset and a generation
// store to it).  `epoch` is the calling CTA's own count, 0 at launch; the
// counter starts at 0.
struct Arrivals {
    unsigned long long n;
    unsigned int err;
};

// One thread per CTA, whose other threads' writes it has seen: arrive as the
// `epoch`-th time and wait for the others.  False: the wait ran out somewhere.
__device__ __forceinline__ bool arrive_and_wait(Arrivals *b, unsigned long long epoch, unsigned long long timeout_ns) {
    __threadfence();
    const unsigned long long target = epoch * gridDim.x;
    volatile unsigned long long *np = &b->n;
    if (atomicAdd(&b->n, 1ull) + 1 < target) {
        const unsigned long long t0 = globaltimer();
        while (*np < target) {
            if (globaltimer() - t0 > timeout_ns) {
                atomicOr(&b->err, DEV_ERR_TIMEOUT);
                break;
            }
            if (*(volatile unsigned int *)&b->err) break;
            __nanosleep(20);
        }
    }
    __threadfence();
    return *(volatile unsigned int *)&b->err == 0;
}

__device__ __forceinline__ bool sync(Arrivals *b, unsigned long long &epoch, unsigned long long timeout_ns) {
    __syncthreads();
    ++epoch;
    return __syncthreads_and(threadIdx.x != 0 || arrive_and_wait(b, epoch, timeout_ns));
}

}  // namespace grid
}  // namespace gg
