// Bounded grid-wide barrier for cooperative persistent kernels.
#pragma once

#include <cuda_runtime.h>

#include "../../include/elhl_prop.h"

namespace elhl {

constexpr unsigned long long kBarrierNs = 5000000000ULL;  // give up after 5 s

__device__ __forceinline__ unsigned long long globaltimer_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Barrier over all CTAs of a cooperative launch on a count that only grows:
// `count` is two 32-bit words read as one 64-bit count (8-byte aligned, zero
// at the launch).  Thread 0 arrives for its CTA by a release add, which
// returns the arrivals before it: all nblocks arrivals of one barrier lie in
// [nblocks e, nblocks (e + 1)), so the CTA polls (relaxed loads, then one
// acquire fence) until the count reaches nblocks (e + 1).  The last arrival
// itself releases the others (no reset, no generation word).  Returns false
// (and sets *err = ELHL_ERR_TIMEOUT) if the other CTAs do not arrive within limit_ns
// (kBarrierNs unless the launch sets a shorter limit), so a stuck launch ends
// with an error instead of hanging.
__device__ __forceinline__ bool grid_barrier(unsigned *count, unsigned nblocks, int *err,
                                             unsigned long long limit_ns = kBarrierNs) {
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long *c = reinterpret_cast<unsigned long long *>(count);
        unsigned long long prev;
        asm volatile("atom.add.release.gpu.global.u64 %0, [%1], 1;" : "=l"(prev) : "l"(c) : "memory");
        const unsigned long long target = (prev / nblocks + 1) * nblocks;
        const unsigned long long t0 = globaltimer_ns();
        while (true) {
            unsigned long long v;
            asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(c) : "memory");
            if (v >= target) break;
            if (globaltimer_ns() - t0 > limit_ns) {
                atomicExch(err, ELHL_ERR_TIMEOUT);
                break;
            }
            __nanosleep(40);
        }
        __threadfence();  // acquire: the other CTAs' writes before their arrivals
    }
    __syncthreads();
    return *(volatile int *)err == 0;
}

// The same count in two halves, for kernels that know how many barriers came
// before (one barrier per round on every CTA): one thread arrives for its CTA
// once the CTA's writes are ordered before it (__syncwarp or __syncthreads), and
// one thread waits for `target` = nblocks x (barriers so far).  Against
// grid_barrier an arrival needs no answer, the poll does not sleep, and *err is
// read by the waiting thread alone, every 64th poll, instead of by every thread
// after each barrier: 3,500 cycles per Taylor round before, 2,750 after (117
// CTAs).  grid_poll returns false on a timeout (which it reports) or when
// another CTA has reported one; the caller broadcasts the answer.
__device__ __forceinline__ void grid_arrive(unsigned *count) {
    asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(count) : "memory");
}
__device__ __forceinline__ bool grid_poll(const unsigned *count, unsigned long long target, int *err,
                                          unsigned long long limit_ns = kBarrierNs) {
    unsigned long long t0 = 0;
    bool ok = true;
    for (unsigned n = 0;; ++n) {
        unsigned long long v;
        asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(count) : "memory");
        if (v >= target) break;
        if ((n & 63u) == 63u) {
            const unsigned long long t = globaltimer_ns();
            if (!t0) t0 = t;
            if (*(volatile int *)err) ok = false;
            else if (t - t0 > limit_ns) {
                atomicExch(err, ELHL_ERR_TIMEOUT);
                ok = false;
            }
            if (!ok) break;
        }
    }
    __threadfence();  // acquire: the other CTAs' writes before their arrivals
    return ok;
}
// One barrier of a block's threads with the grid: `arrivals` counts the grid's
// arrivals so far in every thread, *s_ok (shared memory) carries the answer.
__device__ __forceinline__ bool grid_round(unsigned *count, unsigned long long &arrivals, unsigned nblocks, int *err,
                                           int *s_ok, unsigned long long limit_ns = kBarrierNs) {
    __syncthreads();
    arrivals += nblocks;
    if (threadIdx.x == 0) {
        grid_arrive(count);
        *s_ok = grid_poll(count, arrivals, err, limit_ns);
    }
    __syncthreads();
    return *s_ok;
}

}  // namespace elhl
