// The barrier of a cooperative launch whose CTAs read through L1 what others
// have written (sm_103a).
//
// Thread 0 of each CTA adds to a counter (release) and polls it (acquire, which
// also makes the SM's L1 current).  The wait is bounded by %globaltimer: a CTA
// whose wait runs out sets kErrTimeout and gives up, and so does every other in
// turn.  The counter is only ever added to, a multiple of the CTAs by every launch
// that ends well, so a launch may find it at any such multiple.
#pragma once
#include "logo_device.cuh"
#include "logo_internal.h"

namespace logo {

__device__ __forceinline__ unsigned long long ld_acquire_u64(const unsigned long long* p) {
    unsigned long long v;
    asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    return v;
}

struct GridBarrier {
    unsigned long long* arrived;
    DevState* st;
    bool* ok;  // shared
    unsigned long long wait_ns;
    unsigned long long target = 0;

    // Where the counter need not begin at 0: before the first barrier, in thread 0
    // (that barrier is not passed without this CTA, so fewer than all have arrived).
    __device__ __forceinline__ void start(unsigned int ctas) {
        const unsigned long long now = ld_acquire_u64(arrived);
        target = now - now % ctas;
    }
    // False when the wait ran out (the same in every thread of the CTA).
    __device__ __forceinline__ bool operator()(unsigned int ctas) {
        target += ctas;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u64 [%0], 1;" ::"l"(arrived) : "memory");
            bool fine = true;
            unsigned long long t0 = 0;
            for (uint32_t it = 0; ld_acquire_u64(arrived) < target; ++it) {
                if ((it & 255u) == 255u) {
                    const unsigned long long now = global_timer_ns();
                    if (t0 == 0) t0 = now;
                    if (now - t0 > wait_ns) {
                        atomicOr(&st->status, kErrTimeout);
                        fine = false;
                        break;
                    }
                }
            }
            *ok = fine;
        }
        __syncthreads();
        return *ok;
    }
    __device__ __forceinline__ bool operator()() { return (*this)(gridDim.x); }
};

}  // namespace logo
