// The barriers between a kernel's CTAs that count arrivals over the whole
// launch: the count, its comparison and the bounded wait.
#pragma once

#ifdef __CUDACC__
#define GBG_HOST_DEVICE __host__ __device__
#else
#define GBG_HOST_DEVICE
#endif

namespace gbg {

// A CTA that waits for `target` sees a count less than one barrier's arrivals away
// from it, on either side: the sign of the difference tells which, also where the
// 32 bits wrap (2^32 arrivals are 28 million steps of 152 CTAs in one launch).
GBG_HOST_DEVICE inline bool all_arrived(unsigned count, unsigned target) { return (int)(count - target) >= 0; }

#ifdef __CUDACC__
// *count is at `target`, or false: it did not get there in seconds (then the status
// word is set), or the status word was set elsewhere
__device__ __forceinline__ bool wait_for_arrivals(const unsigned *count, unsigned target, int *status) {
    for (long long spins = 1;; ++spins) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];\n" : "=r"(v) : "l"(count) : "memory");
        if (all_arrived(v, target)) return true;
        if (spins > (1ll << 24)) {
            atomicExch(status, (int)DEV_BARRIER_TIMEOUT);
            return false;
        }
        if ((spins & 1023) == 0 && *(volatile int *)status != DEV_OK) return false;
    }
}
__device__ __forceinline__ void arrive(unsigned *count) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;\n" ::"l"(count) : "memory");
}
#endif

}  // namespace gbg
