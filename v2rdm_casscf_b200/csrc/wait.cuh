// Bounded waits inside one cooperative launch.
#pragma once

#include <cuda_runtime.h>

namespace v2g {

// A wait gives up after two seconds of the device's clock: what it waits for
// takes microseconds to milliseconds (a phase of the CG, other blocks of the same
// projection).  A poll is a load through L2, most of a microsecond, and its
// count is no measure of time, but bounds the wait should the clock stand still.
constexpr unsigned long long kWaitNs = 2000000000ull;
constexpr long kWaitPolls = 1L << 25;

// After n unsuccessful polls: whether to give up, by the time since the wait's
// first look (start, 0 before it) or because another CTA of the launch has (*err
// set: it may be the one waited for).  Looks every 256th poll.
__device__ __forceinline__ bool wait_is_over(long n, unsigned long long& start, const int* err) {
    if ((n & 255) != 255) return false;
    int e;
    unsigned long long now;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(e) : "l"(err) : "memory");
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(now));
    if (start == 0) start = now;
    return e != 0 || now - start >= kWaitNs || n >= kWaitPolls;
}

}  // namespace v2g
