// Time spent in a bounded wait, from the clock readings of its polls.  A gap between two polls counts for
// at most kWaitStepNs: polls come every few microseconds, so a longer gap is one in which the waiting
// threads, and the ones that they wait for, were not running (the whole kernel set aside for
// another context, say), and nobody is late for that.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define WCFD_HD __host__ __device__ __forceinline__
#else
#define WCFD_HD inline
#endif

namespace wcfd {

constexpr uint64_t kWaitStepNs = 1000ull * 1000ull;

struct WaitClock {
    uint64_t last, waited;
    WCFD_HD explicit WaitClock(uint64_t now) : last(now), waited(0) {}
    // one more poll failed; whether the wait has lasted longer than limit
    WCFD_HD bool over(uint64_t now, uint64_t limit) {
        const uint64_t step = now - last;
        waited += step < kWaitStepNs ? step : kWaitStepNs;
        last = now;
        return waited > limit;
    }
};

}  // namespace wcfd
