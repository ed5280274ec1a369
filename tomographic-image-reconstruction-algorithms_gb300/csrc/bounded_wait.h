// bounded_wait.h -- the form of every bounded device wait (async.cuh, resident.cuh); plain C++ beside nvcc, so
// that it can be tested with a clock that jumps.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define TOMO_WAIT_FN __device__ __forceinline__
#else
#define TOMO_WAIT_FN inline
#endif

// Polls ready() until within(start) no longer holds, start being the clock() at the first failed poll.  The clock
// is read before a poll and judged after it: between the two looks the waiting thread may have been off the GPU
// for longer than the limit, and what it waits for be there.
template <typename Ready, typename Clock, typename Within>
TOMO_WAIT_FN bool bounded_wait(Ready ready, Clock clock, Within within) {
    if (ready()) return true;
    const uint64_t start = clock();
    for (;;) {
        const bool more = within(start);
        if (ready()) return true;
        if (!more) return false;
    }
}
