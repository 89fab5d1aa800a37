// The limit on a device wait, apart from what it polls (host code can run it too).
#pragma once

#ifdef __CUDACC__
#define TVMC_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define TVMC_HOST_DEVICE inline
#endif

namespace tvmc {

// Polls until poll() is true; gives up (false) once `limit` ticks of clock() have
// passed since the first miss and one more poll has missed too: a thread that was
// itself held up for that long finds a completed wait completed.
template <class Poll, class Clock>
TVMC_HOST_DEVICE bool bounded_wait(Poll&& poll, Clock&& clock, long long limit) {
    if (poll()) return true;
    const long long t0 = clock();
    while (clock() - t0 < limit)
        if (poll()) return true;
    return poll();
}

}  // namespace tvmc
