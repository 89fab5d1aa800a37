// The limit on a device wait and what follows one that runs out, apart from what it
// polls (host code can run it too).
#pragma once
#include <cstdint>

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

// One thread's waits for its group's MMAs, in order: poll(parity) tells whether the
// phase of that parity of the group's mbarrier is complete.
struct GroupWaits {
    uint32_t phase = 0;  // parity of the next wait
    uint32_t dead = 0;   // 1 + the parity of the wait that ran out: this thread waits, and issues, no more
};
// false: this wait ran out.
template <class Poll, class Clock>
TVMC_HOST_DEVICE bool group_wait(GroupWaits& w, Poll&& poll, Clock&& clock, long long limit) {
    bool ok = true;
    if (!w.dead) {
        ok = bounded_wait([&] { return poll(w.phase); }, clock, limit);
        if (!ok) w.dead = 1 + w.phase;
    }
    w.phase ^= 1;
    return ok;
}
// The issuing thread's last call before its group's memory is given back: an MMA
// whose wait ran out may still be writing its accumulators.
template <class Poll, class Clock>
TVMC_HOST_DEVICE void group_drain(const GroupWaits& w, Poll&& poll, Clock&& clock, long long limit) {
    if (w.dead) bounded_wait([&] { return poll(w.dead - 1); }, clock, limit);
}

}  // namespace tvmc
