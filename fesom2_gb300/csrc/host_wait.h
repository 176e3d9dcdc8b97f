// host_wait.h -- the host's wait for device work, with a time limit.
#pragma once
#include <chrono>
#include <thread>

#include <cuda_runtime.h>

namespace fesom {

// Waits for ev; cudaErrorNotReady past limit_ms (negative: no limit), else the event's status.  The
// first 5 ms are spun: a sleep of 20 us takes 70 with the kernel's timer slack, as long as a whole
// call on a small mesh (a call of three routines on 2.9k nodes waits three times, a step of 16
// instances reads 93 tracers); longer work is waited for in sleeps.  The spin yields every 500 us, so a
// thread of the caller's that waits for this core gets it: no short call meets one (three routines on
// 2.9k nodes: 275 us; yielding every 50 us 279, on every turn 281).
inline cudaError_t wait_event(cudaEvent_t ev, int limit_ms) {
    const auto t0 = std::chrono::steady_clock::now();
    long long yielded = 0;
    for (;;) {
        const cudaError_t q = cudaEventQuery(ev);
        if (q != cudaErrorNotReady) return q;
        const auto us =
            std::chrono::duration_cast<std::chrono::microseconds>(std::chrono::steady_clock::now() - t0).count();
        if (limit_ms >= 0 && us > 1000ll * limit_ms) return cudaErrorNotReady;
        if (us > 5000) {
            std::this_thread::sleep_for(std::chrono::microseconds(us < 10000 ? 20 : 500));
        } else if (us - yielded >= 500) {
            yielded = us;
            std::this_thread::yield();
        }
    }
}

}  // namespace fesom
