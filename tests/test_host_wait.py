"""The host's wait (host_wait.h) on a made-up event: it ends with the event's status or at its limit, and
gives up the core every 500 us before it sleeps, so a thread pinned beside it is not held up."""
from tests import host_cpp

SOURCE = r"""
#include <atomic>
#include <cstdio>
#include <sched.h>
#include "host_wait.h"
static long queries = 0, yields = 0, ready_after = 0;
static cudaError_t answer = cudaSuccess;
extern "C" cudaError_t cudaEventQuery(cudaEvent_t) { return ++queries > ready_after ? answer : cudaErrorNotReady; }
extern "C" int sched_yield() noexcept { yields++; return 0; }
static int bad = 0;
static void check(bool ok, const char *what) { if (!ok) { std::printf("%s: %ld queries, %ld yields\n", what, queries, yields); bad++; } }
int main() {
    using namespace fesom;
    auto reset = [](long n, cudaError_t a) { queries = yields = 0; ready_after = n; answer = a; };
    reset(0, cudaSuccess);
    check(wait_event(nullptr, -1) == cudaSuccess && queries == 1 && yields == 0, "a finished event");
    reset(100, cudaSuccess);
    check(wait_event(nullptr, -1) == cudaSuccess && queries == 101, "a short wait");
    reset(3, cudaErrorInvalidValue);
    check(wait_event(nullptr, -1) == cudaErrorInvalidValue && queries == 4, "an error ends it");
    reset(1l << 60, cudaSuccess);
    const auto t0 = std::chrono::steady_clock::now();
    check(wait_event(nullptr, 30) == cudaErrorNotReady, "the limit ends it");
    const auto ms = std::chrono::duration_cast<std::chrono::milliseconds>(std::chrono::steady_clock::now() - t0).count();
    check(ms >= 30 && ms < 2000, "the limit's time");
    // 5 ms of spinning, then sleeps: one yield in 500 us (fewer where this process has to wait for a core, so
    // a wait without one is tried again)
    long most = yields;
    for (int k = 0; k < 20 && !most; k++) {
        reset(1l << 60, cudaSuccess);
        wait_event(nullptr, 10);
        most = yields;
    }
    check(most >= 1 && most <= 12, "the spin's yields");
    return bad;
}
"""


def test_wait(tmp_path):
    host_cpp.run(tmp_path, SOURCE)
