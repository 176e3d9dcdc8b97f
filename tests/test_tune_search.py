"""The autotuner's search (tune.h) on made-up times: whatever the settings a context comes with, the
result is a setting that was timed, with the time it took."""
from tests import host_cpp

COMMON = r"""
#include <cstdio>
#include <vector>
#include "tune.h"
using namespace fesom;
struct Timed { TuneSetting c; float ms; };
static int bad = 0;
static void check(bool ok, const char *what, int seed) {
    if (!ok) { std::printf("%s (%d)\n", what, seed); bad++; }
}
static TuneSetting defaults() {
    TuneSetting t{};
    t.shape[0].variant = 1;
    return t;
}
"""

PLACE = COMMON + r"""
int main() {
    for (int own = 0; own < 2; own++)          // where the depth puts the diffusion
        for (int set = -1; set < 2; set++)     // and where the context was set to
            for (int seed = 0; seed < 60; seed++) {
                TuneSetting start = defaults();
                start.shape[3].vsep = set;
                if (seed % 3 == 1) start.shape[2].blocks_per_sm = 4;
                std::vector<Timed> timed;
                unsigned r = 77u * seed + 5u * own + set + 1;
                auto time = [&](const TuneSetting &c, float *ms) {
                    r = r * 1664525u + 1013904223u;
                    // the depth's place takes 10 units, the other one 11, the other settings up to 30 % more
                    const int place = c.shape[3].vsep < 0 ? own : c.shape[3].vsep;
                    *ms = (place == own ? 10.f : 11.f) * (1.f + 0.3f * (timed.empty() ? 0.f : (r >> 8) / 16777216.f));
                    timed.push_back({c, *ms});
                    return 0;
                };
                TuneOutcome out{};
                check(tune_search(start, own != 0, 12, time, out) == 0, "error", seed);
                bool found = false;
                for (const Timed &t : timed) found = found || (t.c == out.best && t.ms == out.best_ms);
                check(found, "the best was not timed, or took another time", seed);
                check(out.best.shape[3].vsep == own, "the slower place of the diffusion was kept", seed);
                check(out.def_ms == timed[0].ms && out.candidates == (int)timed.size(), "counts", seed);
            }
    // the first error ends the search
    int calls = 0;
    TuneOutcome out{};
    check(tune_search(defaults(), false, 4, [&](const TuneSetting &, float *ms) { *ms = 1.f; return ++calls == 3 ? 4 : 0; },
                      out) == 4 && calls == 3, "an error does not end the search", 0);
    return bad;
}
"""


def test_the_result_is_a_setting_that_was_timed(tmp_path):
    host_cpp.run(tmp_path, PLACE)
