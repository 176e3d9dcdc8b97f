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
// the same launches: bit 0 of a variant and the edge stage's blocks per SM select nothing
static bool same(const TuneSetting &a, const TuneSetting &b) {
    bool r = a.shape[3].vsep == b.shape[3].vsep;
    for (int k = 0; k < 4; k++)
        r = r && a.stage_tr[k] == b.stage_tr[k] && (k == 1 || a.shape[k].blocks_per_sm == b.shape[k].blocks_per_sm);
    return r;
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
                for (const Timed &t : timed) found = found || (same(t.c, out.best) && t.ms == out.best_ms);
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


INERT = COMMON + r"""
int main() {
    for (int seed = 0; seed < 60; seed++) {
        TuneSetting start = defaults();
        start.shape[3].vsep = -1;
        start.shape[1].blocks_per_sm = seed % 3 ? 4 : 0;  // selects nothing
        start.shape[2].variant = seed % 2;                // selects nothing
        if (seed % 5 == 4) start.stage_tr[1] = 8;         // does
        std::vector<Timed> timed;
        unsigned r = 99u * seed + 1;
        TuneSetting best{};  // the one a candidate is measured against
        float best_ms = 0.f;
        auto time = [&](const TuneSetting &c, float *ms) {
            r = r * 1664525u + 1013904223u;
            *ms = 10.f + 3.f * ((r >> 8) / 16777216.f);
            if (!timed.empty()) check(!same(c, best), "the program of the best was timed again", seed);
            const float margin = timed.size() == 1 && seed % 5 == 4 ? 1.f : 0.99f;  // the start's own settings
            timed.push_back({c, *ms});
            if (timed.size() == 1 || *ms < margin * best_ms) { best = c; best_ms = *ms; }
            return 0;
        };
        TuneOutcome out{};
        tune_search(start, false, 12, time, out);
        check(same(best, out.best) && best_ms == out.best_ms, "another best", seed);
        check(out.best.shape[1].blocks_per_sm == start.shape[1].blocks_per_sm, "the edge stage's blocks were tuned", seed);
        for (int k = 0; k < 4; k++)
            check(out.best.shape[k].variant == start.shape[k].variant, "a variant's bit 0 was changed", seed);
    }
    return bad;
}
"""


def test_no_program_is_timed_against_itself(tmp_path):
    host_cpp.run(tmp_path, INERT)
