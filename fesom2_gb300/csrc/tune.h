// tune.h -- launch settings of the FP32 form, and the autotuner's search over them.
#pragma once

namespace fesom {

// launch shape of the node stages (the autotuner's choices): at most `blocks_per_sm` x 152 blocks
// looping over the tiles (0: one block per tile)
struct LaunchShape {
    int blocks_per_sm = 0;
    int variant = 0;      // bit 0 of fesom_gpu_set_stage_variant (kept and reported; one kernel per stage)
    int vsep = -1;        // the update stage: the implicit vertical diffusion as its own kernel (0, 1; -1: by the depth)
};

struct TuneSetting {
    int stage_tr[4];
    LaunchShape shape[4];
    // whether both launch the same programs: bit 0 of a variant and the edge stage's blocks per SM select nothing
    bool same_launches(const TuneSetting &o) const {
        for (int k = 0; k < 4; k++)
            if (stage_tr[k] != o.stage_tr[k] || (k != 1 && shape[k].blocks_per_sm != o.shape[k].blocks_per_sm) ||
                (k == 3 && shape[k].vsep != o.shape[k].vsep))
                return false;
        return true;
    }
};

struct TuneOutcome {
    TuneSetting best;
    float def_ms, best_ms;
    int candidates;
};

// Times the library defaults and the settings the context came with, then a coordinate descent over the
// stages: the place of the vertical diffusion, blocks per SM, tracers per launch (with more than 8 slots).  A
// candidate replaces the best when it is faster by more than 1 % (timing noise).  own_launch: where the
// mesh's depth puts the diffusion while nothing is set; every setting that is timed names its place, so
// the best is one that was timed.  No two candidates launch the same programs, and what selects nothing
// stays as it was set.  time(setting, &ms) returns an error code; the first one ends the search.
template <class Time>
int tune_search(TuneSetting start, bool own_launch, int slots, Time &&time, TuneOutcome &out) {
    TuneSetting def{};  // the library defaults
    for (int k = 0; k < 4; k++) def.shape[k].variant = start.shape[k].variant;
    def.shape[1].blocks_per_sm = start.shape[1].blocks_per_sm;
    def.shape[3].vsep = own_launch;
    if (start.shape[3].vsep < 0) start.shape[3].vsep = own_launch;
    out = TuneOutcome{def, 0.f, 0.f, 0};
    int rc = time(def, &out.def_ms);
    out.best_ms = out.def_ms;
    out.candidates = 1;
    auto attempt = [&](const TuneSetting &c, float margin) {
        float ms = 0.f;
        if ((rc = time(c, &ms))) return;
        out.candidates++;
        if (ms < margin * out.best_ms) {
            out.best = c;
            out.best_ms = ms;
        }
    };
    if (!rc && !start.same_launches(def)) attempt(start, 1.f);
    const int bps[] = {0, 2, 4};
    for (int k = 0; k < 4 && !rc; k++) {
        // the update: also with the vertical diffusion as its own launch
        const int nvar = k == 3 ? 2 : 1;
        const int ntrs = (k >= 2 && slots > 8) ? 2 : 1;
        for (int v = 0; v < nvar && !rc; v++)
            for (int b : bps)
                for (int q = 0; q < ntrs && !rc; q++) {
                    TuneSetting c = out.best;
                    if (k == 3) c.shape[k].vsep = v;
                    if (k != 1) c.shape[k].blocks_per_sm = b;
                    c.stage_tr[k] = q ? 8 : 0;
                    if (!c.same_launches(out.best)) attempt(c, 0.99f);
                }
    }
    return rc;
}

}  // namespace fesom
