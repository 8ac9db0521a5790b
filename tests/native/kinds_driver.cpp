// The tiling autotuner (runtime/tuner.cu) with both kinds of chunks under the same
// buckets: prints each kind's decision.  Used by tests/test_tuner_kinds.py; no GPU
// needed.
//   kinds_driver decide   feeds both kinds' samples alternately
//   kinds_driver look     only looks the decisions up
#include "runtime/tuner.h"

#include <cstdio>
#include <cstring>

using namespace thy;

static double cost(bool resident, const Tiling &t)
{
    // launched: deep 1 variant 1 and general variant 2 best; resident: deep 2 variant 2
    const double l = (t.deep1 == 1 ? 0.5 : 1.0) + 1.0 + (t.general == 2 ? 0.5 : 1.0);
    const double r = 1.0 + (t.deep2 == 2 ? 0.5 : 1.0) + 1.0;
    return resident ? r : l;
}

int main(int argc, char **argv)
{
    if (argc < 2) return 2;
    const TuneKey key[2] = {{0, 11, 10, false}, {0, 11, 10, true}};
    const bool feed = !std::strcmp(argv[1], "decide");
    int samples[2] = {0, 0};
    for (int n = 0; feed && n < 200; n++) {
        const TuneKey &k = key[n & 1];
        bool sampling = false;
        const Tiling t = tuner_pick(k, &sampling);
        if (!sampling) continue;
        tuner_sample(k, t, cost(k.resident, t));
        samples[n & 1]++;
    }
    for (const TuneKey &k : key) {
        Tiling t;
        const bool done = tuner_decided(k, &t);
        std::printf("%s done=%d tiling=%d,%d,%d samples=%d\n", k.resident ? "resident" : "launched", done ? 1 : 0, t.deep1,
                    t.deep2, t.general, samples[k.resident]);
    }
    return 0;
}
