// For each argument "sms": every work size that a device of that many SMs takes as
// a resident chunk, in every tiling, through thy::resident_rows (kernels/kernels.h).
// Prints the largest such work and the number of choices that break a rule of the
// kernel: rows of 1, 2, 4 or 8 and no more tasks than the launch holds, whatever else
// is stepped on the device (thy::resident_ctas); alone it has every SM.  Used by
// tests/test_resident_rows.py; no GPU needed.
#include "kernels/kernels.h"

#include <cstdio>
#include <cstdlib>

int main(int argc, char **argv)
{
    for (int i = 1; i < argc; i++) {
        const int sms = std::atoi(argv[i]), most = thy::resident_units(sms);
        long long broken = 0;
        for (int units = 1; units <= most; units++) {
            broken += thy::resident_ctas(units, sms, units) != sms;
            for (int w = 0; w < 4 * thy::kTilingVariants * thy::kTilingVariants; w++) {
                const long long others = w % 4 == 0 ? 0 : w % 4 == 1 ? 1 : w % 4 == 2 ? 7ll * units : 1000000000000ll;
                const int v = w / 4;
                const int ctas = thy::resident_ctas(units, sms, units + others), warps = thy::resident_warps(ctas);
                broken += ctas < 1 || ctas > sms;
                thy::Tiling t;
                t.deep2 = v / thy::kTilingVariants;
                t.general = v % thy::kTilingVariants;
                int g = 0, d = 0;
                thy::resident_rows(units, warps, t, &g, &d);
                const bool rows = (g == 1 || g == 2 || g == 4 || g == 8) && (d == 1 || d == 2 || d == 4 || d == 8);
                // a unit is 64 / g general or 32 / d deep tasks
                const long long tasks = rows ? (long long)units * (64 / g > 32 / d ? 64 / g : 32 / d) : 0;
                broken += !rows || tasks > thy::resident_tasks_capacity(warps);
            }
        }
        std::printf("%d %lld\n", most, broken);
    }
    return 0;
}
