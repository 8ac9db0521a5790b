// For each group of three arguments "nx ny sms": the split of a row over the blocks
// of the Okada stage (thy::okada_split, kernels/kernels.h) as "per segs" and 1 when
// every column is some thread's and no thread's columns wrap around.  Used by
// tests/test_okada_split.py; no GPU needed.
#include "kernels/kernels.h"

#include <cstdio>
#include <cstdlib>

int main(int argc, char **argv)
{
    for (int i = 1; i + 2 < argc; i += 3) {
        const int nx = std::atoi(argv[i]), ny = std::atoi(argv[i + 1]);
        const thy::OkadaSplit s = thy::okada_split(nx, ny, std::atoi(argv[i + 2]));
        const unsigned last = s.segs - 1, row = s.per * thy::kOkadaThreads;
        // the last block starts inside the row and ends at or behind its end, in
        // arithmetic that does not wrap
        const unsigned long long first = (unsigned long long)last * row, end = first + row;
        const bool ok = s.segs > 0 && s.per >= 1 && s.per <= 4 && thy::okada_first_cell(s, last) == first &&
                        first < (unsigned long long)nx && end >= (unsigned long long)nx && end < (1ull << 32);
        std::printf("%u %u %d\n", s.per, s.segs, ok ? 1 : 0);
    }
    return 0;
}
