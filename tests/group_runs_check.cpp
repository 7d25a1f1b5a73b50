// Runs of groups over random lists: they follow each other, cover every group, stay within the budget
// unless they are one group, cut a layer only where it does not fit, and stop at the end given.
#include <cassert>
#include <cstdio>
#include <random>
#include <vector>

#include "../porousmediaanalysis_gb300/csrc/group_runs.h"

int main() {
    std::mt19937 rng(5);
    long runs = 0, cuts = 0;
    for (int trial = 0; trial < 20000; ++trial) {
        const size_t per = 1 + rng() % 9, nz = 1 + rng() % 6, n = per * nz;
        const unsigned most = 1u << (rng() % 7);
        std::vector<unsigned long long> off(n + 1, 0), layers(nz + 1);
        for (size_t g = 0; g < n; ++g) off[g + 1] = off[g] + (rng() % 3 ? rng() % (most + 1) : 0);
        for (size_t z = 0; z <= nz; ++z) layers[z] = off[z * per];
        auto groups = [&](size_t z) { return off.data() + z * per; };
        auto walk = [&](size_t from, size_t to, unsigned long long budget, auto each) {
            for (size_t g = from; g < to;) {
                const size_t e = pma::group_run_end(layers.data(), per, g, to, budget, groups);
                assert(e > g && e <= to);
                assert(off[e] - off[g] <= budget || e == g + 1);
                const size_t z = g / per;
                if (g == z * per && (z + 1) * per <= to && layers[z + 1] - layers[z] <= budget) assert(e % per == 0);
                if (e % per && e != to) assert(off[e + 1] - off[g] > budget);  // a cut takes what fits
                cuts += e % per != 0;
                ++runs;
                each(g, e);
                g = e;
            }
        };
        const unsigned long long outer = rng() % 200, inner = rng() % 100;
        walk(0, n, outer, [&](size_t a, size_t b) { walk(a, b, inner, [](size_t, size_t) {}); });
    }
    std::printf("%ld runs, %ld cuts ok\n", runs, cuts);
    return 0;
}
