// A ring of stages whose blocks groups of warps map in turn, on the CPU: copies that land in any order, barriers that are
// waited for by parity, and the waits of the mapping groups as the kernel makes them.  Prints how many blocks a group began
// before their copies had landed, or had mapped twice, and how many runs did not end.
//
//   ring_rounds <stages> <groups> <blocks> <wait for the round before: 0, 1, or 2 = as the kernel does>
#include "sm100.cuh"

#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

int main(int argc, char **argv) {
    if (argc < 5) return 2;
    const int stages = atoi(argv[1]), groups = atoi(argv[2]), blocks = atoi(argv[3]), mode = atoi(argv[4]);
    const bool waits = mode == 2 ? gpx::sm100::ring_rounds_skipped(stages, groups) : mode == 1;
    long wrong = 0, stuck = 0;
    for (unsigned seed = 0; seed < 400; ++seed) {
        std::mt19937 rng(seed);
        // phases that have completed of each stage's barriers
        std::vector<int> full(stages, 0), ready(stages, 0);
        auto passes = [](int completed, int parity) { return (completed & 1) != parity; };  // the phase under way has the other parity
        int asked = 0, used = 0;                // copies asked for; blocks whose products are through
        std::vector<char> landed(blocks, 0);
        std::vector<int> at(groups), mapped(blocks, 0);
        for (int g = 0; g < groups; ++g) at[g] = g;
        for (int idle = 0; used < blocks && idle < 20000; ++idle) {
            const unsigned what = rng() % (unsigned)(groups + 3);
            if (what == 0) {
                if (asked < blocks && asked - used < stages) ++asked, idle = 0;
            } else if (what == 1) {
                // any copy under way lands; now and then the oldest is the last
                const int low = rng() % 8 ? used : used + 1, n = asked - low;
                if (n <= 0) continue;
                const int b = low + (int)(rng() % (unsigned)n);
                if (!landed[b]) landed[b] = 1, ++full[b % stages], idle = 0;
            } else if (what == 2) {
                const int s = used % stages, parity = used / stages & 1;
                if (used < blocks && passes(full[s], parity) && passes(ready[s], parity)) ++used, idle = 0;
            } else {
                int &b = at[what - 3];
                if (b >= blocks) continue;
                const int s = b % stages, parity = b / stages & 1;
                if ((waits && !passes(ready[s], parity ^ 1)) || !passes(full[s], parity)) continue;
                if (!landed[b] || mapped[b]++) ++wrong;
                ++ready[s], idle = 0;
                b += groups;
            }
        }
        if (used < blocks) ++stuck;
    }
    printf("%ld %ld\n", wrong, stuck);
    return 0;
}
