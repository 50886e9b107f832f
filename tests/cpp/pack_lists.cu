// PageRank's packed lists (pack_lists in graphwl.cu) on the CPU, where no thread but the first can allocate: the call
// gives the same lists, and holds every edge once.
#include "graphwl.cu"

#include <cstdio>
#include <cstdlib>
#include <random>

// (first_thread_new.cpp)
extern thread_local bool t_first;
extern bool g_strict;

int main() {
    t_first = true;
    const uint64_t n = 20001;
    const int tile = 64;
    std::mt19937 rng(5);
    std::vector<unsigned long long> row(n + 1, 0);
    std::vector<unsigned> adj;
    for (uint64_t v = 0; v < n; ++v) {
        const unsigned deg = v % 97 == 0 ? 0 : 20 + rng() % 60;
        std::vector<unsigned> ids;
        for (unsigned i = 0; i < deg; ++i) ids.push_back((unsigned)std::min<uint64_t>(n - 1, (v > 500 ? v - 500 : 0) + rng() % 1000));
        std::sort(ids.begin(), ids.end());
        ids.erase(std::unique(ids.begin(), ids.end()), ids.end());
        adj.insert(adj.end(), ids.begin(), ids.end());
        row[v + 1] = adj.size();
    }
    std::vector<uint16_t> packed[2];
    std::vector<unsigned> blk[2];
    std::vector<uint2> win[2];
    int pack[2], win_max[2];
    for (int run = 0; run < 2; ++run) {
        g_strict = run == 1;
        if (!gpx::pack_lists(row, adj, n, tile, pack[run], packed[run], blk[run], win[run], win_max[run])) {
            printf("not packed\n");
            return 1;
        }
    }
    g_strict = false;
    if (packed[0] != packed[1] || blk[0] != blk[1] || pack[0] != pack[1]) {
        printf("differs\n");
        return 1;
    }
    for (uint64_t v = 0; v < n; ++v) {
        const uint2 w = win[0][v / tile];
        std::vector<unsigned> got;
        for (uint64_t i = (uint64_t)blk[0][v] * 32 * pack[0]; i < (uint64_t)blk[0][v + 1] * 32 * pack[0]; ++i)
            if (packed[0][i] != 4 * w.y) got.push_back(packed[0][i] / 4 + w.x);
        std::sort(got.begin(), got.end());
        if (!std::equal(got.begin(), got.end(), adj.begin() + row[v], adj.begin() + row[v + 1])) {
            printf("edges of %llu\n", (unsigned long long)v);
            return 1;
        }
    }
    printf("PASS\n");
    return 0;
}
