// The slots of claimed tiles (claim_slot in blp.cuh), on the CPU: one thread that stores claims and a warp that is as
// late as the barriers let it be, for the order of stores, barriers and reads of a kernel.  Prints how many reads find
// another claim than the one they want.
//
//   claim_slots <layernorm|miniweather_x> <tiles of a CTA>
#include "blp.cuh"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

struct Step {
    enum Kind { Store, Read, Barrier } kind;
    int claim;
};

// What a CTA of that kernel does with its slots, claim by claim.
static std::vector<Step> steps_of(const char *kernel, int tiles) {
    std::vector<Step> s;
    if (!strcmp(kernel, "layernorm"))
        s = {{Step::Store, 0}, {Step::Store, 1}, {Step::Barrier, 0}, {Step::Read, 0}, {Step::Read, 1}};
    else
        s = {{Step::Store, 0}, {Step::Barrier, 0}, {Step::Read, 0}, {Step::Store, 1}, {Step::Barrier, 0}, {Step::Read, 1}};
    for (int claim = 2; claim <= tiles; ++claim) {  // behind a tile, the claim for the tile after next
        s.push_back({Step::Store, claim});
        s.push_back({Step::Barrier, 0});
        s.push_back({Step::Read, claim});
    }
    return s;
}

int main(int argc, char **argv) {
    if (argc < 3) return 2;
    const std::vector<Step> steps = steps_of(argv[1], atoi(argv[2]));
    int slots[gpx::kClaimSlots];
    for (int &v : slots) v = -1;
    // The first thread runs ahead to the next barrier; only then does the late warp run up to it.
    int wrong = 0;
    size_t late = 0;
    for (size_t at = 0; at <= steps.size(); ++at) {
        if (at < steps.size() && steps[at].kind == Step::Store) slots[gpx::claim_slot(steps[at].claim)] = steps[at].claim;
        if (at < steps.size() && steps[at].kind != Step::Barrier) continue;
        for (; late < at; ++late)
            if (steps[late].kind == Step::Read && slots[gpx::claim_slot(steps[late].claim)] != steps[late].claim) ++wrong;
    }
    printf("%d\n", wrong);
    return 0;
}
