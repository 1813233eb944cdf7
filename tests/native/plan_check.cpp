// Host-side sizes of the batched peel, for tests/test_peel_plan.py.
//
//   plan_check scratch LATE n,L,entries,largest_degree ...
//
// prints the scratch bytes of one launch over these graphs, all columns each.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "device.h"

int main(int argc, char** argv) {
    const bool late = atoi(argv[2]) != 0;
    std::vector<fc::PeelSegSpec> specs;
    for (int i = 3; i < argc; i++) {
        unsigned long long n, L, entries, deg;
        if (sscanf(argv[i], "%llu,%llu,%llu,%llu", &n, &L, &entries, &deg) != 4) return 2;
        fc::PeelSegSpec sp{};
        sp.g.n = (uint32_t)n;
        sp.g.L = (uint32_t)L;
        sp.g.entries = entries;
        sp.g.max_level = (uint32_t)deg + 1;
        sp.ncols = sp.g.L;
        specs.push_back(sp);
    }
    printf("%llu\n", (unsigned long long)fc::peel_batch_ws_bytes(specs, late));
    return 0;
}
