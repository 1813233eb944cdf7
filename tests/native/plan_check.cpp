// Host-side sizes of the batched peel, for tests/test_peel_plan.py.
//
//   plan_check scratch LATE n,L,entries,largest_degree ...
//
// prints the scratch bytes of one launch over these graphs, all columns each.
//
//   plan_check admit BUDGET n,L,entries,largest_degree ...
//
// lets the graphs join a server's batch one after another and prints what its
// admission charges for the batch's scratch, whether it runs without the late
// form, the most scratch that its launches take, and the graphs that joined.
//
//   plan_check group BUDGET n,L,entries,largest_degree
//
// prints the columns that a graph's peel takes at once (FC_PEEL_GROUP_MB in the
// environment), their scratch and that of one column more.
#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "device.h"

using namespace fc;

int main(int argc, char** argv) {
    std::vector<PeelSegSpec> specs;
    std::vector<fc_graph*> graphs;
    for (int i = 3; i < argc; i++) {
        unsigned long long n, L, entries, deg;
        if (sscanf(argv[i], "%llu,%llu,%llu,%llu", &n, &L, &entries, &deg) != 4) return 2;
        PeelSegSpec sp{};
        sp.g.n = (uint32_t)n;
        sp.g.L = (uint32_t)L;
        sp.g.entries = entries;
        sp.g.max_level = (uint32_t)deg + 1;
        sp.ncols = sp.g.L;
        specs.push_back(sp);
        fc_graph* const g = new fc_graph;  // the sizes, no rows
        g->n = sp.g.n;
        g->L = sp.g.L;
        if (!g->off.alloc(L * (n + 1))) return 3;
        g->off[L * (n + 1) - 1] = (uint32_t)entries;
        graphs.push_back(g);
    }
    if (!strcmp(argv[1], "scratch")) {
        printf("%llu\n", (unsigned long long)peel_batch_ws_bytes(specs, atoi(argv[2]) != 0));
        return 0;
    }
    if (!strcmp(argv[1], "group")) {
        DeviceGraph d;
        const PeelGraph& g = specs[0].g;
        d.n = g.n;
        d.L = g.L;
        d.entries = g.entries;
        d.max_deg = g.max_level - 1;
        const uint32_t cols = peel_columns_per_group(&d);
        printf("%u %llu %llu\n", cols, (unsigned long long)peel_ws_bytes(g, cols),
               (unsigned long long)peel_ws_bytes(g, std::min(cols + 1, g.L)));
        return 0;
    }
    const uint64_t budget = strtoull(argv[2], nullptr, 10);
    bool lean = false;
    uint64_t charged = 0, taken = 0;
    std::vector<PeelSegSpec> joined;
    std::vector<fc_graph*> batch;
    for (size_t i = 0; i < graphs.size(); i++) {
        batch.push_back(graphs[i]);
        if (batch_scratch(batch.data(), (uint32_t)batch.size(), 0, budget, false, &lean, &charged))
            batch.pop_back();
        else
            joined.push_back(specs[i]);
    }
    for (uint32_t kind = 0; kind < 3; kind++) {
        std::vector<PeelSegSpec> part;
        for (const PeelSegSpec& sp : joined)
            if (peel_kind(sp.g) == kind) part.push_back(sp);
        if (!part.empty()) taken = std::max(taken, peel_batch_ws_bytes(part, !lean));
    }
    printf("%llu %d %llu %zu\n", (unsigned long long)charged, (int)lean, (unsigned long long)taken,
           joined.size());
    return 0;
}
