// Test harness (tests only) of the captured wave graphs' keys.
#include <cstdio>
#include "vkb_graphs.h"

using vkb_host::WaveGraphs;
using vkb_host::WaveKey;

static int check(bool ok, const char* what) {
    if (!ok) std::printf("FAIL %s\n", what);
    return ok ? 0 : 1;
}

int main() {
    int bad = 0;
    WaveGraphs<int> graphs;
    // Two jobs of 7500 paths and three of 4484, 1 sample each (trace 938 and 841 blocks).
    WaveKey two, three;
    two.bounces = three.bounces = 4;
    two.jobs = 2; two.trace = 938; two.split = 15; two.shade = 148;
    three.jobs = 3; three.trace = 841; three.split = 14; three.shade = 148;
    graphs.add(two, 2);
    bad += check(!graphs.find(three), "another job count with other grids is another graph");
    graphs.add(three, 3);
    bad += check(graphs.find(two) && *graphs.find(two) == 2 && *graphs.find(three) == 3, "each key finds its own graph");
    WaveKey each[8] = {two, two, two, two, two, two, two, two};
    each[0].bounces++; each[1].jobs++; each[2].counted = true; each[3].ext = true; each[4].w8 = true; each[5].trace++; each[6].split++; each[7].shade++;
    for (const WaveKey& k : each) bad += check(!graphs.find(k), "every field tells graphs apart");
    if (!bad) std::printf("OK\n");
    return bad;
}
