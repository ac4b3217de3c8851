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
    auto drop = [](int) {};
    graphs.add(two, 2, drop);
    bad += check(!graphs.find(three), "another job count with other grids is another graph");
    graphs.add(three, 3, drop);
    bad += check(graphs.find(two) && *graphs.find(two) == 2 && *graphs.find(three) == 3, "each key finds its own graph");
    WaveKey each[8] = {two, two, two, two, two, two, two, two};
    each[0].bounces++; each[1].jobs++; each[2].counted = true; each[3].ext = true; each[4].w8 = true; each[5].trace++; each[6].split++; each[7].shade++;
    for (const WaveKey& k : each) bad += check(!graphs.find(k), "every field tells graphs apart");
    // Waves of every size up to 64 Mi slots: grids for at least the wave's and less than twice
    // its slots, in few sizes.
    size_t sizes = 0;
    uint32_t last = 0;
    for (uint64_t n = 1; n <= (64u << 20); n += 1 + n / 1000) {
        const uint32_t s = vkb_host::graph_slots(uint32_t(n));
        bad += check(s >= n && (s < 2 * n || s == 1024), "slots cover the wave");
        if (s != last) ++sizes;
        last = s;
    }
    bad += check(sizes == 17, "one size per doubling");
    // A server's life: every wave another key.  The graphs kept are bounded, the one given
    // back is the least recently used, and each is given back once.
    WaveGraphs<int> life;
    std::vector<int> dropped;
    for (int k = 0; k < 1000; ++k) {
        WaveKey key = two;
        key.jobs = uint32_t(k);
        bad += check(!life.find(key), "a new wave has no graph");
        life.add(key, k, [&](int e) { dropped.push_back(e); });
        key.jobs = 0;   // the first one is used between all others
        bad += check(life.find(key) && *life.find(key) == 0, "a graph in use stays");
    }
    bad += check(life.kept.size() == WaveGraphs<int>::KEEP && dropped.size() == 1000 - WaveGraphs<int>::KEEP, "bounded");
    for (size_t k = 0; k < dropped.size(); ++k) bad += check(dropped[k] == int(k) + 1, "the oldest goes first");
    if (!bad) std::printf("OK\n");
    return bad;
}
