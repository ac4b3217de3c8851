// The captured wave graphs of one wave engine: what a capture bakes in, as a key.
// Host-only: compiled into the library and, for its CPU tests, by a plain C++ compiler.
#pragma once
#include <algorithm>
#include <cstdint>
#include <tuple>
#include <utility>
#include <vector>

namespace vkb_host {

// Everything a wave's captured kernels take from the host besides the engine's own buffers:
// the job count (the kernels' searches run over it), the launches (bounces, instrumented or
// not, kernel variants) and their grids.  Compared field by field: a graph of another job
// count would search stale table entries and write past a job's accumulator.
struct WaveKey {
    uint32_t bounces = 0, jobs = 0;
    bool counted = false, ext = false, w8 = false;
    int trace = 0, split = 0, shade = 0;
    auto fields() const { return std::tie(bounces, jobs, counted, ext, w8, trace, split, shade); }
    bool operator==(const WaveKey& o) const { return fields() == o.fields(); }
};

// Path slots that a captured wave's grids are made for: the next power of two, so that the
// waves of a server's life, no two alike, share a graph per doubling (the kernels stride or
// take from a counter: a grid of up to twice the blocks a wave needs does the same work).
inline uint32_t graph_slots(uint32_t paths) {
    uint32_t s = 1024;
    while (s < paths && s < (uint32_t(1) << 31)) s <<= 1;
    return s;
}

// The graphs kept, the least recently used first; at most KEEP, as waves of many job counts
// and depths would otherwise leave one each for as long as the engine lives.
template <class Exec> struct WaveGraphs {
    static constexpr size_t KEEP = 64;
    std::vector<std::pair<WaveKey, Exec>> kept;
    Exec* find(const WaveKey& key) {
        for (size_t k = 0; k < kept.size(); ++k)
            if (kept[k].first == key) {
                std::rotate(kept.begin() + k, kept.begin() + k + 1, kept.end());
                return &kept.back().second;
            }
        return nullptr;
    }
    // drop(exec) gives back the graph that makes room (it may still be running: destroying an
    // executable graph waits for that by itself).
    template <class Drop> Exec* add(const WaveKey& key, Exec exec, Drop drop) {
        if (kept.size() >= KEEP) {
            drop(kept.front().second);
            kept.erase(kept.begin());
        }
        kept.emplace_back(key, exec);
        return &kept.back().second;
    }
};

}  // namespace vkb_host
