// The captured wave graphs of one wave engine: what a capture bakes in, as a key.
// Host-only: compiled into the library and, for its CPU tests, by a plain C++ compiler.
#pragma once
#include <cstdint>
#include <tuple>
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

template <class Exec> struct WaveGraphs {
    std::vector<std::pair<WaveKey, Exec>> kept;
    Exec* find(const WaveKey& key) {
        for (auto& g : kept) if (g.first == key) return &g.second;
        return nullptr;
    }
    Exec* add(const WaveKey& key, Exec exec) {
        kept.emplace_back(key, exec);
        return &kept.back().second;
    }
};

}  // namespace vkb_host
