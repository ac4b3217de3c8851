// Device buffers of one context that outlive the object they were made for, and the one way
// to new device memory.  Host-only and over an allocator (Api), so that a plain C++ compiler
// can test it: Api::alloc(bytes) gives memory or null (out of memory) and throws what else
// goes wrong, Api::out_of_memory() throws that, Api::free(p) takes any pointer it gave.
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <vector>

namespace vkb_host {

// Device buffers that scenes and calls of one context gave back, for the next ones: an
// install takes some forty buffers and a display call three, and cudaMalloc / cudaFree (which
// waits for the device) took most of a small scene's install (20,000 birds on the GPU
// builders, first frame of 640x360: 14-25 ms from process to process, 4.0-4.3 ms with kept
// buffers; a 1080p display call 3.3 -> 2.2 ms in a process that makes it over and over, but
// its time is pageable copies and varies between processes by more than that).  Bounded; a buffer comes back only when no work on any stream still uses it; what
// is idle is freed when the context closes or when an allocation of this library runs out of
// memory (device_alloc).
template <class Api> class DevicePool {
public:
    static constexpr size_t KEEP = size_t(256) << 20;   // idle bytes at most
    DevicePool() { std::lock_guard<std::mutex> g(all_mutex()); all().push_back(this); }
    ~DevicePool() {
        { std::lock_guard<std::mutex> g(all_mutex()); all().erase(std::remove(all().begin(), all().end(), this), all().end()); }
        trim();
    }
    // An idle buffer of at least `bytes`, or null; bytes: its size.  Not twice that and more,
    // nor a MiB more: some forty buffers then hold at most 40 MiB that their scene did not ask for.
    void* take(size_t& bytes) {
        std::lock_guard<std::mutex> g(m_);
        auto it = idle_.lower_bound(bytes);
        if (it == idle_.end() || it->first > bytes + std::min(bytes + (size_t(64) << 10), size_t(1) << 20)) return nullptr;
        void* p = it->second.p;
        bytes = it->first;
        held_ -= bytes;
        idle_.erase(it);
        return p;
    }
    // Keeps the buffer, in place of those idle for longest where the bound asks for it (one
    // large scene's buffers would otherwise keep every later scene's out for good).  False
    // for a buffer above the bound itself: the caller frees it.
    bool give(void* p, size_t bytes) {
        std::lock_guard<std::mutex> g(m_);
        if (bytes > KEEP) return false;
        while (held_ + bytes > KEEP) {
            auto oldest = std::min_element(idle_.begin(), idle_.end(), [](const auto& a, const auto& b) { return a.second.since < b.second.since; });
            Api::free(oldest->second.p);
            held_ -= oldest->first;
            idle_.erase(oldest);
        }
        idle_.emplace(bytes, Idle{p, gives_++});
        held_ += bytes;
        return true;
    }
    void trim() {
        std::lock_guard<std::mutex> g(m_);
        for (auto& b : idle_) Api::free(b.second.p);
        idle_.clear();
        held_ = 0;
    }
    static void trim_all() {
        std::lock_guard<std::mutex> g(all_mutex());
        for (DevicePool* p : all()) p->trim();
    }

private:
    static std::mutex& all_mutex() { static std::mutex m; return m; }
    static std::vector<DevicePool*>& all() { static std::vector<DevicePool*> v; return v; }
    std::mutex m_;
    struct Idle { void* p; uint64_t since; };   // since: the give() it came with
    std::multimap<size_t, Idle> idle_;
    size_t held_ = 0;
    uint64_t gives_ = 0;
};

// New device memory.  Before it gives up, what every context's pool holds idle goes back.
template <class Api> void* device_alloc(size_t bytes) {
    void* p = Api::alloc(bytes);
    if (!p) {
        DevicePool<Api>::trim_all();
        p = Api::alloc(bytes);
    }
    if (!p) Api::out_of_memory();
    return p;
}

}  // namespace vkb_host
