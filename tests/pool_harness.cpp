// Test harness (tests only) of the kept device buffers, over an allocator of 1 GiB.
#include <cstdio>
#include <cstdlib>
#include <map>
#include <stdexcept>
#include "vkb_pool.h"

struct Api {
    static size_t limit, used, calls;
    static std::map<void*, size_t> live;
    static void* alloc(size_t bytes) {
        ++calls;
        if (used + bytes > limit) return nullptr;
        void* p = std::malloc(1);
        live[p] = bytes;
        used += bytes;
        return p;
    }
    [[noreturn]] static void out_of_memory() { throw std::runtime_error("out of memory"); }
    static void free(void* p) {
        auto it = live.find(p);
        if (it == live.end()) { std::printf("FAIL freed twice\n"); std::exit(1); }
        used -= it->second;
        live.erase(it);
        std::free(p);
    }
};
size_t Api::limit = size_t(1) << 30, Api::used = 0, Api::calls = 0;
std::map<void*, size_t> Api::live;
using Pool = vkb_host::DevicePool<Api>;
constexpr size_t MIB = size_t(1) << 20;

static int bad = 0;
static void check(bool ok, const char* what) {
    if (!ok) { std::printf("FAIL %s\n", what); ++bad; }
}
// As an object's buffers: from the pool if it has one, given back to it or freed.
struct Buf { void* p; size_t bytes; };
static Buf take(Pool& pool, size_t bytes) {
    size_t b = bytes;
    void* p = pool.take(b);
    if (!p) p = vkb_host::device_alloc<Api>(b = bytes);
    return {p, b};
}
static void drop(Pool& pool, Buf b) {
    if (!pool.give(b.p, b.bytes)) Api::free(b.p);
}

static void allocations_trim() {
    // 200 MiB idle in each of two pools, 600 MiB in use: 300 MiB more fit once both are emptied.
    Pool a, b;
    drop(a, take(a, 200 * MIB));
    drop(b, take(b, 200 * MIB));
    check(Api::used == 400 * MIB, "idle buffers are kept");
    void* big = vkb_host::device_alloc<Api>(600 * MIB);
    void* p = vkb_host::device_alloc<Api>(300 * MIB);
    check(Api::used == 900 * MIB, "an allocation frees what is idle");
    bool failed = false;
    try { vkb_host::device_alloc<Api>(200 * MIB); } catch (const std::runtime_error&) { failed = true; }
    check(failed && Api::used == 900 * MIB, "and then says that memory is out");
    Api::free(big);
    Api::free(p);
}

static void reuse_is_close_in_size() {
    Pool pool;
    const size_t idle[] = {100, 70000, 300000, 3 * MIB, 40 * MIB};
    for (size_t b : idle) drop(pool, {Api::alloc(b), b});
    const struct { size_t ask, got; } asks[] = {{60, 100}, {60, 60}, {150000, 300000}, {33 * MIB, 33 * MIB}, {3 * MIB - 5, 3 * MIB}, {39 * MIB, 40 * MIB}, {2000, 2000}, {4464, 70000}};
    std::vector<Buf> held;
    size_t before = Api::used;
    for (const auto& a : asks) {
        held.push_back(take(pool, a.ask));
        check(held.back().bytes == (a.ask == 60 && held.size() == 2 ? 60 : a.got), "a buffer of about the size");
        check(Api::live.at(held.back().p) == held.back().bytes, "its size is the allocation's");
    }
    check(Api::used - before == 60 + 33 * MIB + 2000, "the others are new");
    for (const Buf& b : held) drop(pool, b);
}

static void small_scenes_after_a_large_one() {
    // A scene of 300 MiB in buffers of 10 MiB leaves the pool full; scenes of forty small
    // buffers, one after another, then still find theirs.
    Pool pool;
    std::vector<Buf> large;
    for (int k = 0; k < 30; ++k) large.push_back(take(pool, 10 * MIB));
    for (const Buf& b : large) drop(pool, b);
    check(Api::used == 250 * MIB, "as many as the bound allows");
    for (int turn = 0; turn < 4; ++turn) {
        const size_t before = Api::calls;
        std::vector<Buf> small;
        for (size_t k = 1; k <= 40; ++k) small.push_back(take(pool, k * 100000));
        check(turn == 0 || Api::calls == before, "a small scene's buffers are kept");
        for (const Buf& b : small) drop(pool, b);
        check(Api::used <= Pool::KEEP, "within the bound");
    }
    check(!pool.give(large[0].p, Pool::KEEP + 1), "a buffer above the bound is refused");
}

int main() {
    allocations_trim();
    reuse_is_close_in_size();
    small_scenes_after_a_large_one();
    check(Api::used == 0 && Api::live.empty(), "everything is given back");
    if (!bad) std::printf("OK\n");
    return bad;
}
