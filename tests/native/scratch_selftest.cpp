// The growth rule of a stream's scratch (halo_b200/csrc/scratch.h) against a driver that keeps books instead of allocating.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "scratch.h"

using namespace halo_cuda;

#define CHECK(cond)                                                             \
    do {                                                                        \
        if (!(cond)) std::printf("line %d: %s\n", __LINE__, #cond), std::exit(1); \
    } while (0)

constexpr uint64_t MB = 1u << 20;
constexpr int kNoMemory = -2, kRefused = -3;

struct Books {
    bool in_capture = false;
    uint64_t limit = UINT64_MAX;  // an allocation above it fails
    std::set<void*> live;
    int drains = 0, clears = 0;
    uintptr_t next = 0x1000;

    bool capturing() const { return in_capture; }
    int drain() { return in_capture ? kRefused : (++drains, 0); }
    int allocate(void** p, uint64_t bytes) {
        if (bytes > limit) return kNoMemory;
        live.insert(*p = reinterpret_cast<void*>(next++));
        return 0;
    }
    int release(void* p) {
        CHECK(live.erase(p) == 1);
        return 0;
    }
    int clear(void*, uint64_t) { return ++clears, 0; }
    int out_of_host_memory() const { return kNoMemory; }
};

int main() {
    Books d;
    Scratch s;
    void *a = nullptr, *b = nullptr, *c = nullptr;
    // eager calls: one block, released when a larger one replaces it
    CHECK(take_scratch(s, 3, 1, false, false, d, &a) == 0 && s.block[3].bytes == MB && d.live.count(a));
    CHECK(take_scratch(s, 3, MB, false, false, d, &b) == 0 && b == a);
    CHECK(take_scratch(s, 3, MB + 1, false, false, d, &b) == 0 && b != a && !d.live.count(a) && s.block[3].bytes == 2 * MB && s.kept.empty());
    // a graph takes the block's address: growth keeps the block, and at least doubles
    d.in_capture = true;
    CHECK(take_scratch(s, 3, 5, false, false, d, &a) == 0 && a == b);
    CHECK(take_scratch(s, 3, 3 * MB, false, false, d, &c) == kRefused && d.live.count(a) && s.block[3].p == a);  // never grown while capturing
    d.in_capture = false;
    CHECK(take_scratch(s, 3, 2 * MB + 1, false, false, d, &c) == 0 && c != a && d.live.count(a) && s.block[3].bytes == 4 * MB);
    CHECK(s.kept.size() == 1 && s.kept[0].p == a && s.total() == 6 * MB);
    // the new block is in no graph: it goes when it is outgrown
    CHECK(take_scratch(s, 3, 9 * MB, false, false, d, &b) == 0 && !d.live.count(c) && d.live.count(a) && s.block[3].bytes == 9 * MB);
    // another slot of the stream is its own; one that is cleared is cleared whenever it is new
    CHECK(take_scratch(s, 2, 8, true, false, d, &c) == 0 && d.clears == 1 && take_scratch(s, 2, 8, true, false, d, &c) == 0 && d.clears == 1);
    d.in_capture = true;
    CHECK(take_scratch(s, 2, 8, true, false, d, &a) == 0 && a == c && take_scratch(s, 3, MB, false, false, d, &a) == 0 && a == b);
    d.in_capture = false;
    CHECK(take_scratch(s, 2, 2 * MB, true, false, d, &a) == 0 && d.clears == 2 && d.live.count(c));
    // a graph's slot grows by what is needed where twice as much is not to be had, and a refused growth leaves the graph's block alive
    d.limit = 10 * MB;
    CHECK(take_scratch(s, 3, 10 * MB, false, false, d, &a) == 0 && s.block[3].bytes == 10 * MB && d.live.count(b));
    CHECK(take_scratch(s, 3, 11 * MB, false, false, d, &a) == kNoMemory && d.live.count(b) && s.block[3].p == nullptr && s.block[3].bytes == 0);
    CHECK(take_scratch(s, 3, MB, false, false, d, &a) == 0 && s.block[3].bytes == MB);
    d.limit = UINT64_MAX;
    // a slot that may grow during a capture waits for nothing then: what the stream still uses is kept beside what the graph takes
    const int drains = d.drains;
    CHECK(take_scratch(s, 4, MB, false, true, d, &a) == 0 && take_scratch(s, 4, 2 * MB, false, true, d, &b) == 0 && !d.live.count(a) && d.drains > drains);
    const size_t kept = s.kept.size();
    d.in_capture = true;
    CHECK(take_scratch(s, 4, 3 * MB, false, true, d, &c) == 0 && d.live.count(b) && s.kept.size() == kept + 1 && s.block[4].in_graph);
    CHECK(take_scratch(s, 1, 3 * MB, false, true, d, &a) == 0 && s.kept.size() == kept + 1 && s.block[1].in_graph);  // the slot's first block
    d.in_capture = false;
    CHECK(take_scratch(s, 4, 16 * MB, false, true, d, &a) == 0 && d.live.count(c) && s.block[4].bytes == 16 * MB);
    // a growth that fails touches no other slot
    d.limit = 16 * MB;
    a = s.block[3].p;
    CHECK(take_scratch(s, 4, 17 * MB, false, true, d, &b) == kNoMemory && s.block[3].p == a && d.live.count(a));
    const int waited = d.drains;  // nor does it wait for the stream again and again, with nothing left to release
    CHECK(take_scratch(s, 4, 17 * MB, false, true, d, &b) == kNoMemory && d.drains == waited);
    s.each([&](void* p) { d.release(p); });
    CHECK(d.live.empty());
    return 0;
}
