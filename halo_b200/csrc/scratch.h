// One stream's scratch blocks and the rule they grow by.  Host code without CUDA types: the driver calls come in as a parameter, so that the
// rule can be run against a fake.
#pragma once
#include <cstdint>
#include <new>
#include <vector>

namespace halo_cuda {

struct ScratchBlock {
    void* p = nullptr;
    uint64_t bytes = 0;
    bool in_graph = false;  // handed out while its stream was being captured: a graph holds the address
};

/// Slot 0 serves the matmul kernels (staged x), slot 1 the LM head (its logits and argmax partials live across a matmul), slot 2 the row-block
/// counters of the balanced kernels (zeroed when allocated, left zeroed by every kernel), slot 3 their partial sums, slot 4 the partial sums of
/// the prefill GEMM's K splits (its own, so that a prompt that cannot have them leaves what a decode step needs).
struct Scratch {
    static constexpr int kSlots = 5;
    ScratchBlock block[kSlots];
    std::vector<ScratchBlock> kept;  // outgrown blocks whose address a graph holds: they live as long as the stream's scratch

    uint64_t total() const {
        uint64_t n = 0;
        for (const ScratchBlock& b : block) n += b.bytes;
        for (const ScratchBlock& b : kept) n += b.bytes;
        return n;
    }
    template <class Release>
    void each(Release&& release) {
        for (ScratchBlock& b : block)
            if (b.p != nullptr) release(b.p);
        for (ScratchBlock& b : kept) release(b.p);
    }
};

/// A block of at least `bytes` in `slot`.  A larger request replaces the block; its contents are dropped.  The old block is released once the
/// stream has drained, unless a graph holds its address: then it is kept, and the new one is at least twice its size, so that what a slot keeps
/// stays below what it holds.  A stream that is being captured cannot be waited for: `while_capturing` says that the slot grows there too (the
/// old block is kept then), else the request is refused.
/// Driver: capturing(), drain(), allocate(&p, bytes), release(p), clear(p, bytes), out_of_host_memory().
template <class Driver>
int take_scratch(Scratch& set, int slot, uint64_t bytes, bool zeroed, bool while_capturing, Driver& driver, void** out) {
    constexpr uint64_t kUnit = 1u << 20;
    ScratchBlock& b = set.block[slot];
    if (bytes > b.bytes) {
        uint64_t want = (bytes + kUnit - 1) & ~(kUnit - 1), least = want;
        const bool capturing = driver.capturing(), keep = b.p != nullptr && (b.in_graph || (capturing && while_capturing));
        // Work already enqueued on this stream may still read a block that is to be released.
        if (capturing ? !while_capturing : !keep && b.p != nullptr)
            if (int rc = driver.drain()) return rc;
        if (keep) {
            try {
                set.kept.push_back(b);
            } catch (const std::bad_alloc&) {
                return driver.out_of_host_memory();
            }
            want = want < 2 * b.bytes ? 2 * b.bytes : want;
        } else if (b.p != nullptr) {
            if (int rc = driver.release(b.p)) return rc;
        }
        b = ScratchBlock{};
        int rc = driver.allocate(&b.p, want);
        if (rc != 0 && want != least) rc = driver.allocate(&b.p, want = least);
        if (rc != 0) {
            b.p = nullptr;
            return rc;
        }
        b.bytes = want;
        if (zeroed)
            if (int rc2 = driver.clear(b.p, want)) return rc2;
    }
    if (!b.in_graph) b.in_graph = driver.capturing();
    *out = b.p;
    return 0;
}

}  // namespace halo_cuda
