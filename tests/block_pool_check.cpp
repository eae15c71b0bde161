// Host check of the device block pool's bookkeeping (csrc/block_pool.hpp) with a fake device:
// which blocks may be handed out again, what is freed, and when.  test_block_pool.py runs it.
#include <cstdio>
#include <cstdlib>
#include <set>
#include <string>

#include "block_pool.hpp"

namespace {

struct Fake {
    static inline char* next = nullptr;
    static inline std::set<void*> held;
    static inline size_t allocations = 0, bad_frees = 0;
    static inline bool refuse_free = false, out_of_memory = false;
    static void reset() {   // as a device reset: every address is free again
        next = reinterpret_cast<char*>(size_t{1} << 40);   // addresses only, never read
        held.clear();
        allocations = bad_frees = 0;
        refuse_free = out_of_memory = false;
    }
    static void* allocate(int, size_t bytes) {
        if (out_of_memory && !held.empty()) return nullptr;
        void* p = next;
        next += (bytes + 511) / 512 * 512;
        held.insert(p);
        ++allocations;
        return p;
    }
    static bool free(int, void* p) {
        if (refuse_free) return false;
        if (held.erase(p) != 0) return true;
        ++bad_frees;   // not an address of the device's
        return false;
    }
};
using lqcs_b200::block_size;

struct Pool : lqcs_b200::BlockPool<Fake> {
    using Base = lqcs_b200::BlockPool<Fake>;
    uint64_t last = 0;   // era of the block taken last
    void* take(int device, size_t b) { return Base::take(device, b, last); }
    void give(int device, void* p, size_t bytes, bool idle) { Base::give(device, p, bytes, era(), idle); }
    using Base::give;
};

void expect(bool ok, const char* what) {
    if (ok) return;
    std::printf("FAILED: %s\n", what);
    std::exit(1);
}

// A block given back while work on it may be pending (its stream could not be waited for) is not
// handed out again, and does not keep its slab.
void pending_small() {
    Pool pool;
    void* a = pool.take(0, 1000);
    pool.give(0, a, block_size(1000), false);
    for (int i = 0; i < 100; ++i) expect(pool.take(0, 1000) != a, "a pending block was handed out");
    expect(Fake::allocations == 1, "small blocks share a slab");
}
void pending_slab_is_freed() {
    Pool pool;
    void* a = pool.take(0, 1000);
    void* b = pool.take(0, 1000);
    pool.give(0, a, block_size(1000), false);
    pool.clear();
    expect(Fake::held.size() == 1, "a slab with a block in use stays");
    pool.give(0, b, block_size(1000), true);
    pool.clear();
    expect(Fake::held.empty() && Fake::bad_frees == 0, "a slab of pending blocks was not freed");
}
// Larger ones, and frees that the device refuses, are tried again later.
void pending_large() {
    Pool pool;
    const size_t mib2 = size_t{2} << 20;
    const size_t mib64 = size_t{64} << 20;
    void* a = pool.take(0, mib2);
    void* b = pool.take(0, mib2);
    void* c = pool.take(0, mib64);
    Fake::refuse_free = true;   // as during a capture
    pool.give(0, a, mib2, false);
    pool.give(0, c, mib64, false);
    expect(Fake::held.size() == 3, "nothing can be freed now");
    Fake::refuse_free = false;
    pool.give(0, b, mib2, true);
    expect(Fake::held.size() == 1 && Fake::held.count(b) == 1, "refused frees were not tried again");
    expect(pool.take(0, mib2) == b, "an idle block is handed out again");
    expect(pool.take(0, mib2) != a, "a pending block was handed out");
}
// The pool holds little that lies idle, and a failed allocation empties it.
void bounds() {
    Pool pool;
    const size_t mib16 = size_t{16} << 20;
    std::vector<void*> many;
    for (int i = 0; i < 24; ++i) many.push_back(pool.take(0, mib16));
    for (void* p : many) pool.give(0, p, mib16, true);
    expect(Fake::held.size() * mib16 <= lqcs_b200::kIdleMax, "too much lies idle");
    Fake::out_of_memory = true;
    expect(pool.take(0, size_t{32} << 20) != nullptr, "idle blocks were not given up");
}

// What was allocated before the caches were released is not handed out again.  Without a device
// reset in between it is freed with its last block; after one its addresses may be another's.
void released_slab() {
    Pool pool;
    void* a = pool.take(0, 1000);
    void* b = pool.take(0, 1000);
    const uint64_t era = pool.last;
    pool.clear(true);
    void* c = pool.take(0, 1000);
    expect(Fake::allocations == 2, "a block was cut from a retired slab");
    pool.give(0, a, block_size(1000), era, true);
    expect(pool.take(0, 1000) != a, "a block of a retired slab was handed out");
    expect(Fake::held.size() == 2, "a retired slab with a block in use stays");
    pool.give(0, b, block_size(1000), era, true);
    expect(Fake::held.size() == 1 && Fake::bad_frees == 0, "the retired slab was not freed");
    pool.give(0, c, block_size(1000), true);
    expect(pool.take(0, 1000) == c, "a block of this era is handed out again");
}
void released_large() {
    Pool pool;
    const size_t mib2 = size_t{2} << 20;
    void* a = pool.take(0, mib2);
    const uint64_t era = pool.last;
    pool.clear(true);
    pool.give(0, a, mib2, era, true);
    expect(pool.take(0, mib2) != a, "a block from before the release was handed out");
}
void reset_device() {
    Pool pool;
    const size_t mib2 = size_t{2} << 20;
    void* a = pool.take(0, 1000);
    void* b = pool.take(0, 1000);
    void* big = pool.take(0, mib2);
    const uint64_t era = pool.last;
    Fake::reset();
    pool.clear(true);
    void* c = pool.take(0, 1000);   // the same addresses again
    expect(c == a, "the fake device hands out its first address again");
    pool.give(0, a, block_size(1000), era, true);
    pool.give(0, b, block_size(1000), era, true);
    expect(Fake::held.count(c) == 1, "a slab of this era was freed as an old one");
    void* d = pool.take(0, 1000);
    expect(d != c && d != nullptr, "a block in use was handed out twice");
    void* big2 = pool.take(0, mib2);
    expect(big2 == big, "the fake device hands out the same addresses");
    pool.give(0, big, mib2, era, true);
    expect(Fake::held.count(big2) == 1, "a block of this era was freed as an old one");
    expect(Fake::bad_frees == 0, "dead addresses were freed");
    expect(pool.take(0, mib2) != big2, "a block in use was handed out twice");
}

// Idle blocks from before a reset: their free fails, and is not tried again (their addresses may be
// another library's by then).
void reset_with_idle_blocks() {
    Pool pool;
    const size_t mib2 = size_t{2} << 20, mib4 = size_t{4} << 20;
    void* a = pool.take(0, mib2);
    void* b = pool.take(0, 1000);
    pool.give(0, a, mib2, true);
    pool.give(0, b, block_size(1000), true);
    Fake::reset();
    Fake::next += size_t{1} << 30;   // other addresses now
    pool.clear(true);
    expect(Fake::bad_frees == 2, "one try for each");
    void* c = pool.take(0, mib4);
    pool.give(0, c, mib4, true);
    pool.clear();
    pool.clear(true);
    expect(Fake::bad_frees == 2 && Fake::held.empty(), "dead addresses were freed again");
}

}  // namespace

int main() {
    for (auto* check : {pending_small, pending_slab_is_freed, pending_large, bounds, released_slab,
                        released_large, reset_device, reset_with_idle_blocks}) {
        Fake::reset();
        check();
    }
    std::printf("ok\n");
    return 0;
}
