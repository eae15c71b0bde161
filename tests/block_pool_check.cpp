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
    static void reset() {
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
        if (held.erase(p) == 0) ++bad_frees;
        return true;
    }
};
using Pool = lqcs_b200::BlockPool<Fake>;
using lqcs_b200::block_size;

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
    void* a = pool.take(0, mib2);
    void* b = pool.take(0, mib2);
    Fake::refuse_free = true;   // as during a capture
    pool.give(0, a, mib2, false);
    pool.discard(0, Fake::allocate(0, 64));
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

}  // namespace

int main() {
    for (auto* check : {pending_small, pending_slab_is_freed, pending_large, bounds}) {
        Fake::reset();
        check();
    }
    std::printf("ok\n");
    return 0;
}
