// block_pool.hpp — the bookkeeping of the pool of device blocks behind DeviceBuffer (engine.hpp).
//
// Free of CUDA calls: Api makes them, so that a host test can refuse, count and check them.
//     static void* allocate(int device, size_t bytes);   // nullptr: out of memory; else throws
//     static bool free(int device, void* p);             // false: refused (the block stays)
// Api::free waits for the device, as cudaFree does.
#pragma once

#include <algorithm>
#include <cstddef>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace lqcs_b200 {

constexpr size_t kBlockMax = size_t{32} << 20;   // larger blocks are not the pool's
constexpr size_t kIdleMax = size_t{256} << 20;
// Blocks of up to 1 MiB are cut from slabs of 8 MiB: a plan or a program needs a dozen of them.
constexpr size_t kSlabBlockMax = size_t{1} << 20, kSlab = size_t{8} << 20;

// Capacity of a block for b bytes: the next of 4, 5, 6, 7 times a power of two, 512 at least.
inline size_t block_size(size_t b) {
    size_t step = 128;
    while (step * 8 < b) step <<= 1;
    return std::max<size_t>(512, (b + step - 1) / step * step);
}

template <class Api>
class BlockPool {
  public:
    // A block of block_size(b) bytes, b <= kBlockMax; nullptr if the device has no memory left.
    void* take(int device, size_t b) {
        const size_t want = block_size(b);
        const bool slab = want <= kSlabBlockMax;
        {
            std::lock_guard<std::mutex> lk(mu_);
            if (void* p = find(device, want)) return p;
        }
        void* fresh = Api::allocate(device, slab ? kSlab : want);
        if (!fresh) {   // once more without the idle blocks
            clear();
            fresh = Api::allocate(device, slab ? kSlab : want);
        }
        if (fresh && slab) {
            std::lock_guard<std::mutex> lk(mu_);
            slabs_[device].push_back({static_cast<char*>(fresh), want, 1});
        }
        return fresh;
    }

    // A block of `bytes` from take() comes back.  idle: no work on it is pending, it may be
    // handed out again.  Otherwise it never is: it is freed with a later block that is idle, or
    // with its slab once that has no block in use (Api::free waits for the work).
    void give(int device, void* p, size_t bytes, bool idle) {
        Frees drop;
        {
            std::lock_guard<std::mutex> lk(mu_);
            Slab* s = bytes <= kSlabBlockMax ? slab_of(device, p) : nullptr;
            if (s) --s->live;
            if (idle) {
                idle_[{device, bytes}].push_back(p);
                idle_bytes_[device] += bytes;
                if (idle_bytes_[device] > kIdleMax + pinned_[device]) drop = take_idle();
                drop.insert(drop.end(), later_.begin(), later_.end());
                later_.clear();
            } else if (!s) {
                later_.emplace_back(device, p);
            }
        }
        release(drop);
    }

    // Frees memory that is not the pool's: at once, or with a later block where that is refused.
    void discard(int device, void* p) { release({{device, p}}); }

    // Frees the idle blocks and the slabs without a block in use.
    void clear() {
        Frees drop;
        {
            std::lock_guard<std::mutex> lk(mu_);
            drop = take_idle();
            drop.insert(drop.end(), later_.begin(), later_.end());
            later_.clear();
        }
        release(drop);
    }

  private:
    using Frees = std::vector<std::pair<int, void*>>;
    struct Slab {
        char* base;
        size_t used;   // bytes cut so far
        size_t live;   // blocks in use
    };
    std::mutex mu_;
    std::map<std::pair<int, size_t>, std::vector<void*>> idle_;
    std::map<int, size_t> idle_bytes_;
    std::map<int, size_t> pinned_;   // idle bytes the last take_idle left: slabs with blocks in use
    std::map<int, std::vector<Slab>> slabs_;
    Frees later_;                    // to be freed: work was pending, or Api::free refused

    Slab* slab_of(int device, void* p) {
        for (Slab& s : slabs_[device])
            if (p >= s.base && p < s.base + kSlab) return &s;
        return nullptr;
    }

    // An idle block, or one cut from a slab.
    void* find(int device, size_t want) {
        const bool slab = want <= kSlabBlockMax;
        const auto it = idle_.find({device, want});
        if (it != idle_.end() && !it->second.empty()) {
            void* p = it->second.back();
            it->second.pop_back();
            idle_bytes_[device] -= want;
            if (Slab* s = slab ? slab_of(device, p) : nullptr) ++s->live;
            return p;
        }
        if (!slab) return nullptr;
        for (Slab& s : slabs_[device])
            if (s.used + want <= kSlab) {
                void* p = s.base + s.used;
                s.used += want;
                ++s.live;
                return p;
            }
        return nullptr;
    }

    // Idle blocks and slabs without a block in use, taken out of the pool (to be freed).
    Frees take_idle() {
        Frees drop;
        for (auto& [key, ptrs] : idle_) {
            std::vector<void*> keep;
            for (void* p : ptrs) {
                const Slab* s = key.second <= kSlabBlockMax ? slab_of(key.first, p) : nullptr;
                if (s && s->live > 0) {
                    keep.push_back(p);
                    continue;
                }
                idle_bytes_[key.first] -= key.second;
                if (!s) drop.emplace_back(key.first, p);
            }
            ptrs.swap(keep);
        }
        for (auto& [dev, list] : slabs_) {
            std::vector<Slab> keep;
            for (const Slab& s : list) {
                if (s.live > 0) keep.push_back(s);
                else drop.emplace_back(dev, s.base);
            }
            list.swap(keep);
        }
        pinned_ = idle_bytes_;
        return drop;
    }

    void release(const Frees& drop) {
        for (const auto& [dev, p] : drop) {
            if (Api::free(dev, p)) continue;
            std::lock_guard<std::mutex> lk(mu_);
            later_.emplace_back(dev, p);
        }
    }
};

}  // namespace lqcs_b200
