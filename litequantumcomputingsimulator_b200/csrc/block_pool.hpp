// block_pool.hpp — the bookkeeping of the pool of device blocks behind DeviceBuffer (engine.hpp).
//
// Free of CUDA calls: Api makes them, so that a host test can refuse, count and check them.
//     static void* allocate(int device, size_t bytes);   // nullptr: out of memory; else throws
//     static bool free(int device, void* p);             // false: refused (the block stays)
// Api::free waits for the device, as cudaFree does.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace lqcs_b200 {

constexpr size_t kBlockMax = size_t{32} << 20;   // larger blocks are not kept
constexpr size_t kIdleMax = size_t{256} << 20;
// Blocks of up to 1 MiB are cut from slabs of 8 MiB: a plan or a program needs a dozen of them.
constexpr size_t kSlabBlockMax = size_t{1} << 20, kSlab = size_t{8} << 20;

// Capacity of a block for b bytes: the next of 4, 5, 6, 7 times a power of two, 512 at least.
inline size_t block_size(size_t b) {
    size_t step = 128;
    while (step * 8 < b) step <<= 1;
    return std::max<size_t>(512, (b + step - 1) / step * step);
}

// What a buffer for b bytes gets.
inline size_t capacity(size_t b) { return b <= kBlockMax ? block_size(b) : b; }

template <class Api>
class BlockPool {
  public:
    // A block of capacity(b) bytes; nullptr if the device has no memory left.  `era` receives the
    // era it belongs to.
    void* take(int device, size_t b, uint64_t& era) {
        const size_t want = capacity(b);
        const bool slab = want <= kSlabBlockMax;
        {
            std::lock_guard<std::mutex> lk(mu_);
            era = era_;
            if (void* p = find(device, want)) return p;
        }
        void* fresh = Api::allocate(device, slab ? kSlab : want);
        if (!fresh) {   // once more without the idle blocks
            clear();
            fresh = Api::allocate(device, slab ? kSlab : want);
        }
        if (!fresh) return nullptr;
        std::lock_guard<std::mutex> lk(mu_);
        era = owned_[{device, fresh}] = era_;
        if (slab) slabs_[device].push_back({static_cast<char*>(fresh), want, 1, era_});
        return fresh;
    }

    // A block from take() comes back.  idle: no work on it is pending, it may be handed out
    // again, unless it is of an earlier era or larger than the pool keeps.  Otherwise it never
    // is: it is freed with a later block that is idle, or with its slab once that has no block
    // in use (Api::free waits for the work).
    void give(int device, void* p, size_t bytes, uint64_t era, bool idle) {
        std::vector<Free> drop;
        {
            std::lock_guard<std::mutex> lk(mu_);
            const bool now = era == era_;
            Slab* s = bytes > kSlabBlockMax ? nullptr : now ? slab_of(device, p) : retired_slab(device, p, era);
            if (s) --s->live;
            if (bytes > kBlockMax) {
                drop.push_back({device, p, era});
            } else if (!now) {
                if (!s) later_.push_back({device, p, era});
                else if (s->live == 0) drop = drop_retired(s);
            } else if (idle) {
                idle_[{device, bytes}].push_back(p);
                idle_bytes_[device] += bytes;
                if (idle_bytes_[device] > kIdleMax + pinned_[device]) drop = take_idle();
            } else if (!s) {
                later_.push_back({device, p, era});
            }
            if (idle) {
                drop.insert(drop.end(), later_.begin(), later_.end());
                later_.clear();
            }
        }
        release(drop);
    }

    // Frees the idle blocks and the slabs without a block in use.  With `retire` a new era begins:
    // nothing that was allocated before it is handed out any more.  (After a device reset the
    // addresses of blocks in use are no longer theirs.)
    void clear(bool retire = false) {
        std::vector<Free> drop;
        {
            std::lock_guard<std::mutex> lk(mu_);
            drop = take_idle();
            if (retire) {
                ++era_;
                for (auto& [dev, list] : slabs_) {
                    for (const Slab& s : list) retired_.emplace_back(dev, s);
                    list.clear();
                }
                idle_.clear();
                idle_bytes_.clear();
                pinned_.clear();
            }
            drop.insert(drop.end(), later_.begin(), later_.end());
            later_.clear();
        }
        release(drop);
    }

    uint64_t era() {
        std::lock_guard<std::mutex> lk(mu_);
        return era_;
    }

  private:
    struct Free {
        int device;
        void* p;
        uint64_t era;
    };
    struct Slab {
        char* base;
        size_t used;   // bytes cut so far
        size_t live;   // blocks in use
        uint64_t era;
    };
    std::mutex mu_;
    uint64_t era_ = 1;
    std::map<std::pair<int, void*>, uint64_t> owned_;   // allocations, and their eras
    std::map<std::pair<int, size_t>, std::vector<void*>> idle_;
    std::map<int, size_t> idle_bytes_;
    std::map<int, size_t> pinned_;   // idle bytes the last take_idle left: slabs with blocks in use
    std::map<int, std::vector<Slab>> slabs_;
    std::vector<std::pair<int, Slab>> retired_;   // of earlier eras, with blocks in use
    std::vector<Free> later_;        // to be freed: work was pending, or Api::free refused

    Slab* slab_of(int device, void* p) {
        for (Slab& s : slabs_[device])
            if (p >= s.base && p < s.base + kSlab) return &s;
        return nullptr;
    }
    Slab* retired_slab(int device, void* p, uint64_t era) {
        for (auto& [dev, s] : retired_)
            if (dev == device && s.era == era && p >= s.base && p < s.base + kSlab) return &s;
        return nullptr;
    }
    // A retired slab whose last block came back.
    std::vector<Free> drop_retired(const Slab* s) {
        for (size_t i = 0; i < retired_.size(); ++i) {
            if (&retired_[i].second != s) continue;
            const Free f{retired_[i].first, s->base, s->era};
            retired_.erase(retired_.begin() + static_cast<std::ptrdiff_t>(i));
            return {f};
        }
        return {};
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
    std::vector<Free> take_idle() {
        std::vector<Free> drop;
        for (auto& [key, ptrs] : idle_) {
            std::vector<void*> keep;
            for (void* p : ptrs) {
                const Slab* s = key.second <= kSlabBlockMax ? slab_of(key.first, p) : nullptr;
                if (s && s->live > 0) {
                    keep.push_back(p);
                    continue;
                }
                idle_bytes_[key.first] -= key.second;
                if (!s) drop.push_back({key.first, p, era_});
            }
            ptrs.swap(keep);
        }
        for (auto& [dev, list] : slabs_) {
            std::vector<Slab> keep;
            for (const Slab& s : list) {
                if (s.live > 0) keep.push_back(s);
                else drop.push_back({dev, s.base, s.era});
            }
            list.swap(keep);
        }
        pinned_ = idle_bytes_;
        return drop;
    }

    // Frees what is still the pool's (an address of an earlier era may be a later allocation's, of
    // the pool or of others: such a free is tried once only).
    void release(const std::vector<Free>& drop) {
        for (const Free& f : drop) {
            {
                std::lock_guard<std::mutex> lk(mu_);
                const auto it = owned_.find({f.device, f.p});
                if (it == owned_.end() || it->second != f.era) continue;
                owned_.erase(it);
            }
            if (Api::free(f.device, f.p)) continue;
            std::lock_guard<std::mutex> lk(mu_);
            if (f.era != era_) continue;
            owned_.emplace(std::pair{f.device, f.p}, f.era);
            later_.push_back(f);
        }
    }
};

}  // namespace lqcs_b200
