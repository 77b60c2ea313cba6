// Page-locked blocks that the library hands out for downloads and takes back.
// A copy into pageable memory goes through the driver's staging buffer at about 4 GB/s and faults the destination's fresh pages
// (1.28 MB: 320 us); into page-locked memory it is one transfer at link speed (45 us).  Locking pages takes longer than either,
// so released blocks are kept, by power-of-two size, until the last device handle goes.
#pragma once
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace nkb {

// `lock_pages` allocates page-locked memory (null when there is none), `unlock_pages` frees it; both run outside the pool's lock.
class HostPool {
public:
    // Blocks handed out and kept together stay within kBytes.  One block is at most a quarter of that, or two large fields
    // downloaded in turn would push one another out.
    static constexpr size_t kBytes = size_t{256} << 20, kLargest = kBytes / 4u, kSmallest = 4096;
    // A kept block that stands in the way of a new size is given back once this many blocks were taken since its last use.  A
    // sooner one is part of the caller's loop: locking its pages again in every round would cost more than the pageable copy.
    static constexpr uint64_t kIdleTakes = 256;

    HostPool(void* (*lock_pages)(size_t), void (*unlock_pages)(void*)) : lock_pages_(lock_pages), unlock_pages_(unlock_pages) {}

    // A block of at least `bytes`, or null: the caller then copies into memory of its own.
    void* Take(size_t bytes) {
        size_t size = kSmallest;
        while (size < bytes && size < kLargest) size <<= 1;
        if (size < bytes) return nullptr;
        std::vector<void*> idle;
        {
            std::lock_guard<std::mutex> hold(mutex_);
            ++takes_;
            auto& list = kept_[size];
            if (!list.empty()) {
                void* p = list.back();
                list.pop_back();
                blocks_[p].out = true;
                return p;
            }
            if (total_ + size > kBytes) DropIdle(size, idle);
            if (total_ + size > kBytes) return nullptr;
            total_ += size;                                   // reserved while the pages are locked
        }
        for (void* p : idle) unlock_pages_(p);
        void* p = lock_pages_(size);
        std::lock_guard<std::mutex> hold(mutex_);
        if (p == nullptr) { total_ -= size; return nullptr; }
        blocks_[p] = {size, true, 0u};
        return p;
    }

    // Takes a block back; anything else (a foreign pointer, a block released before) is left alone.
    void Give(void* p) {
        {
            std::lock_guard<std::mutex> hold(mutex_);
            const auto it = blocks_.find(p);
            if (it == blocks_.end() || !it->second.out) return;
            if (users_ != 0u) {
                kept_[it->second.size].push_back(p);
                it->second.out = false;
                it->second.used = takes_;
                return;
            }
            total_ -= it->second.size;
            blocks_.erase(it);
        }
        unlock_pages_(p);
    }

    // A pool without users keeps nothing.
    void Join() {
        std::lock_guard<std::mutex> hold(mutex_);
        ++users_;
    }
    void Leave() {
        std::vector<void*> all;
        {
            std::lock_guard<std::mutex> hold(mutex_);
            if (--users_ != 0u) return;
            for (auto& list : kept_)
                for (void* p : list.second) { total_ -= list.first; blocks_.erase(p); all.push_back(p); }
            kept_.clear();
        }
        for (void* p : all) unlock_pages_(p);
    }

private:
    struct Block { size_t size; bool out; uint64_t used; };

    // Gives idle blocks back if that makes room for `size` more bytes.
    void DropIdle(size_t size, std::vector<void*>& dropped) {
        size_t free = 0;
        auto idle = [&](void* p) { return takes_ - blocks_[p].used > kIdleTakes; };
        for (auto& list : kept_) for (void* p : list.second) if (idle(p)) free += list.first;
        if (total_ - free + size > kBytes) return;
        for (auto& list : kept_)
            for (size_t k = 0; k < list.second.size() && total_ + size > kBytes;) {
                void* p = list.second[k];
                if (!idle(p)) { ++k; continue; }
                list.second[k] = list.second.back();
                list.second.pop_back();
                total_ -= list.first;
                blocks_.erase(p);
                dropped.push_back(p);
            }
    }

    void* (*lock_pages_)(size_t);
    void (*unlock_pages_)(void*);
    std::mutex mutex_;
    std::unordered_map<void*, Block> blocks_;                   // every block, handed out or kept
    std::unordered_map<size_t, std::vector<void*>> kept_;
    size_t total_ = 0;
    uint64_t takes_ = 0, users_ = 0;
};

}  // namespace nkb
