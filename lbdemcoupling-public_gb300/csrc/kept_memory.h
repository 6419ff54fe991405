// Device memory that handles keep between calls (the adjoint window's buffers).
//
// A block per owner of at most `each` bytes, `all` bytes in the process; a block is out of here
// while its owner works in it, and its work has finished when it comes back.  So an idle
// block can be freed at any time, from any thread: by its owner, or by an allocation of any
// handle on the device that would fail otherwise.  The freeing stands under the lock, so that
// an allocation that fails meanwhile finds the memory free and not merely gone from here.
#pragma once

#include <cstddef>
#include <mutex>
#include <new>
#include <vector>

namespace lbdem {

class KeptMemory {
public:
    struct Block {
        void* p = nullptr;
        size_t bytes = 0;
        int device = 0;
        const void* owner = nullptr;
    };

    KeptMemory(size_t each, size_t all) : each_(each), all_(all) {}

    // The owner's idle block, which leaves here (p == nullptr: none).
    Block take(const void* owner) {
        std::lock_guard<std::mutex> lock(mutex_);
        for (size_t k = 0; k < idle_.size(); ++k)
            if (idle_[k].owner == owner) {
                const Block b = idle_[k];
                idle_.erase(idle_.begin() + (std::ptrdiff_t)k);
                return b;
            }
        return Block{};
    }
    // Keeps a block; false (the caller frees it) when that would be too much, or the host has
    // no memory for the entry.
    bool keep(const Block& b) {
        std::lock_guard<std::mutex> lock(mutex_);
        size_t sum = b.bytes;
        for (const Block& k : idle_) sum += k.bytes;
        if (b.bytes > each_ || sum > all_) return false;
        try {
            idle_.push_back(b);
        } catch (const std::bad_alloc&) {
            return false;
        }
        return true;
    }
    size_t held(const void* owner) {
        std::lock_guard<std::mutex> lock(mutex_);
        size_t sum = 0;
        for (const Block& k : idle_)
            if (k.owner == owner) sum += k.bytes;
        return sum;
    }
    // Frees every idle block of a device; whether there was one.
    template <typename Free>
    bool give_back(int device, const Free& free_block) {
        std::lock_guard<std::mutex> lock(mutex_);
        bool any = false;
        for (size_t k = idle_.size(); k-- > 0;)
            if (idle_[k].device == device) {
                free_block(idle_[k].p);
                idle_.erase(idle_.begin() + (std::ptrdiff_t)k);
                any = true;
            }
        return any;
    }

private:
    const size_t each_, all_;
    std::mutex mutex_;
    std::vector<Block> idle_;
};

}  // namespace lbdem
