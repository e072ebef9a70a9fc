// Blocks of memory that are slow to get and give back (page-locked host memory), kept for the
// next owner. Backend: static void* get(size_t) (nullptr: none left), static void put(void*),
// static bool alive(void*). Safe with several threads. A block goes to one owner at a time; its
// owner gives it back when nothing uses it any more.
#pragma once

#include <cstddef>
#include <mutex>
#include <vector>

namespace sankhya {
namespace dev {

template <class Backend>
class BlockPool {
public:
    static constexpr size_t kMinBlock = size_t(1) << 12, kMaxBlock = size_t(1) << 20, kMaxKept = size_t(4) << 20;

    // A block of `bytes` rounded up to a power of two (in size); larger ones than kMaxBlock are
    // neither rounded nor kept. nullptr: there is no memory left.
    void* take(size_t bytes, size_t& size) {
        size = bytes;
        if (bytes <= kMaxBlock)
            for (size = kMinBlock; size < bytes;) size *= 2;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            for (size_t k = free_.size(); k-- > 0;) {
                if (free_[k].size != size) continue;
                void* p = free_[k].ptr;
                free_.erase(free_.begin() + static_cast<std::ptrdiff_t>(k));
                kept_ -= size;
                if (Backend::alive(p)) return p;        // else it went with a device reset
            }
        }
        if (void* p = Backend::get(size)) return p;
        trim();
        return Backend::get(size);
    }
    void give(void* p, size_t size) {
        {
            std::lock_guard<std::mutex> lock(mutex_);
            if (size <= kMaxBlock && kept_ + size <= kMaxKept) {
                free_.push_back({p, size});
                kept_ += size;
                return;
            }
        }
        Backend::put(p);
    }
    // Gives back every block that nobody owns.
    void trim() {
        std::vector<Block> blocks;
        {
            std::lock_guard<std::mutex> lock(mutex_);
            blocks.swap(free_);
            kept_ = 0;
        }
        for (const Block& b : blocks)
            if (Backend::alive(b.ptr)) Backend::put(b.ptr);
    }
    size_t kept() {
        std::lock_guard<std::mutex> lock(mutex_);
        return kept_;
    }

private:
    struct Block {
        void* ptr;
        size_t size;
    };
    std::mutex mutex_;
    std::vector<Block> free_;
    size_t kept_ = 0;
};

}  // namespace dev
}  // namespace sankhya
