// Device blocks that handles leave for their next call instead of freeing them.
#pragma once
#include <algorithm>
#include <cstddef>
#include <mutex>
#include <vector>

// Every block in the pool is idle: take() hands it out, keep() brings it back.  All together hold at most `cap` bytes
// (the oldest go first), a handle's block goes with the handle, and an allocation that fails anywhere in the library
// frees the pool and tries again, so a kept block never is the reason why something does not fit.  Mem: static
// void* get(size_t), null where it does not fit, and static void put(void*), which waits for work that uses the block.
template <typename Mem>
class KeepPool {
    struct Block {
        const void* owner;
        void* p;
        size_t bytes;
    };
    std::mutex m_;
    std::vector<Block> idle_;   // oldest first
    const size_t cap_;

    template <typename Pick>
    void free_where(Pick pick) {
        std::vector<Block> out;
        {
            std::lock_guard<std::mutex> lock(m_);
            auto it = std::stable_partition(idle_.begin(), idle_.end(), [&](const Block& b) { return !pick(b); });
            out.assign(it, idle_.end());
            idle_.erase(it, idle_.end());
        }
        for (const Block& b : out) Mem::put(b.p);
    }

public:
    explicit KeepPool(size_t cap) : cap_(cap) {}
    // The owner's block, if it holds `bytes` (its size into *got); a smaller one is freed.
    void* take(const void* owner, size_t bytes, size_t* got) {
        {
            std::lock_guard<std::mutex> lock(m_);
            for (size_t i = 0; i < idle_.size(); i++)
                if (idle_[i].owner == owner && idle_[i].bytes >= bytes) {
                    void* p = idle_[i].p;
                    *got = idle_[i].bytes;
                    idle_.erase(idle_.begin() + (long)i);
                    return p;
                }
        }
        drop(owner);
        return nullptr;
    }
    void keep(const void* owner, void* p, size_t bytes) {
        {
            std::lock_guard<std::mutex> lock(m_);
            idle_.push_back({owner, p, bytes});
        }
        for (;;) {
            size_t sum = 0;
            void* oldest = nullptr;
            {
                std::lock_guard<std::mutex> lock(m_);
                for (const Block& b : idle_) sum += b.bytes;
                if (sum <= cap_) return;
                oldest = idle_.front().p;
            }
            free_where([&](const Block& b) { return b.p == oldest; });
        }
    }
    void drop(const void* owner) {
        free_where([&](const Block& b) { return b.owner == owner; });
    }
    void drop_all() {
        free_where([](const Block&) { return true; });
    }
    size_t idle_bytes() {
        std::lock_guard<std::mutex> lock(m_);
        size_t sum = 0;
        for (const Block& b : idle_) sum += b.bytes;
        return sum;
    }
    // An allocation that gives the pool up before it fails.
    void* get(size_t bytes) {
        void* p = Mem::get(bytes);
        if (p || !idle_bytes()) return p;
        drop_all();
        return Mem::get(bytes);
    }
};
