// pa_arena.h -- host bookkeeping of offsets that are handed out in pieces.
#pragma once

#include <cstdint>
#include <iterator>
#include <map>
#include <unordered_map>

namespace pa {

class Arena {
public:
    static constexpr uint64_t kNone = ~0ull;
    static constexpr uint64_t kAlign = 512;

    // Add free offsets [at, at + len), multiples of kAlign, to the free pieces.
    void add(uint64_t at, uint64_t len)
    {
        if (len == 0) return;
        auto next = free_.lower_bound(at);
        if (next != free_.end() && at + len == next->first) {
            len += next->second;
            next = free_.erase(next);
        }
        if (next != free_.begin()) {
            const auto prev = std::prev(next);
            if (prev->first + prev->second == at) {
                prev->second += len;
                return;
            }
        }
        free_[at] = len;
    }

    // Take offsets [at, at + len), all free, out of the free pieces.
    void cut(uint64_t at, uint64_t len)
    {
        const auto it = std::prev(free_.upper_bound(at));
        const uint64_t lo = it->first, hi = lo + it->second;
        free_.erase(it);
        if (lo < at) free_[lo] = at - lo;
        if (at + len < hi) free_[at + len] = hi - (at + len);
    }

    // The lowest free piece of `bytes` (rounded up to kAlign), or kNone.
    uint64_t take(uint64_t bytes)
    {
        if (bytes == 0 || bytes > (1ull << 62)) return kNone;
        bytes = (bytes + kAlign - 1) & ~(kAlign - 1);
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            if (it->second < bytes) continue;
            const uint64_t at = it->first;
            cut(at, bytes);
            held_[at] = bytes;
            return at;
        }
        return kNone;
    }

    // Take a piece back; false if none is held at this offset.
    bool give(uint64_t at)
    {
        const auto h = held_.find(at);
        if (h == held_.end()) return false;
        const uint64_t len = h->second;
        held_.erase(h);
        add(at, len);
        return true;
    }

    void clear()
    {
        free_.clear();
        held_.clear();
    }
    const std::map<uint64_t, uint64_t> &pieces() const { return free_; }

private:
    std::map<uint64_t, uint64_t> free_;              // offset -> length, no two adjacent
    std::unordered_map<uint64_t, uint64_t> held_;    // offset -> length
};

}  // namespace pa
