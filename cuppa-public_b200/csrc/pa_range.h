// pa_range.h -- a range of device memory that a request server's lane hands out by
// itself, without the driver.
//
// An allocation from a CUDA memory pool may have the driver map memory, move it or
// wait for work that still uses it: milliseconds to seconds on the calling thread.
// take() and give() are host bookkeeping alone (Arena).  Where take() finds no piece
// large enough, regroup() moves the range's free pages together; it calls the driver,
// and is for a moment at which no work is queued.
//
// The pieces are for work of one stream: a piece given back is next used by work
// queued later on that stream.  One thread at a time.
#pragma once

#include <cstdint>
#include <vector>

#include "pa_arena.h"

namespace pa {

class DeviceRange {
public:
    DeviceRange() = default;
    DeviceRange(const DeviceRange &) = delete;
    DeviceRange &operator=(const DeviceRange &) = delete;
    ~DeviceRange() { close(); }

    // Map about `bytes` of the device, which is current; false (and nothing held) if
    // that fails.
    bool open(int device, uint64_t bytes);
    // Unmap everything (no work that uses it is queued).
    void close();

    void *take(uint64_t bytes) { return base_ ? at(arena_.take(bytes)) : nullptr; }
    bool give(void *p)
    {
        const uint64_t off = (uint64_t)((unsigned char *)p - base_);
        return base_ && (unsigned char *)p >= base_ && off < page_ * pages_.size() && arena_.give(off);
    }
    // take(), after whole free pages have been moved together; null if there are too few.
    void *regroup(uint64_t bytes);

private:
    void *at(uint64_t off) { return off == Arena::kNone ? nullptr : base_ + off; }

    int device_ = 0;
    unsigned char *base_ = nullptr;            // reserved addresses, pages_.size() pages of them
    uint64_t page_ = 0;
    std::vector<unsigned long long> pages_;    // memory mapped at each page, 0 for none
    Arena arena_;
};

}  // namespace pa
