// range_allocator.hpp - first-fit allocator of ranges of an arena (units are
// arbitrary; host bookkeeping only).
#pragma once
#include <cstdint>
#include <iterator>
#include <map>

namespace ocm {

class RangeAllocator {
  public:
    explicit RangeAllocator(int64_t cap = 0) { reset(cap); }
    void reset(int64_t cap) {
        cap_ = cap;
        free_.clear();
        if (cap > 0) free_[0] = cap;
    }
    // Offset of a new range, -1 when none is free.
    int64_t alloc(int64_t size, int64_t align = 1) {
        if (size <= 0) size = 1;
        for (auto it = free_.begin(); it != free_.end(); ++it) {
            const int64_t a = (it->first + align - 1) / align * align;
            if (a + size <= it->first + it->second) {
                take(it, a, size);
                return a;
            }
        }
        return -1;
    }
    void release(int64_t off, int64_t size) {
        if (size <= 0) size = 1;
        auto it = free_.emplace(off, size).first;
        auto next = std::next(it);
        if (next != free_.end() && it->first + it->second == next->first) {
            it->second += next->second;
            free_.erase(next);
        }
        if (it != free_.begin()) {
            auto prev = std::prev(it);
            if (prev->first + prev->second == it->first) {
                prev->second += it->second;
                free_.erase(it);
            }
        }
    }
    // Offset of a range of `size` in place of [off, off + old_size), whose
    // room it may use, or -1: the old range is then kept as it was.
    int64_t regrow(int64_t off, int64_t old_size, int64_t size, int64_t align = 1) {
        release(off, old_size);
        const int64_t to = alloc(size, align);
        // the same place, not any free range of that size: what lies in the
        // old range, and whoever knows its offset, stays valid
        if (to < 0) take(std::prev(free_.upper_bound(off)), off, old_size <= 0 ? 1 : old_size);
        return to;
    }
    int64_t capacity() const { return cap_; }

  private:
    // Cuts [off, off + size) out of the free range that holds it.
    void take(std::map<int64_t, int64_t>::iterator it, int64_t off, int64_t size) {
        const int64_t begin = it->first, end = it->first + it->second;
        free_.erase(it);
        if (off > begin) free_[begin] = off - begin;
        if (off + size < end) free_[off + size] = end - (off + size);
    }
    int64_t cap_ = 0;
    std::map<int64_t, int64_t> free_;  // offset -> size
};

}  // namespace ocm
