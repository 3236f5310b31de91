// Checks the arena allocator of the batch: ranges never overlap, a released
// arena becomes whole again, and a range that cannot grow stays exactly where
// it is.  Exit status 0 when every check holds.
#include "range_allocator.hpp"

#include <cstdio>
#include <random>
#include <vector>

using ocm::RangeAllocator;

static int bad = 0;
static void expect(bool ok, const char* what) {
    if (!ok && bad++ < 20) std::printf("failed: %s\n", what);
}

struct Range {
    int64_t off, size;
};

int main() {
    {   // a hole of the old size in front: the old range must not move there
        RangeAllocator a(100);
        const int64_t hole = a.alloc(20), mid = a.alloc(20), old = a.alloc(20), rest = a.alloc(40);
        a.release(hole, 20);
        expect(a.regrow(old, 20, 60) == -1, "a range of 60 does not fit");
        expect(a.alloc(20) == hole, "the hole is free after the failed growth");
        expect(a.alloc(1) == -1, "the old range is still taken");
        a.release(mid, 20);
        expect(a.regrow(old, 20, 40) == mid, "grows into its own room and the free room before it");
        a.release(hole, 20);
        a.release(mid, 40);
        a.release(rest, 40);
        expect(a.alloc(100) == 0, "whole again");
    }
    std::mt19937 g(7);
    for (int round = 0; round < 200; ++round) {
        const int64_t cap = 200 + g() % 2000;
        RangeAllocator a(cap);
        std::vector<Range> live;
        for (int k = 0; k < 300; ++k) {
            const int64_t align = 1 << g() % 4, size = 1 + g() % 120;
            if (live.empty() || g() % 3) {
                const int64_t off = a.alloc(size, align);
                if (off >= 0) {
                    expect(off % align == 0, "aligned");
                    live.push_back({off, size});
                }
            } else if (g() % 2) {
                const size_t i = g() % live.size();
                const Range was = live[i];
                const int64_t off = a.regrow(was.off, was.size, was.size + size, align);
                if (off >= 0) live[i] = {off, was.size + size};
            } else {
                const size_t i = g() % live.size();
                a.release(live[i].off, live[i].size);
                live.erase(live.begin() + (long)i);
            }
            for (size_t i = 0; i < live.size(); ++i) {
                expect(live[i].off >= 0 && live[i].off + live[i].size <= cap, "inside the arena");
                for (size_t j = 0; j < i; ++j)
                    expect(live[i].off + live[i].size <= live[j].off || live[j].off + live[j].size <= live[i].off,
                           "no overlap");
            }
        }
        for (const Range& r : live) a.release(r.off, r.size);
        expect(a.alloc(cap) == 0, "whole again after random use");
    }
    std::printf("%d failures\n", bad);
    return bad == 0 ? 0 : 1;
}
