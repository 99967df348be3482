// Which buffers the launches of a stream may still be writing.
#pragma once
#include <stddef.h>
#include <stdint.h>

#include <vector>

namespace nnb {

// Launches overlap: one starts when every block of the launch before it has begun, and may then fetch its weights before it
// waits for that launch's end.  Because the launch before it may have begun just as early, a weight may be the output of any
// call since the last launch that started only after all work before it (an "ordered" one), however many that are.  So all
// of their outputs are kept; a step or a prompt writes the same few buffers again and again, and when more than `limit` are out,
// the next launch that reads ahead is ordered and the list starts anew.  (MAX covers a 30-layer prompt whose k and v rows go to
// places of their own; one ordered launch costs some 2 us.  While a step is recorded there is no limit: an ordered launch in the
// middle of a run of operators would break it in two, and the recording ends.)
struct InFlight {
    static constexpr size_t MAX = 64;
    struct Range {
        uintptr_t lo, hi;
    };
    std::vector<Range> out;
    size_t limit = MAX;
    bool more = false;   // outputs that are not listed

    void wrote(const void* p, size_t bytes) {
        const uintptr_t a = (uintptr_t)p, b = a + bytes;
        if (!p || !bytes || more) return;
        for (Range& r : out) {
            if (r.lo <= a && b <= r.hi) return;
            if (a <= r.lo && r.hi <= b) {
                r = Range{a, b};
                return;
            }
        }
        if (out.size() >= limit) more = true;
        else out.push_back(Range{a, b});
    }
    bool may_write(const void* p, size_t bytes) const {
        const uintptr_t a = (uintptr_t)p, b = a + bytes;
        bool hit = more;
        for (const Range& r : out) hit |= a < r.hi && r.lo < b;
        return hit && p;
    }
    // What follows starts after everything so far: an ordered launch, a copy, a synchronisation.
    void ordered() {
        out.clear();
        more = false;
    }
    // Outputs that are not known one by one (a replayed recording).
    void wrote_unknown() { more = true; }
};

}  // namespace nnb
