// Which buffers the launches of a stream may still be writing.
#pragma once
#include <stddef.h>
#include <stdint.h>

namespace nnb {

// Launches overlap: one starts when every block of the launch before it has begun, and may then fetch its weights before it
// waits for that launch's end.  Because the launch before it may have begun just as early, a weight may be the output of any
// call since the last launch that started only after all work before it (an "ordered" one), however many that are.  So all
// of their outputs are kept; a step or a prompt writes the same few buffers again and again, and when more than MAX are out,
// the next launch that reads ahead is ordered and the list starts anew.  (MAX covers a 30-layer prompt whose k and v rows go to
// places of their own; one ordered launch costs some 2 us.)
struct InFlight {
    static constexpr int MAX = 64;
    uintptr_t lo[MAX], hi[MAX];
    int n = 0;
    bool more = false;   // outputs that are not listed

    void wrote(const void* p, size_t bytes) {
        const uintptr_t a = (uintptr_t)p, b = a + bytes;
        if (!p || !bytes || more) return;
        for (int i = 0; i < n; ++i) {
            if (lo[i] <= a && b <= hi[i]) return;
            if (a <= lo[i] && hi[i] <= b) {
                lo[i] = a;
                hi[i] = b;
                return;
            }
        }
        if (n == MAX) {
            more = true;
            return;
        }
        lo[n] = a;
        hi[n++] = b;
    }
    bool may_write(const void* p, size_t bytes) const {
        const uintptr_t a = (uintptr_t)p, b = a + bytes;
        bool hit = more;
        for (int i = 0; i < n; ++i) hit |= a < hi[i] && lo[i] < b;
        return hit;
    }
    // What follows starts after everything so far: an ordered launch, a copy, a synchronisation.
    void ordered() {
        n = 0;
        more = false;
    }
    // Outputs that are not known one by one (a replayed recording).
    void wrote_unknown() { more = true; }
};

}  // namespace nnb
