// sbg_ring.h -- where the next block of an upload ring goes (host only).
#pragma once

#include <algorithm>
#include <cstddef>

namespace sbg {

// Blocks follow each other; one that does not fit behind the last starts again
// at offset 0, over blocks handed out before.  So every kernel that reads a
// block has to be queued before the next block is asked for: place() then says
// that the work queued so far must be waited for (WRAP, GROW), and nothing
// still to be queued can read the bytes that are reused.  Blocks that outlive
// other uploads of the same call go to a ring of their own.
struct RingSpace {
    enum Act { FITS, WRAP, GROW };
    size_t cap = 0, head = 0;
    // offset of a block of `bytes`, rounded up to 256.  WRAP: the ring starts
    // again.  GROW: it has to be reallocated first, with `cap` bytes -- four
    // such blocks, at least `min_cap`.
    Act place(size_t bytes, size_t min_cap, size_t* off) {
        const size_t need = rounded(bytes);
        Act act = FITS;
        if (need > cap) {
            act = GROW;
            cap = std::max(need * 4, min_cap);
            head = 0;
        } else if (head + need > cap) {
            act = WRAP;
            head = 0;
        }
        *off = head;
        head += need;
        return act;
    }
    static size_t rounded(size_t bytes) { return (bytes + 255) & ~(size_t)255; }
    void clear() { cap = head = 0; }
};

}  // namespace sbg
