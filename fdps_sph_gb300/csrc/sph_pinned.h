// Which host blocks kernels may read and write in place (plain C++, so that the rule can be checked without a GPU).
#pragma once

#include <cstddef>
#include <cstdint>

namespace sph {

// one allocation or registration of pinned host memory, and where the device sees the byte that was asked for
struct PinnedRange {
    const char *start = nullptr;
    size_t size = 0;
    const char *dev = nullptr;
};

// The device's address of the block [p0, p0 + bytes), or null if the copy engine has to carry it.  A block is taken that
// is aligned to 8 bytes and pinned from its first to its last byte; it may span several registrations (an arena pinned
// in pieces) that leave no gap and that the device sees as far apart as the host does.  Ordinary memory between two
// registrations faults a kernel on a device that does not read pageable memory, and only there: where it does
// (`pageable`), a block with pinned ends is taken whatever lies between them (the engine refuses such a block).
// range(p): the PinnedRange that holds p, of size 0 if p is not pinned.
template <class Range>
const char *reachable_block(const char *p0, size_t bytes, bool pageable, Range range) {
    if (((uintptr_t)p0 & 7) || bytes == 0) return nullptr;
    const PinnedRange first = range(p0), last = range(p0 + bytes - 1);
    if (!first.size || !last.size || last.dev - first.dev != (ptrdiff_t)(bytes - 1)) return nullptr;
    if (pageable) return first.dev;
    const char *p = p0;
    for (int piece = 0; piece < 64; ++piece) {   // (a block in more pieces goes to the engine)
        const PinnedRange r = range(p);
        if (!r.size || p < r.start || p >= r.start + r.size || r.dev - first.dev != p - p0) return nullptr;
        if ((size_t)(p0 + bytes - p) <= (size_t)(r.start + r.size - p)) return first.dev;
        p = r.start + r.size;
    }
    return nullptr;
}

}  // namespace sph
