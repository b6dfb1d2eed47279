// reachable_block (sph_pinned.h) against a block of bytes that says of each byte which registration holds it.
#include <cstdio>
#include <vector>

#include "../../fdps_sph_gb300/csrc/sph_pinned.h"

using sph::PinnedRange;

static int bad = 0;
static char *const HOST = (char *)0x100000;

struct Piece {
    size_t from, to;   // bytes
    ptrdiff_t shift;   // device address minus host address
};

static const char *route(const std::vector<Piece> &pieces, size_t from, size_t bytes, bool pageable) {
    return sph::reachable_block(HOST + from, bytes, pageable, [&](const char *p) {
        const size_t at = p - HOST;
        for (const Piece &q : pieces)
            if (at >= q.from && at < q.to) return PinnedRange{HOST + q.from, q.to - q.from, p + q.shift};
        return PinnedRange{};
    });
}

static void expect(const char *what, const char *got, const char *want) {
    if (got == want) return;
    std::printf("%s: %p instead of %p\n", what, (const void *)got, (const void *)want);
    ++bad;
}

int main() {
    const std::vector<Piece> whole = {{0, 4096, 0}}, gap = {{0, 1024, 0}, {1032, 4096, 0}},
                             adjoin = {{0, 1024, 0}, {1024, 2048, 0}, {2048, 4096, 0}},
                             apart = {{0, 1024, 0}, {1024, 4096, 512}}, back = {{0, 1024, 0}, {1024, 2048, 8}, {2048, 4096, 0}};
    for (bool pageable : {false, true}) {
        expect("whole", route(whole, 0, 4096, pageable), HOST);
        expect("inside", route(whole, 8, 4080, pageable), HOST + 8);
        expect("one byte", route(whole, 4088, 1, pageable), HOST + 4088);
        expect("past the end", route(whole, 8, 4089, pageable), nullptr);
        expect("misaligned", route(whole, 4, 64, pageable), nullptr);
        expect("empty", route(whole, 0, 0, pageable), nullptr);
        expect("not pinned", route({}, 0, 64, pageable), nullptr);
        expect("ends before the gap", route(gap, 0, 1024, pageable), HOST);
        expect("last byte in the gap", route(gap, 0, 1025, pageable), nullptr);
        expect("first byte in the gap", route(gap, 1024, 64, pageable), nullptr);
        expect("adjoining pieces", route(adjoin, 8, 4080, pageable), HOST + 8);
        expect("mapped apart", route(apart, 0, 4096, pageable), nullptr);
    }
    expect("gap, pageable memory out of reach", route(gap, 0, 4096, false), nullptr);
    expect("gap, pageable memory in reach", route(gap, 0, 4096, true), HOST);
    expect("a piece mapped apart", route(back, 0, 4096, false), nullptr);
    std::vector<Piece> many;
    for (size_t k = 0; k < 512; ++k) many.push_back({8 * k, 8 * k + 8, 0});
    expect("64 pieces", route(many, 0, 512, false), HOST);
    expect("65 pieces", route(many, 0, 513, false), nullptr);
    std::printf("%d wrong\n", bad);
    return bad != 0;
}
