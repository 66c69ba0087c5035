// The digit passes' look-back words for counts up to a launch's limit of 2^31 - 1
// keys, and a look-back over tiles whose counts pass 2^30, on the host.
#include <cstdio>

#include "sort.cuh"

using gpma::SortWord;

int main() {
    for (const uint32_t c : {0u, 1u, 4608u, (1u << 30) - 1, 1u << 30, (1u << 30) + 1, (1u << 31) - 1}) {
        const SortWord w = SortWord::upto(c);
        if (!w.published() || !w.is_upto() || w.count() != c)
            return std::printf("count up to a tile: %u\n", c), 1;
    }
    for (const uint32_t c : {0u, 1u, 4608u}) {
        const SortWord w = SortWord::own(c);
        if (!w.published() || w.is_upto() || w.count() != c)
            return std::printf("own count: %u\n", c), 1;
    }
    if (SortWord{0}.published())
        return std::puts("zero is published"), 1;
    // tiles of 4,608 equal keys: each finds its start from the nearest word that
    // holds the count up to its tile, some of them only with their own count
    const uint32_t tiles = 0x7FFFFFFFu / 4608;
    std::vector<SortWord> status(tiles);
    for (uint32_t t = 0; t < tiles; ++t) {
        uint32_t prefix = 0;
        for (uint32_t p = t; p > 0; --p) {
            prefix += status[p - 1].count();
            if (status[p - 1].is_upto())
                break;
        }
        if (prefix != t * 4608u)
            return std::printf("tile %u starts at %u\n", t, prefix), 1;
        status[t] = t % 5 == 0 ? SortWord::upto(prefix + 4608) : SortWord::own(4608);
    }
    std::puts("ok");
    return 0;
}
