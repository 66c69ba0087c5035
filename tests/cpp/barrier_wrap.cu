// The grid barrier's rounds (BarrierRound) against a model of the counter, on the
// host: no CTA may pass before the last one of its round has its ticket, also
// where the counter goes back to zero, and every round starts at a multiple of
// the grid.
#include <cstdio>

#include "gpma_internal.cuh"

int main() {
    for (uint32_t ctas : {1u, 2u, 3u, 152u, 304u, 608u, 760u, 912u, 1216u, 65535u}) {
        const uint32_t last = gpma::BarrierRound::last_ticket(ctas);
        if (last == 0xFFFFFFFFu || (last + 1) % ctas != 0)
            return std::printf("%u CTAs: the counter ends inside a round\n", ctas), 1;
        for (uint32_t start : {0u, last + 1 - 2 * ctas}) {
            uint32_t count = start;
            for (int round = 0; round < 5; ++round) {
                std::vector<gpma::BarrierRound> waiting;
                for (uint32_t c = 0; c < ctas; ++c) {
                    const uint32_t ticket = count;  // atomicInc
                    count = ticket >= last ? 0u : ticket + 1;
                    waiting.emplace_back(ticket, ctas);
                    // the first, the last and one waiting CTA between them
                    for (const uint32_t w : {0u, c / 2, c})
                        if (waiting[w].over_long(count) != (c == ctas - 1))
                            return std::printf("%u CTAs, round %d: CTA %u after arrival %u\n", ctas, round, w, c), 1;
                }
                // a slow poll still sees the end while others take the next round's tickets
                for (uint32_t ahead = 0; ahead < ctas; ++ahead)
                    if (!waiting[0].over_long(count + ahead))
                        return std::printf("%u CTAs, round %d: lost after %u\n", ctas, round, ahead), 1;
            }
        }
    }
    // arrivals that never come keep a round open
    const gpma::BarrierRound stalled(303, 304, 1);
    if (stalled.over(304) || stalled.over_long(304))
        return std::puts("a stalled round ended"), 1;
    std::puts("ok");
    return 0;
}
