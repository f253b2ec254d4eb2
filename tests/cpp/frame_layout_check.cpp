// The block that a frame copies back: nothing overlaps, and the counters that
// searches draw requests from share no 128-byte line with the statistics they
// add to, nor either with the agents' states.
#include <cstdio>

#include "internal.h"

using namespace gmapf_b200;

int main() {
    for (int A : {0, 1, 2, 3, 7, 8, 31, 32, 33, 61, 64, 255, 256, 1000, 4097, 16384, 24001}) {
        const FrameLayout at(A);
        const size_t state_end = at.state + 4 * (size_t)A, counters_end = at.counters + 4 * kCounters;
        const bool ok = at.state >= 8 * (size_t)A && at.counters >= state_end && at.stats >= counters_end &&
                        at.bytes >= at.stats + 8 * ST_COUNT && at.state % 16 == 0 && at.counters % 128 == 0 &&
                        (counters_end - 1) / 128 < at.stats / 128;
        if (!ok) {
            std::printf("A=%d: %zu %zu %zu %zu\n", A, at.state, at.counters, at.stats, at.bytes);
            return 1;
        }
    }
    std::printf("ok\n");
    return 0;
}
