// RoundProgress (csrc/cuda/progress.h) over sequences of round counters: exit code 0 when every
// answer is the expected one, else the number of the failing sequence.
#include "progress.h"

#include <vector>

using gnd::RoundProgress;

struct Read {
    uint32_t iterations;
    uint64_t retired;
    uint32_t inflight;
    bool stuck;
};

static bool holds(uint64_t total, const std::vector<Read>& reads) {
    RoundProgress p;
    for (const Read& r : reads)
        if (p.stuck(r.iterations, r.retired, r.inflight, total) != r.stuck) return false;
    return true;
}

int main() {
    // a render that ends
    if (!holds(100, {{8, 40, 60, false}, {14, 100, 0, false}, {14, 100, 0, false}})) return 1;
    // a round that ends between two passes: nothing in flight, the next pass begins in the next round
    if (!holds(200, {{8, 100, 0, false}, {16, 150, 50, false}, {22, 200, 0, false}})) return 2;
    // long paths: iterations without a retired sample
    if (!holds(10, {{8, 4, 6, false}, {16, 4, 6, false}, {24, 4, 6, false}, {30, 10, 0, false}})) return 3;
    // lost paths: the loop has nothing to run any more
    if (!holds(100, {{8, 90, 0, false}, {8, 90, 0, true}})) return 4;
    // every path lost in the first round
    if (!holds(100, {{2, 0, 0, false}, {2, 0, 0, true}})) return 5;
    // nothing ever started
    if (!holds(100, {{0, 0, 0, true}})) return 6;
    return 0;
}
