// Whether a render's rounds still get anywhere (no CUDA in here).
#pragma once
#include <cstdint>

namespace gnd {

// A round of the device loop runs no iteration once no path is in flight and no work is left
// to hand out. That is the end of a render with every sample retired; with samples missing,
// their paths are on no list any more, and no further round would find them. A limit on the
// iterations does not see this: they no longer grow.
class RoundProgress {
public:
    // Counters of the next round that was read: iterations run and samples retired since the
    // render began, paths in flight. True when the render cannot end.
    bool stuck(uint32_t iterations, uint64_t retired, uint32_t inflight, uint64_t total) {
        const bool still = inflight == 0 && retired < total && iterations == iterations_ && retired == retired_;
        iterations_ = iterations;
        retired_ = retired;
        return still;
    }

private:
    uint32_t iterations_ = 0;
    uint64_t retired_ = 0;
};

}  // namespace gnd
