// The register budget of a kernel whose producer warpgroup hands registers to
// its consumers (setmaxnreg): plain arithmetic, checked on the host before the
// kernel's first launch (reg_split_ok in nova_tma.cuh).
#pragma once

namespace nova {

// regs: registers a thread at launch, as compiled (allocated in units of 8).
// The consumers' setmaxnreg.inc draws on what the block was launched with: a sum
// above that would wait without end.
constexpr bool reg_split_fits(int regs, int consumers, int inc, int producers, int dec)
{
    const int r = (regs + 7) / 8 * 8;
    return dec <= r && r <= inc && consumers * inc + producers * dec <= (consumers + producers) * r;
}

}  // namespace nova
