// Which units a cluster of the expert GEMM computes behind its own: the units of the clusters whose places it takes over.  One
// header for the device code and for the host model of it that the CPU tests run.
#pragma once
#include "layout.hpp"

namespace nep {
namespace gemm {

constexpr int kUnitSlots = 2;  // units handed out ahead of their readers

// `Io` asks for the next cluster's place (its unit, or -1: none was left), waits until the slot of the n-th hand-out may be written, and
// writes it; the first two say whether they came to an end within their time limit.  Every answer below `units` is handed out, in
// whatever order answers come, and "none" once, at the end.  Answers behind the last unit (the offsets may allow more clusters
// than the counts give work) are taken too, so that those clusters need not start.
template <typename Io>
NEP_HD bool hand_out_units(Io& io, int units) {
    int handed = 0, free_slots = kUnitSlots;  // hand-outs so far, and for how many there was a slot
    auto slot = [&]() {
        if (handed < free_slots) return true;
        ++free_slots;
        return io.wait_read(handed);
    };
    for (int unit = 0;;) {
        // Nothing is asked for that would have to wait, or another cluster could have had it sooner.  Clusters are taken over in order
        // (not that anything but time depends on it), so behind an answer past the last unit there is usually no other kind.
        if (unit < units && !slot()) return false;
        if (!io.request(unit)) return false;
        if (unit >= units) continue;
        if (!slot()) return false;
        io.hand_out(handed++, unit);
        if (unit < 0) return true;
    }
}

}  // namespace gemm
}  // namespace nep
