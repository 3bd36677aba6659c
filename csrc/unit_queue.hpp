// Which units a cluster of the expert GEMM computes: those of its own place in the grid, then those of the places that it takes over
// from clusters that have not started.  One header for the device code and for the host model of it that the CPU tests run.
#pragma once
#include "layout.hpp"

namespace nep {
namespace gemm {

constexpr int kUnitSlots = 2;  // units handed out ahead of their readers
constexpr int64_t kFewPlaces = 1024, kManyPlaces = 16384;

// Clusters of a launch, one per place: as many as the offsets allow units, but not many more than rows of at most `largest` per expert
// (0: unknown) could need.  Place p stands for the units p, p + places, p + 2 * places and so on, so every unit has one
// however wrong that expectation is.
// A cluster without a unit costs five nanoseconds to take over: the up-projection of 32 experts with ranges of 4096 rows, 8 of them
// real, 413 us with a place for every unit that the offsets allow, 291 with 1024 (fixed shares 293), at 1024 x 512 instead of
// 7168 x 2048 66 and 31 (31); one expert with rows 224 and 60 (61), 45 and 14.6 (14.6).  A place of several units costs locality: 32 x 4096
// rows 6060-6160 us with a place for each of 8192 units, 6670-6830 with 4096 or 2048 places.  So few places only where
// `largest` says so; without it, 16384 of them are 80 us at worst, underneath the work.
NEP_HD int64_t unit_places(int64_t allowed, int64_t experts, int64_t largest, int64_t tile_tokens, int64_t weight_tiles) {
    int64_t places = largest > 0 ? experts * ((largest + tile_tokens - 1) / tile_tokens) * weight_tiles : kManyPlaces;
    if (places < kFewPlaces) places = kFewPlaces;
    return allowed < places ? allowed : places;
}

// `Io` asks for the next cluster's place (-1: none was left), waits until the slot of the n-th hand-out may be written, and writes it;
// the first two say whether they came to an end within their time limit.  Every unit of the cluster's `own` place but the first and
// all units of every answer are handed out, in whatever order answers come, and "none" once, at the end.  Places behind the last
// unit (the offsets may allow more than the counts give work) are taken too, so that their clusters need not start.
template <typename Io>
NEP_HD bool hand_out_units(Io& io, int units, int places, int own) {
    int handed = 0, free_slots = kUnitSlots;  // hand-outs so far, and for how many there was a slot
    auto slot = [&]() {
        if (handed < free_slots) return true;
        ++free_slots;
        return io.wait_read(handed);
    };
    for (int place = own, unit = own + places;;) {  // the readers start with the first unit of their own place
        for (; unit < units; unit += places) {
            if (!slot()) return false;
            io.hand_out(handed++, unit);
        }
        // Nothing is asked for that would have to wait, or another cluster could have had it sooner.  Clusters are taken over in order
        // (not that anything but time depends on it), so behind an answer past the last unit there is usually no other kind.
        if (place < units && !slot()) return false;
        if (!io.request(place)) return false;
        if (place < 0) break;
        unit = place;
    }
    if (!slot()) return false;
    io.hand_out(handed, -1);
    return true;
}

}  // namespace gemm
}  // namespace nep
