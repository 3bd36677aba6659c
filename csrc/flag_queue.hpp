// A combine's transfer warp announces rows by flags that a publisher warp of the same CTA writes.  This is the order in which
// flags are handed to the publisher; one header for the device code and for the host model of it that the CPU tests run.
#pragma once
#include "layout.hpp"

namespace nep {

constexpr int kFlagRing = 32;       // flags of a transfer warp that the publisher may not have written yet
constexpr int kMaxStoreDepth = 12;  // most bulk stores that a transfer warp may have pending
// Flags that wait: fewer than half a ring of notes, and one per pending store.  A warp whose ring is full has therefore always
// handed something over that the publisher has not written, so the ring empties.
static_assert(kFlagRing / 2 - 1 + kMaxStoreDepth + 1 <= kFlagRing && kMaxStoreDepth < 32, "flag ring");

// `Io` puts a flag on the ring, waits for bulk stores, keeps 32 marks and tells the publisher how many flags it may write.
template <typename Io, typename Flag>
struct FlagQueue {
    Io io;
    int depth;         // bulk stores that may be pending before the warp waits
    int produced = 0;  // flags on the ring
    int handed = 0;    // flags that the publisher may write, and may have written: this never falls
    int groups = 0;    // bulk groups committed; mark g % 32: flags on the ring at the commit of group g

    // Call right after committing the bulk group of the row that `flag` announces.
    NEP_HD void push(Flag flag) {
        io.append(flag, produced++);
        io.set_mark(groups & 31, produced);
        ++groups;
        io.wait_landed(depth);  // everything older than the newest `depth` rows has landed
        // What was on the ring at the commit of the newest of those rows; a note may have handed over more since then.
        if (groups > depth) hand_over(io.mark((groups - 1 - depth) & 31));
    }
    // A flag that announces no bulk store: handed over with the next one that does, or on its own where many have come together.
    NEP_HD void note(Flag flag) {
        io.append(flag, produced++);
        if (produced - handed >= kFlagRing / 2) finish();
    }
    NEP_HD void finish() {
        io.wait_landed(0);
        hand_over(produced);
    }

  private:
    NEP_HD void hand_over(int count) {
        if (count <= handed) return;
        handed = count;
        io.publish_up_to(count);
    }
};

}  // namespace nep
