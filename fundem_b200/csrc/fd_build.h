// fd_build.h -- the build numbers of linked lists on the device (host side).
//
// Cell tables and the reverse index keep, per cell or particle, a list head
// that carries the 32-bit number of the build that wrote it; a head of another
// number reads as empty, so heads are never cleared between steps.  That holds
// as long as no number comes round again while a head can still carry it: a
// small step takes 16 us and one number, so 2^32 of them are gone in a day.
// The clock counts the numbers a run can have used and says when to clear the
// heads and start again.
#pragma once
#include <cstdint>

// well below 2^32: the numbers in use run ahead of the count by a call at most
#ifndef FD_BUILD_LIMIT
#define FD_BUILD_LIMIT (uint64_t(1) << 31)
#endif

namespace fd {

struct BuildClock {
    // numbers a step, or a detection, can use of any one table
    static constexpr uint64_t PER_STEP = 4;
    uint64_t limit = FD_BUILD_LIMIT;
    uint64_t used = 0;

    void restart() { used = 0; }
    // before `steps` steps: true when the heads have to be cleared and the
    // numbers started again first (restart(), then call again)
    bool due(uint64_t steps) const { return used > 0 && used + PER_STEP * steps >= limit; }
    void note(uint64_t steps) { used += PER_STEP * steps; }
};

}  // namespace fd
