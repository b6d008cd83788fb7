// The linked lists' build numbers over a run longer than the numbers last:
// a model of cell_push / cell_first (fd_kernels.cu) with 8-bit numbers, with
// and without the clock that says when to clear the heads.
#include <cstdio>
#include <cstdint>
#include <vector>
#include "fd_build.h"

struct Table {
    struct Head { uint8_t build; int first; };
    std::vector<Head> head;
    uint8_t build[2] = {1, 1};
    Table() : head(8, Head{0, -1}) {}
    void restart() { head.assign(8, Head{0, -1}); build[0] = build[1] = 1; }
};

// steps of one object that mostly stays in cell 0 and visits the others now
// and then; returns how often a cell it is not in held it
static long run(int steps, bool small, bool use_clock)
{
    Table t;
    fd::BuildClock clock;
    clock.limit = 128;
    long wrong = 0;
    for (int k = 0; k < steps; ++k) {
        if (use_clock && clock.due(1)) { t.restart(); clock.restart(); }
        clock.note(1);
        const int par = k & 1, cell = k % 50 == 0 ? 1 + (k / 50) % 7 : 0;
        if (!small) {  // bump_build
            const uint8_t m = t.build[0] > t.build[1] ? t.build[0] : t.build[1];
            t.build[par] = uint8_t(m + 1);
            t.build[par ^ 1] = uint8_t(m + 2);
        }
        t.head[cell] = Table::Head{t.build[par], k};
        for (int c = 0; c < 8; ++c) wrong += c != cell && t.head[c].build == t.build[par] && t.head[c].first >= 0;
        if (small) t.build[par ^ 1] = uint8_t(t.build[par] + 1);
    }
    return wrong;
}

int main()
{
    for (int small = 0; small < 2; ++small)
        std::printf("%s %d %ld\n", small ? "small" : "staged", run(5000, small, true) == 0, run(5000, small, false));
    fd::BuildClock c;
    std::printf("limit %d\n", c.limit + 2 * fd::BuildClock::PER_STEP * 64 < (uint64_t(1) << 32));
    uint64_t resets = 0, numbers = 0, most = 0;
    for (long k = 0; k < (1l << 33) / 64; ++k) {  // 2^33 steps in calls of 64
        if (c.due(64)) { c.restart(); ++resets; numbers = 0; }
        c.note(64);
        numbers += 2 * 64;
        most = numbers > most ? numbers : most;
    }
    std::printf("resets %d most %d\n", resets > 0, most < (uint64_t(1) << 32));
}
