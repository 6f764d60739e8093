// One lane's walk through the ring of copies of narrow_mma.cu, on barriers that know what may not happen to them.
#include "narrow_ring.h"
#include <vector>

namespace {

struct Barrier {
    long phase = 0;        // completed phases
    bool armed = false;    // the present phase expects a copy
};

struct Walk {
    std::vector<Barrier> bars;
    int wrong = 0;
    void arm(int at) {
        if (bars[at].armed) ++wrong;   // a second arrival in an unfinished phase, a second copy into the same bytes
        bars[at].armed = true;
    }
    // The copy lands while the stage is waited for; a parity whose phase is over says so at once, one that nothing completes never does.
    void wait(int at, uint32_t parity) {
        if ((uint32_t)(bars[at].phase & 1) != parity || !bars[at].armed) ++wrong;
        bars[at].armed = false;
        ++bars[at].phase;
    }
};

}  // namespace

// Groups i0 .. i1 - 1, steps a0 .. a1 - 1 of each, as the kernel walks them; the wait of step `fails` (counted through; negative: none) is in vain.  Returns what went wrong:
// misused barriers, copies still under way at the end, copies not waited for that were asked for.
extern "C" int emu_narrow_ring(int stages, int i0, int i1, int rg_shift, int sub_tile, int tiles, int a0, int a1, int fails) {
    Walk w;
    w.bars.resize((size_t)stages);
    const int groups = mk::narrow_live_groups(i0, i1, rg_shift, sub_tile, tiles);
    int wrong = 0;
    for (int i = i0; i < i1; ++i) wrong += (i < i0 + groups) != (((i << rg_shift) + sub_tile) < tiles);
    mk::NarrowRing ring(stages, groups * (a1 - a0));
    auto copy_step = [&] {
        if (!ring.more()) return;
        w.arm(ring.load_stage);
        ring.loaded();
    };
    for (int i = 0; i < stages - 1; ++i) copy_step();
    uint32_t given_up = 0;
    int n = 0;
    for (int i = i0; i < i1; ++i)
        for (int st = a0; st < a1; ++st, ++n) {
            copy_step();
            if (i < i0 + groups && given_up == 0) {
                if (n != fails) w.wait(ring.stage, ring.phase);
                else given_up = ring.give_up((i0 + groups - i) * (a1 - a0) - (st - a0));
            }
            ring.used();
        }
    if (given_up != 0) mk::NarrowRing::drain(stages, given_up, [&](int at, uint32_t parity) { w.wait(at, parity); });
    for (const Barrier& b : w.bars) wrong += b.armed;
    return wrong + w.wrong;
}
