// The waits of one CTA of attention_umma.cu in every order in which its copies can land, its products end and its threads get on.
#include "tile_phases.h"
#include <set>
#include <tuple>
#include <vector>

namespace {

using Phase = mk::TilePhase (*)(int);

// A wait for phase `parity` of a barrier that has gone through `over` phases.
bool passes(int over, uint32_t parity) { return (uint32_t)(over & 1) != parity; }

struct State {
    int issued = 0, ended = 0;      // products in the order of their issue: scores 0, scores 1, output 0, scores 2, output 1, ...; they end in that order
    int asked = 0;                  // copies asked for: keys 0, values 0, keys 1, ...
    unsigned landed = 0;
    int tile = 0, step = 0;         // of the threads that hold the items: 0 waiting for scores, 1 before the rescaling, 2 weights to be handed over
    bool operator<(const State& o) const { return std::tie(issued, ended, asked, landed, tile, step) < std::tie(o.issued, o.ended, o.asked, o.landed, o.tile, o.step); }
};

struct Walk {
    int n, stages;
    Phase outputs;
    std::vector<int> order;         // products: tile of scores, or ~tile of an output
    std::set<State> seen;
    int wrong = 0;

    Walk(int tiles, int st, Phase o) : n(tiles), stages(st), outputs(o) {
        order.push_back(0);
        for (int t = 0; t < n; ++t) {
            if (t + 1 < n) order.push_back(t + 1);
            order.push_back(~t);
        }
    }
    int scores_ended(const State& s, int area) const {
        int k = 0;
        for (int i = 0; i < s.ended; ++i) k += order[i] >= 0 && mk::tile_phase(order[i]).at == area;
        return k;
    }
    int outputs_ended(const State& s, int at) const {   // at < 0: all
        int k = 0;
        for (int i = 0; i < s.ended; ++i) k += order[i] < 0 && (at < 0 || outputs(~order[i]).at == at);
        return k;
    }
    bool score_ended(const State& s, int t) const {
        for (int i = 0; i < s.ended; ++i)
            if (order[i] == t) return true;
        return false;
    }
    int handed_over(const State& s, int area) const {
        int k = 0;
        for (int t = 0; t < s.tile && t < n; ++t) k += mk::tile_phase(t).at == area;
        return k;
    }
    void go(State s) {
        if (!seen.insert(s).second) return;
        if (s.ended < s.issued) { State x = s; ++x.ended; go(x); }
        if (s.asked < 2 * n) {   // the place of a stage is free once the product that read it has ended
            const int t = s.asked / 2 - stages;
            if (t < 0 || (s.asked % 2 == 0 ? score_ended(s, t) : outputs_ended(s, -1) > t)) { State x = s; ++x.asked; go(x); }
        }
        for (int i = 0; i < s.asked; ++i)
            if (!(s.landed >> i & 1)) { State x = s; x.landed |= 1u << i; go(x); }
        if (s.issued < (int)order.size()) {
            const int what = order[s.issued], t = what < 0 ? ~what : what;
            const mk::TilePhase ph = mk::tile_phase(t);
            if (what >= 0 ? (s.landed >> (2 * t) & 1) != 0 : (s.landed >> (2 * t + 1) & 1) != 0 && passes(handed_over(s, ph.at), ph.parity)) {
                if (what < 0 && s.tile <= t) ++wrong;      // weights that are not there
                State x = s;
                ++x.issued;
                go(x);
            }
        }
        if (s.tile == n) {
            const mk::TilePhase last = outputs(n - 1);
            if (s.step == 0 && passes(outputs_ended(s, last.at), last.parity)) {
                if (outputs_ended(s, -1) != n) ++wrong;    // outputs read before they are complete
                State x = s;
                x.step = 1;
                go(x);
            }
        } else if (s.step == 0) {
            const mk::TilePhase ph = mk::tile_phase(s.tile);
            if (passes(scores_ended(s, ph.at), ph.parity)) {
                if (!score_ended(s, s.tile)) ++wrong;
                State x = s;
                x.step = 1;
                go(x);
            }
        } else if (s.step == 1) {
            State x = s;
            x.step = 2;
            if (s.tile == 0) {
                go(x);
            } else {
                go(x);   // the maximum stays: no rescaling, no wait
                const mk::TilePhase ph = outputs(s.tile - 1);
                if (passes(outputs_ended(s, ph.at), ph.parity) && outputs_ended(s, -1) != s.tile) ++wrong;   // rescaled under a product that adds to them
            }
        } else {
            State x = s;
            ++x.tile;
            x.step = 0;
            go(x);
        }
    }
};

int walk(int tiles, int stages, Phase outputs) {
    Walk w(tiles, stages, outputs);
    w.go(State{});
    bool ends = false;
    for (const State& s : w.seen) ends |= s.tile == tiles && s.step == 1;
    return ends ? w.wrong : -1;
}

}  // namespace

extern "C" int emu_tile_phases(int tiles, int stages) { return walk(tiles, stages, mk::tile_phase); }
// One barrier for the output products of all tiles, though only some are waited for.
extern "C" int emu_one_output_barrier(int tiles, int stages) {
    return walk(tiles, stages, [](int t) { return mk::TilePhase{0, (uint32_t)(t & 1)}; });
}
