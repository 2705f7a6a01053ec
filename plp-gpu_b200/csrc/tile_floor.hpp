// tile_floor.hpp -- depths that the batches of a handle turned out to need, where
// its tile is chosen per batch. A batch whose restarts outgrew their tile would
// have its like run twice as well, so the next batches start at the depth it
// needed; each floor holds for its engine and kind of batch, no deeper than a
// batch can need, and falls again, so that one odd instance does not cost all
// later batches their residency.
#pragma once

#include <algorithm>

namespace plpb {

struct Floor {
    int P = 0, C = 0;
};

class TileFloors {
public:
    // batches that a floor outlives the one that last raised it: a retry in 64
    // costs a handle that needs the floor 2 %
    static constexpr int BATCHES = 64;

    Floor get(int engine, int wave) const { return at(engine, wave).f; }
    // after a batch that started at `from` and had to go to `to`
    void raise(int engine, int wave, const Floor& from, const Floor& to) {
        Entry& e = at(engine, wave);
        if (to.P <= from.P && to.C <= from.C) {
            if (e.left > 0 && --e.left == 0) e.f = Floor{};
            return;
        }
        if (to.P > from.P) e.f.P = std::max(e.f.P, to.P);
        if (to.C > from.C) e.f.C = std::max(e.f.C, to.C);
        e.left = BATCHES;
    }

private:
    struct Entry {
        Floor f;
        int left = 0;
    };
    Entry e_[2][2];   // [engine][0: one wave, 1: several]
    const Entry& at(int engine, int wave) const { return e_[engine == 1][wave == 1]; }
    Entry& at(int engine, int wave) { return e_[engine == 1][wave == 1]; }
};

// A tile's depth with a floor under it: a pass places at most a box per step and
// adds at most seven points with each.
inline Floor floored(const Floor& depth, const Floor& f, int steps) {
    return {std::max(depth.P, std::min(f.P, (steps + 15) & ~15)),
            std::max(depth.C, std::min(f.C, (1 + 7 * steps + 31) & ~31))};
}

}  // namespace plpb
