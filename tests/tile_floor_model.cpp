// Prints what a handle's tile floors say after batches that outgrew their tiles,
// one line per question (test_tile_floors.py).
#include <cstdio>

#include "tile_floor.hpp"

using plpb::Floor;

static void show(const Floor& f) { std::printf("%d %d\n", f.P, f.C); }

int main() {
    plpb::TileFloors t;
    t.raise(0, 1, {256, 192}, {256, 1536});
    t.raise(0, 1, {256, 1536}, {1024, 1536});
    for (int engine = 0; engine < 2; engine++)
        for (int wave = 0; wave < 2; wave++) show(t.get(engine, wave));
    // under a batch of 20 steps and one of 2000
    show(plpb::floored({32, 128}, t.get(0, 1), 20));
    show(plpb::floored({256, 192}, t.get(0, 1), 2000));
    // batches of the other kinds leave it; its own kind lets it fall
    for (int k = 0; k < 1000; k++) t.raise(1, 1, {128, 192}, {128, 192});
    show(t.get(0, 1));
    for (int k = 1; k < plpb::TileFloors::BATCHES; k++) t.raise(0, 1, {1024, 1536}, {1024, 1536});
    show(t.get(0, 1));
    t.raise(0, 1, {1024, 1536}, {1024, 1536});
    show(t.get(0, 1));
    return 0;
}
