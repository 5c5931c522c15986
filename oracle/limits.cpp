// limits.cpp — test infrastructure: the library's sizes and index arithmetic at the limits of a
// scene (diffvg-rs_b200/csrc/limits.hpp), called by tests/test_limits.py.
#include "../diffvg-rs_b200/csrc/limits.hpp"

// Shared-memory bytes of a forward launch over scenes of these filter radii; *all: whether every
// scene accumulates there.
extern "C" size_t limits_splat(const int* ri, int n, int* all) {
    dvgb::SplatPlan p;
    for (int i = 0; i < n; ++i) p.add(ri[i]);
    *all = p.all;
    return p.bytes();
}

// The place in the tile list that the kernels read back from entry `place` of a walk.
extern "C" int limits_place(int listed, int place, int flags) {
    return dvgb::entry_place(listed != 0, place, dvgb::entry_word(listed != 0, place, flags));
}
extern "C" int limits_cell_list_max() { return dvgb::CELL_LIST_MAX; }

// `tiles` requests of `need` places each of `cap`, as k_cells makes them.  Returns the requests
// granted; -1 if a grant reaches past `cap` or into an earlier one.
extern "C" long long limits_room(long long tiles, int need, int cap) {
    unsigned long long taken = 0;
    long long granted = 0, end = 0;
    for (long long i = 0; i < tiles; ++i) {
        const int at = dvgb::room_at(taken, need, cap);
        taken += (unsigned long long)need;
        if (at < 0) continue;
        if (at < end || (long long)at + need > cap) return -1;
        end = (long long)at + need;
        granted += 1;
    }
    return granted;
}

// The room of a scene's cell lists: out = entries, items, their offsets, the counters' offset, bytes.
extern "C" void limits_cell_room(uint64_t tiles, uint64_t tile_entries, uint64_t items, uint64_t budget, uint64_t* out) {
    const dvgb::CellRoom r = dvgb::cell_room(tiles, tile_entries, items, budget);
    const uint64_t v[6] = {r.ents, r.items, r.at_ents, r.at_items, r.at_counters, r.bytes};
    for (int k = 0; k < 6; ++k) out[k] = v[k];
}

extern "C" int limits_entry_steps(int pairs, int curves, int hard, int strokes) {
    return dvgb::entry_steps(pairs, curves, hard, strokes);
}
