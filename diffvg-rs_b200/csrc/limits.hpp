// limits.hpp — sizes and index arithmetic whose limits no test can reach on a device, in plain
// functions that oracle/limits.cpp runs on the CPU (tests/test_limits.py).
#pragma once
#include <algorithm>
#include <cstddef>
#include <cstdint>

#ifdef __CUDACC__
#define DVG_LIM_HD __host__ __device__ __forceinline__
#else
#define DVG_LIM_HD inline
#endif

namespace dvgb {

// Filter radii up to this (ceil) use the shared-memory tile+halo splat.
constexpr int MAX_SMEM_RI = 8;
constexpr int SPLAT_TILE = 16;

// The forward splat of one launch over scenes of several filter radii.  Each scene accumulates
// in shared memory if its own radius fits, so the launch has room for the largest that does,
// whether or not others do not; the lane-group splat, which works in shared memory only, needs
// all of them to fit.
struct SplatPlan {
    int ri = -1;      // the largest radius that fits, -1: none
    bool all = true;  // every scene fits
    void add(int scene_ri) {
        if (scene_ri > MAX_SMEM_RI) all = false;
        else if (scene_ri > ri) ri = scene_ri;
    }
    size_t bytes() const {
        const size_t w = SPLAT_TILE + 2 * (size_t)(ri < 0 ? 0 : ri);
        return ri < 0 ? 0 : w * w * 5 * sizeof(float);
    }
};

// The word of a cell entry: its group's place in the tile list above eight flags.  Longer tile
// lists than CELL_LIST_MAX get no cell lists; a walk over the list itself (`listed` false) has
// any length, and the place is the step of the walk.
constexpr int CELL_LIST_MAX = 1 << 22;
DVG_LIM_HD int entry_word(bool listed, int place, int flags) { return listed ? (place << 8) | flags : flags; }
DVG_LIM_HD int entry_place(bool listed, int step, int word) { return listed ? word >> 8 : step; }

// A cell is heavy from this many steps in its lists: pairs of rows, curves, one-point segments and
// stroke segments.  The kernels are bound by instruction fetch: where the lists are long, a CTA's
// warps take them one entry at a time, so that they run the same code together (forward of the
// large 1024x1024 scene 18.5 -> 14.7 ms, edge pass 62.9 -> 48.0 when it came in).  Against 24, from
// 12 on: batch of 64 icons 5.25 -> 5.58 ms, large render 15.9 -> 15.7; from 40 on: large render
// 16.7, its step 69.6 -> 71.5 ms.
constexpr int CELL_HEAVY = 24;
// A primitive whose edge crosses the cell (`hard` says so: one formula, no segments) makes it heavy
// by itself: its code is a detour from the segments' that the warps had better take together.
// Mixed 512x512 step: edge pass 0.432 ms against 0.476 where it counts as one step, forward
// 0.846 against 0.831.
constexpr int CELL_PRIMITIVE = 63;
DVG_LIM_HD int entry_steps(int pairs, int curves, int hard, int strokes) {
    return pairs + curves + (hard == CELL_PRIMITIVE ? CELL_HEAVY : hard) + strokes;
}

// Where a request for `need` of `cap` places begins when `taken` were asked for before it, or -1:
// no room.  `taken` goes on counting when the room is used up (the host reads what a scene
// would have needed), in 64 bits: in 32 it came round to small numbers after 2^28 tile entries, and
// places were handed out twice.
DVG_LIM_HD int room_at(unsigned long long taken, int need, int cap) {
    return taken + (unsigned long long)need <= (unsigned long long)cap ? (int)taken : -1;
}

// The memory of one scene's cell lists: 8 bytes per cell, 32 per entry (at most one per tile-list
// entry and cell of its tile), 16 per item.  Within `budget` bytes: all that is wanted, or four
// fifths of the rest for entries at most and what is left for items (a tile without entries is
// walked, an entry without items keeps the full queries).  bytes 0: no lists.
constexpr int TILE_CELLS = 16;
struct CellRoom {
    size_t ents = 0, items = 0, at_ents = 0, at_items = 0, at_counters = 0, bytes = 0;
};
inline CellRoom cell_room(uint64_t tiles, uint64_t tile_entries, uint64_t want_items, uint64_t budget) {
    constexpr uint64_t most = 1ull << 30, pad = 3 * 256 + 16;
    const uint64_t info = tiles * TILE_CELLS * 8;
    CellRoom r;
    if (tiles == 0 || budget < info + pad + 48) return r;
    const uint64_t rest = budget - info - pad;
    const uint64_t want_ents = std::min(std::max<uint64_t>(tile_entries, 1) * TILE_CELLS, most);
    want_items = std::min(std::max<uint64_t>(want_items, 1), most);
    uint64_t ents = want_ents, items = want_items;
    if (ents * 32 + items * 16 > rest) {
        ents = std::min(want_ents, rest / 5 * 4 / 32);
        items = std::min(want_items, (rest - ents * 32) / 16);
    }
    if (ents == 0 || items == 0) return r;
    r.ents = (size_t)ents;
    r.items = (size_t)items;
    r.at_ents = (size_t)((info + 255) & ~255ull);
    r.at_items = r.at_ents + (size_t)ents * 32;
    r.at_counters = (size_t)((r.at_items + items * 16 + 255) & ~255ull);
    r.bytes = r.at_counters + 16;
    return r;
}

}  // namespace dvgb
