// limits.hpp — sizes and index arithmetic whose limits no test can reach on a device, in plain
// functions that oracle/limits.cpp runs on the CPU (tests/test_limits.py).
#pragma once
#include <cstddef>

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

// Where a request for `need` of `cap` places begins when `taken` were asked for before it, or -1:
// no room.  `taken` goes on counting when the room is used up (the host reads what a scene
// would have needed), in 64 bits: in 32 it came round to small numbers after 2^28 tile entries, and
// places were handed out twice.
DVG_LIM_HD int room_at(unsigned long long taken, int need, int cap) {
    return taken + (unsigned long long)need <= (unsigned long long)cap ? (int)taken : -1;
}

}  // namespace dvgb
