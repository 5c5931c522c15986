// limits.hpp — sizes and index arithmetic whose limits no test can reach on a device, in plain
// functions that oracle/limits.cpp runs on the CPU (tests/test_limits.py).
#pragma once
#include <cstddef>

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

}  // namespace dvgb
