// cells.cuh — per-cell lists of what a sample point still has to test (built by cells.cu).
//
// Each 16x16 tile's group list is split over the tile's sixteen 4x4-pixel cells.  A cell keeps
// an entry, in group order, for every group that can cover one of its sample points, with the
// tests that are left there (cell_classify.cuh): none at all when the fill covers the whole
// cell; else a winding number summed beforehand, the rows at which it steps, the curves
// x(y) that stand for pieces crossing the cell and the few segments that are solved per sample; and
// the segments that a stroke can reach the cell from, the nearest first.  Groups that the lists
// do not describe (several shapes, styled strokes, strokes of ellipses and rectangles) keep the
// full query.
#pragma once
#include "device.cuh"
#include "limits.hpp"

namespace dvgb {

constexpr int CELL = 4;               // cell edge in pixels
constexpr int CELLS = 16;             // cells per tile
constexpr int CELL_MAX_SEGS = 512;    // longer paths keep the full query

// Entry flags (low 8 bits of an entry's first word, entry_word).
enum : int {
    CE_FILL = 1,         // the fill covers every sample point of the cell
    CE_FILL_TEST = 2,    // winding = base + the entry's levels and fill segments
    CE_FILL_ANY = 4,     // full query (group_inside)
    CE_STROKE_TEST = 8,  // the entry's stroke segments
    CE_STROKE_ANY = 16,  // full query (group_within)
    CE_BOX = 32,         // the tests hold inside the group's root box only
    CE_ODD = 64,         // even-odd rule
    CE_STROKE = 128      // the stroke covers every sample point of the cell
};
// Two int4 per entry: {index << 8 | flags, group, fill paint, stroke paint} and {shape,
// winding base of the fast tests | base of the slow ones << 16, first item, counts}.  The items
// (int4 each):
//   a header {middle row yc} when there are fill tests,
//   level pairs {row, tolerance, row, tolerance}, each tolerance with (step + 2) in its low three
//     bits: the winding steps where py passes the row,
//   curves {c0, c1, c2, c3 as a half | the upper half of the band with (sign + 2) in its low three
//     bits},
//   segments {path BVH leaf whose box is to be tested or -1, segment, e1, e2}: the first `hard`
//     are tested by every sample (cell_winding_point with their extrema, the crate's solve where
//     that is not certain), all of them solved (with the slow base, without levels and
//     curves) for a sample within a tolerance or a band,
//   stroke segments {leaf or -1, segment, miss, hit}: a CellStroke, with k0 in the low four bits
//     of miss and k1 in the low five of hit.
// counts: level pairs, curves, hard segments, segments, stroke segments, six bits each; hard =
// CELL_PRIMITIVE: the shape is a circle, an ellipse or a rectangle.
constexpr int CELL_MAX_ITEMS = 48;  // of each kind
struct CellCounts {
    int pairs, curves, hard, segs, strokes;
    __device__ __forceinline__ explicit CellCounts(int w)
        : pairs(w & 63), curves((w >> 6) & 63), hard((w >> 12) & 63), segs((w >> 18) & 63), strokes((w >> 24) & 63) {}
};
struct CellTable {
    int2* info;     // per cell: first entry, entries (-1: none were kept, walk the tile's list)
    int4* entries;
    int4* items;
    unsigned long long* counters;  // entries and items asked for so far (room_at)
    int cap_entries, cap_items;
};

// The full queries, out of line: with the lists they run for few entries, and their code
// inside the sample loop costs every sample instruction fetches.
static __device__ __noinline__ bool group_within_any(const DevScene& S, int g, float2 lp) {
    return group_within(S, g, lp);
}
static __device__ __noinline__ bool group_inside_any(const DevScene& S, int g, float2 lp) {
    return group_inside(S, g, lp, __ldg(&S.g_info[g].z));
}

// A heavy cell (CELL_HEAVY) is marked next to its number of entries.
constexpr int CELL_HEAVY_BIT = 1 << 30;

// The groups to visit at one cell: the cell's entries, or the tile's whole list.
struct CellWalk {
    const int4* ent;
    const int* list;
    int n;
    bool heavy;  // its items take CELL_HEAVY steps or more
};
__device__ __forceinline__ CellWalk cell_walk(const DevScene& S, int tile, int cell) {
    CellWalk w;
    const int2 info = S.cell_info ? __ldg(&S.cell_info[tile * CELLS + cell]) : make_int2(0, -1);
    if (info.y >= 0) {
        w.ent = S.cell_entries + 2 * (size_t)info.x;
        w.list = nullptr;
        w.n = info.y & ~CELL_HEAVY_BIT;
        w.heavy = info.y & CELL_HEAVY_BIT;
    } else {
        const int off = S.tile_offsets[tile];
        w.ent = nullptr;
        w.list = S.tile_entries + off;
        w.n = S.tile_offsets[tile + 1] - off;
        w.heavy = false;
    }
    return w;
}
__device__ __forceinline__ int4 cell_entry(const DevScene& S, const CellWalk& w, int k) {
    if (w.ent) return __ldg(&w.ent[2 * k]);
    const int g = __ldg(&w.list[k]);
    const int4 gi = __ldg(&S.g_info[g]);
    const int flags = (gi.x >= 0 ? CE_FILL_ANY : 0) | (gi.y >= 0 ? CE_STROKE_ANY : 0);
    return make_int4(entry_word(false, k, flags), g, gi.x, gi.y);
}
// The place of entry k (first words A) in the tile list.
__device__ __forceinline__ int cell_place(const CellWalk& w, int k, int4 A) { return entry_place(w.ent != nullptr, k, A.x); }
// Whether the stroke and the fill of entry k (first words A) cover canvas point pt: the
// decisions of group_within / group_inside.
__device__ __forceinline__ void cell_hits(const DevScene& S, const CellWalk& w, int k, int4 A, float2 pt, bool* stroke,
                                          bool* fill) {
    const int flags = A.x & 255;
    *stroke = (flags & CE_STROKE) != 0;
    *fill = (flags & CE_FILL) != 0;
    if (!(flags & ~(CE_FILL | CE_STROKE))) return;
    const float2 lp = xf9(S.g_c2s + 9 * A.y, pt);
    if (flags & CE_STROKE_ANY) *stroke = group_within_any(S, A.y, lp);
    if (flags & CE_FILL_ANY) *fill = group_inside_any(S, A.y, lp);
    if (!(flags & (CE_FILL_TEST | CE_STROKE_TEST))) return;
    if (flags & CE_BOX) {
        const float4 b = __ldg(&S.gn_bounds[__ldg(&S.g_bvh[A.y].x)]);
        if (!(lp.x >= b.x && lp.x <= b.z && lp.y >= b.y && lp.y <= b.w)) return;
    }
    const int4 B = __ldg(&w.ent[2 * k + 1]);
    const float2 p = shape_local_dist(S, B.x, lp);
    const CellCounts n(B.w);
    const int4* items = S.cell_items + B.z;
    if (flags & CE_FILL_TEST) {
        const float v = p.y - __int_as_float(__ldg(&items[0].x));
        ++items;
        int wind = (short)(B.y & 0xffff);
        bool close = false;
#pragma unroll 1
        for (int j = 0; j < n.pairs; ++j) {
            const int4 it = __ldg(&items[j]);
            const float d0 = p.y - __int_as_float(it.x), d1 = p.y - __int_as_float(it.z);
            if (d0 > 0.0f) wind += (it.y & 7) - 2;
            if (d1 > 0.0f) wind += (it.w & 7) - 2;
            close = close || fabsf(d0) <= __int_as_float(it.y & ~7) || fabsf(d1) <= __int_as_float(it.w & ~7);
        }
        items += n.pairs;
#pragma unroll 1
        for (int j = 0; j < n.curves; ++j) {
            const int4 it = __ldg(&items[j]);
            const float c1 = __int_as_float(it.y), c2 = __int_as_float(it.z);
            const float c3 = __half2float(__ushort_as_half((unsigned short)(it.w & 0xffff)));
            const float d = p.x - (__int_as_float(it.x) + (c1 + (c2 + c3 * v) * v) * v);
            if (d < 0.0f) wind += ((it.w >> 16) & 7) - 2;
            close = close || fabsf(d) <= __int_as_float(it.w & 0xfff80000);
        }
        items += n.curves;
        if (n.hard == CELL_PRIMITIVE) {
            wind = winding_primitive(__ldg(&S.s_info[B.x].x), __ldg(&S.s_params[B.x]), p);
        } else {
            if (close) wind = B.y >> 16;
            const int solve = close ? n.segs : n.hard;
#pragma unroll 1
            for (int j = 0; j < solve; ++j) {
                const int4 it = __ldg(&items[j]);
                if (it.x >= 0) {
                    const float4 b = __ldg(&S.pn_bounds[it.x]);
                    if (p.y < b.y || p.y > b.w || p.x > b.z) continue;
                }
                SegGeom sg;
                load_seg(S, it.y, sg);
                const float e1 = __int_as_float(it.z);
                int w;
                if (!close && e1 >= 0.0f &&
                    cell_winding_point(sg.kind, sg.q, e1, __int_as_float(it.w), p.x, p.y, &w))
                    wind += w;
                else if (!ray_misses_segment(sg, p))
                    wind += winding_segment(sg, p);
            }
        }
        items += n.segs;
        *fill = fill_hit(flags & CE_ODD ? 1 : 0, wind);
    }
    if (flags & CE_STROKE_TEST) {
        const bool approx = __ldg(&S.p_info[2 * __ldg(&S.s_info[B.x].z) + 1].w) & PF_APPROX;
#pragma unroll 1
        for (int j = 0; j < n.strokes; ++j) {
            const int4 it = __ldg(&items[j]);
            if (it.x >= 0) {
                const float4 b = __ldg(&S.pn_bounds[it.x]);
                if (!(p.x >= b.x && p.x <= b.z && p.y >= b.y && p.y <= b.w)) continue;
            }
            SegGeom sg;
            load_seg(S, it.y, sg);
            const int k1 = it.w & 31;
            if (k1) {
                const float d2 = cell_chords_d2(cell_chords(sg.kind, sg.q), p.x, p.y, it.z & 15, k1);
                if (d2 > __int_as_float(it.z & ~15)) continue;
                if (d2 <= __int_as_float(it.w & ~31)) {
                    *stroke = true;
                    break;
                }
            } else if (stroke_misses_segment(sg, p)) {
                continue;
            }
            // one radius: the first candidate within it decides (1e-6 below the rounding of seg_radius)
            const bool even = sg.r[0] == sg.r[1] && sg.r[0] == sg.r[2] && sg.r[0] == sg.r[3];
            const CPRes c = seg_closest_plain(sg, p, approx, even ? sg.r[0] * (1.0f - 1.0e-6f) : 0.0f);
            if (c.dist < seg_radius(sg, c.t)) {
                *stroke = true;
                break;
            }
        }
    }
}

// A tile's pixels in cell order (sixteen pixels of a cell, row by row, then the next cell), so
// that the lanes of a warp share a cell's list.
__device__ __forceinline__ int cell_of_pix(int pix) { return pix >> 4; }
__device__ __forceinline__ int2 pix_xy(int pix) {
    const int c = pix >> 4;
    return make_int2((c & 3) * CELL + (pix & 3), (c >> 2) * CELL + ((pix >> 2) & 3));
}

// Builds a scene's table (asynchronous; T.counters are zeroed by the caller on the stream).
int launch_cells(const DevScene& S, const CellTable& T, cudaStream_t stream);

}  // namespace dvgb
