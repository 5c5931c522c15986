// cell_stress.cpp — test infrastructure: the library's per-cell decisions
// (diffvg-rs_b200/csrc/cell_classify.cuh) against the oracle's restatement of the crate's
// per-sample computation, at random points of random boxes.  Built into
// oracle/_build/libcell_stress.so by the Makefile; driven by tests/test_cells.py.
#include "oracle.cpp"

#include "../diffvg-rs_b200/csrc/cell_classify.cuh"

namespace {
struct SplitMix {
    uint64_t s;
    uint64_t next() {
        uint64_t z = (s += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        return z ^ (z >> 31);
    }
    double uni() { return (double)(next() >> 11) * (1.0 / 9007199254740992.0); }
    float range(float lo, float hi) { return (float)((double)lo + (double)(hi - lo) * uni()); }
};

// One random segment of the given kind (0 line, 1 quadratic, 2 cubic) and mode:
// 0 uniform control points; 1 integer control points; 2 near-degenerate (elevated lines and
// quadratics, cusps, tiny loops, with perturbations of 10^U[-7, -1]); 3 coordinates up to
// 4096; 4 small segments (extent 0.5 to 8) far from the origin; 5 nearly flat in y.
void random_segment(SplitMix& rng, int kind, int mode, V2* p) {
    const float scale = mode == 3 ? rng.range(64.0f, 4096.0f) : 64.0f;
    for (int k = 0; k < 4; ++k) p[k] = mk(rng.range(-1.0f, 1.0f) * scale, rng.range(-1.0f, 1.0f) * scale);
    if (mode == 1)
        for (int k = 0; k < 4; ++k) p[k] = mk(std::floor(rng.range(-16.0f, 17.0f)), std::floor(rng.range(-16.0f, 17.0f)));
    if (mode == 2 && kind > 0) {
        const int how = (int)(rng.next() % 4);
        const float eps = (float)std::pow(10.0, -7.0 + 6.0 * rng.uni());
        if (kind == 1) {
            p[1] = lerp(p[0], p[2], how == 0 ? 0.5f : rng.range(0.0f, 1.0f));
        } else if (how == 0) {
            V2 q1 = mk(rng.range(-64, 64), rng.range(-64, 64));
            p[1] = p[0] + (q1 - p[0]) * (2.0f / 3.0f);
            p[2] = p[3] + (q1 - p[3]) * (2.0f / 3.0f);
        } else if (how == 1) {
            p[1] = lerp(p[0], p[3], 1.0f / 3.0f);
            p[2] = lerp(p[0], p[3], 2.0f / 3.0f);
        } else if (how == 2) {
            p[1] = lerp(p[0], p[3], 0.7f);
            p[2] = lerp(p[0], p[3], 0.3f);
        } else {
            p[1] = p[3] + mk(rng.range(-4, 4), rng.range(-4, 4));
            p[2] = p[0] + mk(rng.range(-4, 4), rng.range(-4, 4));
        }
        for (int k = 1; k <= kind; ++k) p[k] = p[k] + mk(rng.range(-1, 1) * eps * 64.0f, rng.range(-1, 1) * eps * 64.0f);
    }
    if (mode == 4) {
        const V2 c = mk(rng.range(-600, 600), rng.range(-600, 600));
        const float e = rng.range(0.5f, 8.0f);
        for (int k = 0; k < 4; ++k) p[k] = c + mk(rng.range(-e, e), rng.range(-e, e));
    }
    if (mode == 5) {
        const float e = (float)std::pow(10.0, -4.0 + 5.0 * rng.uni());
        for (int k = 0; k < 4; ++k) p[k].y = p[0].y + rng.range(-1, 1) * e;
    }
    for (int k = kind + 2; k < 4; ++k) p[k] = p[kind + 1];
}
// A box near the segment: its centre on the curve or anywhere in the grown hull, half sizes
// 10^U[-3, 1.2].
dvgb::CellBox random_box(SplitMix& rng, int kind, const V2* p) {
    V2 lo = vmin(vmin(p[0], p[1]), vmin(p[2], p[3])), hi = vmax(vmax(p[0], p[1]), vmax(p[2], p[3]));
    V2 c = mk(rng.range(lo.x - 8, hi.x + 4), rng.range(lo.y - 2, hi.y + 2));
    if (rng.next() % 3 == 0) {
        const float t = (float)rng.uni(), u = 1.0f - t;
        if (kind == 0) c = p[0] * u + p[1] * t;
        if (kind == 1) c = p[0] * (u * u) + p[1] * (2 * u * t) + p[2] * (t * t);
        if (kind == 2) c = p[0] * (u * u * u) + p[1] * (3 * u * u * t) + p[2] * (3 * u * t * t) + p[3] * (t * t * t);
        c = c + mk(rng.range(-6, 6), rng.range(-6, 6));
    }
    const float hx = (float)std::pow(10.0, -3.0 + 4.2 * rng.uni()), hy = (float)std::pow(10.0, -3.0 + 4.2 * rng.uni());
    return dvgb::CellBox{c.x - hx, c.y - hy, c.x + hx, c.y + hy};
}
// A point of the box: uniform, or on an edge or corner; rows at the segment's end points and
// y extremum levels when the box has them.
V2 random_point(SplitMix& rng, const dvgb::CellBox& b, const V2* p) {
    float x = rng.range(b.x0, b.x1), y = rng.range(b.y0, b.y1);
    const int e = (int)(rng.next() % 8);
    if (e == 0) x = b.x0;
    if (e == 1) x = b.x1;
    if (e == 2) y = b.y0;
    if (e == 3) y = b.y1;
    if (e == 4) {
        const float ye = rng.next() % 2 ? p[0].y : p[3].y;
        if (ye >= b.y0 && ye <= b.y1) y = ye;
    }
    return mk(std::fmin(std::fmax(x, b.x0), b.x1), std::fmin(std::fmax(y, b.y0), b.y1));
}
// The per-sample culling of the kernels (ray_misses_segment in device.cuh).
bool culled(const V2* p, V2 q) {
    float m = std::fmax(std::fabs(q.x), std::fabs(q.y));
    for (int k = 0; k < 4; ++k) m = std::fmax(m, std::fmax(std::fabs(p[k].x), std::fabs(p[k].y)));
    m = 1.0e-3f * (1.0f + m);
    const V2 lo = vmin(vmin(p[0], p[1]), vmin(p[2], p[3])), hi = vmax(vmax(p[0], p[1]), vmax(p[2], p[3]));
    return q.y < lo.y - m || q.y > hi.y + m || q.x > hi.x + m;
}
}  // namespace

// out: boxes, boxes decided, decided with a level to compare, points compared, points left to
// the per-sample test (a row too close to a level), points whose per-sample winding differs
// from the box's.
extern "C" void cell_winding_stress(int kind, int mode, uint64_t seed, uint64_t n, int points,
                                    unsigned long long* out) {
    SplitMix rng{seed * 0x2545f4914f6cdd1dull + (uint64_t)(mode * 3 + kind)};
    for (int k = 0; k < 6; ++k) out[k] = 0;
    for (uint64_t i = 0; i < n; ++i) {
        V2 p[4];
        random_segment(rng, kind, mode, p);
        const dvgb::CellBox b = random_box(rng, kind, p);
        const float q[8] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y, p[3].x, p[3].y};
        dvgb::CellSeg r;
        out[0] += 1;
        if (!dvgb::cell_winding(kind, q, b, &r)) continue;
        out[1] += 1;
        float lev[4];
        int nl = 0;
        if (r.start) lev[nl++] = q[1];
        if (r.end) lev[nl++] = q[7];
        for (int k = 0; k < r.ne; ++k) lev[nl++] = r.ext[k];
        if (nl || r.nc) out[2] += 1;
        for (int k = 0; k < points; ++k) {
            V2 pt = random_point(rng, b, p);
            if (nl && rng.next() % 2) {  // just outside the tolerance of a level
                const float l = lev[rng.next() % (uint64_t)nl];
                const float y = l + (rng.next() % 2 ? 1.0f : -1.0f) * r.tol * rng.range(1.0f, 1.5f);
                if (y >= b.y0 && y <= b.y1) pt.y = y;
            }
            if (r.nc && rng.next() % 2) {  // just outside the band of a curve
                const dvgb::CellCurve& c = r.curve[rng.next() % (uint64_t)r.nc];
                const float v = pt.y - dvgb::cc_row_centre(b);
                const float x = c.c0 + (c.c1 + (c.c2 + c.c3 * v) * v) * v + (rng.next() % 2 ? 1.0f : -1.0f) * c.band * rng.range(1.0f, 1.5f);
                if (x >= b.x0 && x <= b.x1) pt.x = x;
            }
            bool close = false;
            for (int j = 0; j < nl; ++j) close = close || std::fabs(pt.y - lev[j]) <= r.tol;
            int w = r.base;
            for (int j = 0; j < r.nc; ++j) {
                const float v = pt.y - dvgb::cc_row_centre(b);
                const float dx = pt.x - (r.curve[j].c0 + (r.curve[j].c1 + (r.curve[j].c2 + r.curve[j].c3 * v) * v) * v);
                close = close || std::fabs(dx) <= r.curve[j].band;
                if (dx < 0.0f) w += r.curve[j].sign;
            }
            if (close) {
                out[4] += 1;
                continue;
            }
            if (r.start && pt.y > q[1]) w += 1;
            if (r.end && pt.y > q[7]) w -= 1;
            if (r.twice) w *= 2;
            const int ref = culled(p, pt) ? 0 : winding_number_segment((uint8_t)kind, p[0], p[1], p[2], p[3], pt);
            out[3] += 1;
            if (ref != w) out[5] += 1;
        }
    }
}

// The one-point version: points, points decided, decided with a crossing, decided and different
// from the crate's winding.
extern "C" void cell_point_stress(int kind, int mode, uint64_t seed, uint64_t n, int points, unsigned long long* out) {
    SplitMix rng{seed * 0x2545f4914f6cdd1dull + (uint64_t)(mode * 3 + kind) + 177};
    for (int k = 0; k < 4; ++k) out[k] = 0;
    for (uint64_t i = 0; i < n; ++i) {
        V2 p[4];
        random_segment(rng, kind, mode, p);
        const dvgb::CellBox b = random_box(rng, kind, p);
        const float q[8] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y, p[3].x, p[3].y};
        float e1, e2;
        dvgb::cell_extrema(kind, q, dvgb::cc_max8(q), &e1, &e2);
        for (int k = 0; k < points; ++k) {
            V2 pt = random_point(rng, b, p);
            if (rng.next() % 2) {  // near the curve or near an end's row
                const float t = (float)rng.uni(), u = 1.0f - t, mag = (float)std::pow(10.0, -6.0 + 6.0 * rng.uni());
                V2 on = kind == 0 ? p[0] * u + p[1] * t
                        : kind == 1 ? p[0] * (u * u) + p[1] * (2 * u * t) + p[2] * (t * t)
                                    : p[0] * (u * u * u) + p[1] * (3 * u * u * t) + p[2] * (3 * u * t * t) + p[3] * (t * t * t);
                pt = on + mk(rng.range(-mag, mag), rng.range(-mag, mag));
                if (rng.next() % 4 == 0) pt.y = (rng.next() % 2 ? p[0].y : p[3].y) + rng.range(-mag, mag);
            }
            out[0] += 1;
            int w = 0;
            if (!(e1 >= 0.0f) || !dvgb::cell_winding_point(kind, q, e1, e2, pt.x, pt.y, &w)) continue;
            out[1] += 1;
            if (w) out[2] += 1;
            if (w != winding_number_segment((uint8_t)kind, p[0], p[1], p[2], p[3], pt)) out[3] += 1;
        }
    }
}

// The stroke tests: boxes, far boxes, full boxes, points tested, points the chords call a miss
// or a hit, wrong misses (a far box's or a missed point within r by the crate's closest point),
// wrong hits (a full box's or a hit point that is not).
extern "C" void cell_stroke_stress(int kind, int mode, uint64_t seed, uint64_t n, int points,
                                   unsigned long long* out) {
    SplitMix rng{seed * 0x2545f4914f6cdd1dull + (uint64_t)(mode * 3 + kind) + 77};
    for (int k = 0; k < 7; ++k) out[k] = 0;
    for (uint64_t i = 0; i < n; ++i) {
        V2 p[4];
        random_segment(rng, kind, mode, p);
        const dvgb::CellBox b = random_box(rng, kind, p);
        const float q[8] = {p[0].x, p[0].y, p[1].x, p[1].y, p[2].x, p[2].y, p[3].x, p[3].y};
        const float r = (float)std::pow(10.0, -1.0 + 2.0 * rng.uni()), rad[4] = {r, r, r, r};
        const dvgb::CellStroke s = dvgb::cell_stroke(kind, q, rad, b, false);
        const dvgb::CellChords ch = dvgb::cell_chords(kind, q);
        out[0] += 1;
        if (s.far) out[1] += 1;
        if (s.full) out[2] += 1;
        for (int k = 0; k < points; ++k) {
            const V2 pt = random_point(rng, b, p);
            CP c;
            if (kind == 0) distance_to_segment(pt, p[0], p[1], &c.dist, &c.cp, &c.t);
            else if (kind == 1) c = closest_point_quadratic(pt, p[0], p[1], p[2], false);
            else c = closest_point_cubic(pt, p[0], p[1], p[2], p[3], false);
            bool miss = s.far, hit = s.full;
            if (!s.far && s.k1) {
                const float d2 = dvgb::cell_chords_d2(ch, pt.x, pt.y, s.k0, s.k1);
                miss = d2 > s.miss;
                hit = hit || d2 <= s.hit;
            }
            out[3] += 1;
            if (miss || hit) out[4] += 1;
            if (miss && c.dist < r) out[5] += 1;
            if (hit && !(c.dist < r)) out[6] += 1;
        }
    }
}

// One stroke segment (eight coordinates, four radii), one box and one point of it.  out: the
// decision of the lists (0 left to the crate's search, 1 a miss, 2 a hit, 3 a box that is full),
// whether the crate's closest point is within its radius.
extern "C" void cell_stroke_point(int kind, const float* q, const float* rad, const float* box, const float* pt, int approx,
                                  int* out) {
    const dvgb::CellBox b{box[0], box[1], box[2], box[3]};
    const dvgb::CellStroke s = dvgb::cell_stroke(kind, q, rad, b, approx != 0);
    const V2 p[4] = {mk(q[0], q[1]), mk(q[2], q[3]), mk(q[4], q[5]), mk(q[6], q[7])}, at = mk(pt[0], pt[1]);
    out[0] = s.full ? 3 : s.far ? 1 : 0;
    if (!s.full && !s.far && s.k1) {
        const float d2 = dvgb::cell_chords_d2(dvgb::cell_chords(kind, q), at.x, at.y, s.k0, s.k1);
        out[0] = d2 > s.miss ? 1 : d2 <= s.hit ? 2 : 0;
    }
    CP c;
    float r;
    if (kind == 0) {
        distance_to_segment(at, p[0], p[1], &c.dist, &c.cp, &c.t);
        r = rad[0] + c.t * (rad[1] - rad[0]);
    } else if (kind == 1) {
        c = closest_point_quadratic(at, p[0], p[1], p[2], approx != 0);
        const float u = 1.0f - c.t;
        r = u * u * rad[0] + 2.0f * u * c.t * rad[1] + c.t * c.t * rad[2];
    } else {
        c = closest_point_cubic(at, p[0], p[1], p[2], p[3], approx != 0);
        const float u = 1.0f - c.t;
        r = u * u * u * rad[0] + 3.0f * u * u * c.t * rad[1] + 3.0f * u * c.t * c.t * rad[2] + c.t * c.t * c.t * rad[3];
    }
    out[1] = c.dist < r ? 1 : 0;
}
