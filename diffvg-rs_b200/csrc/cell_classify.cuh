// cell_classify.cuh — what a segment contributes to the sample points of a small box.
//
// The render kernels look at the scene through lists kept for every 4x4-pixel cell of the
// canvas (cells.cu).  A list holds, per group, only the segments that come near the cell; the
// winding contribution of the others is summed beforehand, up to a few comparisons of the
// sample's row with the rows where it steps.  The functions here decide which is which, for a
// box that holds every point the cell's samples can have in shape space (their f32 rounding
// included).
//
// Certainty.  The crate adds, per segment, the sign of y'(t) of each computed root t in [0, 1]
// of y(t) = py with x(t) > px (winding.rs:118-192).  Let m be the largest coordinate of the
// segment and the box.  The polynomial that it solves has f32-rounded coefficients and lies
// within 4.6e-6 m of the curve on [0, 1]; its f64 roots carry the error of its root formula.
// Take the monotone pieces of y(t) that meet the box's rows, and the parameter range in which
// each is inside them (bracketed by evaluation).  When every such range of the curve lies
// left of the box by more than M = 1e-4 (1 + m), the segment adds nothing; where it lies right
// of the box by more than M, the piece from level l0 to l1 adds [py > l0] - [py > l1].  At an
// extremum between two such pieces that cancels; what remains is a constant and a step at each
// end point inside the rows.  A piece that crosses all of the rows near the box is replaced by
// a cubic x(y) through four of its points, with a bound on the distance in x between the two:
// it counts where px lies left of that curve by more than the bound, and not where it lies
// right of it by as much.  The crate's computed sum is this number when
//  * py is farther than T = 1e-5 (1 + m) from every level inside the rows (end points and
//    extrema): the sample loop compares, and runs the full query otherwise;
//  * |y'| >= M at an inflection, so that |y'| is small near extrema only;
//  * a cubic is well conditioned: |b|, |c|, |d| <= 64 |a|, so that the crate's normalised
//    coefficients are at most 64, or its a is below the 1e-6 at which the crate solves a
//    quadratic.
// Then with D = T - 4.6e-6 m > 5e-6 m the distance in y to the next level of the crate's own
// polynomial, its roots are off by p / |y'| with p = 24 m 64^2 eps < 1.1e-11 m from the rounding
// of its normalised coefficients.  Next to an extremum, |y'| dt = 2 D for the distance dt to it,
// so the error is below 1.1e-6 dt; next to an end point the root is at least D / |y'| away from
// it, 4e5 times the error.  The trigonometric formula adds 4 sqrt(q) 8 eps / sqrt(1 - x^2), below
// 1e-7 for roots that are sqrt(2 D / 24 m) apart.  So every computed root is on the same side of
// 0, of 1, of px (M against 6 m times the error) and of every extremum as the exact one.
// The bound holds the interpolation error (the fourth derivative of X - Q(Y) over the bracket)
// and T moved in y and in x, for the rounded coefficients and the root.
// Anything else is left to the per-sample test.  A segment whose control points miss the rays
// of the whole box by the per-sample culling margin (ray_misses_segment in device.cuh)
// contributes nothing, as there.
//
// Host and device share this code: oracle/cell_stress.cpp runs it against the oracle's f64
// decisions at random points of random boxes.
#pragma once
#include <cmath>
#ifdef __CUDACC__
#include <cuda_fp16.h>
#endif

#ifdef __CUDACC__
#define DVG_CC_HD __host__ __device__ __forceinline__
#else
#define DVG_CC_HD inline
#endif

namespace dvgb {

struct CellBox {
    float x0, y0, x1, y1;
};

DVG_CC_HD float cc_max8(const float* q) {
    float m = 0.0f;
    for (int k = 0; k < 8; ++k) m = std::fmax(m, std::fabs(q[k]));
    return m;
}
DVG_CC_HD float cc_poly(float a, float b, float c, float d, float t) { return ((a * t + b) * t + c) * t + d; }

// The box as seen through an affine map (rows m[0..2], m[3..5]), grown by the f32 rounding of
// the map at its points.
DVG_CC_HD CellBox cc_map_box(const float* m, CellBox b) {
    const float cx = 0.5f * (b.x0 + b.x1), cy = 0.5f * (b.y0 + b.y1);
    const float hx = 0.5f * (b.x1 - b.x0), hy = 0.5f * (b.y1 - b.y0);
    const float ax = std::fmax(std::fabs(b.x0), std::fabs(b.x1)), ay = std::fmax(std::fabs(b.y0), std::fabs(b.y1));
    CellBox r;
    float v = m[0] * cx + m[1] * cy + m[2];
    float h = std::fabs(m[0]) * hx + std::fabs(m[1]) * hy;
    h += 2.0e-6f * (std::fabs(m[0]) * ax + std::fabs(m[1]) * ay + std::fabs(m[2])) + 1.0e-30f;
    r.x0 = v - h;
    r.x1 = v + h;
    v = m[3] * cx + m[4] * cy + m[5];
    h = std::fabs(m[3]) * hx + std::fabs(m[4]) * hy;
    h += 2.0e-6f * (std::fabs(m[3]) * ax + std::fabs(m[4]) * ay + std::fabs(m[5])) + 1.0e-30f;
    r.y0 = v - h;
    r.y1 = v + h;
    return r;
}

// A segment's winding contribution over a box: base + start [py > y(0)] - end [py > y(1)] for
// rows farther than `tol` from y(0) (if start), y(1) (if end) and ext[0 .. ne).
// Each of the nc curves adds its sign where px < c0 + (c1 + (c2 + c3 v) v) v - band, v = py - yc
// with yc the middle of the box's rows, and nothing where px is as far to the other side (c3 is
// rounded to a half-precision number).
DVG_CC_HD float cc_round_half(float v) {
#ifdef __CUDA_ARCH__
    return __half2float(__float2half_rn(v));
#else
    if (!(std::fabs(v) < 65504.0f)) return v;
    int e;
    std::frexp(v, &e);
    const int q = e - 11 < -24 ? -24 : e - 11;
    return std::ldexp(std::nearbyint(std::ldexp(v, -q)), q);
#endif
}
struct CellCurve {
    float c0, c1, c2, c3, band;
    int sign;
};
struct CellSeg {
    int base, start, end, ne, nc;
    float ext[2];
    CellCurve curve[3];
    float tol;
    int twice;  // the crate counts each crossing twice
};
DVG_CC_HD double cc_polyd(float a, float b, float c, float d, double t) {
    return (((double)a * t + (double)b) * t + (double)c) * t + (double)d;
}
DVG_CC_HD float cc_row_centre(CellBox b) { return 0.5f * (b.y0 + b.y1); }
// x as a cubic polynomial of the row through the piece's points at the four Chebyshev nodes of
// [u0, v1] (y monotone there).
DVG_CC_HD bool cell_curve(float a, float b, float c, float d, float ax, float bx, float cx, float dx, float u0, float v1,
                          float T, CellBox box, CellCurve* r) {
    const float yc = cc_row_centre(box);
    const double mid = 0.5 * ((double)u0 + (double)v1), half = 0.5 * ((double)v1 - (double)u0);
    const double node[4] = {-0.92387953251128674, -0.38268343236508977, 0.38268343236508977, 0.92387953251128674};
    double y[4], f[4];
    for (int k = 0; k < 4; ++k) {
        const double t = mid + half * node[k];
        y[k] = cc_polyd(a, b, c, d, t) - (double)yc;
        f[k] = cc_polyd(ax, bx, cx, dx, t);
    }
    for (int j = 1; j < 4; ++j)  // divided differences
        for (int k = 3; k >= j; --k) f[k] = (f[k] - f[k - 1]) / (y[k] - y[k - j]);
    // Newton form to powers of the row
    double p0 = f[3], p1 = 0.0, p2 = 0.0, p3 = 0.0;
    for (int k = 2; k >= 0; --k) {
        p3 = p2 - y[k] * p3;
        p2 = p1 - y[k] * p2;
        p1 = p0 - y[k] * p1;
        p0 = f[k] - y[k] * p0;
    }
    r->c0 = (float)p0;
    r->c1 = (float)p1;
    r->c2 = (float)p2;
    r->c3 = cc_round_half((float)p3);
    // fourth derivative of X - c1 Y - c2 Y^2 - c3 Y^3 over the bracket (Y relative to yc)
    const float H = (float)half, tm = (float)mid;
    const float yb = std::fmax(std::fabs(box.y1 - yc), std::fmax(std::fabs((float)(cc_polyd(a, b, c, d, u0) - (double)yc)),
                                                                 std::fabs((float)(cc_polyd(a, b, c, d, v1) - (double)yc))));
    const float d3 = 6.0f * std::fabs(a), d2 = std::fabs(6.0f * a * tm + 2.0f * b) + d3 * H;
    const float d1 = std::fabs((3.0f * a * tm + 2.0f * b) * tm + c) + d2 * H;
    const float fb = std::fabs(r->c1), fg = std::fabs(r->c2), fh = std::fabs((float)p3);
    const float R4 = fg * (8.0f * d1 * d3 + 6.0f * d2 * d2) +
                     fh * (24.0f * yb * d1 * d3 + 18.0f * yb * d2 * d2 + 36.0f * d1 * d1 * d2);
    const float fit = H * H * H * H * (1.0f / 192.0f) * R4 * 1.01f + std::fabs(r->c3 - (float)p3) * yb * yb * yb;
    const float slope = fb + (2.0f * fg + 3.0f * fh * yb) * yb;
    const float band = fit + T * (1.0f + slope) + 1.0e-6f * (std::fabs(r->c0) + (fb + (fg + fh * yb) * yb) * yb);
    // Worth it while few samples fall into the band: one that does costs its warp the solves
    // that the lists are there to avoid.
    if (!(band < 0.004f * (box.x1 - box.x0) && fh < 6.0e4f)) return false;  // (NaN: no)
    r->band = band;
    return true;
}
// Fills *r for a segment (kind 0 line, 1 quadratic, 2 cubic; q: four control points, lines and
// quadratics repeat their last one), or returns false: test it per sample.
DVG_CC_HD bool cell_winding(int kind, const float* q, CellBox bx, CellSeg* r) {
    r->base = r->start = r->end = r->ne = r->nc = r->twice = 0;
    const float m = std::fmax(std::fmax(cc_max8(q), std::fmax(std::fabs(bx.x0), std::fabs(bx.x1))),
                              std::fmax(std::fabs(bx.y0), std::fabs(bx.y1)));
    if (!(m < 1.0e6f)) return false;  // also NaN and infinities
    const float M1 = 1.0e-3f * (1.0f + m), M = 1.0e-4f * (1.0f + m);
    r->tol = 1.0e-5f * (1.0f + m);
    const float ymin = std::fmin(std::fmin(q[1], q[3]), std::fmin(q[5], q[7]));
    const float ymax = std::fmax(std::fmax(q[1], q[3]), std::fmax(q[5], q[7]));
    const float xmin = std::fmin(std::fmin(q[0], q[2]), std::fmin(q[4], q[6]));
    const float xmax = std::fmax(std::fmax(q[0], q[2]), std::fmax(q[4], q[6]));
    if (bx.y1 < ymin - M1 || bx.y0 > ymax + M1 || bx.x0 > xmax + M1) return true;
    const bool hull_right = xmin > bx.x1 + M;
    const float lo = bx.y0 - M, hi = bx.y1 + M;
    // power coefficients of y(t) and x(t), as the crate forms them
    float a = 0.0f, b = 0.0f, c, d = q[1], ax = 0.0f, bxc = 0.0f, cx, dx = q[0];
    if (kind == 0) {
        c = q[3] - q[1];
        cx = q[2] - q[0];
    } else if (kind == 1) {
        b = q[1] - 2.0f * q[3] + q[5];
        c = -2.0f * q[1] + 2.0f * q[3];
        bxc = q[0] - 2.0f * q[2] + q[4];
        cx = -2.0f * q[0] + 2.0f * q[2];
    } else {
        a = -q[1] + 3.0f * q[3] - 3.0f * q[5] + q[7];
        b = 3.0f * q[1] - 6.0f * q[3] + 3.0f * q[5];
        c = -3.0f * q[1] + 3.0f * q[3];
        ax = -q[0] + 3.0f * q[2] - 3.0f * q[4] + q[6];
        bxc = 3.0f * q[0] - 6.0f * q[2] + 3.0f * q[4];
        cx = -3.0f * q[0] + 3.0f * q[2];
        if (std::fabs(a) < 0.9e-6f) {
            a = 0.0f;  // the crate solves the quadratic
            // ... and below 1e-12 the linear equation, whose root its quadratic solver returns twice
            r->twice = std::fabs(b) < 1.0e-12f ? 1 : 0;
        } else {
            const float dm = std::fmax(std::fabs(d - bx.y0), std::fabs(d - bx.y1));
            const float k = std::fmax(std::fmax(std::fabs(b), std::fabs(c)), dm);
            if (!(std::fabs(a) > 1.1e-6f && k <= 64.0f * std::fabs(a))) return false;
        }
    }
    // extrema of y in (0, 1): roots of 3a t^2 + 2b t + c
    float e1 = 2.0f, e2 = 2.0f;
    const float disc = b * b - 3.0f * a * c;
    if (a != 0.0f) {
        const float ti = -b / (3.0f * a);
        if (ti > -0.05f && ti < 1.05f && !(std::fabs(disc) >= 3.0f * std::fabs(a) * M)) return false;
    }
    if (disc > 0.0f) {
        const float s = -(b + (b < 0.0f ? -std::sqrt(disc) : std::sqrt(disc)));
        if (a != 0.0f) e1 = s / (3.0f * a);
        if (s != 0.0f) e2 = c / s;
        if (!(e1 > 0.0f && e1 < 1.0f)) e1 = 2.0f;
        if (!(e2 > 0.0f && e2 < 1.0f)) e2 = 2.0f;
        if (e2 < e1) {
            const float t = e1;
            e1 = e2;
            e2 = t;
        }
    }
    float t0 = 0.0f, l0 = d;
    for (int i = 0; i < 3; ++i) {
        const float te = i == 0 ? e1 : (i == 1 ? e2 : 1.0f);
        if (te > 1.0f) continue;  // no such extremum
        const float ts = t0, t1 = te, ls = l0;
        // an extremum's level in f64: the sample rows are compared with it
        const float l1 = i == 2 ? q[7]
                                : (float)((((double)a * (double)te + (double)b) * (double)te + (double)c) * (double)te +
                                          (double)d);
        t0 = t1;
        l0 = l1;
        if (std::fmax(ls, l1) < lo || std::fmin(ls, l1) > hi) continue;
        const bool up = l1 > ls;
        const bool in0 = ls >= lo && ls <= hi, in1 = l1 >= lo && l1 <= hi;
        if (!hull_right) {
            // the parameter range inside the rows: a piece end, or the outer end of a bracket
            // around the row limit that the piece crosses
            float u0 = ts, u1 = in0 ? ts : t1, v0 = in1 ? t1 : ts, v1 = t1;
            const float lin = up ? lo : hi, lout = up ? hi : lo;
            for (int it = 0; it < 11; ++it) {
                const float tu = 0.5f * (u0 + u1), tv = 0.5f * (v0 + v1);
                const float yu = cc_poly(a, b, c, d, tu), yv = cc_poly(a, b, c, d, tv);
                if ((yu < lin) == up) u0 = tu; else u1 = tu;
                if ((yv < lout) == up) v0 = tv; else v1 = tv;
            }
            if (in0) u0 = ts;
            if (in1) v1 = t1;
            const float tm = 0.5f * (u0 + v1), h = 0.5f * (v1 - u0) + 1.0e-6f;
            const float x = cc_poly(ax, bxc, cx, dx, tm);
            const float dxx = (3.0f * ax * tm + 2.0f * bxc) * tm + cx, ddx = 6.0f * ax * tm + 2.0f * bxc;
            const float rx = ((std::fabs(ax) * h + 0.5f * std::fabs(ddx)) * h + std::fabs(dxx)) * h * 1.0001f;
            if (x + rx < bx.x0 - M) continue;
            if (!(x - rx > bx.x1 + M)) {
                if (in0 || in1 ||
                    !cell_curve(a, b, c, d, ax, bxc, cx, dx, u0, v1, r->tol, bx, &r->curve[r->nc]))
                    return false;
                r->curve[r->nc++].sign = up ? 1 : -1;
                continue;
            }
        }
        // [py > ls] - [py > l1]; an extremum's two halves cancel
        if (in0) {
            if (i == 0 || ts == 0.0f) r->start = 1;
        } else if (ls < lo) {
            r->base += 1;
        }
        if (in1) {
            if (i == 2) r->end = 1;
            else r->ext[r->ne++] = l1;
        } else if (l1 < lo) {
            r->base -= 1;
        }
    }
    return true;
}

// The extrema of y(t) in (0, 1) for cell_winding_point (2: none), or e1 < 0 when a segment does
// not meet the conditions on its coefficients (its inflection, its |a| against |b| and |c|).
DVG_CC_HD void cell_extrema(int kind, const float* q, float m, float* e1, float* e2) {
    *e1 = *e2 = 2.0f;
    if (kind == 0) return;
    float a = 0.0f, b, c;
    if (kind == 1) {
        b = q[1] - 2.0f * q[3] + q[5];
        c = -2.0f * q[1] + 2.0f * q[3];
    } else {
        a = -q[1] + 3.0f * q[3] - 3.0f * q[5] + q[7];
        b = 3.0f * q[1] - 6.0f * q[3] + 3.0f * q[5];
        c = -3.0f * q[1] + 3.0f * q[3];
        if (!(std::fabs(a) > 1.1e-6f && std::fmax(std::fabs(b), std::fabs(c)) <= 64.0f * std::fabs(a))) {
            *e1 = -1.0f;
            return;
        }
    }
    const float disc = b * b - 3.0f * a * c;
    if (a != 0.0f) {
        const float ti = -b / (3.0f * a);
        if (ti > -0.05f && ti < 1.05f && !(std::fabs(disc) >= 3.0f * std::fabs(a) * 1.0e-4f * (1.0f + m))) {
            *e1 = -1.0f;
            return;
        }
    }
    if (!(disc > 0.0f)) return;
    const float s = -(b + (b < 0.0f ? -std::sqrt(disc) : std::sqrt(disc)));
    float t1 = a != 0.0f ? s / (3.0f * a) : 2.0f, t2 = s != 0.0f ? c / s : 2.0f;
    if (!(t1 > 0.0f && t1 < 1.0f)) t1 = 2.0f;
    if (!(t2 > 0.0f && t2 < 1.0f)) t2 = 2.0f;
    *e1 = std::fmin(t1, t2);
    *e2 = std::fmax(t1, t2);
}
DVG_CC_HD float cc_quick_div(float a, float b) {
#ifdef __CUDA_ARCH__
    return __fdividef(a, b);
#else
    return a / b;
#endif
}
// cell_winding for the box of one point, with the extrema of cell_extrema (e1 >= 0): the
// winding contribution at (px, py) in *w, or false when it is not certain.  The coefficients
// are the crate's own (rounded to f32), so its polynomial is met exactly here: a piece that py
// passes has one root, found by f32 Newton steps kept inside a bracket and two f64 steps.  The
// crate's root lies within et = 1e-7 + 2e-11 (1 + m) / |y'| of it while py is T from every
// extremum (the bounds at the top, with 2 D = T); et moves the end-point tests by 2 et |y'| and
// x by et |x'|.  (Lines are the crate's in f32 throughout: T there.)
DVG_CC_HD bool cell_winding_point(int kind, const float* q, float e1, float e2, float px, float py, int* w) {
    *w = 0;
    const float m = std::fmax(cc_max8(q), std::fmax(std::fabs(px), std::fabs(py)));
    const float T = 1.0e-5f * (1.0f + m), tiny = 1.0e-9f * (1.0f + m);
    float a = 0.0f, b = 0.0f, c, ax = 0.0f, bx = 0.0f, cx;
    const float d = q[1] - py, dx = q[0] - px;
    if (kind == 0) {
        c = q[3] - q[1];
        cx = q[2] - q[0];
    } else if (kind == 1) {
        b = q[1] - 2.0f * q[3] + q[5];
        c = -2.0f * q[1] + 2.0f * q[3];
        bx = q[0] - 2.0f * q[2] + q[4];
        cx = -2.0f * q[0] + 2.0f * q[2];
    } else {
        a = -q[1] + 3.0f * q[3] - 3.0f * q[5] + q[7];
        b = 3.0f * q[1] - 6.0f * q[3] + 3.0f * q[5];
        c = -3.0f * q[1] + 3.0f * q[3];
        ax = -q[0] + 3.0f * q[2] - 3.0f * q[4] + q[6];
        bx = 3.0f * q[0] - 6.0f * q[2] + 3.0f * q[4];
        cx = -3.0f * q[0] + 3.0f * q[2];
        if (!(std::fabs(d) <= 64.0f * std::fabs(a))) return false;
    }
    float t0 = 0.0f, l0 = d;
    if (!(std::fabs(d) > (kind == 0 ? T : 1.0e-6f * std::fabs(c) + tiny))) return false;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
    for (int i = 0; i < 3; ++i) {
        const float te = i == 0 ? e1 : (i == 1 ? e2 : 1.0f);
        if (te > 1.0f) continue;  // no such extremum
        const float ls = l0, l1 = (float)cc_polyd(a, b, c, d, te);
        float lo = t0, hi = te;
        t0 = te;
        l0 = l1;
        const float Te = i < 2 || kind == 0 ? T : 1.0e-6f * std::fabs(3.0f * a + 2.0f * b + c) + tiny;
        if (!(std::fabs(l1) > Te)) return false;
        if ((ls < 0.0f) == (l1 < 0.0f)) continue;
        const bool up = l1 > 0.0f;
        float t = lo + (hi - lo) * cc_quick_div(ls, ls - l1), dy = 0.0f;
#ifdef __CUDA_ARCH__
#pragma unroll 1
#endif
        for (int it = 0; it < 12; ++it) {
            const float y = cc_poly(a, b, c, d, t);
            dy = (3.0f * a * t + 2.0f * b) * t + c;
            if (std::fabs(y) <= 0.3f * T) break;
            if ((y < 0.0f) == up) lo = t; else hi = t;
            t = t - cc_quick_div(y, dy);
            if (!(t > lo && t < hi)) t = 0.5f * (lo + hi);
        }
        const float inv = cc_quick_div(1.0f, dy);
        const double s1 = cc_polyd(a, b, c, d, t) * (double)inv, ta = (double)t - s1;
        const double s2 = cc_polyd(a, b, c, d, ta) * (double)inv, tr = ta - s2;
        // the slope within 5 % over the first step, so the second leaves 0.06 |s2| at most
        const float h = std::fabs((float)s1), ddy = std::fabs(6.0f * a * t + 2.0f * b);
        if (!((ddy + 6.0f * std::fabs(a) * h) * h <= 0.05f * std::fabs(dy) && std::fabs(s2) <= 1.0e-7)) return false;
        const float et = (kind == 0 ? 1.0e-6f : 1.1e-7f) + (kind == 0 ? T : 2.0f * 1.0e-2f * tiny) * std::fabs(inv);
        if (!(tr > 2.0 * (double)et && tr < 1.0 - 2.0 * (double)et)) return false;
        const double x = cc_polyd(ax, bx, cx, dx, tr);
        const float tf = (float)tr, xs = std::fabs((3.0f * ax * tf + 2.0f * bx) * tf + cx);
        const float xss = std::fabs(6.0f * ax * tf + 2.0f * bx) + 6.0f * std::fabs(ax) * et;
        if (!(std::fabs(x) > (double)((xs + xss * et) * et * 1.01f + (kind == 0 ? T : tiny)))) return false;
        if (x > 0.0) *w += up ? 1 : -1;
    }
    return true;
}

// A segment's 16-chord polyline (a line is its own chord), within `dev` of the curve at equal
// parameters: (1 / (8 n^2)) max|B''|.
struct CellChords {
    float ax, ay, bx, by, cx, cy, dx, dy, ex, ey;  // power coefficients, end point
    float dev;
    int n;
};
DVG_CC_HD CellChords cell_chords(int kind, const float* q) {
    CellChords c{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, q[0], q[1], q[6], q[7], 0.0f, 16};
    if (kind == 0) {
        c.cx = q[2] - q[0];
        c.cy = q[3] - q[1];
        c.n = 1;
    } else if (kind == 1) {
        c.bx = q[0] - 2.0f * q[2] + q[4];
        c.by = q[1] - 2.0f * q[3] + q[5];
        c.cx = 2.0f * (q[2] - q[0]);
        c.cy = 2.0f * (q[3] - q[1]);
        c.dev = (1.0f / 1024.0f) * std::sqrt(c.bx * c.bx + c.by * c.by);  // |B''| = 2 |b|
    } else {
        c.ax = -q[0] + 3.0f * q[2] - 3.0f * q[4] + q[6];
        c.ay = -q[1] + 3.0f * q[3] - 3.0f * q[5] + q[7];
        c.bx = 3.0f * q[0] - 6.0f * q[2] + 3.0f * q[4];
        c.by = 3.0f * q[1] - 6.0f * q[3] + 3.0f * q[5];
        c.cx = 3.0f * (q[2] - q[0]);
        c.cy = 3.0f * (q[3] - q[1]);
        const float s0x = q[0] - 2.0f * q[2] + q[4], s0y = q[1] - 2.0f * q[3] + q[5];
        const float s1x = q[2] - 2.0f * q[4] + q[6], s1y = q[3] - 2.0f * q[5] + q[7];
        c.dev = (3.0f / 1024.0f) * std::sqrt(std::fmax(s0x * s0x + s0y * s0y, s1x * s1x + s1y * s1y));
    }
    return c;
}
DVG_CC_HD void cell_chord_point(const CellChords& c, int k, float px, float py, float* x, float* y) {
    const float t = (float)k * (1.0f / 16.0f);
    *x = (k == c.n ? c.ex : cc_poly(c.ax, c.bx, c.cx, c.dx, t)) - px;
    *y = (k == c.n ? c.ey : cc_poly(c.ay, c.by, c.cy, c.dy, t)) - py;
}
// Squared distance of the origin to the chord v -> w.
DVG_CC_HD float cell_chord_d2(float vx, float vy, float wx, float wy) {
    const float dx = wx - vx, dy = wy - vy, ee = dx * dx + dy * dy, de = -(vx * dx + vy * dy);
    if (de <= 0.0f || ee <= 0.0f) return vx * vx + vy * vy;
    if (de >= ee) return wx * wx + wy * wy;
    const float cr = vx * dy - vy * dx;
    return cr * cr / ee;
}
// Squared distance from (px, py) to chords k0 .. k1 - 1.
DVG_CC_HD float cell_chords_d2(const CellChords& c, float px, float py, int k0, int k1) {
    float best = INFINITY, vx, vy;
    cell_chord_point(c, k0, px, py, &vx, &vy);
    for (int k = k0 + 1; k <= k1; ++k) {
        float wx, wy;
        cell_chord_point(c, k, px, py, &wx, &wy);
        best = std::fmin(best, cell_chord_d2(vx, vy, wx, wy));
        vx = wx;
        vy = wy;
    }
    return best;
}

// A stroke segment over a box: the samples' tests on chords k0 .. k1 - 1 (the others are out of
// every point's reach; k1 = 0: no chord test), on their squared distance d2.
//   d2 > miss: the crate's closest point is farther than the radius, by the culling margin of
//     the per-sample tests and the chord deviation;
//   d2 <= hit: the crate finds a point nearer than the radius (hit < 0: never taken).
// `hit` is for quadratics.  There the curve has a point within sqrt(d2) + dev, and the crate's
// closest point is at most a little farther.  Its candidates are the end points and the roots in
// [0, 1] of the cubic D'(t) / 4 = A t^3 + B t^2 + C t + D of the squared distance D(t), A = |a|^2
// with a half the second derivative.  In f64 its formula returns the sign-changing roots of a cubic
// within E = 500 eps S^3 of the monic one on [0, 1], S = B / A + sqrt(C / A) + cbrt(D / A) from the
// norms of the coefficients' terms (a double root that it misses changes no sign), and moves
// them by 1e-6 at most (the term that it drops for |ar| <= 1e-6).  Between candidates D is off by
// 8 A E, and a moved root adds 4 A (3 + 2 S + S^2) 1e-12; below A = 1e-6 the crate solves the
// quadratic, which is off by 2 A.  All of that, and the rounding of the coefficients to f32, is
// taken off r^2.
// A cubic's closest point comes from brackets that need not part the roots of its quintic: with
// the control points (-11, -15), (5, 9), (-3, 15), (1, 3) the crate passes over the nearest root
// for whole areas of points.  No threshold on the chord distance decides as it does, so cubics
// have no `hit`; their samples run the crate's search, which ends at its first candidate within the
// radius.  Its first candidates are the end points: a box within r of one is full.
struct CellStroke {
    bool far;   // no point of the box is in reach
    bool full;  // every point of the box is a hit
    float key;  // distance of the box centre less the radius
    float miss, hit;
    int k0, k1;
};
DVG_CC_HD CellStroke cell_stroke(int kind, const float* q, const float* rad, CellBox b, bool approx) {
    CellStroke s{false, false, 0.0f, INFINITY, -1.0f, 0, 0};
    const float m = std::fmax(std::fmax(cc_max8(q), std::fmax(std::fabs(b.x0), std::fabs(b.x1))),
                              std::fmax(std::fabs(b.y0), std::fabs(b.y1)));
    if (!(m < 1.0e6f)) return s;
    const float r = std::fmax(std::fmax(rad[0], rad[1]), std::fmax(rad[2], rad[3]));
    const float rm = r + 1.0e-3f * (1.0f + m) + 1.0e-5f * std::fabs(r);
    const float xmin = std::fmin(std::fmin(q[0], q[2]), std::fmin(q[4], q[6]));
    const float xmax = std::fmax(std::fmax(q[0], q[2]), std::fmax(q[4], q[6]));
    const float ymin = std::fmin(std::fmin(q[1], q[3]), std::fmin(q[5], q[7]));
    const float ymax = std::fmax(std::fmax(q[1], q[3]), std::fmax(q[5], q[7]));
    s.far = b.x1 < xmin - rm || b.x0 > xmax + rm || b.y1 < ymin - rm || b.y0 > ymax + rm;
    if (s.far || (kind == 2 && approx)) return s;  // (approximate cubic: the hull test only)
    const CellChords c = cell_chords(kind, q);
    const float px = 0.5f * (b.x0 + b.x1), py = 0.5f * (b.y0 + b.y1);
    const float hx = 0.5f * (b.x1 - b.x0), hy = 0.5f * (b.y1 - b.y0);
    const float hd = std::sqrt(hx * hx + hy * hy) * 1.00001f;
    const float reach = rm + c.dev + hd;
    float best = INFINITY, vx, vy;
    int k0 = 16, k1 = 0;
    cell_chord_point(c, 0, px, py, &vx, &vy);
    for (int k = 1; k <= c.n; ++k) {
        float wx, wy;
        cell_chord_point(c, k, px, py, &wx, &wy);
        const float d2 = cell_chord_d2(vx, vy, wx, wy);
        best = std::fmin(best, d2);
        if (!(d2 > reach * reach)) {
            if (k0 == 16) k0 = k - 1;
            k1 = k;
        }
        vx = wx;
        vy = wy;
    }
    const float d = std::sqrt(best);
    s.key = d - r;
    if (k1 == 0) {
        s.far = true;
        return s;
    }
    if (kind == 0 || approx) return s;
    s.k0 = k0;
    s.k1 = k1;
    s.miss = (rm + c.dev) * (rm + c.dev) * 1.00001f;
    if (!(rad[0] > 0.0f && rad[0] == rad[1] && rad[0] == rad[2] && rad[0] == rad[3])) return s;
    if (kind == 2) {
        const float ex = std::fmin(std::hypot(q[0] - px, q[1] - py), std::hypot(q[6] - px, q[7] - py));
        s.full = ex + hd <= r - 1.0e-5f * (1.0f + m);
        return s;
    }
    float slack = 2.0e-4f * (1.0f + m) * r + 1.0e-5f;
    const float A = c.bx * c.bx + c.by * c.by;
    if (!(A < 0.9e-6f)) {
        const float a = std::sqrt(A), b = 0.5f * std::sqrt(c.cx * c.cx + c.cy * c.cy);
        const float R = std::hypot(q[0] - px, q[1] - py) + hd;
        const float S = 1.001f * (3.0f * b / a + std::sqrt((2.0f * b * b + a * R) / A) + std::cbrt(b * R / A));
        slack += 1.0e-12f * A * S * S * S + 1.0e-11f * A * (S + 2.0f) * (S + 2.0f);
    }
    const float in = r * r - slack;
    const float h = in > 0.0f ? std::sqrt(in) - c.dev : -1.0f;
    if (h > 0.0f) {
        s.hit = h * h * 0.99999f;
        s.full = d + hd <= h;
    }
    return s;
}

}  // namespace dvgb
