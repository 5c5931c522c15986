// cells.cu — builds the per-cell lists (cells.cuh), for the first call that reads a scene's and
// after each on-device parameter step.  Built with -fmad=false like kernels.cu.
//
// One CTA per tile walks the tile's groups; for a path group its 256 threads take the
// (cell, segment) pairs, sixteen cells of one segment next to each other, so a pair costs one
// classification where the sample loop used to test the segment at each of the cell's
// 16 * spp sample points.  The sample kernels are bound by instruction issue on those tests
// (f64 root solves): on the mixed 512x512 scene a sample met 49 segments of 5.3 groups, and
// with the lists 1.2 segments, 1.5 curves and 2.7 rows of 2.2 groups are left (large
// 1024x1024 scene: 199 -> 18, 6, 26).  The lists took the forward from 3.43 to 1.23 ms and the
// edge pass from 1.31 to 0.81 ms on the mixed scene at 4x4 spp, from 76 to 34 ms and from 216 to
// 136 ms on the large one (with the steps taken since: 0.83, 0.43, 15.9 and 49.2 ms).  4x4
// pixels: the 16 samples per pixel of a CTA share one list; cells of a whole tile leave 8
// segments.  The build itself is bound by latency, a few barriers per group at 12-24 % occupancy:
// 55 us on a 128x128 scene of 8 shapes, 0.23 ms on the mixed scene, 3.0 ms on the large one.
#include "cells.cuh"
#include "kernels.cuh"

namespace dvgb {

namespace {
enum : uint8_t { SEG_START = 1, SEG_END = 2, SEG_TWICE = 4 };  // levels of a segment at a cell
enum : int { BOX_OUT = 0, BOX_IN = 1, BOX_MIXED = 2 };

__device__ __forceinline__ int box_state(const CellBox& b, float4 r) {
    if (b.x1 < r.x || b.x0 > r.z || b.y1 < r.y || b.y0 > r.w) return BOX_OUT;
    return b.x0 >= r.x && b.x1 <= r.z && b.y0 >= r.y && b.y1 <= r.w ? BOX_IN : BOX_MIXED;
}
// Fill of a circle, ellipse or rectangle over the box: 1 covered, 0 not, -1 varies (the
// strict tests of winding_shape, with a margin far above their f32 rounding).
__device__ __forceinline__ int primitive_fill(int kind, float4 prm, const CellBox& b) {
    const float m = fmaxf(fmaxf(fmaxf(fabsf(b.x0), fabsf(b.x1)), fmaxf(fabsf(b.y0), fabsf(b.y1))),
                          fmaxf(fmaxf(fabsf(prm.x), fabsf(prm.y)), fmaxf(fabsf(prm.z), fabsf(prm.w))));
    if (!(m < 1.0e6f)) return -1;
    const float M = 1.0e-4f * (1.0f + m);
    if (kind == K_RECT) {
        if (b.x0 > prm.x + M && b.x1 < prm.z - M && b.y0 > prm.y + M && b.y1 < prm.w - M) return 1;
        return b.x1 < prm.x - M || b.x0 > prm.z + M || b.y1 < prm.y - M || b.y0 > prm.w + M ? 0 : -1;
    }
    const float rx = kind == K_CIRCLE ? fabsf(prm.z) : fmaxf(fabsf(prm.z), 1.0e-6f);
    const float ry = kind == K_CIRCLE ? rx : fmaxf(fabsf(prm.w), 1.0e-6f);
    const float x0 = b.x0 - prm.x, x1 = b.x1 - prm.x, y0 = b.y0 - prm.y, y1 = b.y1 - prm.y;
    if (!(rx > 2.0f * M && ry > 2.0f * M)) return -1;
    const float fx = (fmaxf(fabsf(x0), fabsf(x1)) + M) / rx, fy = (fmaxf(fabsf(y0), fabsf(y1)) + M) / ry;
    if (fx * fx + fy * fy < 0.9999f) return 1;
    const float nx = fmaxf((x0 <= 0.0f && x1 >= 0.0f ? 0.0f : fminf(fabsf(x0), fabsf(x1))) - M, 0.0f) / rx;
    const float ny = fmaxf((y0 <= 0.0f && y1 >= 0.0f ? 0.0f : fminf(fabsf(y0), fabsf(y1))) - M, 0.0f) / ry;
    return nx * nx + ny * ny > 1.0001f ? 0 : -1;
}
// A tolerance (rounded up) with a step of -2 .. 2 in its low bits.
__device__ __forceinline__ int coded(float tol, int step) { return ((__float_as_int(tol) + 7) & ~7) | (step + 2); }
// A curve's band (rounded up to its upper half's leading bits), step and c3 in one word.
__device__ __forceinline__ int coded_curve(const CellCurve& q, int step) {
    const unsigned band = ((unsigned)__float_as_int(q.band) + 0x7ffffu) & 0xfff80000u;
    return (int)(band | ((unsigned)(step + 2) << 16) | (unsigned)__half_as_ushort(__float2half_rn(q.c3)));
}
}  // namespace

__global__ void __launch_bounds__(256) k_cells(const __grid_constant__ DevScene S, const CellTable T) {
    __shared__ CellBox cbox[CELLS], pbox[CELLS];
    __shared__ int state[CELLS], base[CELLS], kept[CELLS], steps[CELLS], ent_base;
    __shared__ short leaf_of[CELL_MAX_SEGS];  // from the path's first node
    __shared__ uint8_t levels_of[CELL_MAX_SEGS][CELLS];
    // an entry's items, per cell (segments as leaf slots; stroke segments with their distance)
    __shared__ int n_lev[CELLS], n_cur[CELLS], n_hard[CELLS], n_soft[CELLS], n_str[CELLS], base_slow[CELLS];
    __shared__ int2 lev[CELLS][CELL_MAX_ITEMS];
    __shared__ int4 cur[CELLS][CELL_MAX_ITEMS];
    __shared__ short hard[CELLS][CELL_MAX_ITEMS], soft[CELLS][CELL_MAX_ITEMS], str[CELLS][CELL_MAX_ITEMS];
    __shared__ float str_key[CELLS][CELL_MAX_ITEMS], str_miss[CELLS][CELL_MAX_ITEMS], str_hit[CELLS][CELL_MAX_ITEMS];
    __shared__ int full[CELLS];
    const int tile = blockIdx.x, tid = threadIdx.x;
    const int tx = tile % S.tiles_x, ty = tile / S.tiles_x;
    const int off = S.tile_offsets[tile], n = S.tile_offsets[tile + 1] - off;
    if (tid == 0) {
        ent_base = n > 0 && n < CELL_LIST_MAX
                       ? room_at(atomicAdd(&T.counters[0], (unsigned long long)(CELLS * n)), CELLS * n, T.cap_entries)
                       : (n > 0 ? -1 : 0);
    }
    if (tid < CELLS) {
        // Every point that is looked up in the cell: its pixels' samples, and edge samples,
        // whose two sides lie 1e-4 of the canvas off a point of the pixel (truncation puts
        // points up to a pixel left of or above the canvas into its first pixels).
        const int x0 = tx * TILE + (tid & 3) * CELL, y0 = ty * TILE + (tid >> 2) * CELL;
        const float px = 1.01e-4f * (float)S.width + 0.01f, py = 1.01e-4f * (float)S.height + 0.01f;
        cbox[tid] = CellBox{(float)x0 - px - (x0 == 0 ? 1.0f : 0.0f), (float)y0 - py - (y0 == 0 ? 1.0f : 0.0f),
                            (float)(x0 + CELL) + px, (float)(y0 + CELL) + py};
        kept[tid] = steps[tid] = 0;
    }
    __syncthreads();
    if (ent_base < 0) {
        if (tid < CELLS) T.info[tile * CELLS + tid] = make_int2(0, -1);
        return;
    }
    for (int e = 0; e < n; ++e) {
        const int g = __ldg(&S.tile_entries[off + e]);
        const int4 gi = __ldg(&S.g_info[g]);
        const int4 gb = __ldg(&S.g_bvh[g]);
        if (gb.y == 0) continue;  // no shape with points: nothing to cover (an empty box is in the list of a one-tile canvas)
        const int4 root = __ldg(&S.gn_meta[gb.x]);
        const bool single = gb.y == 1 && root.z == 1;
        const int s = single ? __ldg(&S.gl_shapes[root.y]) : 0;
        const int4 si = single ? __ldg(&S.s_info[s]) : make_int4(-1, 0, -1, 0);
        const bool is_path = si.x == K_PATH && si.z >= 0;
        const int4 pi = is_path ? __ldg(&S.p_info[2 * si.z]) : make_int4(0, 0, 0, 0);
        const int pflags = is_path ? __ldg(&S.p_info[2 * si.z + 1].w) : 0;
        const bool listed = is_path && pi.y <= CELL_MAX_SEGS;  // (so node offsets and bases fit in 16 bits)
        const bool want_fill = gi.x >= 0;
        const bool want_stroke = gi.y >= 0 && !(single && !(__ldg(&S.s_stroke[s]) > 0.0f));
        const bool list_stroke = want_stroke && listed && !(pflags & PF_STYLED);
        const int nseg = listed ? pi.y : 0;
        const int k0 = listed && pi.w > 0 ? __ldg(&S.pn_meta[pi.z].y) : 0;  // the path's first leaf slot
        __syncthreads();  // the previous group's masks are written out
        if (tid < CELLS) {
            const CellBox lb = cc_map_box(S.g_c2s + 9 * g, cbox[tid]);
            state[tid] = box_state(lb, __ldg(&S.gn_bounds[gb.x]));
            pbox[tid] = single && (si.y & (SF_IDENTITY | SF_INVERTIBLE)) == SF_INVERTIBLE ? cc_map_box(S.s_inv + 6 * s, lb) : lb;
            full[tid] = base[tid] = base_slow[tid] = n_lev[tid] = n_cur[tid] = n_hard[tid] = n_soft[tid] = n_str[tid] = 0;
        }
        if (listed)
            for (int nd = pi.z + tid; nd < pi.z + pi.w; nd += blockDim.x) {
                const int4 m = __ldg(&S.pn_meta[nd]);
                for (int k = m.y; k < m.y + m.z; ++k) leaf_of[k - k0] = (short)(nd - pi.z);
            }
        __syncthreads();
        for (int i = tid; i < CELLS * nseg; i += blockDim.x) {
            const int c = i & 15, k = i >> 4;
            if (state[c] == BOX_OUT) continue;
            const CellBox b = pbox[c];
            SegGeom sg;
            const int sidx = __ldg(&S.pl_segs[k0 + k]);
            load_seg(S, sidx, sg);
            const float4 lb = __ldg(&S.pn_bounds[pi.z + leaf_of[k]]);
            uint8_t lv = 0;
            if (want_fill && !(b.y1 < lb.y || b.y0 > lb.w || b.x0 > lb.z)) {
                CellSeg r;
                if (!cell_winding(sg.kind, sg.q, b, &r)) {
                    const int o = atomicAdd(&n_hard[c], 1);
                    if (o < CELL_MAX_ITEMS) hard[c][o] = (short)k;
                } else {
                    const int mult = r.twice ? 2 : 1;
                    if (r.base) atomicAdd(&base[c], mult * r.base);
                    lv = (uint8_t)((r.start ? SEG_START : 0) | (r.end ? SEG_END : 0) | (r.twice ? SEG_TWICE : 0));
                    for (int j = 0; j < r.ne; ++j) {
                        const int o = atomicAdd(&n_lev[c], 1);
                        if (o < CELL_MAX_ITEMS) lev[c][o] = make_int2(__float_as_int(r.ext[j]), coded(r.tol, 0));
                    }
                    for (int j = 0; j < r.nc; ++j) {
                        const CellCurve& q = r.curve[j];
                        const int o = atomicAdd(&n_cur[c], 1);
                        if (o < CELL_MAX_ITEMS)
                            cur[c][o] = make_int4(__float_as_int(q.c0), __float_as_int(q.c1), __float_as_int(q.c2),
                                                  coded_curve(q, mult * q.sign));
                    }
                    if (r.start || r.end || r.ne || r.nc) {  // not one number over the cell
                        const int o = atomicAdd(&n_soft[c], 1);
                        if (o < CELL_MAX_ITEMS) soft[c][o] = (short)k;
                    } else if (r.base) {
                        atomicAdd(&base_slow[c], mult * r.base);
                    }
                }
            }
            levels_of[sidx - pi.x][c] = lv;
            if (list_stroke && box_state(b, lb) != BOX_OUT) {
                const CellStroke st = cell_stroke(sg.kind, sg.q, sg.r, b, pflags & PF_APPROX);
                if (!st.far) {
                    if (st.full && box_state(b, lb) == BOX_IN && state[c] == BOX_IN) full[c] = 1;
                    const int o = atomicAdd(&n_str[c], 1);
                    if (o < CELL_MAX_ITEMS) {
                        str[c][o] = (short)k;
                        str_key[c][o] = st.key;
                        // (rounded up and down to make room for the chord range)
                        str_miss[c][o] = __int_as_float(((__float_as_int(st.miss) + 15) & ~15) | st.k0);
                        str_hit[c][o] = __int_as_float((__float_as_int(st.hit) & ~31) | st.k1);
                    }
                }
            }
        }
        __syncthreads();
        // The steps at the segments' ends.  A vertex between two segments that both step there
        // is one level (their steps cancel unless one of them counts twice).
        if (want_fill)
            for (int i = tid; i < CELLS * nseg; i += blockDim.x) {
                const int c = i & 15, k = i >> 4;
                if (state[c] == BOX_OUT) continue;
                const int lv = levels_of[k][c];
                if (!lv) continue;
                const float4 p0 = __ldg(&S.seg_p[2 * (pi.x + k)]), p1 = __ldg(&S.seg_p[2 * (pi.x + k) + 1]);
                const CellBox b = pbox[c];
                const float m = fmaxf(fmaxf(fmaxf(fabsf(b.x0), fabsf(b.x1)), fmaxf(fabsf(b.y0), fabsf(b.y1))),
                                      fmaxf(fmaxf(fmaxf(fabsf(p0.x), fabsf(p0.y)), fmaxf(fabsf(p0.z), fabsf(p0.w))),
                                            fmaxf(fmaxf(fabsf(p1.x), fabsf(p1.y)), fmaxf(fabsf(p1.z), fabsf(p1.w)))));
                float tol = 1.0e-5f * (1.0f + m);  // cell_winding's
                const int mult = lv & SEG_TWICE ? 2 : 1;
                if (lv & SEG_START) {
                    int step = mult;
                    const int kp = k > 0 ? k - 1 : nseg - 1;
                    const float4 q1 = __ldg(&S.seg_p[2 * (pi.x + kp) + 1]);
                    const int lp = levels_of[kp][c];
                    if (kp != k && (lp & SEG_END) && q1.z == p0.x && q1.w == p0.y) {
                        step -= lp & SEG_TWICE ? 2 : 1;
                        const float4 q0 = __ldg(&S.seg_p[2 * (pi.x + kp)]);
                        tol = fmaxf(tol, 1.0e-5f * (1.0f + fmaxf(fmaxf(fmaxf(fabsf(q0.x), fabsf(q0.y)),
                                                                       fmaxf(fabsf(q0.z), fabsf(q0.w))),
                                                                 fmaxf(fabsf(q1.x), fabsf(q1.y)))));
                    }
                    const int o = atomicAdd(&n_lev[c], 1);
                    if (o < CELL_MAX_ITEMS) lev[c][o] = make_int2(__float_as_int(p0.y), coded(tol, step));
                }
                if (lv & SEG_END) {
                    const int kn = k + 1 < nseg ? k + 1 : 0;
                    const float4 q0 = __ldg(&S.seg_p[2 * (pi.x + kn)]);
                    if (!(kn != k && (levels_of[kn][c] & SEG_START) && q0.x == p1.z && q0.y == p1.w)) {
                        const int o = atomicAdd(&n_lev[c], 1);
                        if (o < CELL_MAX_ITEMS) lev[c][o] = make_int2(__float_as_int(p1.w), coded(tol, -mult));
                    }
                }
            }
        __syncthreads();
        if (tid >= 32) continue;
        const int c = tid & 15;
        int nl = 0, nc = 0, nh = 0, nf = 0, ns = 0, flags = 0;
        if (tid < CELLS && state[c] != BOX_OUT) {
            const bool in = state[c] == BOX_IN;
            if (want_fill) {
                const bool fits = n_lev[c] <= CELL_MAX_ITEMS && n_cur[c] <= CELL_MAX_ITEMS &&
                                  n_hard[c] + n_soft[c] <= CELL_MAX_ITEMS;
                if (!single || (is_path && !(listed && fits))) {
                    flags |= CE_FILL_ANY;
                } else if (is_path) {
                    nl = (n_lev[c] + 1) >> 1;
                    nc = n_cur[c];
                    nh = n_hard[c];
                    nf = nh + n_soft[c];
                    if (nf > 0)
                        flags |= CE_FILL_TEST;
                    else if (fill_hit(gi.z, base[c]))
                        flags |= in ? CE_FILL : CE_FILL_TEST;
                } else if (si.x != K_PATH) {
                    const int w = primitive_fill(si.x, __ldg(&S.s_params[s]), pbox[c]);
                    if (w < 0 || (w == 1 && !in)) {
                        flags |= CE_FILL_TEST;
                        nh = CELL_PRIMITIVE;
                    } else if (w == 1 && fill_hit(gi.z, 1)) {
                        flags |= CE_FILL;
                    }
                }
            }
            if (full[c]) {
                flags |= CE_STROKE;
            } else if (list_stroke && n_str[c] <= CELL_MAX_ITEMS) {
                ns = n_str[c];
                if (ns > 0) flags |= CE_STROKE_TEST;
            } else if (want_stroke && !(single && si.x == K_PATH && !is_path)) {
                flags |= CE_STROKE_ANY;
            }
            if (!in && (flags & (CE_FILL_TEST | CE_STROKE_TEST))) flags |= CE_BOX;
            if (gi.z == 1) flags |= flags & CE_FILL_TEST ? CE_ODD : 0;
        }
        // room for the sixteen cells' items at once
        const int head = flags & CE_FILL_TEST ? 1 : 0;
        const int need = head + nl + nc + nf + ns;
        int upto = need;
        for (int o = 1; o < 16; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (tid >= o) upto += v;
        }
        const int total = __shfl_sync(0xffffffffu, upto, 15);
        int at = 0;
        if (tid == 0 && total > 0) at = room_at(atomicAdd(&T.counters[1], (unsigned long long)total), total, T.cap_items);
        at = __shfl_sync(0xffffffffu, at, 0);
        const bool room = at >= 0;
        at += upto - need;
        if (tid >= CELLS || !flags) continue;
        if (!room && need > 0) {  // no room left: the full queries
            if (flags & CE_FILL_TEST) flags = (flags & ~CE_FILL_TEST) | CE_FILL_ANY;
            if (flags & CE_STROKE_TEST) flags = (flags & ~CE_STROKE_TEST) | CE_STROKE_ANY;
            flags &= ~(CE_BOX | CE_ODD);
            nl = nc = nh = nf = ns = 0;
        }
        const CellBox b = pbox[c];
        int o = at;
        if (flags & CE_FILL_TEST) T.items[o++] = make_int4(__float_as_int(cc_row_centre(b)), 0, 0, 0);
        for (int j = 0; j < nl; ++j) {
            const int2 l0 = lev[c][2 * j];
            const int2 l1 = 2 * j + 1 < n_lev[c] ? lev[c][2 * j + 1] : make_int2(__float_as_int(INFINITY), coded(0.0f, 0));
            T.items[o++] = make_int4(l0.x, l0.y, l1.x, l1.y);
        }
        for (int j = 0; j < nc; ++j) T.items[o++] = cur[c][j];
        for (int j = 0; j < nf; ++j) {
            const int k = j < nh ? hard[c][j] : soft[c][j - nh], leaf = pi.z + leaf_of[k];
            const int sidx = __ldg(&S.pl_segs[k0 + k]);
            const float4 lb = __ldg(&S.pn_bounds[leaf]);
            const bool all = b.y0 >= lb.y && b.y1 <= lb.w && b.x1 <= lb.z;
            float e1 = -1.0f, e2 = -1.0f;
            if (j < nh) {
                SegGeom sg;
                load_seg(S, sidx, sg);
                const float m = fmaxf(fmaxf(fmaxf(fabsf(b.x0), fabsf(b.x1)), fmaxf(fabsf(b.y0), fabsf(b.y1))), cc_max8(sg.q));
                if (m < 1.0e6f) cell_extrema(sg.kind, sg.q, m, &e1, &e2);
            }
            T.items[o++] = make_int4(all ? -1 : leaf, sidx, __float_as_int(e1), __float_as_int(e2));
        }
        for (int j = 0; j < ns; ++j) {  // nearest first: a sample stops at its first hit
            int best = j;
            for (int i = j + 1; i < ns; ++i)
                if (str_key[c][i] < str_key[c][best]) best = i;
            const int k = str[c][best], leaf = pi.z + leaf_of[k];
            const bool all = box_state(b, __ldg(&S.pn_bounds[leaf])) == BOX_IN;
            T.items[o++] = make_int4(all ? -1 : leaf, __ldg(&S.pl_segs[k0 + k]), __float_as_int(str_miss[c][best]),
                                     __float_as_int(str_hit[c][best]));
            str[c][best] = str[c][j];
            str_key[c][best] = str_key[c][j];
            str_miss[c][best] = str_miss[c][j];
            str_hit[c][best] = str_hit[c][j];
        }
        int4* E = T.entries + 2 * ((size_t)ent_base + (size_t)c * n + kept[c]);
        E[0] = make_int4(entry_word(true, e, flags), g, gi.x, gi.y);
        E[1] = make_int4(s, (base[c] & 0xffff) | (base_slow[c] << 16), at,
                         nl | (nc << 6) | (nh << 12) | (nf << 18) | (ns << 24));
        kept[c] += 1;
        steps[c] += entry_steps(nl, nc, nh, ns);
    }
    __syncthreads();
    if (tid < CELLS) T.info[tile * CELLS + tid] = make_int2(ent_base + tid * n, kept[tid] | (steps[tid] >= CELL_HEAVY ? CELL_HEAVY_BIT : 0));
}

int launch_cells(const DevScene& S, const CellTable& T, cudaStream_t stream) {
    const int tiles = S.tiles_x * S.tiles_y;
    if (tiles == 0) return 0;
    k_cells<<<tiles, 256, 0, stream>>>(S, T);
    return 1;
}

}  // namespace dvgb
