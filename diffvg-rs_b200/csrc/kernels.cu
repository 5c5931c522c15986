// kernels.cu — sm_100a kernels of the render / backward hot path.
//
//   k_bin_count / k_bin_scan / k_bin_write  tile binning of groups (group order kept)
//   k_forward      per (tile, sub-sample) CTA: scene evaluation + filtered splat
//                  into a shared-memory tile+halo accumulator, flushed once
//   k_weights      filter-weight image only (backward without a preceding forward)
//   k_resolve      Σ(c·w)/Σw and un-premultiply            (forward.rs:294-334)
//   k_interior     interior adjoint per sample             (backward/render.rs:95-169)
//   k_interior_cached  the same for samples whose fragments the forward cached
//   k_boundary     edge sampling adjoint per boundary sample (backward/boundary.rs:141-196)
//   k_l2           L2 loss and d_render
//
// Built with -fmad=false (see device.cuh).
#include <algorithm>

#include "cells.cuh"
#include "device.cuh"
#include "kernels.cuh"

// Minimum resident CTAs per SM for the scene-evaluation kernels (register cap =
// 65536 / (threads * value)); chosen by measurement on B200.
#ifndef DVG_MINB_FWD
#define DVG_MINB_FWD 5  // 48 registers: mixed 512x512 forward 0.86 -> 0.82 ms against 4 (large scene 14.3 -> 14.7)
#endif
#ifndef DVG_MINB_INT
#define DVG_MINB_INT 2
#endif
// The edge evaluation is bound by instruction fetch: 512 threads of a CTA that take a heavy cell's
// entries together, at 40 registers, against 128 threads at 32 that run apart: edge pass of the
// large 1024x1024 scene 62.0 -> 48.0 ms, mixed 0.43 -> 0.41 (49.2 and 0.43 now; together: 128 threads 59.9 ms, 256
// 52.4, 512 at 32 registers 49.8 and at 64 51.7, 1024 at 64 59.1).
#ifndef DVG_BND_THREADS
#define DVG_BND_THREADS 512
#endif
#ifndef DVG_MINB_BND
#define DVG_MINB_BND 3
#endif
#ifndef DVG_MINB_LEAN
#define DVG_MINB_LEAN 4
#endif

namespace dvgb {

// ------------------------------------------------------------------ tile binning
// One CTA per tile scans all group boxes; the crate bins on the GPU and sorts on
// the host (src/renderer/renderer.rs:254-384); scanning in group order keeps the
// compositing order without a sort.  Edge tiles extend to infinity so that any
// point clamped to an edge tile is covered.
__device__ __forceinline__ bool tile_hits(const DevScene& S, int tile, float4 b) {
    int tx = tile % S.tiles_x, ty = tile / S.tiles_x;
    float x0 = tx == 0 ? -INFINITY : (float)(tx * TILE);
    float y0 = ty == 0 ? -INFINITY : (float)(ty * TILE);
    float x1 = tx == S.tiles_x - 1 ? INFINITY : (float)((tx + 1) * TILE);
    float y1 = ty == S.tiles_y - 1 ? INFINITY : (float)((ty + 1) * TILE);
    return !(b.z < x0 || b.x > x1 || b.w < y0 || b.y > y1);
}
__global__ void __launch_bounds__(256) k_bin_count(DevScene S, const float4* g_bbox, int* counts) {
    int tile = blockIdx.x;
    int total = 0;
#pragma unroll 1
    for (int base = 0; base < S.num_groups; base += blockDim.x) {
        int g = base + threadIdx.x;
        bool hit = false;
        if (g < S.num_groups) {
            int4 gi = S.g_info[g];
            hit = (gi.x >= 0 || gi.y >= 0) && tile_hits(S, tile, g_bbox[g]);
        }
        total += __syncthreads_count(hit);
    }
    if (threadIdx.x == 0) counts[tile] = total;
}
// Exclusive scan of tile counts (single CTA of 1024 threads, any length).
__global__ void __launch_bounds__(1024) k_bin_scan(const int* counts, int n, int* offsets) {
    __shared__ int warp_sums[32];
    __shared__ int carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 1
    for (int base = 0; base < n; base += 1024) {
        int i = base + threadIdx.x;
        int v = i < n ? counts[i] : 0;
        int x = v;
        for (int o = 1; o < 32; o <<= 1) {
            int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int w = warp_sums[lane];
            for (int o = 1; o < 32; o <<= 1) {
                int y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            warp_sums[lane] = w;
        }
        __syncthreads();
        int excl = carry + (wid > 0 ? warp_sums[wid - 1] : 0) + x - v;
        if (i < n) offsets[i] = excl;
        __syncthreads();
        if (threadIdx.x == 1023) carry = excl + v;
        __syncthreads();
    }
    if (threadIdx.x == 0) offsets[n] = carry;
}
// Two-level exclusive scan for long count arrays (the boundary sort's buckets): each
// CTA scans 4096 counts and leaves its total in part[], one CTA scans the totals, a
// third pass adds each CTA's base.  offsets[n] receives the grand total.
constexpr int SCAN_CHUNK = 4096;
__global__ void __launch_bounds__(1024) k_scan_chunks(const int* counts, int n, int* offsets, int* part) {
    __shared__ int warp_sums[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int base = blockIdx.x * SCAN_CHUNK + 4 * threadIdx.x;
    int v[4], t = 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        v[k] = base + k < n ? counts[base + k] : 0;
        t += v[k];
    }
    int x = t;
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_sums[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int w = warp_sums[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    int excl = (wid > 0 ? warp_sums[wid - 1] : 0) + x - t;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        if (base + k < n) offsets[base + k] = excl;
        excl += v[k];
    }
    if (threadIdx.x == 1023) part[blockIdx.x] = warp_sums[31];
}
__global__ void __launch_bounds__(1024) k_scan_add(int* offsets, int n, const int* part_offsets) {
    const int i = blockIdx.x * SCAN_CHUNK + 4 * threadIdx.x;
    const int add = part_offsets[blockIdx.x];
#pragma unroll
    for (int k = 0; k < 4; ++k)
        if (i + k < n) offsets[i + k] += add;
}
// Exclusive scan of counts[n] into offsets[n + 1]; part: scratch of scan_part_ints(n) ints.
inline int scan_chunks(int n) { return (n + SCAN_CHUNK - 1) / SCAN_CHUNK; }
int launch_scan(const int* counts, int n, int* offsets, int* part, cudaStream_t stream) {
    const int c = scan_chunks(n);
    if (c <= 1) {
        k_bin_scan<<<1, 1024, 0, stream>>>(counts, n, offsets);
        return 1;
    }
    k_scan_chunks<<<c, 1024, 0, stream>>>(counts, n, offsets, part);
    k_bin_scan<<<1, 1024, 0, stream>>>(part, c, part + c);  // part + c: the chunks' bases, then the total
    k_scan_add<<<c, 1024, 0, stream>>>(offsets, n, part + c);
    cudaMemcpyAsync(offsets + n, part + 2 * c, sizeof(int), cudaMemcpyDeviceToDevice, stream);
    return 3;
}

__global__ void __launch_bounds__(256) k_bin_write(DevScene S, const float4* g_bbox, const int* offsets,
                                                   int* entries) {
    __shared__ int warp_counts[8];
    int tile = blockIdx.x;
    int cursor = offsets[tile];
    int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll 1
    for (int base = 0; base < S.num_groups; base += blockDim.x) {
        int g = base + threadIdx.x;
        bool hit = false;
        if (g < S.num_groups) {
            int4 gi = S.g_info[g];
            hit = (gi.x >= 0 || gi.y >= 0) && tile_hits(S, tile, g_bbox[g]);
        }
        unsigned m = __ballot_sync(0xffffffffu, hit);
        if (lane == 0) warp_counts[wid] = __popc(m);
        __syncthreads();
        int before = 0, total = 0;
        for (int w = 0; w < 8; ++w) {
            if (w < wid) before += warp_counts[w];
            total += warp_counts[w];
        }
        if (hit) entries[cursor + before + __popc(m & ((1u << lane) - 1u))] = g;
        cursor += total;
        __syncthreads();
    }
}

// ------------------------------------------------------------------ forward
// One CTA = 256 samples of one 16x16 tile.  Pixels are numbered cell by cell (pix_xy), so a
// warp's samples share one cell list (or two): entry loads are uniform.  When the CTA's
// samples lie in one cell (layout 1, spp a power of two from 16 to 256), its splat
// accumulator covers that cell and its halo only.  G: the splat's lane groups (splat_group: the
// samples per pixel, 4 or 16, with layout 1), 0: a shared-memory atomic per sample and value.
// Gaussian r = 1, 4x4 spp, mixed 512x512 scene: 0.55 of the forward's 1.23 ms were those atomics;
// 0.93 ms with the groups (0.82 with the steps taken since).
template <int G>
__device__ __forceinline__ void forward_body(const DevScene& S, const SampleParams& sp, int tile, int round,
                                             float* accum, float* wsum, float* sm) {
    const int ri = S.filter_ri;
    const bool use_sm = ri <= MAX_SMEM_RI;
    const int tx = tile % S.tiles_x, ty = tile / S.tiles_x;
    const int spp = sp.sxn * sp.syn;
    const int s_in_tile = round * 256 + (int)threadIdx.x;
    const int pix = sp.layout ? s_in_tile / spp : (int)threadIdx.x, sub = sp.layout ? s_in_tile % spp : round;
    const int2 pxy = pix_xy(pix);
    const int x = tx * TILE + pxy.x, y = ty * TILE + pxy.y;
    const bool one_cell = sp.layout && spp >= 16 && 256 % spp == 0;
    const int HW = (one_cell ? CELL : TILE) + 2 * ri;
    const int ox = (one_cell ? x & ~(CELL - 1) : tx * TILE) - ri, oy = (one_cell ? y & ~(CELL - 1) : ty * TILE) - ri;
    if (use_sm)
#pragma unroll 1
        for (int i = threadIdx.x; i < HW * HW * 5; i += blockDim.x) sm[i] = 0.0f;
    __syncthreads();
    const bool valid = x < S.width && y < S.height;
    float2 pt = make_float2(0.0f, 0.0f);
    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (valid) {
        const int sx = sub % sp.sxn, sy = sub / sp.sxn;
        pt = sample_pos(x, y, sx, sy, sp.sxn, sp.syn, S.width, sp.seed, sp.jitter);
        const CellWalk walk = cell_walk(S, tile, cell_of_pix(pix));
        // Fragment cache (see SampleParams): kept only where the interior pass, which
        // normalises the sample point by the canvas size and scales it back
        // (src/backward/render.rs:111, src/backward/sampling.rs:91), tests the same point.
        const size_t fstride = (size_t)S.tiles_x * S.tiles_y * spp * 256;
        const size_t sid = ((size_t)tile * spp + round) * 256 + threadIdx.x;
        const bool cache = sp.frag != nullptr &&
                           S.tile_offsets[tile + 1] - S.tile_offsets[tile] <= FRAG_MAX_ENTRIES &&
                           (pt.x / (float)S.width) * (float)S.width == pt.x &&
                           (pt.y / (float)S.height) * (float)S.height == pt.y;
        int nf = 0;
        acc = background_premul(S, y * S.width + x);
        // one list for the CTA, and all of its threads here: entry by entry if the list is heavy
        const bool step = one_cell && walk.heavy && (tx + 1) * TILE <= S.width && (ty + 1) * TILE <= S.height;
#pragma unroll 1
        for (int k = 0; k < walk.n; ++k) {
            if (step) __syncthreads();
            // stroke first, then fill; one paint call site for both
            const int4 A = cell_entry(S, walk, k);
            bool hit[2];
            cell_hits(S, walk, k, A, pt, &hit[0], &hit[1]);
#pragma unroll 1
            for (int which = 0; which < 2; ++which)
                if (which ? hit[1] : hit[0]) {
                    over(acc, paint_color(S, which ? A.z : A.w, pt));
                    if (cache) {
                        if (nf < sp.frag_slots) sp.frag[(size_t)nf * fstride + sid] = (uint16_t)(2 * cell_place(walk, k, A) + which);
                        ++nf;
                    }
                }
        }
        if (sp.frag) sp.frag_n[sid] = cache && nf <= sp.frag_slots ? (uint8_t)nf : FRAG_NONE;
    }
    if constexpr (G > 0)
        splat_group<G>(S, x, y, ox, oy, ri, HW, valid, pt, acc, sm);
    else if (valid)
        splat_sample(S, x, y, ox, oy, ri, HW, use_sm, pt, acc, sm, accum, wsum);
    if (!use_sm) return;
    __syncthreads();
    flush_splat(S, ox, oy, HW, sm, accum, wsum);
}
template <int G>
__global__ void __launch_bounds__(256, DVG_MINB_FWD) k_forward(const __grid_constant__ DevScene S, SampleParams sp,
                                                               float* accum, float* wsum) {
    extern __shared__ float sm[];
    forward_body<G>(S, sp, sp.tile_base + blockIdx.x, blockIdx.y, accum, wsum, sm);
}
// Batched forward: one flat grid over every (scene, tile, sub-sample) work item.
template <int G>
__global__ void __launch_bounds__(256, DVG_MINB_FWD) k_forward_batch(const BatchEntry* __restrict__ B,
                                                                     const int2* __restrict__ work, int items,
                                                                     int* counter) {
    extern __shared__ float sm[];
    for_each_item(items, counter, [&](int i) {
        const int2 wk = work[i];  // (scene, tile + tiles * sub-sample round)
        const BatchEntry& E = B[wk.x];
        const int tiles = E.S.tiles_x * E.S.tiles_y;
        forward_body<G>(E.S, E.sp, wk.y % tiles, wk.y / tiles, E.accum, E.wsum, sm);
    });
}

// Weight image only (rasterize_weights_f32, forward.rs:1505-1564).
__global__ void __launch_bounds__(256) k_weights(DevScene S, SampleParams sp, float* wsum) {
    const int tile = sp.tile_base + blockIdx.x, sub = blockIdx.y;
    const int tx = tile % S.tiles_x, ty = tile / S.tiles_x;
    const int x = tx * TILE + (threadIdx.x % TILE), y = ty * TILE + (threadIdx.x / TILE);
    if (x >= S.width || y >= S.height) return;
    const int ri = S.filter_ri;
    const int sx = sub % sp.sxn, sy = sub / sp.sxn;
    const float2 pt = sample_pos(x, y, sx, sy, sp.sxn, sp.syn, S.width, sp.seed, sp.jitter);
#pragma unroll 1
    for (int dy = -ri; dy <= ri; ++dy)
#pragma unroll 1
        for (int dx = -ri; dx <= ri; ++dx) {
            int xx = x + dx, yy = y + dy;
            if (xx < 0 || yy < 0 || xx >= S.width || yy >= S.height) continue;
            float w = filter_weight(S.filter_type, S.filter_radius, (float)xx + 0.5f - pt.x, (float)yy + 0.5f - pt.y);
            if (w > 0.0f) atomicAdd(wsum + (size_t)yy * S.width + xx, w);
        }
}

__global__ void k_resolve(DevScene S, const float* accum, const float* wsum, float* out) {
    size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (size_t)S.width * S.height) return;
    float r = S.bg[0], g = S.bg[1], b = S.bg[2], a = S.bg[3];
    float w = wsum[p];
    if (w > 0.0f) {
        float4 c = reinterpret_cast<const float4*>(accum)[p];
        r = c.x / w;
        g = c.y / w;
        b = c.z / w;
        a = c.w / w;
    }
    if (a > 1.0e-8f) {
        r = r / a;
        g = g / a;
        b = b / a;
    }
    reinterpret_cast<float4*>(out)[p] = make_float4(r, g, b, a);
}

// ------------------------------------------------------------------ backward helpers
// ------------------------------------------------------------------ interior backward
// Per sample: gather d_color (filters.rs:70-103), recompute the fragments of
// sample_color (sampling.rs:76-224) and back-propagate through compositing,
// paints, background and the filter (filters.rs:106-156).  The fragment list comes
// from the forward's fragment cache or is rebuilt from the BVHs; only (fragment
// code, transmittance) pairs live in per-thread local memory.  The adjoint loop
// walks the tile's group list in the same order on every lane so solid-paint
// gradients reduce across the warp before one atomic.
//
// LEAN: the kernel takes only the samples with cached fragments and carries no hit
// tests (fewer registers, more resident warps for its load chains); otherwise it
// takes every sample without a cache entry (all samples when there is no cache).
// Each sample is handled by exactly one of the two launches.
template <bool LEAN>
__device__ __forceinline__ void interior_body(const DevScene& S, const SampleParams& sp, int tile, int round,
                                              const float* d_render, const float* wsum, const GradPtrs& G,
                                              unsigned* status) {
    __shared__ float red[8][6];
    const int tx = tile % S.tiles_x, ty = tile / S.tiles_x;
    const int spp = sp.sxn * sp.syn;
    const int s_in_tile = round * 256 + (int)threadIdx.x;
    const int pix = sp.layout ? s_in_tile / spp : (int)threadIdx.x, sub = sp.layout ? s_in_tile % spp : round;
    const int2 pxy = pix_xy(pix);
    const int x = tx * TILE + pxy.x, y = ty * TILE + pxy.y;
    const size_t fstride = (size_t)S.tiles_x * S.tiles_y * spp * 256;
    const size_t sid = ((size_t)tile * spp + round) * 256 + threadIdx.x;
    const bool inside = x < S.width && y < S.height;
    const int cn = inside && sp.frag ? (int)__ldcs(&sp.frag_n[sid]) : (int)FRAG_NONE;
    const bool valid = inside && (LEAN ? cn != (int)FRAG_NONE : cn == (int)FRAG_NONE);
    if (!__syncthreads_or(valid)) return;  // uniform per CTA
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int* list = S.tile_entries + S.tile_offsets[tile];
    const int W = S.width, H = S.height;

    float2 ps = make_float2(0.0f, 0.0f), pt = make_float2(0.0f, 0.0f);
    int pixel = 0;
    float4 dcol = make_float4(0, 0, 0, 0), bg = make_float4(0, 0, 0, 0), rad = bg;
    if (valid) {
        const int sx = sub % sp.sxn, sy = sub / sp.sxn;
        ps = sample_pos(x, y, sx, sy, sp.sxn, sp.syn, W, sp.seed, sp.jitter);
        float2 npt = make_float2(ps.x / (float)W, ps.y / (float)H);  // render.rs:111
        pt = make_float2(npt.x * (float)W, npt.y * (float)H);       // sampling.rs:91
        pixel = y * W + x;
        bg = background_premul(S, pixel);
        dcol = gather_d_color_radius(S, d_render, wsum, ps, &rad);
    }
    // Pass 1: fragments in order (stroke before fill within a group).
    int code[MAX_FRAGMENTS];
    float tr[MAX_FRAGMENTS];
    int nf = 0;
    bool overflow = false;
    float4 acc = bg;
    if (valid) {
        // Either the forward's cached fragment codes (one fragment per step) or the
        // cell's entries with both hit tests (up to two fragments per step).
        CellWalk walk{};
        if constexpr (!LEAN) walk = cell_walk(S, tile, cell_of_pix(pix));
        const int steps = LEAN ? cn : walk.n;
#pragma unroll 1
        for (int k = 0; k < steps; ++k) {
            int e, hitp[2];
            if constexpr (LEAN) {
                const int c0 = __ldcs(&sp.frag[(size_t)k * fstride + sid]);
                e = c0 >> 1;
                const int4 gi = __ldg(&S.g_info[__ldg(&list[e])]);
                hitp[0] = (c0 & 1) ? -1 : gi.y;
                hitp[1] = (c0 & 1) ? gi.x : -1;
            } else {
                const int4 A = cell_entry(S, walk, k);
                bool st, fi;
                cell_hits(S, walk, k, A, pt, &st, &fi);
                e = cell_place(walk, k, A);
                hitp[0] = st ? A.w : -1;
                hitp[1] = fi ? A.z : -1;
            }
#pragma unroll 1
            for (int which = 0; which < 2; ++which) {
                if (hitp[which] < 0) continue;
                float4 c = paint_color(S, hitp[which], pt);
                over(acc, c);
                if (nf < MAX_FRAGMENTS) {
                    code[nf] = 2 * e + which;
                    tr[nf] = c.w;
                } else {
                    overflow = true;
                }
                ++nf;
            }
        }
    }
    if (overflow) {
        atomicOr(status, ST_FRAGMENT_OVERFLOW);
        nf = 0;
    }
    __syncthreads();  // the CTA's warps fetch one pass's instructions at a time: 0.874 -> 0.836 ms (mixed scene)
    const bool active = valid && !overflow;
    // Final colour and the adjoint at the end of compositing (sampling.rs:161-174).
    float4 ret = bg;
    float dcr = dcol.x, dcg = dcol.y, dcb = dcol.z, dca = dcol.w;
    if (nf > 0) {
        float fa = acc.w, fr = acc.x, fg = acc.y, fb = acc.z;
        if (fa > 1.0e-6f) {
            float s = 1.0f / fa;
            fr = fr * s;
            fg = fg * s;
            fb = fb * s;
            float dfr = dcr, dfg = dcg, dfb = dcb;
            dcr = dcr * s;
            dcg = dcg * s;
            dcb = dcb * s;
            dca -= (dfr * fr + dfg * fg + dfb * fb) / fa;
        }
        ret = make_float4(fr, fg, fb, fa);
        // Pass 2: transmittance after each fragment, T_i = prod_{j>i}(1 - a_j).
        float run = 1.0f;
        for (int i = nf - 1; i >= 0; --i) {
            float a = tr[i];
            tr[i] = run;
            run = run * (1.0f - a);
        }
        // background adjoint after all fragments
        float4 dbg = make_float4(dcr * run, dcg * run, dcb * run, dca * run);
        if (S.bg_image) {
            float* b = G.d_background_image;
            if (b) {
                add_if(b + 4 * (size_t)pixel + 0, dbg.x);
                add_if(b + 4 * (size_t)pixel + 1, dbg.y);
                add_if(b + 4 * (size_t)pixel + 2, dbg.z);
                add_if(b + 4 * (size_t)pixel + 3, dbg.w);
            }
            dbg = make_float4(0, 0, 0, 0);
        }
        dcol = dbg;  // reused below as this sample's constant-background adjoint
    } else if (active) {
        // no fragment: accumulate_background_grad(d_color) (sampling.rs:121-127)
        if (S.bg_image) {
            float* b = G.d_background_image;
            if (b) {
                add_if(b + 4 * (size_t)pixel + 0, dcol.x);
                add_if(b + 4 * (size_t)pixel + 1, dcol.y);
                add_if(b + 4 * (size_t)pixel + 2, dcol.z);
                add_if(b + 4 * (size_t)pixel + 3, dcol.w);
            }
            dcol = make_float4(0, 0, 0, 0);
        }
    }
    if (!active) dcol = make_float4(0, 0, 0, 0);

    // Pass 3: forward over the fragments with the compositing adjoint (sampling.rs:175-210).
    // The warp visits only the (group, stroke/fill) entries some lane hit: each round
    // takes the smallest next fragment code over the warp, so lanes stay in step for
    // the warp-reduced solid-paint gradients while entries nobody hit cost nothing.
    int cur = 0;
    float4 prev = bg;
    while (true) {
        const int mine = cur < nf ? code[cur] : 0x7fffffff;
        const int nxt = __reduce_min_sync(0xffffffffu, mine);
        if (nxt == 0x7fffffff) break;
        const int e = nxt >> 1, which = nxt & 1;  // code = 2 * entry + (0 stroke, 1 fill)
        const int g = __ldg(&list[e]);
        const int4 gi = __ldg(&S.g_info[g]);
        const int p = which == 0 ? gi.y : gi.x;
        const bool has = mine == nxt;
        float4 dv = make_float4(0, 0, 0, 0);
        if (has) {
            const float4 c = paint_color(S, p, pt);
            float T = tr[cur];
            float r_ = dcr * T, g_ = dcg * T, b_ = dcb * T, a_ = dca * T;
            float d_alpha = a_ * (1.0f - prev.w);
            d_alpha += r_ * (c.x - prev.x) + g_ * (c.y - prev.y) + b_ * (c.z - prev.z);
            dv = make_float4(r_ * c.w, g_ * c.w, b_ * c.w, d_alpha);
            over(prev, c);
            ++cur;
        }
        const int kind = __ldg(&S.paint_info[p].x);
        if (kind == P_SOLID) {
            float s0 = warp_sum(dv.x), s1 = warp_sum(dv.y), s2 = warp_sum(dv.z), s3 = warp_sum(dv.w);
            if (lane == 0) {
                float* d = G.d_paint_params + 4 * p;
                add_if(d + 0, s0);
                add_if(d + 1, s1);
                add_if(d + 2, s2);
                add_if(d + 3, s3);
            }
        } else {
            float2 dtr = make_float2(0.0f, 0.0f);
            d_gradient_paint_warp(S, G, p, pt, dv, has, &dtr);
            if (has && G.d_translation) {
                add_if(G.d_translation + 2 * (size_t)pixel, dtr.x);
                add_if(G.d_translation + 2 * (size_t)pixel + 1, dtr.y);
            }
        }
    }
    // Filter-radius adjoint (filters.rs:106-156) and the constant-background adjoint.
    float dradius = 0.0f;
    if (active)
        dradius = S.filter_type == F_PARABOLIC ? filter_radius_adjoint(S, d_render, wsum, ps, ret)
                                               : rad.x * ret.x + rad.y * ret.y + rad.z * ret.z + rad.w * ret.w;
    float v[5] = {dcol.x, dcol.y, dcol.z, dcol.w, dradius};
#pragma unroll
    for (int k = 0; k < 5; ++k) v[k] = warp_sum(v[k]);
    if (lane == 0)
        for (int k = 0; k < 5; ++k) red[wid][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 5) {
        float s = 0.0f;
        for (int w = 0; w < 8; ++w) s += red[w][threadIdx.x];
        if (threadIdx.x < 4)
            add_if(G.d_background + threadIdx.x, s);
        else
            add_if(G.d_filter_radius, s);
    }
}

__global__ void __launch_bounds__(256, DVG_MINB_INT) k_interior(const __grid_constant__ DevScene S, SampleParams sp, const float* d_render,
                                                                const float* wsum, GradPtrs G, unsigned* status) {
    interior_body<false>(S, sp, sp.tile_base + blockIdx.x, blockIdx.y, d_render, wsum, G, status);
}
__global__ void __launch_bounds__(256, DVG_MINB_LEAN) k_interior_cached(DevScene S, SampleParams sp,
                                                                        const float* d_render, const float* wsum,
                                                                        GradPtrs G, unsigned* status) {
    interior_body<true>(S, sp, sp.tile_base + blockIdx.x, blockIdx.y, d_render, wsum, G, status);
}
__global__ void __launch_bounds__(256, DVG_MINB_INT) k_interior_batch(const BatchEntry* __restrict__ B,
                                                                      const int2* __restrict__ work, int items,
                                                                      int* counter, unsigned* status) {
    for_each_item(items, counter, [&](int i) {
        const int2 wk = work[i];  // (scene, tile + tiles * sub-sample round)
        const BatchEntry& E = B[wk.x];
        const int tiles = E.S.tiles_x * E.S.tiles_y;
        interior_body<false>(E.S, E.sp, wk.y % tiles, wk.y / tiles, E.d_render, E.wsum, E.G, status);
    });
}
__global__ void __launch_bounds__(256, DVG_MINB_LEAN) k_interior_cached_batch(const BatchEntry* __restrict__ B,
                                                                              const int2* __restrict__ work, int items,
                                                                              int* counter, unsigned* status) {
    for_each_item(items, counter, [&](int i) {
        const int2 wk = work[i];  // (scene, tile + tiles * sub-sample round)
        const BatchEntry& E = B[wk.x];
        if (!E.sp.frag) return;  // uniform per item
        const int tiles = E.S.tiles_x * E.S.tiles_y;
        interior_body<true>(E.S, E.sp, wk.y % tiles, wk.y / tiles, E.d_render, E.wsum, E.G, status);
    });
}

// ------------------------------------------------------------------ boundary sampling
// The queried shape's own tests, out of line (run where no fragment decides the hit).
static __device__ __noinline__ bool within_shape_any(const DevScene& S, int s, float2 lp, float r) {
    return within_shape(S, s, lp, r);
}
static __device__ __noinline__ int winding_shape_any(const DevScene& S, int s, float2 sp) {
    return winding_shape(S, s, sp, true);
}
// Whether the group tests above, which found no hit of the queried group, are the queried
// shape's own tests at lp: the group has no other shape, lp lies in its box (so the tests were
// made) and both take the same point (shape_local_dist's identity shortcut is exact).  Half of
// the samples' points end here, each with a walk over the whole path: 128x128 adjoint scene,
// the edge pass 0.53 -> 0.40 ms (128x128 scene of 8 outlines, 262,144 samples).
__device__ __forceinline__ bool edge_tests_done(const DevScene& S, int g, int s, float2 lp) {
    const int4 gb = __ldg(&S.g_bvh[g]);
    if (gb.y != 1 || __ldg(&S.gn_meta[gb.x].z) != 1) return false;
    const float4 b = __ldg(&S.gn_bounds[gb.x]);
    if (!(lp.x >= b.x && lp.x <= b.z && lp.y >= b.y && lp.y <= b.w)) return false;
    const int4 si = __ldg(&S.s_info[s]);
    if (si.x == K_PATH && (si.z < 0 || (__ldg(&S.p_info[2 * si.z + 1].w) & PF_STYLED))) return false;
    if (!(si.y & SF_IDENTITY)) return true;
    const float* v = S.s_inv + 6 * s;
    return v[0] == 1.0f && v[1] == 0.0f && v[2] == 0.0f && v[3] == 0.0f && v[4] == 1.0f && v[5] == 0.0f;
}
// sample_color with an EdgeQuery (sampling.rs:76-224, 485-552) at canvas point pt.
// Returns the un-premultiplied colour (or the premultiplied background when no
// fragment covers pt) and whether the queried shape is the visible boundary.
// All threads of the CTA call it (`valid` false: no point).
__device__ __forceinline__ float4 edge_color(const DevScene& S, bool valid, int tile, int cell, float2 pt, float4 bg,
                                             int eq_group, int eq_shape, bool* hit_out) {
    CellWalk walk{};
    if (valid) walk = cell_walk(S, tile, cell);
    const bool step = __syncthreads_or(walk.heavy);  // (the CTA's samples share a cell or neighbouring ones)
    float4 acc = bg;
    int nfrag = 0, ev = 0;  // ev: 0 none, 1 last event sets the hit, 2 last event clears it
#pragma unroll 1
    for (int k = 0; step ? __syncthreads_or(k < walk.n) : k < walk.n; ++k) {
        if (k >= walk.n) continue;
        // stroke first, then fill; one paint call site for both
        const int4 A = cell_entry(S, walk, k);
        bool hit[2];
        cell_hits(S, walk, k, A, pt, &hit[0], &hit[1]);
#pragma unroll 1
        for (int which = 0; which < 2; ++which) {
            if (!(which ? hit[1] : hit[0])) continue;
            const float4 c = paint_color(S, which ? A.z : A.w, pt);
            over(acc, c);
            ++nfrag;
            if (c.w >= 1.0f) ev = 2;
            if (A.y == eq_group) ev = 1;
        }
    }
    if (!valid) return bg;
    if (ev != 0) {
        *hit_out = ev == 1;
    } else {  // no deciding fragment: the edge tests on the queried shape alone
              // (within_distance_edge / is_inside_edge)
        bool hit0 = false;
        const int4 gi = __ldg(&S.g_info[eq_group]);
        const float2 lp = xf9(S.g_c2s + 9 * eq_group, pt);
        if (!edge_tests_done(S, eq_group, eq_shape, lp)) {
            if (gi.y >= 0) {
                float sw = __ldg(&S.s_stroke[eq_shape]);
                if (sw > 0.0f && within_shape_any(S, eq_shape, lp, sw)) hit0 = true;
            }
            if (gi.x >= 0) {
                float2 sp = shape_local_bwd(S, eq_shape, lp);
                if (fill_hit(gi.z, winding_shape_any(S, eq_shape, sp))) hit0 = true;
            }
        }
        *hit_out = hit0;
    }
    if (nfrag == 0) return bg;
    float fa = acc.w, fr = acc.x, fg = acc.y, fb = acc.z;
    if (fa > 1.0e-6f) {
        float s = 1.0f / fa;
        fr = fr * s;
        fg = fg * s;
        fb = fb * s;
    }
    return make_float4(fr, fg, fb, fa);
}

__device__ __forceinline__ int lower_bound_cdf(const float* cdf, int n, float u) {
    // first idx with !(u > cdf[idx]) — the crate's linear scan (boundary.rs:454-469)
    int lo = 0, hi = n;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (u > __ldg(&cdf[mid]))
            lo = mid + 1;
        else
            hi = mid;
    }
    return lo;
}
__device__ __forceinline__ float cdf_local_t(const float* cdf, int n, int idx, float u) {
    float prev = idx == 0 ? 0.0f : __ldg(&cdf[idx - 1]);
    float denom = fmaxf(__ldg(&cdf[idx]) - prev, 1.0e-6f);
    return clampf((u - prev) / denom, 0.0f, 1.0f);
}
__device__ __forceinline__ bool path_pt(const DevScene& S, int po, int pc, bool closed, long idx, float2* p) {
    if (pc == 0) return false;
    long i;
    if (closed)
        i = idx % pc;
    else if (idx >= pc)
        return false;
    else
        i = idx;
    *p = S.points[po + i];
    return true;
}
__device__ __forceinline__ bool path_pt_r(const DevScene& S, int po, int pc, bool closed, bool thick, long idx,
                                          float def_r, float2* p, float* r) {
    if (!path_pt(S, po, pc, closed, idx, p)) return false;
    long i = closed ? idx % pc : idx;
    *r = (thick && i < pc) ? S.thickness[po + i] * 1.0f : def_r;
    return true;
}
struct BData {
    int base_point_id, point_id;
    float t;
    bool is_stroke;
};
__device__ __forceinline__ float2 nrm2(float2 v) {
    float l = len2(v.x, v.y);
    return l == 0.0f ? make_float2(0.0f, 0.0f) : make_float2(v.x / l, v.y / l);
}
// Join and cap edges of a stroke with non-round joins or caps (the polygons
// join_cap_hit tests), sampled as part of its boundary: uniform over the sites (the
// non-round joins, and for open paths with non-round caps the two ends), then by
// length along the site's edges.  Like the crate's offset-curve samples, a point
// moves with its centreline point (the vertex): data->point_id is the vertex's path
// point, data->t the radius derivative (p - v) . n / r (every site polygon scales
// about v with the radius), and base_point_id = -1 marks the sample.
__device__ float2 sample_join_cap(const DevScene& S, int path, float t, float2* normal, float* pdf, BData* data) {
    const int4 pi = __ldg(&S.p_info[2 * path]);
    const int4 pi2 = __ldg(&S.p_info[2 * path + 1]);
    const bool closed = pi2.w & PF_CLOSED;
    const int join = (pi2.w >> PF_JOIN_SHIFT) & 3, cap = (pi2.w >> PF_CAP_SHIFT) & 3;
    const int off = pi.x, n = pi.y;
    const int nj = join != JOIN_ROUND ? (closed ? n : n - 1) : 0;
    const int ncap = !closed && cap != CAP_ROUND ? 2 : 0;
    const int sites = nj + ncap;
    if (n <= 0 || sites <= 0) {
        *pdf = 0.0f;
        return make_float2(0, 0);
    }
    int k = (int)(t * (float)sites);
    if (k > sites - 1) k = sites - 1;
    const float u = t * (float)sites - (float)k;
    *pdf /= (float)sites;
    float2 e[4], v;
    int ne = 0, pid = 0;
    float r = 0.0f;
    float2 capdir = make_float2(0, 0);
    if (k < nj) {
        const int vb = closed ? k : k + 1, va = vb > 0 ? vb - 1 : n - 1;
        const float4 a0 = __ldg(&S.seg_p[2 * (off + va)]), a1 = __ldg(&S.seg_p[2 * (off + va) + 1]);
        const float4 b0 = __ldg(&S.seg_p[2 * (off + vb)]), b1 = __ldg(&S.seg_p[2 * (off + vb) + 1]);
        v = make_float2(b0.x, b0.y);
        r = __ldg(&S.seg_r[off + vb]).x;
        pid = __ldg(&S.seg_meta[off + vb]).z;
        float2 din = seg_dir1(a0, a1), dout = seg_dir0(b0, b1);
        const float li = sqrtf(din.x * din.x + din.y * din.y), lo = sqrtf(dout.x * dout.x + dout.y * dout.y);
        if (!(li > 0.0f) || !(lo > 0.0f) || !(r > 0.0f)) {
            *pdf = 0.0f;
            return make_float2(0, 0);
        }
        din = make_float2(din.x / li, din.y / li);
        dout = make_float2(dout.x / lo, dout.y / lo);
        const float cr = cross2f(din.x, din.y, dout.x, dout.y);
        if (fabsf(cr) < 1.0e-6f) {  // no outer corner: no edge here
            *pdf = 0.0f;
            return make_float2(0, 0);
        }
        const float sg = cr > 0.0f ? 1.0f : -1.0f;
        e[0] = make_float2(v.x + r * sg * din.y, v.y - r * sg * din.x);
        const float2 b = make_float2(v.x + r * sg * dout.y, v.y - r * sg * dout.x);
        ne = 1;
        if (join == JOIN_MITER) {
            const float sm = cross2f(b.x - e[0].x, b.y - e[0].y, dout.x, dout.y) / cr;
            const float2 m = make_float2(e[0].x + sm * din.x, e[0].y + sm * din.y);
            const float ml = sqrtf((m.x - v.x) * (m.x - v.x) + (m.y - v.y) * (m.y - v.y));
            if (ml <= __ldg(&S.p_miter[path]) * r) e[ne++] = m;
        }
        e[ne] = b;
    } else {
        const bool start = k == nj;
        const int sidx = start ? 0 : n - 1;
        const float4 q0 = __ldg(&S.seg_p[2 * (off + sidx)]), q1 = __ldg(&S.seg_p[2 * (off + sidx) + 1]);
        float2 d;
        if (start) {
            const float2 d0 = seg_dir0(q0, q1);
            d = make_float2(-d0.x, -d0.y);
            v = make_float2(q0.x, q0.y);
            r = __ldg(&S.seg_r[off]).x;
            pid = __ldg(&S.seg_meta[off]).z;
        } else {
            d = seg_dir1(q0, q1);
            v = make_float2(q1.z, q1.w);
            r = __ldg(&S.seg_r[off + n - 1]).w;
            pid = pi2.y - 1;
        }
        const float l = sqrtf(d.x * d.x + d.y * d.y);
        if (!(l > 0.0f) || !(r > 0.0f)) {
            *pdf = 0.0f;
            return make_float2(0, 0);
        }
        d = make_float2(d.x / l, d.y / l);
        capdir = d;
        const float2 np = make_float2(-d.y, d.x);
        e[0] = make_float2(v.x - r * np.x, v.y - r * np.y);
        if (cap == CAP_SQUARE) {
            e[1] = make_float2(e[0].x + r * d.x, e[0].y + r * d.y);
            e[2] = make_float2(v.x + r * np.x + r * d.x, v.y + r * np.y + r * d.y);
            e[3] = make_float2(v.x + r * np.x, v.y + r * np.y);
            ne = 3;
        } else {
            e[1] = make_float2(v.x + r * np.x, v.y + r * np.y);
            ne = 1;
        }
    }
    float len[3], total = 0.0f;
#pragma unroll 1
    for (int i = 0; i < ne; ++i) {
        len[i] = len2(e[i + 1].x - e[i].x, e[i + 1].y - e[i].y);
        total += len[i];
    }
    if (!(total > 0.0f)) {
        *pdf = 0.0f;
        return make_float2(0, 0);
    }
    float sl = u * total;
    int i = 0;
    while (i < ne - 1 && sl > len[i]) sl -= len[i++];
    const float f = len[i] > 0.0f ? fminf(sl / len[i], 1.0f) : 0.0f;
    const float2 p = make_float2(e[i].x + f * (e[i + 1].x - e[i].x), e[i].y + f * (e[i + 1].y - e[i].y));
    float2 nn = nrm2(make_float2(-(e[i + 1].y - e[i].y), e[i + 1].x - e[i].x));
    const float mx = 0.5f * (e[i].x + e[i + 1].x) - v.x, my = 0.5f * (e[i].y + e[i + 1].y) - v.y;
    const float side = (mx == 0.0f && my == 0.0f) ? nn.x * capdir.x + nn.y * capdir.y : nn.x * mx + nn.y * my;
    if (side < 0.0f) nn = make_float2(-nn.x, -nn.y);
    *pdf /= total;
    *normal = nn;
    (void)pid;
    data->base_point_id = -1 - k;  // the site
    data->point_id = i;            // the edge of the site's polygon
    data->t = f;                   // the position along that edge
    return p;
}

// Normal velocity of the join / cap edge point sampled at (site, edge, f):
// w[k] = dp/dtheta_k . n for theta = (v, qa, qb, r); ids = path points of v, qa, qb
// (-1: not used).  Out of line: it runs only for those samples.
static __device__ __noinline__ bool join_cap_velocity(const int4* p_info, const float* p_miter, const float4* seg_p,
                                                     const float4* seg_r, const int4* seg_meta, int path, int site,
                                                     int edge, float f, float nx, float ny, float* w, int* ids) {
    const int4 pi = __ldg(&p_info[2 * path]);
    const int4 pi2 = __ldg(&p_info[2 * path + 1]);
    const bool closed = pi2.w & PF_CLOSED;
    const int join = (pi2.w >> PF_JOIN_SHIFT) & 3, cap = (pi2.w >> PF_CAP_SHIFT) & 3;
    const int off = pi.x, nseg = pi.y, pc = pi2.y;
    const int nj = join != JOIN_ROUND ? (closed ? nseg : nseg - 1) : 0;
    ids[0] = ids[1] = ids[2] = -1;
    DV e[4];
    int ne = 0;
    if (site < nj) {
        const int vb = closed ? site : site + 1, va = vb > 0 ? vb - 1 : nseg - 1;
        const float4 a0 = __ldg(&seg_p[2 * (off + va)]), a1 = __ldg(&seg_p[2 * (off + va) + 1]);
        const float4 b0 = __ldg(&seg_p[2 * (off + vb)]), b1 = __ldg(&seg_p[2 * (off + vb) + 1]);
        const int sa = seg_dir1_slot(a0, a1), sb = seg_dir0_slot(b0, b1);
        const float2 v = make_float2(b0.x, b0.y), qa = seg_slot(a0, a1, sa), qb = seg_slot(b0, b1, sb);
        const int4 ma = __ldg(&seg_meta[off + va]), mb = __ldg(&seg_meta[off + vb]);
        ids[0] = mb.z;
        ids[1] = seg_slot_point(ma, sa, closed, pc);
        ids[2] = seg_slot_point(mb, sb, closed, pc);
        const DV V{dl_var(v.x, 0), dl_var(v.y, 1)}, QA{dl_var(qa.x, 2), dl_var(qa.y, 3)},
            QB{dl_var(qb.x, 4), dl_var(qb.y, 5)};
        const Dl R = dl_var(__ldg(&seg_r[off + vb]).x, 6);
        const DV din = dv_unit(dv_sub(V, QA)), dout = dv_unit(dv_sub(QB, V));
        const Dl cr = din.x * dout.y - din.y * dout.x;
        if (fabsf(cr.v) < 1.0e-6f) return false;
        const Dl sg = dl_const(cr.v > 0.0f ? 1.0f : -1.0f);
        e[0] = DV{V.x + R * sg * din.y, V.y - R * sg * din.x};
        const DV b{V.x + R * sg * dout.y, V.y - R * sg * dout.x};
        ne = 1;
        if (join == JOIN_MITER) {
            const Dl sm = ((b.x - e[0].x) * dout.y - (b.y - e[0].y) * dout.x) / cr;
            const DV m = dv_add(e[0], dv_scale(din, sm));
            const float ml = sqrtf((m.x.v - v.x) * (m.x.v - v.x) + (m.y.v - v.y) * (m.y.v - v.y));
            if (ml <= __ldg(&p_miter[path]) * R.v) e[ne++] = m;
        }
        e[ne] = b;
    } else {
        const bool start = site == nj;
        const int si = start ? 0 : nseg - 1;
        const float4 q0 = __ldg(&seg_p[2 * (off + si)]), q1 = __ldg(&seg_p[2 * (off + si) + 1]);
        const int sq = start ? seg_dir0_slot(q0, q1) : seg_dir1_slot(q0, q1);
        const float2 v = start ? make_float2(q0.x, q0.y) : make_float2(q1.z, q1.w), q = seg_slot(q0, q1, sq);
        const int4 m = __ldg(&seg_meta[off + si]);
        ids[0] = start ? m.z : pc - 1;
        ids[start ? 2 : 1] = seg_slot_point(m, sq, closed, pc);
        const DV V{dl_var(v.x, 0), dl_var(v.y, 1)};
        const DV Q = start ? DV{dl_var(q.x, 4), dl_var(q.y, 5)} : DV{dl_var(q.x, 2), dl_var(q.y, 3)};
        const float4 rr = __ldg(&seg_r[off + si]);
        const Dl R = dl_var(start ? rr.x : rr.w, 6);
        const DV d = dv_unit(dv_sub(V, Q));  // outward along the end
        const DV np{dl_const(0.0f) - d.y, d.x};
        e[0] = dv_sub(V, dv_scale(np, R));
        if (cap == CAP_SQUARE) {
            e[1] = dv_add(e[0], dv_scale(d, R));
            e[2] = dv_add(dv_add(V, dv_scale(np, R)), dv_scale(d, R));
            e[3] = dv_add(V, dv_scale(np, R));
            ne = 3;
        } else {
            e[1] = dv_add(V, dv_scale(np, R));
            ne = 1;
        }
    }
    if (edge >= ne) return false;
    const DV p = dv_add(e[edge], dv_scale(dv_sub(e[edge + 1], e[edge]), dl_const(f)));
#pragma unroll
    for (int k = 0; k < 7; ++k) w[k] = p.x.d[k] * nx + p.y.d[k] * ny;
    return true;
}

// sample_boundary_path (boundary.rs:630-842)
__device__ float2 sample_boundary_path(const DevScene& S, int shape, float path_len, float t, float2* normal,
                                       float* pdf, BData* data, float dir, float srad) {
    const int path = __ldg(&S.s_info[shape].z);
    const int4 pi2 = __ldg(&S.p_info[2 * path + 1]);
    const int po = pi2.x, pc = pi2.y, co = pi2.z;
    const bool closed = pi2.w & PF_CLOSED;
    const bool thick = pi2.w & PF_THICK;
    const int4 cinfo = __ldg(&S.path_cdf_info[shape]);
    const int nb = cinfo.y;
    if (pc == 0 || nb == 0) {
        *pdf = 0.0f;
        return make_float2(0, 0);
    }
    const bool styled = dir != 0.0f && (pi2.w & PF_STYLED);
    if (styled) {  // a share of the samples on the join / cap edges (both sides draw them)
        const float q = JOIN_CAP_SHARE;
        if (t < q) {
            *pdf *= 2.0f * q;
            return sample_join_cap(S, path, t / q, normal, pdf, data);
        }
        t = (t - q) / (1.0f - q);
        *pdf *= 1.0f - q;
    }
    if (dir != 0.0f && !closed && (!styled || ((pi2.w >> PF_CAP_SHIFT) & 3) == CAP_ROUND)) {
        float cap = 0.0f;
        if (thick)
            cap = PI_F * (S.thickness[po] + S.thickness[po + pc - 1]);
        else
            cap = 2.0f * PI_F * srad;
        float denom = cap + path_len;
        if (denom > 0.0f) {
            float cp = cap / denom;
            if (t < cp) {
                t /= cp;
                *pdf *= cp;
                float r0 = srad, r1 = srad;
                if (thick) {
                    r0 = S.thickness[po];
                    r1 = S.thickness[po + pc - 1];
                }
                float ang = 2.0f * PI_F * t;
                if (dir < 0.0f) {
                    float2 o = make_float2(r0 * dvg_cosf(ang), r0 * dvg_sinf(ang));
                    *normal = nrm2(o);
                    *pdf /= 2.0f * PI_F * r0;
                    data->base_point_id = 0;
                    data->point_id = 0;
                    data->t = 0.0f;
                    float2 p0 = S.points[po];
                    return make_float2(p0.x + o.x, p0.y + o.y);
                }
                float2 o = make_float2(r1 * dvg_cosf(ang), r1 * dvg_sinf(ang));
                *normal = nrm2(o);
                *pdf /= 2.0f * PI_F * r1;
                data->base_point_id = nb - 1;
                int controls = S.ncp[co + nb - 1];
                data->point_id = pc >= 2 + controls ? pc - (2 + controls) : 0;
                data->t = 1.0f;
                float2 pl = S.points[po + pc - 1];
                return make_float2(pl.x + o.x, pl.y + o.y);
            }
            t = (t - cp) / (1.0f - cp);
            *pdf *= 1.0f - cp;
        }
    }
    const float* cdf = S.path_cdf + cinfo.x;
    int sid = lower_bound_cdf(cdf, nb, t);
    if (sid >= nb) sid = nb - 1;
    float lt = cdf_local_t(cdf, nb, sid, t);
    int pid = S.path_pid[cinfo.x + sid];
    data->base_point_id = sid;
    data->point_id = pid;
    data->t = lt;
    if (lt < -1.0e-3f || lt > 1.0f + 1.0e-3f) {
        *pdf = 0.0f;
        return make_float2(0, 0);
    }
    int nc = S.ncp[co + sid];
    float pmf = S.path_pmf[cinfo.x + sid];
    auto nxt = [&](long i) -> long { return closed ? i % pc : (i < pc - 1 ? i : pc - 1); };
    float2 q[4];
    float r[4];
    int np = nc + 2;
    if (nc > 2) {
        *pdf = 0.0f;
        return make_float2(0, 0);
    }
#pragma unroll 1
    for (int k = 0; k < np; ++k) {
        long idx = (k == np - 1) ? nxt(pid + k) : (long)(pid + k);
        if (!path_pt_r(S, po, pc, closed, thick, idx, srad, &q[k], &r[k])) {
            *pdf = 0.0f;
            return make_float2(0, 0);
        }
    }
    float tt = 1.0f - lt;
    float2 ev, tg;
    float rr;
    if (nc == 0) {
        tg = make_float2(q[1].x - q[0].x, q[1].y - q[0].y);
        ev = make_float2(q[0].x + tg.x * lt, q[0].y + tg.y * lt);
        rr = r[0] + lt * (r[1] - r[0]);
    } else if (nc == 1) {
        float w0 = tt * tt, w1 = 2.0f * tt * lt, w2 = lt * lt;
        ev = make_float2(q[0].x * w0 + q[1].x * w1 + q[2].x * w2, q[0].y * w0 + q[1].y * w1 + q[2].y * w2);
        float a = 2.0f * tt, b = 2.0f * lt;
        tg = make_float2((q[1].x - q[0].x) * a + (q[2].x - q[1].x) * b, (q[1].y - q[0].y) * a + (q[2].y - q[1].y) * b);
        rr = r[0] * w0 + r[1] * w1 + r[2] * w2;
    } else {
        float w0 = tt * tt * tt, w1 = 3.0f * tt * tt * lt, w2 = 3.0f * tt * lt * lt, w3 = lt * lt * lt;
        ev = make_float2(q[0].x * w0 + q[1].x * w1 + q[2].x * w2 + q[3].x * w3,
                         q[0].y * w0 + q[1].y * w1 + q[2].y * w2 + q[3].y * w3);
        float a = 3.0f * tt * tt, b = 6.0f * tt * lt, c = 3.0f * lt * lt;
        tg = make_float2((q[1].x - q[0].x) * a + (q[2].x - q[1].x) * b + (q[3].x - q[2].x) * c,
                         (q[1].y - q[0].y) * a + (q[2].y - q[1].y) * b + (q[3].y - q[2].y) * c);
        rr = r[0] * w0 + r[1] * w1 + r[2] * w2 + r[3] * w3;
    }
    float tl = len2(tg.x, tg.y);
    if (tl == 0.0f) {
        *pdf = 0.0f;
        return make_float2(0, 0);
    }
    *normal = make_float2(-tg.y / tl, tg.x / tl);
    *pdf *= pmf / tl;
    if (dir != 0.0f) {
        ev.x += normal->x * (dir * rr);
        ev.y += normal->y * (dir * rr);
        if (dir < 0.0f) *normal = make_float2(normal->x * -1.0f, normal->y * -1.0f);
    }
    return ev;
}
// sample_boundary_point (boundary.rs:472-627)
__device__ bool sample_boundary_point(const DevScene& S, int shape, int group, float t, float shape_len,
                                      float2* pt_out, float2* normal_out, float* pdf_out, BData* data) {
    const int4 gi = __ldg(&S.g_info[group]);
    const bool has_fill = gi.x >= 0, has_stroke = gi.y >= 0;
    if (!has_fill && !has_stroke) return false;
    float pdf = 1.0f, lt = t;
    bool stroke = false;
    if (has_fill && has_stroke) {
        if (lt < 0.5f) {
            lt *= 2.0f;
        } else {
            stroke = true;
            lt = 2.0f * (lt - 0.5f);
        }
        pdf = 0.5f;
    } else if (has_stroke) {
        stroke = true;
    }
    float dir = 0.0f;
    if (stroke) {
        if (lt < 0.5f) {
            dir = -1.0f;
            lt *= 2.0f;
        } else {
            dir = 1.0f;
            lt = 2.0f * (lt - 0.5f);
        }
        pdf *= 0.5f;
    }
    data->base_point_id = 0;
    data->point_id = 0;
    data->t = 0.0f;
    data->is_stroke = stroke;
    const int4 si = __ldg(&S.s_info[shape]);
    const float4 prm = __ldg(&S.s_params[shape]);
    const float sw = __ldg(&S.s_stroke[shape]);
    float2 normal = make_float2(0, 0), out;
    if (si.x == K_CIRCLE) {
        float r = fabsf(prm.z);
        if (r <= 0.0f) return false;
        float ang = 2.0f * PI_F * lt;
        float2 o = make_float2(r * dvg_cosf(ang), r * dvg_sinf(ang));
        normal = nrm2(o);
        pdf /= 2.0f * PI_F * r;
        out = make_float2(prm.x + o.x, prm.y + o.y);
    } else if (si.x == K_ELLIPSE) {
        float rx = fabsf(prm.z), ry = fabsf(prm.w);
        if (rx <= 0.0f || ry <= 0.0f) return false;
        float ang = 2.0f * PI_F * lt;
        float s = dvg_sinf(ang), c = dvg_cosf(ang);
        float dxdt = -rx * s * 2.0f * PI_F, dydt = ry * c * 2.0f * PI_F;
        normal = nrm2(make_float2(dydt, -dxdt));
        pdf /= sqrtf(dxdt * dxdt + dydt * dydt);
        out = make_float2(prm.x + rx * c, prm.y + ry * s);
    } else if (si.x == K_RECT) {
        float w = prm.z - prm.x, h = prm.w - prm.y;
        if (w == 0.0f && h == 0.0f) return false;
        pdf /= 2.0f * (w + h);
        if (lt <= w / (w + h)) {
            lt *= (w + h) / w;
            if (lt < 0.5f) {
                normal = make_float2(0.0f, -1.0f);
                out = make_float2(prm.x + 2.0f * lt * (prm.z - prm.x), prm.y + 0.0f);
            } else {
                normal = make_float2(0.0f, 1.0f);
                out = make_float2(prm.x + 2.0f * (lt - 0.5f) * (prm.z - prm.x), prm.w + 0.0f);
            }
        } else {
            lt = (lt - w / (w + h)) * (w + h) / h;
            if (lt < 0.5f) {
                normal = make_float2(-1.0f, 0.0f);
                out = make_float2(prm.x + 0.0f, prm.y + 2.0f * lt * (prm.w - prm.y));
            } else {
                normal = make_float2(1.0f, 0.0f);
                out = make_float2(prm.z + 0.0f, prm.y + 2.0f * (lt - 0.5f) * (prm.w - prm.y));
            }
        }
    } else {
        if (si.z < 0) return false;
        const int4 ci = __ldg(&S.path_cdf_info[shape]);
        if (!ci.z) return false;
        if (S.path_len[shape] <= 0.0f) return false;
        out = sample_boundary_path(S, shape, shape_len, lt, &normal, &pdf, data, dir, sw);
        dir = 0.0f;  // the path sampler applies the stroke offset itself
    }
    if (dir != 0.0f) {
        out.x += normal.x * (dir * sw);
        out.y += normal.y * (dir * sw);
        if (dir < 0.0f) normal = make_float2(normal.x * -1.0f, normal.y * -1.0f);
    }
    if (!isfinite(pdf) || pdf <= 0.0f) return false;
    *pt_out = out;
    *normal_out = normal;
    *pdf_out = pdf;
    return true;
}
// The gradient of one join / cap edge sample (out of line with scalar arguments: the
// boundary kernel is instruction-fetch bound and these samples are few).
static __device__ __noinline__ void accumulate_join_cap(const int4* p_info, const float* p_miter,
                                                       const float4* seg_p, const float4* seg_r,
                                                       const int4* seg_meta, float* d_points, float* d_thickness,
                                                       float* d_stroke_width, int path, int po, int site, int edge,
                                                       float f, float nx, float ny, float contrib) {
    float w[7];
    int ids[3];
    if (!join_cap_velocity(p_info, p_miter, seg_p, seg_r, seg_meta, path, site, edge, f, nx, ny, w, ids)) return;
    for (int j = 0; j < 3; ++j)
        if (ids[j] >= 0) {
            add_if(d_points + 2 * (po + ids[j]), w[2 * j] * contrib);
            add_if(d_points + 2 * (po + ids[j]) + 1, w[2 * j + 1] * contrib);
        }
    if (d_thickness)
        add_if(d_thickness + po + ids[0], w[6] * contrib);
    else
        add_if(d_stroke_width, w[6] * contrib);
}
__device__ __forceinline__ void mul33(const float* a, const float* b, float* o) {  // Mat3::mul
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) o[3 * r + c] = a[3 * r] * b[c] + a[3 * r + 1] * b[3 + c] + a[3 * r + 2] * b[6 + c];
}
// accumulate_boundary_gradient (boundary.rs:970-1148)
// STYLED: the scene has strokes with non-round joins or caps (join / cap edge samples,
// base_point_id < 0); the kernels of other scenes carry none of that code.
template <bool STYLED>
__device__ void accumulate_boundary(const DevScene& S, const GradPtrs& G, int shape, int group, float contrib,
                                    float t, float2 n, const BData& bd, float2 local_pt) {
    const int4 si = __ldg(&S.s_info[shape]);
    int po = 0, pc = 0, co = 0, pflags = 0;
    if (si.x == K_PATH && si.z >= 0) {
        int4 pi2 = __ldg(&S.p_info[2 * si.z + 1]);
        po = pi2.x;
        pc = pi2.y;
        co = pi2.z;
        pflags = pi2.w;
    }
    const bool closed = pflags & PF_CLOSED;
    int nc = 0;  // num_control_points.get(base_point_id).unwrap_or(0)
    if (si.x == K_PATH && (!STYLED || bd.base_point_id >= 0)) {
        int ctrl_count = __ldg(&S.path_cdf_info[shape].y);
        nc = bd.base_point_id < ctrl_count ? S.ncp[co + bd.base_point_id] : 0;
    }
    if (STYLED && bd.base_point_id < 0) {  // a join / cap edge sample: the exact normal velocity
        accumulate_join_cap(S.p_info, S.p_miter, S.seg_p, S.seg_r, S.seg_meta, G.d_points,
                            (pflags & PF_THICK) ? G.d_thickness : nullptr, G.d_shape_stroke_width + shape, si.z, po,
                            -1 - bd.base_point_id, bd.point_id, bd.t, n.x, n.y, contrib);
    } else if (bd.is_stroke) {
        if (si.x == K_PATH && (pflags & PF_THICK)) {
            float t2 = bd.t, tt = 1.0f - t2;
            int pid = bd.point_id;
            auto addt = [&](long i, float v) {
                if (i < pc) add_if(G.d_thickness + po + i, v);
            };
            if (nc == 0) {
                addt(pid, (1.0f - t2) * contrib);
                addt(closed ? (pid + 1) % pc : pid + 1, t2 * contrib);
            } else if (nc == 1) {
                addt(pid, tt * tt * contrib);
                addt(pid + 1, 2.0f * tt * t2 * contrib);
                addt(closed ? (pid + 2) % pc : pid + 2, t2 * t2 * contrib);
            } else if (nc == 2) {
                addt(pid, tt * tt * tt * contrib);
                addt(pid + 1, 3.0f * tt * tt * t2 * contrib);
                addt(pid + 2, 3.0f * tt * t2 * t2 * contrib);
                addt(closed ? (pid + 3) % pc : pid + 3, t2 * t2 * t2 * contrib);
            }
        } else {
            add_if(G.d_shape_stroke_width + shape, contrib);
        }
    }
    float* dp = G.d_shape_params + 4 * shape;
    if (si.x == K_CIRCLE) {
        add_if(dp + 0, n.x * contrib);
        add_if(dp + 1, n.y * contrib);
        add_if(dp + 2, contrib);
    } else if (si.x == K_ELLIPSE) {
        add_if(dp + 0, n.x * contrib);
        add_if(dp + 1, n.y * contrib);
        float ang = 2.0f * PI_F * t;
        add_if(dp + 2, dvg_cosf(ang) * n.x * contrib);
        add_if(dp + 3, dvg_sinf(ang) * n.y * contrib);
    } else if (si.x == K_PATH && (!STYLED || bd.base_point_id >= 0)) {
        float t2 = bd.t, tt = 1.0f - t2;
        int pid = bd.point_id;
        auto addp = [&](long idx, float w) {
            long i = closed ? idx % pc : idx;
            if (i < pc) {
                add_if(G.d_points + 2 * (po + i), n.x * (w * contrib));
                add_if(G.d_points + 2 * (po + i) + 1, n.y * (w * contrib));
            }
        };
        if (nc == 0) {
            addp(pid, 1.0f - t2);
            addp(pid + 1, t2);
        } else if (nc == 1) {
            addp(pid, tt * tt);
            addp(pid + 1, 2.0f * tt * t2);
            addp(pid + 2, t2 * t2);
        } else if (nc == 2) {
            addp(pid, tt * tt * tt);
            addp(pid + 1, 3.0f * tt * tt * t2);
            addp(pid + 2, 3.0f * tt * t2 * t2);
            addp(pid + 3, t2 * t2 * t2);
        }
    } else if (si.x == K_RECT) {
        if (n.x == -1.0f && n.y == 0.0f)
            add_if(dp + 0, -contrib);
        else if (n.x == 1.0f && n.y == 0.0f)
            add_if(dp + 2, contrib);
        else if (n.x == 0.0f && n.y == -1.0f)
            add_if(dp + 1, -contrib);
        else if (n.x == 0.0f && n.y == 1.0f)
            add_if(dp + 3, contrib);
    }
    // transforms (boundary.rs:1132-1147) with d_xform_pt (backward/math.rs:109-128)
    const float* gs = S.g_s2c + 9 * group;
    const float* sx = S.s_xform + 9 * shape;
    float m[9];
    mul33(gs, sx, m);
    const float2 dout = make_float2(n.x * contrib, n.y * contrib);
    const float2 p = local_pt;
    float t0 = m[0] * p.x + m[1] * p.y + m[2];
    float t1 = m[3] * p.x + m[4] * p.y + m[5];
    float t2 = m[6] * p.x + m[7] * p.y + m[8];
    float ox = t0 / t2, oy = t1 / t2;
    float d0 = dout.x / t2, d1 = dout.y / t2, d2 = -(dout.x * ox + dout.y * oy) / t2;
    float dm[9] = {d0 * p.x, d0 * p.y, d0, d1 * p.x, d1 * p.y, d1, d2 * p.x, d2 * p.y, d2};
    // d_group = dm * shape_xform^T ; d_shape = group_s2c^T * dm
#pragma unroll
    for (int r = 0; r < 3; ++r)
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            float dg = dm[3 * r] * sx[3 * c] + dm[3 * r + 1] * sx[3 * c + 1] + dm[3 * r + 2] * sx[3 * c + 2];
            float ds = gs[r] * dm[c] + gs[3 + r] * dm[3 + c] + gs[6 + r] * dm[6 + c];
            add_if(G.d_group_transform + 9 * group + 3 * r + c, dg);
            add_if(G.d_shape_transform + 9 * shape + 3 * r + c, ds);
        }
}

// Boundary pass, stage 1: draw every edge sample (boundary.rs:141-175), keep
// the valid ones with the tile of their boundary pixel as sort key.
__device__ __forceinline__ void boundary_gen_one(const DevScene& S, uint64_t idx, uint64_t slot, uint32_t seed,
                                                 int rng_kind, int tile_off, int seg_off, int scene, int cell,
                                                 float pdf_scale, BSample* out, int2* key, int* tile_counts,
                                                 int* seg_bucket) {
    key[slot] = make_int2(-1, -1);
    float u, t;
    if (rng_kind == 1) {
        uint4 r = philox4x32_10(make_uint4((uint32_t)idx, (uint32_t)(idx >> 32), 0u, 0u), make_uint2(seed, 0u));
        u = unit_from_u32(r.x);
        t = unit_from_u32(r.y);
    } else {
        Pcg32 rng(idx, (uint64_t)seed);
        u = rng.next_f32();
        t = rng.next_f32();
    }
    int sid = lower_bound_cdf(S.bcdf, S.bcdf_n, u);
    if (sid >= S.bcdf_n) sid = S.bcdf_n - 1;
    const int shape = S.b_shape[sid], group = S.b_group[sid];
    const float pmf = S.bpmf[sid];
    if (pmf <= 0.0f) return;
    float2 local_pt, normal;
    float bpdf;
    BData bd;
    if (!sample_boundary_point(S, shape, group, t, S.shape_len[shape], &local_pt, &normal, &bpdf, &bd)) return;
    if (bpdf <= 0.0f) return;
    float s2c[9];
    mul33(S.g_s2c + 9 * group, S.s_xform + 9 * shape, s2c);
    float2 bpt = xf9(s2c, local_pt);
    float sinv[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1};
    if (__ldg(&S.s_info[shape].y) & SF_INVERTIBLE) {
        const float* iv = S.s_inv + 6 * shape;
        for (int k = 0; k < 6; ++k) sinv[k] = iv[k];
    }
    float cinv[9];
    mul33(sinv, S.g_c2s + 9 * group, cinv);
    float2 nc = nrm2(make_float2(cinv[0] * normal.x + cinv[3] * normal.y, cinv[1] * normal.x + cinv[4] * normal.y));
    const float W = (float)S.width, H = (float)S.height;
    bpt.x /= W;
    bpt.y /= H;
    const float pdf = pmf * bpdf * pdf_scale;
    if (pdf <= 0.0f) return;
    const int bx = f2i(bpt.x * W), by = f2i(bpt.y * H);
    if (bx < 0 || bx >= S.width || by < 0 || by >= S.height) return;
    BSample r;
    r.bx = bpt.x;
    r.by = bpt.y;
    r.nx = nc.x;
    r.ny = nc.y;
    r.lx = local_pt.x;
    r.ly = local_pt.y;
    r.pdf = pdf;
    r.t = t;
    r.shape = shape;
    r.group = group;
    r.pixel = by * S.width + bx;
    r.base_point_id = bd.base_point_id;
    r.point_id = bd.point_id;
    r.bt = bd.t;
    r.is_stroke = bd.is_stroke ? 1 : 0;
    r.scene = scene;
    out[slot] = r;
    // sort bucket: the cell of the boundary pixel inside its tile, so that a warp
    // evaluates edge points that lie close together (coherent group walks), then the
    // sample's class, so that it mostly runs one sampling / gradient code path
    const int tile = tile_off + (by / TILE) * S.tiles_x + (bx / TILE);
    const int per_row = TILE / cell;
    const int cls = (bd.is_stroke ? 2 : 0) + (__ldg(&S.s_info[shape]).x == K_PATH ? 1 : 0);
    const int bucket =
        (tile * (per_row * per_row) + ((by % TILE) / cell) * per_row + (bx % TILE) / cell) * BND_CLASSES + cls;
    // second bucket: the path segment, or the shape, whose parameters the sample's gradient goes to
    const int4 si = __ldg(&S.s_info[shape]);
    const int2 ps = si.x == K_PATH && si.z >= 0 ? make_int2(__ldg(&S.p_info[2 * si.z].x), __ldg(&S.p_info[2 * si.z].y))
                                                : make_int2(0, 0);
    const int seg = bd.base_point_id >= 0 && bd.base_point_id < ps.y ? ps.x + bd.base_point_id : S.num_segs + shape;
    key[slot] = make_int2(bucket, seg_off + seg);
    atomicAdd(tile_counts + bucket, 1);
    *seg_bucket = seg_off + seg;
}
// Counts of the segment buckets that a CTA's samples fall in, in shared memory while they span
// at most SEG_SPAN buckets (a scene of few shapes has all its samples in a few dozen, and L2
// serialises their atomics: edge pass of a 128x128 scene of 8 outlines 0.40 -> 0.33 ms).
constexpr int SEG_SPAN = 4096;
constexpr int GEN_ITEMS = 4;  // samples per thread
struct SegSpan {
    int lo, hi;
};
__device__ __forceinline__ SegSpan seg_span(const int* bucket, int2* range) {
    if (threadIdx.x == 0) *range = make_int2(0x7fffffff, -1);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GEN_ITEMS; ++k)
        if (bucket[k] >= 0) {
            atomicMin(&range->x, bucket[k]);
            atomicMax(&range->y, bucket[k]);
        }
    __syncthreads();
    return SegSpan{range->x, range->y};
}
// Adds the CTA's buckets (-1: none) to the counts.
__device__ __forceinline__ void seg_count(const int* bucket, int* seg_counts, int* hist, int2* range) {
    const SegSpan sp = seg_span(bucket, range);
    const int n = sp.hi - sp.lo + 1;
    if (sp.hi < 0) return;
    if (n > SEG_SPAN) {
#pragma unroll
        for (int k = 0; k < GEN_ITEMS; ++k)
            if (bucket[k] >= 0) atomicAdd(seg_counts + bucket[k], 1);
        return;
    }
    for (int i = threadIdx.x; i < n; i += blockDim.x) hist[i] = 0;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GEN_ITEMS; ++k)
        if (bucket[k] >= 0) atomicAdd(hist + (bucket[k] - sp.lo), 1);
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += blockDim.x)
        if (hist[i]) atomicAdd(seg_counts + sp.lo + i, hist[i]);
}
__global__ void __launch_bounds__(256) k_boundary_gen(const __grid_constant__ DevScene S, BoundaryParams bp, BSample* out,
                                                      int2* key, int* tile_counts, int* seg_counts) {
    __shared__ int hist[SEG_SPAN];
    __shared__ int2 range;
    int bucket[GEN_ITEMS];
#pragma unroll 1
    for (int k = 0; k < GEN_ITEMS; ++k) {
        const uint64_t idx = ((uint64_t)blockIdx.x * GEN_ITEMS + k) * blockDim.x + threadIdx.x + bp.sample_base;
        int b = -1;
        if (idx < bp.num_samples)
            boundary_gen_one(S, idx, idx - bp.slot_base, bp.seed, bp.rng, 0, 0, 0, bp.cell, bp.pdf_scale, out, key,
                             tile_counts, &b);
#pragma unroll
        for (int j = 0; j < GEN_ITEMS; ++j)
            if (j == k) bucket[j] = b;
    }
    seg_count(bucket, seg_counts, hist, &range);
}
// Batched stage 1: one flat index over all scenes' boundary samples; the scene is
// found by binary search over the per-scene sample offsets.
__global__ void __launch_bounds__(256) k_boundary_gen_batch(const BatchEntry* __restrict__ B, int nscenes,
                                                            uint64_t total, int cell, BSample* out, int2* key,
                                                            int* tile_counts, int* seg_counts) {
    __shared__ int hist[SEG_SPAN];
    __shared__ int2 range;
    int bucket[GEN_ITEMS];
#pragma unroll 1
    for (int k = 0; k < GEN_ITEMS; ++k) {
        const uint64_t g = ((uint64_t)blockIdx.x * GEN_ITEMS + k) * blockDim.x + threadIdx.x;
        int b = -1;
        if (g < total) {
            int lo = 0, hi = nscenes - 1;
            while (lo < hi) {
                int mid = (lo + hi + 1) >> 1;
                if (B[mid].b_off <= g)
                    lo = mid;
                else
                    hi = mid - 1;
            }
            const BatchEntry& E = B[lo];
            key[g] = make_int2(-1, -1);
            if (E.S.boundary_ok && g - E.b_off < E.nb)
                boundary_gen_one(E.S, g - E.b_off, g, E.bseed, E.rng, E.tile_off, E.seg_off, lo, cell, E.bscale, out,
                                 key, tile_counts, &b);
        }
#pragma unroll
        for (int j = 0; j < GEN_ITEMS; ++j)
            if (j == k) bucket[j] = b;
    }
    seg_count(bucket, seg_counts, hist, &range);
}
// Stage 2: counting-sort scatter of sample slots, by cell and by segment (the latter through a
// CTA's own counts, as in stage 1: one cursor atomic per bucket and CTA).
__global__ void __launch_bounds__(256) k_boundary_scatter(const int2* key, uint64_t n, int* cursor, int* order,
                                                          int* seg_cursor, int* seg_order) {
    __shared__ int hist[SEG_SPAN];
    __shared__ int2 range;
    int bucket[GEN_ITEMS];
    const uint64_t first = (uint64_t)blockIdx.x * GEN_ITEMS * blockDim.x + threadIdx.x;
#pragma unroll
    for (int k = 0; k < GEN_ITEMS; ++k) {
        const uint64_t i = first + (uint64_t)k * blockDim.x;
        const int2 q = i < n ? key[i] : make_int2(-1, -1);
        bucket[k] = q.y;
        if (q.x >= 0) order[atomicAdd(cursor + q.x, 1)] = (int)i;
    }
    const SegSpan sp = seg_span(bucket, &range);
    const int w = sp.hi - sp.lo + 1;
    if (sp.hi < 0) return;
    if (w > SEG_SPAN) {
#pragma unroll
        for (int k = 0; k < GEN_ITEMS; ++k)
            if (bucket[k] >= 0) seg_order[atomicAdd(seg_cursor + bucket[k], 1)] = (int)(first + (uint64_t)k * blockDim.x);
        return;
    }
    for (int i = threadIdx.x; i < w; i += blockDim.x) hist[i] = 0;
    __syncthreads();
    int rank[GEN_ITEMS];
#pragma unroll
    for (int k = 0; k < GEN_ITEMS; ++k)
        rank[k] = bucket[k] >= 0 ? atomicAdd(hist + (bucket[k] - sp.lo), 1) : 0;
    __syncthreads();
    for (int i = threadIdx.x; i < w; i += blockDim.x)
        if (hist[i]) hist[i] = atomicAdd(seg_cursor + sp.lo + i, hist[i]);
    __syncthreads();
#pragma unroll
    for (int k = 0; k < GEN_ITEMS; ++k)
        if (bucket[k] >= 0) seg_order[hist[bucket[k] - sp.lo] + rank[k]] = (int)(first + (uint64_t)k * blockDim.x);
}
// Stage 3: evaluate both sides of every edge sample in tile order, so that the
// lanes of a warp share one group list (render_edge_sample, boundary.rs:845-967).
// Two lanes per sample: the even lane of a pair takes the colour inside, the odd lane
// the colour outside.  The two points are 2e-4 of the canvas apart, so a pair walks
// the same BVH nodes and segment tests in lockstep; the even lane receives the odd
// lane's colour and hit by shuffle and finishes the sample alone.  Every lane of the
// warp reaches the shuffles (`valid` false: a pair past the last sample).  The sample's
// contribution goes back into its record (pdf), with the normal turned outwards: stage 4
// adds it to the gradients.
__device__ __forceinline__ void boundary_eval_pair(const DevScene& S, const BSample& r, bool valid,
                                                   const float* d_render, const float* wsum, float* d_translation,
                                                   BSample* out) {
    const float W = (float)S.width, H = (float)S.height;
    const int side = threadIdx.x & 1;
    float4 cs = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool hs = false;
    float4 bg = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    int tile = 0, cell = 0;
    float2 q = make_float2(0.0f, 0.0f);
    if (valid) {
        bg = background_premul(S, r.pixel);
        const int bx = r.pixel % S.width, by = r.pixel / S.width;
        tile = (by / TILE) * S.tiles_x + bx / TILE;
        cell = (by % TILE) / CELL * (TILE / CELL) + (bx % TILE) / CELL;
        const float o = side == 0 ? -1.0e-4f : 1.0e-4f;
        q = make_float2(r.bx + r.nx * o, r.by + r.ny * o);
    }
    cs = edge_color(S, valid, tile, cell, make_float2(q.x * W, q.y * H), bg, r.group, r.shape, &hs);
    float4 co;
    co.x = __shfl_xor_sync(0xffffffffu, cs.x, 1);
    co.y = __shfl_xor_sync(0xffffffffu, cs.y, 1);
    co.z = __shfl_xor_sync(0xffffffffu, cs.z, 1);
    co.w = __shfl_xor_sync(0xffffffffu, cs.w, 1);
    const bool ho = __shfl_xor_sync(0xffffffffu, (int)hs, 1) != 0;
    if (!valid || side != 0) return;
    float2 nc = make_float2(r.nx, r.ny);
    float4 ci = cs;
    const bool hi = hs;
    if (!hi && !ho) {
        out->pdf = 0.0f;
        return;
    }
    if (!hi) {
        nc = make_float2(nc.x * -1.0f, nc.y * -1.0f);
        out->nx = nc.x;
        out->ny = nc.y;
        float4 tmp = ci;
        ci = co;
        co = tmp;
    }
    // gather_d_color at the boundary pixel, divided by W*H (boundary.rs:913-929)
    const float2 sb = make_float2(r.bx * W, r.by * H);
    float4 dc = make_float4(0, 0, 0, 0);
    {
        const int px = f2i(floorf(sb.x)), py = f2i(floorf(sb.y)), ri = S.filter_ri;
#pragma unroll 1
        for (int dy = -ri; dy <= ri; ++dy)
#pragma unroll 1
            for (int dx = -ri; dx <= ri; ++dx) {
                int xx = px + dx, yy = py + dy;
                if (xx < 0 || yy < 0 || xx >= S.width || yy >= S.height) continue;
                float w = filter_weight(S.filter_type, S.filter_radius, (float)xx + 0.5f - sb.x,
                                        (float)yy + 0.5f - sb.y);
                size_t q = (size_t)yy * S.width + xx;
                float ws = wsum[q];
                if (ws > 0.0f) {
                    float4 d = reinterpret_cast<const float4*>(d_render)[q];
                    float k = w / ws;
                    dc.x += k * d.x;
                    dc.y += k * d.y;
                    dc.z += k * d.z;
                    dc.w += k * d.w;
                }
            }
    }
    const float norm = W * H;
    if (norm > 0.0f) {
        dc.x /= norm;
        dc.y /= norm;
        dc.z /= norm;
        dc.w /= norm;
    }
    const float contrib =
        ((ci.x - co.x) * dc.x + (ci.y - co.y) * dc.y + (ci.z - co.z) * dc.z + (ci.w - co.w) * dc.w) / r.pdf;
    out->pdf = isfinite(contrib) ? contrib : 0.0f;
    if (d_translation && isfinite(contrib)) {
        add_if(d_translation + 2 * (size_t)r.pixel, nc.x * contrib);
        add_if(d_translation + 2 * (size_t)r.pixel + 1, nc.y * contrib);
    }
}
// Two threads per sample (boundary_eval_pair): launch 2 * samples threads.
__global__ void __launch_bounds__(DVG_BND_THREADS, DVG_MINB_BND) k_boundary_eval(const __grid_constant__ DevScene S,
                                                                     BSample* samples, const int* order,
                                                                     const int* offsets, int tiles,
                                                                     const float* d_render, const float* wsum,
                                                                     float* d_translation) {
    const int64_t i = (int64_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 1);
    const bool valid = i < offsets[tiles];
    BSample r{};
    const int at = valid ? order[i] : 0;
    if (valid) r = samples[at];
    boundary_eval_pair(S, r, valid, d_render, wsum, d_translation, samples + at);
}
__global__ void __launch_bounds__(DVG_BND_THREADS, DVG_MINB_BND) k_boundary_eval_batch(const BatchEntry* __restrict__ B,
                                                                           BSample* samples, const int* order,
                                                                           const int* offsets, int tiles) {
    const int64_t i = (int64_t)(((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 1);
    const bool valid = i < offsets[tiles];
    BSample r{};
    const int at = valid ? order[i] : 0;
    if (valid) r = samples[at];
    const BatchEntry& E = B[valid ? r.scene : 0];
    boundary_eval_pair(E.S, r, valid, E.d_render, E.wsum, E.G.d_translation, samples + at);
}

// Stage 4: the samples' gradients (accumulate_boundary), in segment order.  A warp takes
// ACC_SAMPLES consecutive samples, 32 at a time.  While they share a segment, group and side,
// every lane keeps its own sums of the terms below; the sums are transposed over the warp (31
// shuffles, lane i receives term i) and added with one atomic per parameter, instead of some
// thirty per sample on the same few addresses.  The group's and the shape's transform gradient
// are both linear in the nine entries of dm, so dm is what is summed.
constexpr int ACC_SAMPLES = 128;
enum : int { ACC_DM = 0, ACC_PTS = 9, ACC_RAD = 17, ACC_PRM = 21, ACC_TERMS = 32 };
struct AccKey {
    int shape, group, base_point_id, point_id, is_stroke, scene;
    __device__ __forceinline__ bool operator==(const AccKey& o) const {
        return shape == o.shape && group == o.group && base_point_id == o.base_point_id &&
               point_id == o.point_id && is_stroke == o.is_stroke && scene == o.scene;
    }
};
// The terms of one sample (the formulas of accumulate_boundary).
__device__ __forceinline__ void boundary_terms(const DevScene& S, const BSample& r, float* v) {
    const float contrib = r.pdf;
    const float2 n = make_float2(r.nx, r.ny);
    const int4 si = __ldg(&S.s_info[r.shape]);
    int co = 0, pflags = 0, nc = 0;
    const bool path = si.x == K_PATH;
    if (path && si.z >= 0) {
        const int4 pi2 = __ldg(&S.p_info[2 * si.z + 1]);
        co = pi2.z;
        pflags = pi2.w;
    }
    if (path) nc = r.base_point_id < __ldg(&S.path_cdf_info[r.shape].y) ? S.ncp[co + r.base_point_id] : 0;
    const float t2 = r.bt, tt = 1.0f - t2;
    float w[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (path) {
        if (nc == 0) {
            w[0] = 1.0f - t2;
            w[1] = t2;
        } else if (nc == 1) {
            w[0] = tt * tt;
            w[1] = 2.0f * tt * t2;
            w[2] = t2 * t2;
        } else if (nc == 2) {
            w[0] = tt * tt * tt;
            w[1] = 3.0f * tt * tt * t2;
            w[2] = 3.0f * tt * t2 * t2;
            w[3] = t2 * t2 * t2;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            v[ACC_PTS + 2 * j] += n.x * (w[j] * contrib);
            v[ACC_PTS + 2 * j + 1] += n.y * (w[j] * contrib);
        }
    }
    if (r.is_stroke) {
        if (path && (pflags & PF_THICK)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[ACC_RAD + j] += w[j] * contrib;
        } else {
            v[ACC_RAD] += contrib;
        }
    }
    if (si.x == K_CIRCLE) {
        v[ACC_PRM] += n.x * contrib;
        v[ACC_PRM + 1] += n.y * contrib;
        v[ACC_PRM + 2] += contrib;
    } else if (si.x == K_ELLIPSE) {
        const float ang = 2.0f * PI_F * r.t;
        v[ACC_PRM] += n.x * contrib;
        v[ACC_PRM + 1] += n.y * contrib;
        v[ACC_PRM + 2] += dvg_cosf(ang) * n.x * contrib;
        v[ACC_PRM + 3] += dvg_sinf(ang) * n.y * contrib;
    } else if (si.x == K_RECT) {
        if (n.x == -1.0f && n.y == 0.0f) v[ACC_PRM] -= contrib;
        else if (n.x == 1.0f && n.y == 0.0f) v[ACC_PRM + 2] += contrib;
        else if (n.x == 0.0f && n.y == -1.0f) v[ACC_PRM + 1] -= contrib;
        else if (n.x == 0.0f && n.y == 1.0f) v[ACC_PRM + 3] += contrib;
    }
    float m[9];
    mul33(S.g_s2c + 9 * r.group, S.s_xform + 9 * r.shape, m);
    const float2 dout = make_float2(n.x * contrib, n.y * contrib);
    const float px = r.lx, py = r.ly;
    const float t0 = m[0] * px + m[1] * py + m[2], t1 = m[3] * px + m[4] * py + m[5], tw = m[6] * px + m[7] * py + m[8];
    const float d0 = dout.x / tw, d1 = dout.y / tw, d2 = -(dout.x * (t0 / tw) + dout.y * (t1 / tw)) / tw;
    const float dm[9] = {d0 * px, d0 * py, d0, d1 * px, d1 * py, d1, d2 * px, d2 * py, d2};
#pragma unroll
    for (int k = 0; k < 9; ++k) v[ACC_DM + k] += dm[k];
}
// Adds the warp's sums of one key to the gradients and clears them.
__device__ __forceinline__ void boundary_flush(const DevScene& S, const GradPtrs& G, const AccKey& k, float* v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int s = 16; s > 0; s >>= 1)
#pragma unroll
        for (int i = 0; i < s; ++i) {
            const float keep = lane & s ? v[i + s] : v[i], send = lane & s ? v[i] : v[i + s];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, s);
        }
    const float sum = v[0];
    float dm[9];
#pragma unroll
    for (int i = 0; i < 9; ++i) dm[i] = __shfl_sync(0xffffffffu, sum, ACC_DM + i);
#pragma unroll
    for (int i = 0; i < ACC_TERMS; ++i) v[i] = 0.0f;
    const int4 si = __ldg(&S.s_info[k.shape]);
    int po = 0, pc = 0, pflags = 0, pid = 0, np = 0;
    const bool path = si.x == K_PATH;
    if (path && si.z >= 0) {
        const int4 pi2 = __ldg(&S.p_info[2 * si.z + 1]);
        po = pi2.x;
        pc = pi2.y;
        pflags = pi2.w;
        np = 2 + (k.base_point_id < __ldg(&S.path_cdf_info[k.shape].y) ? S.ncp[pi2.z + k.base_point_id] : 0);
        pid = k.point_id;
    }
    // lanes 0-17: the two transforms
    if (lane < 18) {
        const int o = lane < 9 ? lane : lane - 9, r = o / 3, c = o % 3;
        const float* gs = S.g_s2c + 9 * k.group;
        const float* sx = S.s_xform + 9 * k.shape;
        float a = 0.0f;
        if (lane < 9)
            a = (r == 0 ? dm[0] : r == 1 ? dm[3] : dm[6]) * sx[3 * c] + (r == 0 ? dm[1] : r == 1 ? dm[4] : dm[7]) * sx[3 * c + 1] +
                (r == 0 ? dm[2] : r == 1 ? dm[5] : dm[8]) * sx[3 * c + 2];
        else
            a = gs[r] * (c == 0 ? dm[0] : c == 1 ? dm[1] : dm[2]) + gs[3 + r] * (c == 0 ? dm[3] : c == 1 ? dm[4] : dm[5]) +
                gs[6 + r] * (c == 0 ? dm[6] : c == 1 ? dm[7] : dm[8]);
        add_if(lane < 9 ? G.d_group_transform + 9 * k.group + o : G.d_shape_transform + 9 * k.shape + o, a);
    }
    // lanes 9-24: points, radius or thickness, shape parameters
    if (lane >= ACC_PTS && lane < ACC_RAD) {
        const int j = (lane - ACC_PTS) >> 1;
        if (path && j < np && pc > 0) {
            const bool closed = pflags & PF_CLOSED;
            const int i = closed ? (pid + j) % pc : pid + j;
            if (i < pc) add_if(G.d_points + 2 * (po + i) + ((lane - ACC_PTS) & 1), sum);
        }
    } else if (lane >= ACC_RAD && lane < ACC_PRM) {
        const int j = lane - ACC_RAD;
        if (path && (pflags & PF_THICK)) {
            // the last point of a closed path's segment wraps around, as the points do
            const int i = (pflags & PF_CLOSED) && j == np - 1 ? (pid + j) % pc : pid + j;
            if (j < np && i < pc) add_if(G.d_thickness + po + i, sum);
        } else if (j == 0) {
            add_if(G.d_shape_stroke_width + k.shape, sum);
        }
    } else if (lane >= ACC_PRM && lane < ACC_PRM + 4) {
        add_if(G.d_shape_params + 4 * k.shape + (lane - ACC_PRM), sum);
    }
}
template <bool STYLED, typename SceneOf, typename GradsOf>
__device__ __forceinline__ void boundary_accum(const BSample* samples, const int* order, int64_t n, SceneOf&& scene,
                                               GradsOf&& grads) {
    const int lane = threadIdx.x & 31;
    const int64_t base = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * ACC_SAMPLES;
    float v[ACC_TERMS];
#pragma unroll
    for (int i = 0; i < ACC_TERMS; ++i) v[i] = 0.0f;
    AccKey run{-1, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (int64_t i0 = base; i0 < base + ACC_SAMPLES && i0 < n; i0 += 32) {
        const bool in = i0 + lane < n;
        BSample r{};
        if (in) r = samples[order[i0 + lane]];
        const bool has = in && r.pdf != 0.0f;
        const AccKey mine{r.shape, r.group, r.base_point_id, r.point_id, r.is_stroke, r.scene};
        const unsigned m = __ballot_sync(0xffffffffu, has);
        if (!m) continue;
        const int l = __ffs(m) - 1;
        const AccKey key{__shfl_sync(0xffffffffu, mine.shape, l), __shfl_sync(0xffffffffu, mine.group, l),
                         __shfl_sync(0xffffffffu, mine.base_point_id, l), __shfl_sync(0xffffffffu, mine.point_id, l),
                         __shfl_sync(0xffffffffu, mine.is_stroke, l), __shfl_sync(0xffffffffu, mine.scene, l)};
        const bool join = STYLED && key.base_point_id < 0;
        if (__all_sync(0xffffffffu, !has || mine == key) && !join) {
            if (run.shape >= 0 && !(run == key)) boundary_flush(scene(run.scene), grads(run.scene), run, v);
            run = key;
            if (has) boundary_terms(scene(r.scene), r, v);
        } else if (has) {  // the warp spans segments: each lane adds its own
            BData bd;
            bd.base_point_id = r.base_point_id;
            bd.point_id = r.point_id;
            bd.t = r.bt;
            bd.is_stroke = r.is_stroke != 0;
            accumulate_boundary<STYLED>(scene(r.scene), grads(r.scene), r.shape, r.group, r.pdf, r.t,
                                        make_float2(r.nx, r.ny), bd, make_float2(r.lx, r.ly));
        }
    }
    if (run.shape >= 0) boundary_flush(scene(run.scene), grads(run.scene), run, v);
}
template <bool STYLED>
__global__ void __launch_bounds__(256) k_boundary_accum(const __grid_constant__ DevScene S, const BSample* samples,
                                                        const int* order, const int* total,
                                                        const __grid_constant__ GradPtrs G) {
    boundary_accum<STYLED>(samples, order, *total, [&](int) -> const DevScene& { return S; },
                           [&](int) -> const GradPtrs& { return G; });
}
template <bool STYLED>
__global__ void __launch_bounds__(256) k_boundary_accum_batch(const BatchEntry* __restrict__ B, const BSample* samples,
                                                              const int* order, const int* total) {
    boundary_accum<STYLED>(samples, order, *total, [&](int k) -> const DevScene& { return B[k].S; },
                           [&](int k) -> const GradPtrs& { return B[k].G; });
}

// ------------------------------------------------------------------ background finalisation (background.rs:29-61)
__global__ void k_finalize_background(DevScene S, GradPtrs G) {
    size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (S.bg_image) {
        if (!G.d_background_image || p >= (size_t)S.width * S.height) return;
        const float* im = S.bg_image + 4 * p;
        float* c = G.d_background_image + 4 * p;
        float dr = c[0] * im[3], dg = c[1] * im[3], db = c[2] * im[3];
        float da = c[0] * im[0] + c[1] * im[1] + c[2] * im[2] + c[3];
        c[0] = dr;
        c[1] = dg;
        c[2] = db;
        c[3] = da;
        return;
    }
    if (p != 0) return;
    float* d = G.d_background;
    float r = S.bg[0], g = S.bg[1], b = S.bg[2], a = S.bg[3];
    float nr = d[0] * a, ng = d[1] * a, nb = d[2] * a;
    float na = d[0] * r + d[1] * g + d[2] * b + d[3];
    d[0] = nr;
    d[1] = ng;
    d[2] = nb;
    d[3] = na;
}

// Image::solid / background image copy for scenes without groups (renderer.rs:57-66).
__global__ void k_fill_background(DevScene S, float* out) {
    size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (size_t)S.width * S.height) return;
    float4 v = S.bg_image ? reinterpret_cast<const float4*>(S.bg_image)[p]
                          : make_float4(S.bg[0], S.bg[1], S.bg[2], S.bg[3]);
    reinterpret_cast<float4*>(out)[p] = v;
}

// ------------------------------------------------------------------ L2 loss
__global__ void k_l2(const float* img, const float* target, size_t n, float* d_render, float* loss) {
    __shared__ float red[8];
    float s = 0.0f;
#pragma unroll 1
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float d = img[i] - target[i];
        d_render[i] = 2.0f * d;
        s += d * d;
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0 && loss) {
        float t = 0.0f;
#pragma unroll 1
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        atomicAdd(loss, t);
    }
}

// ------------------------------------------------------------------ batched per-pixel kernels (grid.y = scene)
__global__ void k_resolve_batch(const BatchEntry* __restrict__ B) {
    const BatchEntry& E = B[blockIdx.y];
    size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= (size_t)E.S.width * E.S.height) return;
    float r = E.S.bg[0], g = E.S.bg[1], b = E.S.bg[2], a = E.S.bg[3];
    float w = E.wsum[p];
    if (w > 0.0f) {
        float4 c = reinterpret_cast<const float4*>(E.accum)[p];
        r = c.x / w;
        g = c.y / w;
        b = c.z / w;
        a = c.w / w;
    }
    if (a > 1.0e-8f) {
        r = r / a;
        g = g / a;
        b = b / a;
    }
    reinterpret_cast<float4*>(E.image)[p] = make_float4(r, g, b, a);
}
__global__ void k_l2_batch(const BatchEntry* __restrict__ B) {
    __shared__ float red[8];
    const BatchEntry& E = B[blockIdx.y];
    const size_t n = (size_t)E.S.width * E.S.height * 4;
    float s = 0.0f;
#pragma unroll 1
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        float d = E.image[i] - E.target[i];
        E.d_render[i] = 2.0f * d;
        s += d * d;
    }
    s = warp_sum(s);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.0f;
#pragma unroll 1
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        atomicAdd(E.loss, t);
    }
}
__global__ void k_finalize_background_batch(const BatchEntry* __restrict__ B) {
    const BatchEntry& E = B[blockIdx.y];
    size_t p = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (E.S.bg_image) {
        if (!E.G.d_background_image || p >= (size_t)E.S.width * E.S.height) return;
        const float* im = E.S.bg_image + 4 * p;
        float* c = E.G.d_background_image + 4 * p;
        float dr = c[0] * im[3], dg = c[1] * im[3], db = c[2] * im[3];
        float da = c[0] * im[0] + c[1] * im[1] + c[2] * im[2] + c[3];
        c[0] = dr;
        c[1] = dg;
        c[2] = db;
        c[3] = da;
        return;
    }
    if (p != 0) return;
    float* d = E.G.d_background;
    float r = E.S.bg[0], g = E.S.bg[1], b = E.S.bg[2], a = E.S.bg[3];
    float nr = d[0] * a, ng = d[1] * a, nb = d[2] * a;
    float na = d[0] * r + d[1] * g + d[2] * b + d[3];
    d[0] = nr;
    d[1] = ng;
    d[2] = nb;
    d[3] = na;
}

}  // namespace dvgb

// ------------------------------------------------------------------ launchers
namespace dvgb {

int launch_binning(const DevScene& S, const float4* g_bbox, int* counts, int* offsets, int* entries,
                   cudaStream_t stream) {
    const int tiles = S.tiles_x * S.tiles_y;
    if (!entries) {
        k_bin_count<<<tiles, 256, 0, stream>>>(S, g_bbox, counts);
        k_bin_scan<<<1, 1024, 0, stream>>>(counts, tiles, offsets);
        return 2;
    }
    k_bin_write<<<tiles, 256, 0, stream>>>(S, g_bbox, offsets, entries);
    return 1;
}
// Lane groups of the forward's splat: 4 or 16 samples of a pixel next to each other in a warp.
static int splat_lanes(const SampleParams& sp) {
    const int spp = sp.sxn * sp.syn;
    return sp.layout && (spp == 4 || spp == 16) ? spp : 0;
}
int launch_forward(const DevScene& S, const SampleParams& sp, float* accum, float* wsum, cudaStream_t stream) {
    SplatPlan splat;
    splat.add(S.filter_ri);
    const size_t smem = splat.bytes();
    dim3 grid(launch_tiles(S, sp), sp.sxn * sp.syn);
    const int g = splat.all ? splat_lanes(sp) : 0;
    if (g == 16)
        k_forward<16><<<grid, 256, smem, stream>>>(S, sp, accum, wsum);
    else if (g == 4)
        k_forward<4><<<grid, 256, smem, stream>>>(S, sp, accum, wsum);
    else
        k_forward<0><<<grid, 256, smem, stream>>>(S, sp, accum, wsum);
    return 1;
}
int launch_weights(const DevScene& S, const SampleParams& sp, float* wsum, cudaStream_t stream) {
    dim3 grid(launch_tiles(S, sp), sp.sxn * sp.syn);
    k_weights<<<grid, 256, 0, stream>>>(S, sp, wsum);
    return 1;
}
int launch_resolve(const DevScene& S, const float* accum, const float* wsum, float* out, cudaStream_t stream) {
    size_t n = (size_t)S.width * S.height;
    k_resolve<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(S, accum, wsum, out);
    return 1;
}
int launch_interior(const DevScene& S, const SampleParams& sp, const float* d_render, const float* wsum,
                    const GradPtrs& G, unsigned* status, cudaStream_t stream) {
    dim3 grid(launch_tiles(S, sp), sp.sxn * sp.syn);
    if (sp.frag) k_interior_cached<<<grid, 256, 0, stream>>>(S, sp, d_render, wsum, G, status);
    k_interior<<<grid, 256, 0, stream>>>(S, sp, d_render, wsum, G, status);
    return sp.frag ? 2 : 1;
}
static unsigned gen_grid(uint64_t n) { return (unsigned)((n + 256 * GEN_ITEMS - 1) / (256 * GEN_ITEMS)); }
// Stages 2 to 4 for the n drawn samples in sc (counts filled by stage 1).
template <typename Eval, typename Accum>
static int boundary_stages(const BoundaryScratch& sc, uint64_t n, int tiles, int segs, cudaStream_t stream, Eval eval,
                           Accum accum) {
    int* offsets = sc.counts + tiles;  // tiles + 1 entries
    int* seg_counts = sc.seg_counts;
    int* seg_offsets = seg_counts + segs;
    int launches = launch_scan(sc.counts, tiles, offsets, sc.counts + 2 * (size_t)tiles + 1, stream);
    launches += launch_scan(seg_counts, segs, seg_offsets, seg_counts + 2 * (size_t)segs + 1, stream);
    // reuse the count arrays as the scatter cursors (copies of the exclusive offsets)
    cudaMemcpyAsync(sc.counts, offsets, sizeof(int) * (size_t)tiles, cudaMemcpyDeviceToDevice, stream);
    cudaMemcpyAsync(seg_counts, seg_offsets, sizeof(int) * (size_t)segs, cudaMemcpyDeviceToDevice, stream);
    k_boundary_scatter<<<gen_grid(n), 256, 0, stream>>>(sc.key, n, sc.counts, sc.order, seg_counts,
                                                                       sc.seg_order);
    eval(offsets, (unsigned)((2 * n + DVG_BND_THREADS - 1) / DVG_BND_THREADS));
    accum(seg_offsets + segs, (unsigned)((n + 8 * ACC_SAMPLES - 1) / (8 * ACC_SAMPLES)));
    return launches + 3;
}
int launch_boundary(const DevScene& S, const BoundaryParams& bp, const float* d_render, const float* wsum,
                    const GradPtrs& G, const BoundaryScratch& sc, uint64_t capacity, cudaStream_t stream) {
    const uint64_t n = bp.num_samples;  // samples [bp.sample_base, n)
    const int tiles = S.tiles_x * S.tiles_y * bnd_buckets(bp.cell);  // sort buckets
    const int segs = S.num_segs + S.num_shapes;
    int launches = 0;
#pragma unroll 1
    for (uint64_t base = bp.sample_base; base < n; base += capacity) {
        const uint64_t cnt = base + capacity < n ? capacity : n - base;
        BoundaryParams b = bp;
        b.sample_base = base;
        b.slot_base = base;
        b.num_samples = base + cnt;
        cudaMemsetAsync(sc.counts, 0, sizeof(int) * (2 * (size_t)tiles + 1), stream);
        cudaMemsetAsync(sc.seg_counts, 0, sizeof(int) * (2 * (size_t)segs + 1), stream);
        k_boundary_gen<<<gen_grid(cnt), 256, 0, stream>>>(S, b, sc.samples, sc.key, sc.counts,
                                                                         sc.seg_counts);
        launches += 1 + boundary_stages(
            sc, cnt, tiles, segs, stream,
            [&](const int* offsets, unsigned grid) {
                k_boundary_eval<<<grid, DVG_BND_THREADS, 0, stream>>>(S, sc.samples, sc.order, offsets, tiles, d_render, wsum,
                                                          G.d_translation);
            },
            [&](const int* total, unsigned grid) {
                if (S.styled)
                    k_boundary_accum<true><<<grid, 256, 0, stream>>>(S, sc.samples, sc.seg_order, total, G);
                else
                    k_boundary_accum<false><<<grid, 256, 0, stream>>>(S, sc.samples, sc.seg_order, total, G);
            });
    }
    return launches;
}
int launch_finalize_background(const DevScene& S, const GradPtrs& G, cudaStream_t stream) {
    size_t n = S.bg_image ? (size_t)S.width * S.height : 1;
    k_finalize_background<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(S, G);
    return 1;
}
// Batched step launchers (one launch per stage for all scenes).
// CTAs of a persistent launch: as many as the GPU holds at once (and no more than items).
template <typename K>
int persistent_grid(K kernel, size_t smem, int items) {
    int dev = 0, sms = 0, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, smem);
    return std::max(1, std::min(items, std::max(per_sm, 1) * std::max(sms, 1)));
}
int launch_forward_batch(const BatchEntry* B, const SampleParams& sp, const int2* work, int items, int* counter,
                         const SplatPlan& splat, cudaStream_t stream) {
    const size_t smem = splat.bytes();
    auto go = [&](auto kernel) {
        kernel<<<counter ? persistent_grid(kernel, smem, items) : items, 256, smem, stream>>>(B, work, items, counter);
    };
    const int g = splat.all ? splat_lanes(sp) : 0;  // (one set of options, and of a batch one layout, for all its scenes)
    if (g == 16)
        go(k_forward_batch<16>);
    else if (g == 4)
        go(k_forward_batch<4>);
    else
        go(k_forward_batch<0>);
    return 1;
}
int launch_pixels_batch(const BatchEntry* B, int nscenes, size_t max_pixels, int which, cudaStream_t stream) {
    if (which == 0) {
        dim3 grid((unsigned)((max_pixels + 255) / 256), nscenes);
        k_resolve_batch<<<grid, 256, 0, stream>>>(B);
    } else if (which == 1) {
        unsigned bx = (unsigned)((max_pixels * 4 + 255) / 256);
        if (bx > 512) bx = 512;
        dim3 grid(bx, nscenes);
        k_l2_batch<<<grid, 256, 0, stream>>>(B);
    } else {
        dim3 grid((unsigned)((max_pixels + 255) / 256), nscenes);
        k_finalize_background_batch<<<grid, 256, 0, stream>>>(B);
    }
    return 1;
}
int launch_interior_batch(const BatchEntry* B, const int2* work, int items, int* counters, unsigned* status,
                          cudaStream_t stream) {
    int* c0 = counters ? counters : nullptr;
    int* c1 = counters ? counters + 1 : nullptr;
    k_interior_cached_batch<<<c0 ? persistent_grid(k_interior_cached_batch, 0, items) : items, 256, 0, stream>>>(
        B, work, items, c0, status);
    k_interior_batch<<<c1 ? persistent_grid(k_interior_batch, 0, items) : items, 256, 0, stream>>>(B, work, items, c1,
                                                                                                  status);
    return 2;
}
int launch_boundary_batch(const BatchEntry* B, int nscenes, uint64_t total, int total_tiles, int total_segs, int cell,
                          bool styled, const BoundaryScratch& sc, cudaStream_t stream) {
    if (total == 0) return 0;
    total_tiles *= bnd_buckets(cell);  // sort buckets
    cudaMemsetAsync(sc.counts, 0, sizeof(int) * (2 * (size_t)total_tiles + 1), stream);
    cudaMemsetAsync(sc.seg_counts, 0, sizeof(int) * (2 * (size_t)total_segs + 1), stream);
    k_boundary_gen_batch<<<gen_grid(total), 256, 0, stream>>>(B, nscenes, total, cell, sc.samples,
                                                                              sc.key, sc.counts, sc.seg_counts);
    return 1 + boundary_stages(
        sc, total, total_tiles, total_segs, stream,
        [&](const int* offsets, unsigned grid) {
            k_boundary_eval_batch<<<grid, DVG_BND_THREADS, 0, stream>>>(B, sc.samples, sc.order, offsets, total_tiles);
        },
        [&](const int* tot, unsigned grid) {
            if (styled)
                k_boundary_accum_batch<true><<<grid, 256, 0, stream>>>(B, sc.samples, sc.seg_order, tot);
            else
                k_boundary_accum_batch<false><<<grid, 256, 0, stream>>>(B, sc.samples, sc.seg_order, tot);
        });
}

int launch_fill_background(const DevScene& S, float* out, cudaStream_t stream) {
    size_t n = (size_t)S.width * S.height;
    k_fill_background<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(S, out);
    return 1;
}
int launch_l2(const float* img, const float* target, size_t n, float* d_render, float* loss, cudaStream_t stream) {
    unsigned blocks = (unsigned)((n + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    if (blocks == 0) blocks = 1;
    k_l2<<<blocks, 256, 0, stream>>>(img, target, n, d_render, loss);
    return 1;
}

}  // namespace dvgb
