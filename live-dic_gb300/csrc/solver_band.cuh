// Banded IC-GN solver: complete B-spline windows with 16 or 32 lanes per
// subset (reference operations as in solver_impl.cuh, whose reduction and
// update this shares; results are bit-identical to solve_group's).
//
// The reference's order fixes which lane accumulates a pixel and when, not
// which lane samples it, so an iteration goes over the window in bands of
// `band.rows` rows, each in two phases with the band's samples in shared
// memory between them:
//
//   sample      every lane walks vertical runs of `band.run` pixels, two at a
//               time (the halves of the packed FP32 pairs), neighbouring lanes
//               in neighbouring columns.  Consecutive pixels of a run are one
//               row apart, so their 4 x 4 footprints share three tap rows: the
//               taps stay in a ring of four register rows and a pixel loads
//               the four taps of its new row only.  A footprint that did not
//               move by exactly one row (a run's first pixel, a column or row
//               crossing under the warp's gradient) reloads its sixteen.
//   accumulate  lane p mod LANES adds pixel p in increasing p, as the
//               reference does: the same operations in the same order on the
//               same samples, so the sums are bit-identical.
//
// Two 16-lane groups of a warp rarely need the same number of iterations:
// once one of them is done its lanes adopt the other's subset and sample it
// too (the accumulation stays on 16 lanes).  Launches that would not fill the
// SMs with two subsets a warp start out that way, one subset to a warp.  What
// a subset needs only between the pixel loops (its row of the metadata, the
// inverse Hessian, stop counters) lives in shared memory, which keeps the
// loops free of spills (quadratic with 16 lanes: 8 bytes).
//
// What bounds it.  The direct loop (solver_impl.cuh) gathers 16 taps and a
// 16-byte plane entry for every pixel: 32 L1 wavefronts per warp and pixel,
// 70 % of the L1 data pipe.  Here it is 16 to 20 (35 to 45 %): the taps come
// from the ring, and f and (gx, gy) from planes of their own (a misaligned
// 16-byte entry costs twice its wavefronts).  The FMA pipe (57 to 59 %, an
// FFMA2 of three register pairs takes three cycles of operand reads) and the
// latency of L2 reads at 20 warps per SM remain: 371 cycles of a warp's time
// per pixel go to sampling, 206 to accumulating, 80 to the update (affine,
// S 31).  ncu, 1920 x 1080 S 31 / s 8 affine: 302 against 322 M instructions.
// Measured (solver launch, CUPTI, direct -> banded): UHD S 31 / s 8 affine
// 1,874 -> 1,630 us; the 12 launches of four pyramid frames 5,368 -> 4,763;
// UHD S 41 / s 10 quadratic 3,877 -> 3,229; 1280 x 720 S 21 / s 7 affine
// 250 -> 219; 512 x 512 S 21 / s 10 80 -> 57; 2560 x 1440 S 31 / s 8
// translation 666 -> 471; 400 x 300 S 41 / s 20 (234 subsets) quadratic
// 149 -> 105.  (Grids of few affine or translation windows take a block each,
// solver_partial.cu.)
//
// Tried and not kept: smaller bands (more L1 left, but every band restarts the
// rings: 1,826 us with 16-row bands); six CTAs per SM (80 registers, spills);
// four (128); per-SM queues of window tiles (L1 reuse, but the end of the
// launch cost more); the next block's plane loads ahead of the current sums
// (masks on every pixel: 1,914); a whole warp's lanes sharing the affine
// update (shuffles: 1,739).
#pragma once

#include <type_traits>

#include "solver_impl.cuh"


namespace gbdic {

// Resident CTAs per SM the kernels are compiled for (96 and 128 registers),
// and pixels whose loads are issued together.
constexpr int kBandBlocks = 5, kBandQuadBlocks = 4;
constexpr int kBandPixels = 8, kBandQuadPixels = 4;
constexpr int kMaxBandFloats = 1100;        // largest band: 8 subsets of a CTA stay below 48 KB
constexpr unsigned kFloorBits = 0x4b000000u;  // 2^23: floor(x) + 2^23 keeps the integer in the low mantissa bits

// Taps of one run slot (HI: the pair's second half) of the ring's window at
// rotation ROT: window row j is ring[(ROT + j) & 3].
template <int ROT, int J, bool HI>
__device__ __forceinline__ void ring_row(float2 (&ring)[4][4], const float *__restrict__ p) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        if (HI) ring[(ROT + J) & 3][i].y = __ldg(p + i);
        else ring[(ROT + J) & 3][i].x = __ldg(p + i);
    }
}

// The two pixels a lane walks (A in .x, B in .y): where they are, and the
// next row of each.
struct Walk {
    float2 lx, ly, xo, yo;     // local and integer coordinates of the row to come
    float2 tx, ty;             // fractions of the current sample positions
    unsigned ia, ib;           // plane index of the current footprints' first taps
    unsigned nexta, nextb;     // the index at which the ring's rows are the footprint's upper three
};

// Moves to the next row: its positions, and the bottom tap row of its
// footprints into ring row (ROT + 3) & 3.  The row after a run's last one is
// looked up as well; the bound keeps its load inside the plane.
template <int MODEL, int ROT>
__device__ __forceinline__ void walk_next(Walk &k, float2 (&ring)[4][4], const SolveArgs &a, const Warp &w) {
    float2 dx, dy;
    if (MODEL == kModelQuadratic) {
        const float2 half2 = pair(0.5f);
        const float2 hx2 = mul2(mul2(half2, k.lx), k.lx), xy = mul2(k.lx, k.ly), hy2 = mul2(mul2(half2, k.ly), k.ly);
        dx = add2(pair(w.t0), fma2(pair(w.l0), k.lx, mul2(pair(w.l1), k.ly)));
        dy = add2(pair(w.t1), fma2(pair(w.l2), k.lx, mul2(pair(w.l3), k.ly)));
        dx = add2(dx, fma2(pair(w.c0), hx2, fma2(pair(w.c1), xy, mul2(pair(w.c2), hy2))));
        dy = add2(dy, fma2(pair(w.c3), hx2, fma2(pair(w.c4), xy, mul2(pair(w.c5), hy2))));
    } else {
        // in scalars: as packed operands the warp's parameters would take a register pair each
        displacement<MODEL>(w, k.lx.x, k.ly.x, 0.0f, 0.0f, 0.0f, dx.x, dy.x);
        displacement<MODEL>(w, k.lx.y, k.ly.y, 0.0f, 0.0f, 0.0f, dx.y, dy.y);
    }
    const float2 px = add2(k.xo, dx), py = add2(k.yo, dy);
    const float2 big = pair(8388608.0f), m1 = pair(-1.0f);
    const float2 ix = __fadd2_rd(px, big), iy = __fadd2_rd(py, big);
    k.tx = fma2(add2(ix, pair(-8388608.0f)), m1, px);
    k.ty = fma2(add2(iy, pair(-8388608.0f)), m1, py);
    // plane index of the first tap: (by - 1) W + bx - 1 from the floors' bits
    const unsigned W = (unsigned)a.W, origin = kFloorBits * W + kFloorBits + W + 1u, most = ((unsigned)a.H - 3u) * W - 4u;
    k.ia = min(__float_as_uint(iy.x) * W + (__float_as_uint(ix.x) - origin), most);
    k.ib = min(__float_as_uint(iy.y) * W + (__float_as_uint(ix.y) - origin), most);
    const float *bottom = a.coef + 3 * (size_t)W;
    ring_row<ROT, 3, false>(ring, bottom + k.ia);
    ring_row<ROT, 3, true>(ring, bottom + k.ib);
    k.ly = add2(k.ly, pair(1.0f));
    k.yo = add2(k.yo, pair(1.0f));
}

// Samples the current row of both pixels (the arithmetic of
// sample_bspline_pair) into *ga and *gb and moves on: once the top tap row is
// summed, its registers take the bottom row of the next footprints, whose
// loads then have the rest of this step and the next one's weights to land.
template <int MODEL, int ROT>
__device__ __forceinline__ void walk_step(Walk &k, float2 (&ring)[4][4], const SolveArgs &a, const Warp &w, float *&ga,
                                          float *&gb) {
    const unsigned W = (unsigned)a.W;
    const bool jumpa = k.ia != k.nexta, jumpb = k.ib != k.nextb;
    // warp-uniform: no divergence on the sliding path
    if (__any_sync(kFullMask, jumpa || jumpb)) {
        const float *pa = a.coef + k.ia, *pb = a.coef + k.ib;
        if (jumpa) {
            ring_row<ROT, 0, false>(ring, pa);
            ring_row<ROT, 1, false>(ring, pa + W);
            ring_row<ROT, 2, false>(ring, pa + 2 * (size_t)W);
        }
        if (jumpb) {
            ring_row<ROT, 0, true>(ring, pb);
            ring_row<ROT, 1, true>(ring, pb + W);
            ring_row<ROT, 2, true>(ring, pb + 2 * (size_t)W);
        }
    }
    k.nexta = k.ia + W;
    k.nextb = k.ib + W;
    float2 wx[4], wy[4];
    bspline_weights2(k.tx, wx);
    bspline_weights2(k.ty, wy);
    float2 row = pair(0.0f);
#pragma unroll
    for (int i = 0; i < 4; ++i) row = fma2(wx[i], ring[ROT & 3][i], row);
    float2 value = fma2(wy[0], row, pair(0.0f));
    walk_next<MODEL, ROT + 1>(k, ring, a, w);
    // Tap columns outside, rows inside: independent sums, and the column
    // weight stays in the operand cache (an FFMA2 of three register pairs
    // issues every third cycle, with one of them cached every second one).
    float2 rows[3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
        for (int j = 1; j < 4; ++j) rows[j - 1] = fma2(wx[i], ring[(ROT + j) & 3][i], i == 0 ? pair(0.0f) : rows[j - 1]);
    }
#pragma unroll
    for (int j = 1; j < 4; ++j) value = fma2(wy[j], rows[j - 1], value);
    *ga = value.x;
    *gb = value.y;
    ga += a.S;
    gb += a.S;
}

// warp_inside with one control point on each lane `sl` of a 16-lane segment
// (called by the lanes in `mask`).
template <int MODEL>
__device__ __forceinline__ bool warp_inside_lanes(const Warp &w, int px0, int py0, int S, float half,
                                            int W, int H, int sl, unsigned mask) {
    const float xmax = (float)W - 3.0f, ymax = (float)H - 3.0f;
    if (MODEL == kModelTranslation) {
        float x0 = (float)px0 + w.t0, y0 = (float)py0 + w.t1;
        float x1 = (float)(px0 + S - 1) + w.t0, y1 = (float)(py0 + S - 1) + w.t1;
        return x0 >= 2.0f && y0 >= 2.0f && x1 <= xmax && y1 <= ymax;
    }
    float lx, ly;
    if (MODEL == kModelQuadratic) {
        const int p = sl < 9 ? sl : 0;
        lx = (float)(p % 3 - 1) * half;
        ly = (float)(p / 3 - 1) * half;
    } else {
        lx = (sl & 1) ? half : -half;
        ly = (sl & 2) ? half : -half;
    }
    float dx, dy;
    displacement<MODEL>(w, lx, ly, 0.5f * lx * lx, lx * ly, 0.5f * ly * ly, dx, dy);
    const float px = ((float)px0 + (half + lx)) + dx;
    const float py = ((float)py0 + (half + ly)) + dy;
    return __all_sync(mask, px >= 2.0f && py >= 2.0f && px <= xmax && py <= ymax);
}

// v / S for v <= 64 (S <= 1100).
__device__ __forceinline__ int div_subset(const SolveArgs &a, int v) { return (int)(((unsigned)v * a.band.magic) >> 20); }

// Samples of the band whose first row is `row0` into `buf` (band.rows x S),
// by `samplers` lanes of which this is lane `sl`.  Run q covers column q mod
// S, rows (q / S) band.run ...; the last run of a column ends at the band's
// last row (rows shared with the run above are sampled twice, alike), and
// lanes beyond the last run repeat it.
template <int MODEL>
__device__ __forceinline__ void sample_band(const SolveArgs &a, const Warp &w, float *buf, int row0, int sl,
                                            int samplers, int px0, int py0, float half) {
    const bool all = samplers == 32;
    const int S = a.S, L = all ? a.band.run32 : a.band.run, R = a.band.rows;
    const int segments = all ? a.band.segments32 : a.band.segments, runs = segments * S;
    const int sdiv = div_subset(a, samplers), smod = samplers - sdiv * S;
    int seg = div_subset(a, sl), col = sl - seg * S;
    for (int q = 0; q < runs; q += 2 * samplers) {
        int segb = seg + sdiv, colb = col + smod;
        if (colb >= S) { colb -= S; ++segb; }
        int nseg = segb + sdiv, ncol = colb + smod;
        if (ncol >= S) { ncol -= S; ++nseg; }
        const int sa = min(seg, segments - 1), ca = seg < segments ? col : S - 1;
        const int sb = min(segb, segments - 1), cb = segb < segments ? colb : S - 1;
        const int ra = min(sa * L, R - L), rb = min(sb * L, R - L);
        Walk k;
        k.lx = make_float2((float)ca - half, (float)cb - half);
        k.ly = make_float2((float)(row0 + ra) - half, (float)(row0 + rb) - half);
        k.xo = make_float2((float)(px0 + ca), (float)(px0 + cb));
        k.yo = make_float2((float)(py0 + row0 + ra), (float)(py0 + row0 + rb));
        k.nexta = k.nextb = 0xffffffffu;  // no footprint's index: the first step loads all its taps
        float *ga = buf + ra * S + ca, *gb = buf + rb * S + cb;
        float2 ring[4][4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) ring[j][i] = pair(0.0f);
        walk_next<MODEL, 0>(k, ring, a, w);
        int left = L;
        for (; left >= 4; left -= 4) {
            walk_step<MODEL, 0>(k, ring, a, w, ga, gb);
            walk_step<MODEL, 1>(k, ring, a, w, ga, gb);
            walk_step<MODEL, 2>(k, ring, a, w, ga, gb);
            walk_step<MODEL, 3>(k, ring, a, w, ga, gb);
        }
        if (left > 0) walk_step<MODEL, 0>(k, ring, a, w, ga, gb);
        if (left > 1) walk_step<MODEL, 1>(k, ring, a, w, ga, gb);
        if (left > 2) walk_step<MODEL, 2>(k, ring, a, w, ga, gb);
        seg = nseg;
        col = ncol;
    }
}

// sample_band pixel by pixel with clamped taps, for quadratic warps that may
// bulge over the plane's border inside the window.
template <int MODEL>
__device__ __forceinline__ void sample_band_clamped(const SolveArgs &a, const Warp &w, float *buf, int row0, int sl,
                                                    int samplers, int px0, int py0, float half) {
    const int S = a.S, sdiv = div_subset(a, samplers), smod = samplers - sdiv * S;
    int row = div_subset(a, sl), col = sl - row * S;
    while (row < a.band.rows) {
        const float lx = (float)col - half, ly = (float)(row0 + row) - half;
        float dx, dy;
        displacement<MODEL>(w, lx, ly, 0.5f * lx * lx, lx * ly, 0.5f * ly * ly, dx, dy);
        buf[row * S + col] = sample_target<kInterpBspline, true>(a.coef, a.img, a.W, a.H, (float)(px0 + col) + dx,
                                                                 (float)(py0 + row0 + row) + dy);
        row += sdiv;
        col += smod;
        if (col >= S) { col -= S; ++row; }
    }
}

// Every sample of the window lies at least one pixel inside the taps' reach:
// the bounds check guarantees it for affine and translation warps; a
// quadratic one is bounded by the sizes of its terms.
template <int MODEL>
__device__ __forceinline__ bool taps_inside(const SolveArgs &a, const Warp &w, int px0, int py0, float half) {
    if (MODEL != kModelQuadratic) return true;
    const float h2 = half * half;
    const float ex = half * (1.0f + fabsf(w.l0) + fabsf(w.l1)) + h2 * (0.5f * fabsf(w.c0) + fabsf(w.c1) + 0.5f * fabsf(w.c2)) + 1.0f;
    const float ey = half * (1.0f + fabsf(w.l2) + fabsf(w.l3)) + h2 * (0.5f * fabsf(w.c3) + fabsf(w.c4) + 0.5f * fabsf(w.c5)) + 1.0f;
    const float cx = (float)px0 + half + w.t0, cy = (float)py0 + half + w.t1;
    return cx - ex >= 1.0f && cy - ey >= 1.0f && cx + ex <= (float)(a.W - 3) && cy + ey <= (float)(a.H - 3);
}

// reduce_warp with the sums split over the lanes: at every stride the two
// halves of a segment swap the halves of their sums and add one each, so a
// sum sees the additions of the pairwise tree (an addition's operand order
// does not change its result) at about half the shuffles.
__host__ __device__ constexpr int split_lane(int value, int count, int stride) {
    return stride == 0 ? 0
           : value >= (count + 1) / 2 && count > 1
               ? stride + split_lane(value - (count + 1) / 2, (count + 1) / 2, stride / 2)
               : split_lane(value, (count + 1) / 2, stride / 2);
}

template <int STRIDE, int COUNT, int N>
__device__ __forceinline__ void split_step(float (&s)[N], int lane) {
    if constexpr (STRIDE > 0) {
        constexpr int kept = (COUNT + 1) / 2;
        const bool upper = (lane & STRIDE) != 0;
#pragma unroll
        for (int k = 0; k < kept; ++k) {
            float mine = s[k], other = s[k];
            if constexpr (COUNT > 1) {
                const float high = k + kept < COUNT ? s[k + kept] : s[k];
                other = upper ? s[k] : high;
                mine = upper ? high : s[k];
            }
            s[k] = mine + __shfl_xor_sync(kFullMask, other, STRIDE);
        }
        split_step<STRIDE / 2, kept, N>(s, lane);
    }
}

template <int LANES, int N, int K = 0>
__device__ __forceinline__ void split_gather(float (&out)[N], float total, int lane) {
    if constexpr (K < N) {
        out[K] = __shfl_sync(kFullMask, total, split_lane(K, N, LANES / 2), LANES);
        split_gather<LANES, N, K + 1>(out, total, lane);
    }
}

template <int LANES, int N>
__device__ __forceinline__ void reduce_split(float (&s)[N], int lane) {
    split_step<LANES / 2, N, N>(s, lane);
    split_gather<LANES, N>(s, s[0], lane);
}

// Adds the band's pixels p (rows first .. last - 1, p mod LANES == glane) to
// the lane's sums in increasing p; g[p]: their samples.  A pixel's local
// coordinates, weight and plane offset come from the level's pixel table
// (the same 16 bytes for every window, so they stay in L1).
template <int MODEL, int LANES, bool GAUSS, int N>
__device__ __forceinline__ void accumulate_band(float (&s)[N], const SolveArgs &a, const float *g, int first, int last,
                                                int glane, int px0, int py0, float mean) {
    const int end = last * a.S;
    int p = first * a.S + ((glane - first * a.S) & (LANES - 1));
    const size_t origin = (size_t)py0 * a.W + px0;
    const float *plane_f = a.plane_f + origin;
    const float2 *plane_grad = a.plane_grad + origin;
    // C pixels, their loads ahead of the sums.  `tail`: pixels beyond the
    // band's end count as zeros, which leave every sum as it is.
    auto pixels = [&](auto count, auto tail) {
        constexpr int C = decltype(count)::value;
        constexpr bool kTail = decltype(tail)::value;
        float f[C], v[C];
        float2 grad[C];
        float4 px[C];  // lx, ly, weight, offset
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const int q = kTail ? min(p + k * LANES, end - 1) : p + k * LANES;
            px[k] = __ldg(a.pixel_table + q);
            v[k] = g[q];
        }
#pragma unroll
        for (int k = 0; k < C; ++k) {
            f[k] = __ldg(plane_f + __float_as_uint(px[k].w));
            grad[k] = __ldg(plane_grad + __float_as_uint(px[k].w));
        }
#pragma unroll
        for (int k = 0; k < C; ++k) {
            const float x = px[k].x, y = px[k].y;
            float hx2 = 0.0f, xy = 0.0f, hy2 = 0.0f;
            if (MODEL == kModelQuadratic) {
                hx2 = 0.5f * x * x;
                xy = x * y;
                hy2 = 0.5f * y * y;
            }
            const bool on = !kTail || p + k * LANES < end;
            accumulate_values<MODEL, GAUSS, N>(s, on ? v[k] : 0.0f, on ? f[k] - mean : 0.0f, on ? grad[k].x : 0.0f,
                                               on ? grad[k].y : 0.0f, px[k].z, x, y, hx2, xy, hy2);
        }
        p += C * LANES;
    };
    constexpr int kBlockPx = MODEL == kModelQuadratic ? kBandQuadPixels : kBandPixels;
    using Block = std::integral_constant<int, kBlockPx>;
    using Half = std::integral_constant<int, kBlockPx / 2>;
    while (p + (kBlockPx - 1) * LANES < end) pixels(Block{}, std::false_type{});
    if (__any_sync(kFullMask, p + (kBlockPx / 2) * LANES < end)) pixels(Block{}, std::true_type{});
    else if (__any_sync(kFullMask, p < end)) pixels(Half{}, std::true_type{});
}

// Shared-memory words of one group beside its band buffer (a multiple of the
// 32 banks).
enum { kColdIndex, kColdFlags, kColdIterations, kColdPrevious, kColdStalled, kColdMean, kColdWsum, kColdMeta = 8 };
__host__ __device__ constexpr int cold_words(int model) {
    return (kColdMeta + meta_stride(model) + parameter_count(model) * parameter_count(model) + 31) / 32 * 32;
}

// Shared memory of a warp: its groups, and the lanes' sums between bands.
__host__ __device__ inline int band_warp_floats(const SolveArgs &a, int model, int lanes) {
    const int sums = model == kModelQuadratic ? 15 : (model == kModelTranslation ? 5 : 9);
    return (32 / lanes) * (cold_words(model) + a.band.pitch) + (a.band.rows < a.S ? 32 * sums : 0);
}

__device__ __forceinline__ void copy_async4(float *dst, const float *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}

// Solves subset `idx` (where it `exists`) on each LANES lanes of the warp;
// `warp_smem`: band_warp_floats floats, per group cold_words(MODEL) words then
// band.pitch floats.
template <int MODEL, int LANES, bool GAUSS>
__device__ __forceinline__ void solve_band(const SolveArgs &a, int idx, bool exists, int lane, float *warp_smem) {
    constexpr int N = SumCount<MODEL>::value;
    constexpr int n = parameter_count(MODEL);
    constexpr int kGroups = 32 / LANES;
    const int glane = lane & (LANES - 1);
    const int pitch = cold_words(MODEL) + a.band.pitch;
    volatile float *cold = warp_smem + (LANES == 16 ? (lane >> 4) * pitch : 0);
    const unsigned seg_mask = LANES == 16 ? (0xffffu << (lane & 16)) : kFullMask;
    const int S = a.S;
    const float half = 0.5f * ((float)S - 1.0f);
    Warp w = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    float status;
    bool done;
    int px0, py0;
    {
        const int sidx = exists ? idx : 0;
        const float *md = a.meta + (size_t)sidx * meta_stride(MODEL);
        const float *hi = a.inv + (size_t)sidx * (n * n);
        float *dst = const_cast<float *>(cold) + kColdMeta;
#pragma unroll
        for (int k = 0; k < (meta_stride(MODEL) + LANES - 1) / LANES; ++k)
            if (k * LANES + glane < meta_stride(MODEL)) copy_async4(dst + k * LANES + glane, md + k * LANES + glane);
        dst += meta_stride(MODEL);
#pragma unroll
        for (int k = 0; k < (n * n + LANES - 1) / LANES; ++k)
            if (k * LANES + glane < n * n) copy_async4(dst + k * LANES + glane, hi + k * LANES + glane);
        bool enabled = exists;
        if (a.seed != nullptr && exists) {
            const float4 *s = reinterpret_cast<const float4 *>(a.seed + (size_t)sidx * state_stride(MODEL));
            const float4 s0 = __ldg(s), s1 = __ldg(s + 1);
            w.t0 = s0.x; w.l0 = s0.y; w.l1 = s0.z; w.t1 = s0.w;
            w.l2 = s1.x; w.l3 = s1.y;
            if (MODEL == kModelQuadratic) {
                const float4 s2 = __ldg(s + 2);
                w.c0 = s1.z; w.c1 = s1.w; w.c2 = s2.x; w.c3 = s2.y; w.c4 = s2.z; w.c5 = s2.w;
            }
            enabled = __ldg(a.active + sidx) != 0u;
        }
        if (MODEL == kModelTranslation) { w.l0 = w.l1 = w.l2 = w.l3 = 0.0f; }
        const float mvalid = __ldg(md + 1);
        const float rejected = a.roi_enabled ? fminf(-1.0f, mvalid) : -1.0f;
        status = enabled && mvalid >= 0.5f ? 0.0f : rejected;
        done = !exists;
        px0 = (sidx % a.grid_w) * a.stride;
        py0 = (sidx / a.grid_w) * a.stride;
        if (glane == 0) {
            cold[kColdIndex] = __int_as_float(idx);
            cold[kColdFlags] = __int_as_float((exists ? 1 : 0) | (exists && (enabled || !a.preserve_disabled) ? 2 : 0));
            cold[kColdIterations] = 0.0f;
            cold[kColdPrevious] = 3.402823e38f;
            cold[kColdStalled] = __uint_as_float(0u);
            cold[kColdMean] = a.use_mean ? __ldg(md + 2 + 2 * n) : 0.0f;
            cold[kColdWsum] = GAUSS ? __ldg(md + 3 + 2 * n) : (float)(S * S);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        __syncwarp();
    }
    bool helper = false;   // lanes whose own subset is done, sampling the other group's
    int samplers = LANES;
    auto finish = [&]() {
        const int flags = __float_as_int(cold[kColdFlags]);
        const float iters = cold[kColdIterations];
        if (glane != 0) return;
        if (a.iteration_total != nullptr && (flags & 1) && iters > 0.0f)
            atomicAdd(a.iteration_total, (unsigned long long)iters);
        if (flags & 2) {
            const float final_status = (a.div_patience != 0 && status == 3.0f) ? 0.0f : status;
            float4 *o = reinterpret_cast<float4 *>(a.state + (size_t)__float_as_int(cold[kColdIndex]) * state_stride(MODEL));
            o[0] = make_float4(w.t0, w.l0, w.l1, w.t1);
            if (MODEL == kModelQuadratic) {
                o[1] = make_float4(w.l2, w.l3, w.c0, w.c1);
                o[2] = make_float4(w.c2, w.c3, w.c4, w.c5);
                o[3] = make_float4(final_status, iters, 0.0f, 0.0f);
            } else {
                o[1] = make_float4(w.l2, w.l3, final_status, iters);
            }
        }
    };

    for (int it = 0; it < 30; ++it) {
        if (!done) {
            if (!(a.div_patience != 0 && status == 3.0f)) {
                if (!warp_inside_lanes<MODEL>(w, px0, py0, S, half, a.W, a.H, lane & 15, seg_mask)) {
                    if (!a.roi_enabled || status > -2.5f) status = -1.0f;
                }
            }
            if (it >= a.iterations || fabsf(status) > 0.5f) done = true;
        }
        const unsigned live_lanes = __ballot_sync(kFullMask, !done);
        if (live_lanes == 0u) break;
        if (LANES == 16 && samplers == 16 && ((live_lanes & 0xffffu) == 0u || (live_lanes >> 16) == 0u)) {
            if (done) finish();
            helper = done;
            const int from = (live_lanes & 0xffffu) ? 0 : 16;
            w.t0 = __shfl_sync(kFullMask, w.t0, from); w.t1 = __shfl_sync(kFullMask, w.t1, from);
            w.l0 = __shfl_sync(kFullMask, w.l0, from); w.l1 = __shfl_sync(kFullMask, w.l1, from);
            w.l2 = __shfl_sync(kFullMask, w.l2, from); w.l3 = __shfl_sync(kFullMask, w.l3, from);
            if (MODEL == kModelQuadratic) {
                w.c0 = __shfl_sync(kFullMask, w.c0, from); w.c1 = __shfl_sync(kFullMask, w.c1, from);
                w.c2 = __shfl_sync(kFullMask, w.c2, from); w.c3 = __shfl_sync(kFullMask, w.c3, from);
                w.c4 = __shfl_sync(kFullMask, w.c4, from); w.c5 = __shfl_sync(kFullMask, w.c5, from);
            }
            px0 = __shfl_sync(kFullMask, px0, from);
            py0 = __shfl_sync(kFullMask, py0, from);
            status = 0.0f;  // a live subset's
            cold = warp_smem + (from >> 4) * pitch;
            done = false;
            samplers = 32;
        }
        // Every live lane has work here: the band's samples, then the lane's
        // pixels of the band in order, a block at a time with their
        // loads ahead of the sums.  Nothing of the accumulation stays in
        // registers while a band is sampled.
        float s[N];
        float *buf = const_cast<float *>(cold) + cold_words(MODEL);
        float *sums = warp_smem + kGroups * pitch + lane;
        const bool inside = __all_sync(kFullMask, taps_inside<MODEL>(a, w, px0, py0, half));
        for (int first = 0; first < S; first += a.band.rows) {
            const int top = min(first, S - a.band.rows);
            __syncwarp();
            if (inside) sample_band<MODEL>(a, w, buf, top, samplers == 32 ? lane : glane, samplers, px0, py0, half);
            else sample_band_clamped<MODEL>(a, w, buf, top, samplers == 32 ? lane : glane, samplers, px0, py0, half);
            __syncwarp();
            if (first == 0) {
#pragma unroll
                for (int k = 0; k < N; ++k) s[k] = 0.0f;
            } else {
#pragma unroll
                for (int k = 0; k < N; ++k) s[k] = sums[k * 32];
            }
            const int last = min(first + a.band.rows, S);
            accumulate_band<MODEL, LANES, GAUSS, N>(s, a, buf - top * S, first, last, glane, px0, py0,
                                                    cold[kColdMean]);
            if (last < S) {
#pragma unroll
                for (int k = 0; k < N; ++k) sums[k * 32] = s[k];
            }
        }
        reduce_split<LANES, N>(s, lane);
        const float *md = const_cast<const float *>(cold) + kColdMeta;
        float previous = cold[kColdPrevious];
        unsigned stalled = __float_as_uint(cold[kColdStalled]);
        __syncwarp();
        status = gn_update<MODEL, true>(a, s, md, md + meta_stride(MODEL), cold[kColdWsum], half, (unsigned)(it + 1), w,
                                  previous, stalled, lane & 15, seg_mask);
        if (glane == 0) {
            cold[kColdIterations] = (float)(it + 1);
            cold[kColdPrevious] = previous;
            cold[kColdStalled] = __uint_as_float(stalled);
        }
        __syncwarp();
    }
    if (!helper) finish();
    __syncwarp();
}

template <int MODEL, int LANES, bool GAUSS>
__global__ void __launch_bounds__(128, MODEL == kModelQuadratic ? kBandQuadBlocks : kBandBlocks)
    icgn_band_kernel(SolveArgs a) {
    constexpr int kGroups = 32 / LANES;
    extern __shared__ float band_smem[];
    const int tid = threadIdx.x, lane = tid & 31, group_in_warp = LANES == 16 ? lane >> 4 : 0;
    float *warp_smem = band_smem + (tid >> 5) * band_warp_floats(a, MODEL, LANES);
    // Small launches give every subset a warp: two to a warp would leave SMs
    // idle, and the second half's lanes sample too.
    const int per_warp = LANES == 16 && !a.persistent && a.count <= a.band.solo_count ? 1 : kGroups;
    const long long unit = (long long)blockIdx.x * 4 + (tid >> 5);
    const int count = a.list_count != nullptr ? min(a.count, (int)__ldg(a.list_count)) : a.count;
    for (;;) {
        int base;
        if (a.persistent) {
            int v = 0;
            if (lane == 0) v = (int)atomicAdd(a.work_counter, (unsigned)kGroups);
            base = __shfl_sync(kFullMask, v, 0);
        } else {
            base = unit * per_warp < (long long)count ? (int)(unit * per_warp) : count;
        }
        if (base >= count) break;
        const int group = base + group_in_warp;
        const bool exists = group < count && group_in_warp < per_warp;
        solve_band<MODEL, LANES, GAUSS>(a, a.subset_list != nullptr && exists ? __ldg(a.subset_list + group) : group, exists,
                                        lane, warp_smem);
        if (!a.persistent) break;
    }
}

}  // namespace gbdic
