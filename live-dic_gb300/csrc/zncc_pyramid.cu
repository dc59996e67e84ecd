// Final ZNCC (reference: shaders/affine_zncc.wgsl:57-99) and the pyramid /
// temporal kernels (reference: shaders/full_pyramid.wgsl).
#include "gbdic_common.cuh"
#include "gbdic_kernels.h"
#include "solver_band.cuh"

namespace gbdic {

namespace {

// ------------------------------------------------------------ final ZNCC
// 64 lanes per subset (two subsets per 128-thread CTA); sums over the valid
// warped pixels of [f, g, f^2, g^2, f g, count], pairwise tree over lanes.
template <int INTERP>
__global__ void __launch_bounds__(128) final_zncc_kernel(ZnccArgs a) {
    __shared__ float red[2][6][64];
    const int sub = threadIdx.x >> 6, lane = threadIdx.x & 63;
    const int index = blockIdx.x * 2 + sub;
    const bool exists = index < a.count;
    const int sidx = exists ? index : 0;
    const float4 *st = reinterpret_cast<const float4 *>(a.state + (size_t)sidx * 8);
    const float4 p = st[0], q = st[1];
    const bool active = exists && q.z == 1.0f;
    float s[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (active) {
        const int S = a.S;
        const int gx = sidx % a.grid_w, gy = sidx / a.grid_w;
        const float half = ((float)S - 1.0f) * 0.5f;
        for (int k = lane; k < S * S; k += 64) {
            const int col = k % S, row = k / S;
            const int px = gx * a.stride + col, py = gy * a.stride + row;
            const float lx = (float)col - half, ly = (float)row - half;
            const float tx = (float)px + (p.x + fmaf(p.y, lx, p.z * ly));
            const float ty = (float)py + (p.w + fmaf(q.x, lx, q.y * ly));
            if (tx >= 2.0f && ty >= 2.0f && tx <= (float)(a.W - 3) && ty <= (float)(a.H - 3)) {
                const float g = sample_target<INTERP, true>(a.coef, a.img, a.W, a.H, tx, ty);
                const float f = a.plane[(size_t)py * a.W + px].x;
                s[0] = s[0] + f;
                s[1] = s[1] + g;
                s[2] = fmaf(f, f, s[2]);
                s[3] = fmaf(g, g, s[3]);
                s[4] = fmaf(f, g, s[4]);
                s[5] = s[5] + 1.0f;
            }
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) red[sub][k][lane] = s[k];
    __syncthreads();
    if (lane < 32) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            float v = red[sub][k][lane] + red[sub][k][lane + 32];
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_down_sync(kFullMask, v, off);
            s[k] = v;
        }
    }
    if (!exists || lane != 0) return;
    if (!active) {
        a.out[index] = -2.0f;
        return;
    }
    const float n = s[5], nn = fmaxf(n, 1.0f);
    const float vf = s[2] - s[0] * s[0] / nn;
    const float vg = s[3] - s[1] * s[1] / nn;
    if (n == (float)(a.S * a.S) && vf > 1e-9f && vg > 1e-9f) {
        const float r = (s[4] - s[0] * s[1] / n) / sqrtf(vf * vg);
        a.out[index] = fminf(fmaxf(r, -1.0f), 1.0f);
    } else {
        a.out[index] = -2.0f;
    }
}

// final_zncc_kernel of B-spline windows, a warp to a subset: the window is
// sampled as by the banded solver loop (sample_band: tap rows in a register
// ring, two runs to a lane), then every lane adds the pixels of the two of
// the 64 lanes it stands for, in their order.  The value is defined only if
// every pixel lands in [2, W-3] x [2, H-3], so the check is made on the four
// corner pixels; pixels between corners that lie inside by a margin lie
// inside too (an affine map, rounded far below the margin), and a window
// closer to the bound is checked pixel by pixel.
// FMA-bound as the solver's sampling (96 registers, 44 bytes of spills).  UHD S 31 / s 8 (127,359 subsets): 1,011
// us with sixteen clamped taps gathered and two integer divisions per pixel
// (final_zncc_kernel), 517 us here.
__global__ void __launch_bounds__(128, kBandBlocks) final_zncc_band_kernel(SolveArgs a, const float *f_plane, int f_pitch,
                                                                           float *out) {
    extern __shared__ float band_smem[];
    const int lane = threadIdx.x & 31, index = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (index >= a.count) return;  // warp-uniform
    float *buf = band_smem + (threadIdx.x >> 5) * a.band.pitch;
    const float4 *st = reinterpret_cast<const float4 *>(a.state + (size_t)index * 8);
    const float4 p = __ldg(st), q = __ldg(st + 1);
    const Warp w = {p.x, p.w, p.y, p.z, q.x, q.y, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    const int S = a.S, W = a.W, H = a.H;
    const int px0 = (index % a.grid_w) * a.stride, py0 = (index / a.grid_w) * a.stride;
    const float half = ((float)S - 1.0f) * 0.5f;
    auto position = [&](int col, int row, float &tx, float &ty) {
        const float lx = (float)col - half, ly = (float)row - half;
        float dx, dy;
        displacement<kModelAffine>(w, lx, ly, 0.0f, 0.0f, 0.0f, dx, dy);
        tx = (float)(px0 + col) + dx;
        ty = (float)(py0 + row) + dy;
    };
    auto inside = [&](float tx, float ty, float m) {
        return tx >= 2.0f + m && ty >= 2.0f + m && tx <= (float)(W - 3) - m && ty <= (float)(H - 3) - m;
    };
    float tx, ty;
    position((lane & 1) * (S - 1), ((lane >> 1) & 1) * (S - 1), tx, ty);
    bool valid = q.z == 1.0f && __all_sync(kFullMask, inside(tx, ty, 0.0f));
    if (valid && !__all_sync(kFullMask, inside(tx, ty, 0.0625f + 1e-6f * (float)(W + H)))) {
        bool all = true;
        for (int k = lane; k < S * S; k += 32) {
            position(k % S, k / S, tx, ty);
            all = all && inside(tx, ty, 0.0f);
        }
        valid = __all_sync(kFullMask, all);
    }
    if (!valid) {
        if (lane == 0) out[index] = -2.0f;
        return;
    }
    float s[2][5];
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int k = 0; k < 5; ++k) s[h][k] = 0.0f;
    const int rows = a.band.rows;
    const float *f_window = f_plane + ((size_t)py0 * W + px0) * f_pitch;
    for (int first = 0; first < S; first += rows) {
        const int top = min(first, S - rows), last = min(first + rows, S);
        __syncwarp();
        sample_band<kModelAffine>(a, w, buf, top, lane, 32, px0, py0, half);
        __syncwarp();
        const float *g = buf - top * S;
        // pixel 32 m + lane belongs to lane 32 (m & 1) + lane of the 64
        const int end = last * S;
        int m = first * S / 32;
        int k = 32 * m + lane;
        int row = k / S, col = k - row * S;
        const int sdiv = div_subset(a, 32), smod = 32 - sdiv * S;
        auto add = [&](float (&t)[5]) {
            if (k >= first * S && k < end) {
                const float fv = __ldg(f_window + (size_t)(row * W + col) * f_pitch), gv = g[k];
                t[0] = t[0] + fv;
                t[1] = t[1] + gv;
                t[2] = fmaf(fv, fv, t[2]);
                t[3] = fmaf(gv, gv, t[3]);
                t[4] = fmaf(fv, gv, t[4]);
            }
            k += 32;
            row += sdiv;
            col += smod;
            if (col >= S) { col -= S; ++row; }
        };
        if (m & 1) {
            add(s[1]);
            ++m;
        }
#pragma unroll 4
        for (; 32 * m < end; m += 2) {
            add(s[0]);
            add(s[1]);
        }
    }
    float t[5];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
        float v = s[0][k] + s[1][k];
#pragma unroll
        for (int off = 16; off >= 1; off >>= 1) v = v + __shfl_down_sync(kFullMask, v, off);
        t[k] = v;
    }
    if (lane != 0) return;
    const float n = (float)(S * S), nn = fmaxf(n, 1.0f);
    const float vf = t[2] - t[0] * t[0] / nn;
    const float vg = t[3] - t[1] * t[1] / nn;
    float value = -2.0f;
    if (vf > 1e-9f && vg > 1e-9f) {
        const float r = (t[4] - t[0] * t[1] / n) / sqrtf(vf * vg);
        value = fminf(fmaxf(r, -1.0f), 1.0f);
    }
    out[index] = value;
}

// ------------------------------------------------------------ reduction
// full_pyramid.wgsl:218-249: exact integer 5x5 [1 4 6 4 1]^2 sum over the
// reflected source, truncating division by 256.  Integer sums are exact in any
// order, so the separable form equals the 5x5 one.
// A thread has 4 x 4 outputs: for each of its 11 source rows the four
// horizontal sums as byte dot products of 16 bytes loaded as words, added into
// the rows' vertical sums as they come; nothing goes through shared memory.
// A border thread mends its one reflected word from the neighbouring one, so
// that the words' warps do not diverge; where rows are not whole words, and in
// the last thread of a row that its outputs do not fill, bytes are gathered
// (a kernel of its own for the former: the word loads beside it cost it 10 to 20 %).
// By bytes through shared memory -> here, us a launch: 3840 x 2160 21.2 -> 7.3
// (8.3 MB read: 1.2), 1920 x 1080 7.4 -> 4.6, 640 x 360 7.0 -> 4.8, 160 x 90
// 5.8 -> 4.2; of bytes 3839 x 2159 21.2 -> 15.3, 1919 x 1080 7.4 -> 6.5, 321 x 181
// 7.1 -> 5.3, 81 x 45 5.1 -> 4.6.  With the border threads gathering bytes beside
// the others' words a warp took both ways: 1920 x 1080 8.2, 640 x 360 8.1.
constexpr int kRX = 4, kRY = 4;

template <bool WORDS>  // rows are whole words
__global__ void __launch_bounds__(128) reduce_half_kernel(const uint8_t *__restrict__ src, int W, int H,
                                                          uint8_t *__restrict__ dst) {
    const int W2 = W / 2, H2 = H / 2;
    const int X = kRX * (int)(blockIdx.x * 32 + threadIdx.x), Y = kRY * (int)(blockIdx.y * 4 + threadIdx.y);
    if (X >= W2 || Y >= H2) return;
    const int c0 = 2 * X - 4;  // the words cover columns c0 .. c0 + 15; the sums use c0 + 2 .. c0 + 12
    const bool words = WORDS && c0 + 12 <= W;
    const int first = c0 < 0 ? 1 : 0, last = c0 + 16 <= W ? 3 : 2;  // words inside the row
    unsigned acc[kRY][kRX] = {};
#pragma unroll
    for (int k = 0; k < 2 * kRY + 3; ++k) {
        const uint8_t *row = src + (size_t)mirror_clamp(2 * Y - 2 + k, H) * W;
        uint32_t w[4];
        if (words) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                w[q] = __ldg(reinterpret_cast<const uint32_t *>(row + c0) + min(max(q, first), last));
            if (first == 1) w[0] = __byte_perm(w[1], 0u, 0x1244);  // columns -1, -2 are 1, 2
            if (last == 2) w[3] = __byte_perm(w[2], 0u, 0x4442);   // column W is W - 2
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                w[q] = 0u;
#pragma unroll
                for (int b = 0; b < 4; ++b) w[q] |= (uint32_t)__ldg(row + mirror_clamp(c0 + 4 * q + b, W)) << (8 * b);
            }
        }
        // five bytes from column c0 + 2 + 2 i: four by the weights 1 4 6 4, and one
        const uint32_t four = 0x04060401u;
        unsigned h[kRX];
        h[0] = __dp4a(__byte_perm(w[0], w[1], 0x5432), four, __dp4a(w[1], 0x00010000u, 0u));
        h[1] = __dp4a(w[1], four, w[2] & 0xffu);
        h[2] = __dp4a(__byte_perm(w[1], w[2], 0x5432), four, __dp4a(w[2], 0x00010000u, 0u));
        h[3] = __dp4a(w[2], four, w[3] & 0xffu);
#pragma unroll
        for (int y = 0; y < kRY; ++y) {
            const int tap = k - 2 * y;
            if (tap < 0 || tap > 4) continue;
            const unsigned weight = tap == 2 ? 6u : (tap & 1) ? 4u : 1u;
#pragma unroll
            for (int x = 0; x < kRX; ++x) acc[y][x] += weight * h[x];
        }
    }
    const bool store_words = X + kRX <= W2 && (W2 & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 3) == 0;
#pragma unroll
    for (int y = 0; y < kRY; ++y) {
        if (Y + y >= H2) break;
        uint8_t *o = dst + (size_t)(Y + y) * W2 + X;
        if (store_words) {
            *reinterpret_cast<uint32_t *>(o) = (acc[y][0] >> 8) | (acc[y][1] >> 8) << 8 | (acc[y][2] >> 8) << 16 |
                                               (acc[y][3] >> 8) << 24;
        } else {
#pragma unroll
            for (int x = 0; x < kRX; ++x)
                if (X + x < W2) o[x] = (uint8_t)(acc[y][x] >> 8);
        }
    }
}

// ------------------------------------------------------------ seed transfer
// full_pyramid.wgsl:251-308
__device__ void accumulate_seed(const SeedArgs &a, int sidx, float weight, float spx, float spy,
                                float dpx, float dpy, float tscale, float *acc, float &wsum) {
    const int ss = state_stride(a.model);
    const float *s = a.source + (size_t)sidx * ss;
    const float status = s[status_slot(a.model)];
    if (status < -0.5f) return;
    const float dx = dpx - spx, dy = dpy - spy;
    float tu = fmaf(s[2], dy, fmaf(s[1], dx, s[0]));
    float tv = fmaf(s[5], dy, fmaf(s[4], dx, s[3]));
    float ux = s[1], uy = s[2], vx = s[4], vy = s[5];
    if (a.model == kModelQuadratic) {
        tu = tu + fmaf(s[8], 0.5f * dy * dy, fmaf(s[7], dx * dy, s[6] * (0.5f * dx * dx)));
        tv = tv + fmaf(s[11], 0.5f * dy * dy, fmaf(s[10], dx * dy, s[9] * (0.5f * dx * dx)));
        ux = ux + fmaf(s[7], dy, s[6] * dx);
        uy = uy + fmaf(s[8], dy, s[7] * dx);
        vx = vx + fmaf(s[10], dy, s[9] * dx);
        vy = vy + fmaf(s[11], dy, s[10] * dx);
    }
    acc[0] = fmaf(weight * tu, tscale, acc[0]);
    acc[1] = fmaf(weight, ux, acc[1]);
    acc[2] = fmaf(weight, uy, acc[2]);
    acc[3] = fmaf(weight * tv, tscale, acc[3]);
    acc[4] = fmaf(weight, vx, acc[4]);
    acc[5] = fmaf(weight, vy, acc[5]);
    if (a.model == kModelQuadratic) {
        const float cs = 1.0f / tscale;
        for (int k = 6; k < 12; ++k) acc[k] = fmaf(weight * s[k], cs, acc[k]);
    }
    wsum = wsum + weight;
}

// full_pyramid.wgsl:310-395: bilinear blend of the permitted source corners
// at the destination centre (normalised); returns the weight sum.  `lx`,
// `ly` receive the lower source corner.
__device__ float interpolate_seed(const SeedArgs &a, int i, unsigned perm, float (&acc)[12], int &lx, int &ly) {
    for (int k = 0; k < 12; ++k) acc[k] = 0.0f;
    float wsum = 0.0f;
    const int dxg = i % a.dst_grid_w, dyg = i / a.dst_grid_w;
    const float soff = (1.0f - a.src_scale) * 0.5f, doff = (1.0f - a.dst_scale) * 0.5f;
    const float dcx = fmaf(a.subset_stride, (float)dxg, 0.5f * a.subset_size);
    const float dcy = fmaf(a.subset_stride, (float)dyg, 0.5f * a.subset_size);
    const float scx = fmaf(a.dst_scale, dcx, doff - soff) / a.src_scale;
    const float scy = fmaf(a.dst_scale, dcy, doff - soff) / a.src_scale;
    const float gxf = (scx - 0.5f * a.subset_size) / a.subset_stride;
    const float gyf = (scy - 0.5f * a.subset_size) / a.subset_stride;
    const int maxx = a.src_grid_w - 2 > 0 ? a.src_grid_w - 2 : 0;
    const int maxy = a.src_grid_h - 2 > 0 ? a.src_grid_h - 2 : 0;
    lx = clampi((int)floorf(gxf), 0, maxx);
    ly = clampi((int)floorf(gyf), 0, maxy);
    const float fx = fminf(fmaxf(gxf - (float)lx, 0.0f), 1.0f);
    const float fy = fminf(fmaxf(gyf - (float)ly, 0.0f), 1.0f);
    const float tscale = a.src_scale / a.dst_scale;
    for (int corner = 0; corner < 4; ++corner) {
        if ((perm & (1u << corner)) == 0u) continue;
        const int ox = corner & 1, oy = corner >> 1;
        const int sx = lx + ox, sy = ly + oy;
        if (sx >= a.src_grid_w || sy >= a.src_grid_h) continue;
        const float wx = ox ? fx : 1.0f - fx, wy = oy ? fy : 1.0f - fy;
        const float spx = fmaf(a.subset_stride, (float)sx, 0.5f * a.subset_size);
        const float spy = fmaf(a.subset_stride, (float)sy, 0.5f * a.subset_size);
        accumulate_seed(a, sy * a.src_grid_w + sx, wx * wy, spx, spy, scx, scy, tscale, acc, wsum);
    }
    const unsigned fallback = perm >> 5;
    if (wsum == 0.0f && fallback != 0u) {
        const int sidx = (int)fallback - 1;
        const float st = a.source[(size_t)sidx * state_stride(a.model) + status_slot(a.model)];
        if (st >= 0.5f) {
            const int sx = sidx % a.src_grid_w, sy = sidx / a.src_grid_w;
            const float spx = fmaf(a.subset_stride, (float)sx, 0.5f * a.subset_size);
            const float spy = fmaf(a.subset_stride, (float)sy, 0.5f * a.subset_size);
            accumulate_seed(a, sidx, 1.0f, spx, spy, scx, scy, tscale, acc, wsum);
        }
    }
    if (wsum > 0.0f)
        for (int k = 0; k < 12; ++k) acc[k] = acc[k] / wsum;
    return wsum;
}

// full_pyramid.wgsl:397-450 (transfer_seed, transfer_seed_roi and, with a
// projection counter, project_temporal_seed).
__global__ void transfer_seed_kernel(SeedArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool projected = false;
    if (i < a.dst_count) {
        const unsigned perm = a.links ? a.links[i] : 31u;
        float acc[12];
        int lx, ly;
        const float wsum = interpolate_seed(a, i, perm, acc, lx, ly);
        float4 *d = reinterpret_cast<float4 *>(a.seed + (size_t)i * state_stride(a.model));
        d[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
        if (a.model == kModelQuadratic) {
            d[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
            d[2] = make_float4(acc[8], acc[9], acc[10], acc[11]);
            d[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        } else {
            d[1] = make_float4(acc[4], acc[5], 0.0f, 0.0f);
        }
        projected = wsum > 0.0f && (perm & 16u) != 0u;
        float *status = a.seed + (size_t)i * state_stride(a.model) + status_slot(a.model);
        if (a.track) *status = wsum >= 0.99999f ? 0.0f : -1.0f;
        if (a.mark_missing && wsum == 0.0f) *status = -1.0f;
        if (a.track && a.projected && !projected) *status = -1.0f;
        a.active[i] = (perm >> 4) & 1u;
    }
    if (a.projected) {
        const int count = __syncthreads_count(projected);
        if (threadIdx.x == 0 && count > 0) atomicAdd(a.projected, (unsigned)count);
    }
}

// full_pyramid.wgsl:452-506.  Runs after the ordinary coarse-to-fine
// transfer into `seed` (with availability markers); `source` is the coarse
// accepted history, `history` the fine one.
__global__ void refine_temporal_seed_kernel(SeedArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.dst_count) return;
    if (a.active[i] == 0u) return;
    const unsigned age = a.history_ages[i];
    if (age == 0xffffffffu || age > a.max_age) return;
    const int ss = state_stride(a.model);
    float *seed = a.seed + (size_t)i * ss;
    if (seed[status_slot(a.model)] < -0.5f) return;
    const unsigned perm = a.links ? a.links[i] : 31u;
    float predicted[12];
    int lx, ly;
    // The lower corner is the one interpolate_seed uses; every permitted
    // corner's coarse history must date from the fine history's frame.
    const float wsum = interpolate_seed(a, i, perm, predicted, lx, ly);
    for (int corner = 0; corner < 4; ++corner) {
        if ((perm & (1u << corner)) == 0u) continue;
        const int sx = lx + (corner & 1), sy = ly + (corner >> 1);
        if (sx >= a.src_grid_w || sy >= a.src_grid_h) continue;
        if (a.source_ages[sy * a.src_grid_w + sx] != age) return;
    }
    if (wsum < 0.99999f) return;
    const float *h = a.history + (size_t)i * ss;
    // a = (tu, ux, uy, tv), b.xy = (vx, vy); quadratic: b.zw and c are the
    // curvature terms.  Markers and iteration slots keep the transfer's.
    const int n = a.model == kModelQuadratic ? 12 : 6;
    for (int k = 0; k < n; ++k) seed[k] = h[k] + (seed[k] - predicted[k]);
}

// ------------------------------------------------------------ temporal
// States move as vectors: a row of NV = 2 (translation, affine) or 4 (quadratic)
// float4, all of a subset's rows loaded together.  A float at a time these were
// chains of strided loads: UHD (127,359 subsets) prediction 11-15 us -> 2.9,
// previous history 7.7 -> 3.1, merge 6.9 -> 3.2.
template <int NV>
__device__ __forceinline__ float row_status(const float4 (&v)[NV]) {
    return NV == 4 ? v[3].x : v[1].z;  // status_slot 12 or 6
}

template <int NV>
__device__ __forceinline__ void load_row(float4 (&v)[NV], const float *states, int i) {
#pragma unroll
    for (int k = 0; k < NV; ++k) v[k] = reinterpret_cast<const float4 *>(states)[(size_t)i * NV + k];
}

template <int NV>
__device__ __forceinline__ void store_row(float *states, int i, const float4 (&v)[NV]) {
#pragma unroll
    for (int k = 0; k < NV; ++k) reinterpret_cast<float4 *>(states)[(size_t)i * NV + k] = v[k];
}

// full_pyramid.wgsl:83-122 velocity prediction into `prediction`.
template <int NV>
__global__ void temporal_predict_kernel(TemporalArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool predicted = false;
    if (i < a.count) {
        float4 c[NV], p[NV];
        load_row(c, a.history, i);
        load_row(p, a.prev_history, i);
        predicted = a.ages[i] == 0u && a.prev_ages[i] == 0u && row_status(c) >= 0.5f && row_status(p) >= 0.5f;
        if (predicted) {
            // the last vector keeps its status and iterations (quadratic: all of it)
#pragma unroll
            for (int k = 0; k < (NV == 4 ? 3 : 2); ++k) {
                c[k].x = fmaf(2.0f, c[k].x, -p[k].x);
                c[k].y = fmaf(2.0f, c[k].y, -p[k].y);
                if (NV == 4 || k == 0) {
                    c[k].z = fmaf(2.0f, c[k].z, -p[k].z);
                    c[k].w = fmaf(2.0f, c[k].w, -p[k].w);
                }
            }
        }
        store_row(a.prediction, i, c);
    }
    const int count = __syncthreads_count(predicted);
    if (threadIdx.x == 0 && count > 0) atomicAdd(a.counters + 2, (unsigned)count);
}

// full_pyramid.wgsl:126-148
template <int NV>
__global__ void temporal_save_previous_kernel(TemporalArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.count) return;
    constexpr int ss = 4 * NV, sat = NV == 4 ? 12 : 6;
    const float rs = a.raw[(size_t)i * ss + sat], fs = a.output[(size_t)i * ss + sat];
    float4 h[NV];
    load_row(h, a.history, i);
    const unsigned current = a.ages[i], previous = a.prev_ages[i];
    if ((rs == 1.0f || rs == 2.0f) && (fs == 1.0f || fs == 2.0f)) {
        store_row(a.prev_history, i, h);
        a.prev_ages[i] = current;
    } else if (previous != 0xffffffffu) {
        a.prev_ages[i] = (previous < 0xfffffffdu ? previous : 0xfffffffdu) + 1u;
    }
}

// full_pyramid.wgsl:508-575
template <int NV>
__global__ void temporal_merge_kernel(TemporalArgs a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    bool accepted = false, expired = false;
    if (i < a.count) {
        constexpr int ss = 4 * NV, sat = NV == 4 ? 12 : 6;
        float4 src[NV];
        load_row(src, a.use_filtered ? a.output : a.raw, i);
        const float rs = a.raw[(size_t)i * ss + sat], fs = a.output[(size_t)i * ss + sat];
        const unsigned current = a.ages[i];
        const bool raw_ok = rs == 1.0f || rs == 2.0f, fin_ok = fs == 1.0f || fs == 2.0f;
        if (fin_ok && (a.use_filtered || raw_ok)) {
            store_row(a.history, i, src);
            a.ages[i] = 0u;
            accepted = true;
        } else if (current != 0xffffffffu) {
            const unsigned age = (current < 0xfffffffdu ? current : 0xfffffffdu) + 1u;
            a.ages[i] = age;
            if (age > a.max_age) {
                a.history[(size_t)i * ss + sat] = -1.0f;
                expired = age == a.max_age + 1u;
            }
        }
    }
    const int na = __syncthreads_count(accepted);
    const int ne = __syncthreads_count(expired);
    if (threadIdx.x == 0 && a.counters) {
        if (na > 0) atomicAdd(a.counters + 1, (unsigned)na);
        if (ne > 0 && a.report_expiry) atomicAdd(a.counters + 3, (unsigned)ne);
    }
}
static_assert(state_stride(kModelAffine) == 8 && status_slot(kModelAffine) == 6 && state_stride(kModelTranslation) == 8 &&
                  status_slot(kModelTranslation) == 6 && state_stride(kModelQuadratic) == 16 &&
                  status_slot(kModelQuadratic) == 12, "rows of vectors");

}  // namespace

cudaError_t launch_final_zncc(const ZnccArgs &a, cudaStream_t stream) {
    if (a.count <= 0) return cudaSuccess;
    if (a.band.rows > 0) {
        SolveArgs b{};
        b.coef = a.coef;
        b.state = const_cast<float *>(a.state);
        b.W = a.W; b.H = a.H; b.grid_w = a.grid_w; b.count = a.count; b.S = a.S; b.stride = a.stride;
        b.band = a.band;
        final_zncc_band_kernel<<<(a.count + 3) / 4, 128, 4 * (size_t)a.band.pitch * sizeof(float), stream>>>(
            b, a.plane_f ? a.plane_f : reinterpret_cast<const float *>(a.plane), a.plane_f ? 1 : 4, a.out);
        return cudaGetLastError();
    }
    const int grid = (a.count + 1) / 2;
    switch (a.interp) {
    case kInterpLinear: final_zncc_kernel<kInterpLinear><<<grid, 128, 0, stream>>>(a); break;
    case kInterpKeys: final_zncc_kernel<kInterpKeys><<<grid, 128, 0, stream>>>(a); break;
    default: final_zncc_kernel<kInterpBspline><<<grid, 128, 0, stream>>>(a); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_reduce_half(const uint8_t *src, int W, int H, uint8_t *dst, cudaStream_t stream) {
    const int W2 = W / 2, H2 = H / 2;
    if (W2 <= 0 || H2 <= 0) return cudaSuccess;
    const int cx = 32 * kRX, cy = 4 * kRY;
    const dim3 grid((W2 + cx - 1) / cx, (H2 + cy - 1) / cy), block(32, 4);
    if ((W & 3) == 0 && (reinterpret_cast<uintptr_t>(src) & 3) == 0)
        reduce_half_kernel<true><<<grid, block, 0, stream>>>(src, W, H, dst);
    else
        reduce_half_kernel<false><<<grid, block, 0, stream>>>(src, W, H, dst);
    return cudaGetLastError();
}

cudaError_t launch_transfer_seed(const SeedArgs &a, cudaStream_t stream) {
    if (a.dst_count <= 0) return cudaSuccess;
    transfer_seed_kernel<<<(a.dst_count + 255) / 256, 256, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_refine_temporal_seed(const SeedArgs &a, cudaStream_t stream) {
    if (a.dst_count <= 0) return cudaSuccess;
    refine_temporal_seed_kernel<<<(a.dst_count + 255) / 256, 256, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_temporal_predict(const TemporalArgs &a, cudaStream_t stream) {
    const int grid = (a.count + 255) / 256;
    if (a.model == kModelQuadratic) temporal_predict_kernel<4><<<grid, 256, 0, stream>>>(a);
    else temporal_predict_kernel<2><<<grid, 256, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_temporal_save_previous(const TemporalArgs &a, cudaStream_t stream) {
    const int grid = (a.count + 255) / 256;
    if (a.model == kModelQuadratic) temporal_save_previous_kernel<4><<<grid, 256, 0, stream>>>(a);
    else temporal_save_previous_kernel<2><<<grid, 256, 0, stream>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_temporal_merge(const TemporalArgs &a, cudaStream_t stream) {
    const int grid = (a.count + 255) / 256;
    if (a.model == kModelQuadratic) temporal_merge_kernel<4><<<grid, 256, 0, stream>>>(a);
    else temporal_merge_kernel<2><<<grid, 256, 0, stream>>>(a);
    return cudaGetLastError();
}

namespace {

// Every subset seeded with the translation (shift[0], shift[1]) * inv_scale
// (zero gradients), active where ROI-selected.
__global__ void uniform_seed_kernel(float *seed, uint32_t *active, const uint8_t *selected, int count, int ss,
                                    const float *shift, float inv_scale) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    float *s = seed + (size_t)i * ss;
    for (int k = 0; k < ss; ++k) s[k] = 0.0f;
    s[0] = shift[0] * inv_scale;
    s[3] = shift[1] * inv_scale;
    active[i] = selected ? (selected[i] ? 1u : 0u) : 1u;
}

}  // namespace

cudaError_t launch_uniform_seed(float *seed, uint32_t *active, const uint8_t *selected, int count, int model,
                                const float *shift, float inv_scale, cudaStream_t stream) {
    if (count <= 0) return cudaSuccess;
    uniform_seed_kernel<<<(count + 255) / 256, 256, 0, stream>>>(seed, active, selected, count, state_stride(model),
                                                                shift, inv_scale);
    return cudaGetLastError();
}

}  // namespace gbdic
