// A block to a window: IC-GN over partial-support ROI windows, and over the
// complete windows of a launch too small to fill the chip otherwise (reference: solve_partial /
// solve_partial_seeded / retry_partial_seeded, shaders/icgn.wgsl:1042-1085):
// for those, the complete-window solver's iteration with the window's support bits,
// support box and partial metadata (validity -4, partial mean and weight
// sum).  One launch over the partial windows, after the complete-window launch
// of the same frame.
//
// Partial windows are the few along an ROI's edge, so a launch of one group of
// lanes to a window leaves the chip nearly idle and lasts as long as one
// window's chain: every lane took its pixels one after the other, each with its
// taps' latency.  Here a block of 256 threads has the window.  All of them
// sample the supported pixels and leave each pixel's factors in shared memory;
// then lane l of the reference's LANES accumulates its pixels from there in the
// reference's order, the sums dealt out over the 256 / LANES threads that share
// the lane, and one warp takes the update.  Each sum's chain and the reduction
// tree are the reference's, so the result is the same bit for bit.
// 1279 x 717, S 25 / s 12 Gaussian, 349 partial windows, 16 lanes: 208 us ->
// 119 with the factors formed in the accumulation and 128 threads -> 53.
#include "gbdic_kernels.h"
#include "solver_impl.cuh"

namespace gbdic {
namespace {

constexpr int kPartialThreads = 256;
// Complete windows of a launch up to which a block has one too.  Device time of a
// frame, other loops -> blocks (16 lanes): affine B-spline S 21, 324 windows 81 ->
// 73 us, 676 120 -> 110, 1,156 126 -> 133; S 31 88 -> 58, 103 -> 77, 101 -> 92,
// 1,764 134 -> 127, 2,704 128 -> 161; affine linear S 21 (direct loop) 676 98 -> 64,
// 1,764 124 -> 93, 2,704 125 -> 119, 4,356 138 -> 154; translation linear S 15 676
// 73 -> 53, 1,764 75 -> 66, 2,704 77 -> 79.
constexpr int kBlockWindowsBspline = 912, kBlockWindows = 2128;
// Pixels sampled between two accumulations: a multiple of the lane counts (lanes
// keep their pixels); a whole window up to S = 32.  The arrays' pitch puts the
// two halves of a warp, which read different arrays, on different banks.
constexpr int kPartialChunk = 1024, kPartialPitch = kPartialChunk + 16;
// Factors of a pixel: weighted g and f, weighted g times the two gradients, g,
// and the local coordinates.
enum { kWc, kWf, kGxg, kGyg, kG, kLx, kLy, kFactors };

// Running (column, row, plane index) of pixels p, p + STEP, ... of a window.
template <int STEP>
struct PixelWalk {
    float col, row, size, dcol, drow;
    unsigned index, step, wrap;
    __device__ __forceinline__ PixelWalk(int p, int S, int W, unsigned origin) {
        const int r = p / S, c = p % S;
        col = (float)c;
        row = (float)r;
        size = (float)S;
        dcol = (float)(STEP % S);
        drow = (float)(STEP / S);
        index = origin + (unsigned)r * (unsigned)W + (unsigned)c;
        step = (unsigned)(STEP % S) + (unsigned)(STEP / S) * (unsigned)W;
        wrap = (unsigned)(W - S);
    }
    __device__ __forceinline__ void next() {
        col += dcol;
        row += drow;
        index += step;
        if (col >= size) { col -= size; row += 1.0f; index += wrap; }
    }
};

// Sum k of accumulate_values is s = fma(x, y, s) of two of a pixel's factors (y
// one: a plain addition).
template <int MODEL>
__device__ __forceinline__ int factor_x(int k) {
    if (MODEL == kModelTranslation) return k < 2 ? kWc : k == 2 ? kWf : k == 3 ? kGxg : kGyg;
    return k < 2 ? kWc : k == 2 ? kWf : k < 6 ? kGxg : kGyg;
}
template <int MODEL>
__device__ __forceinline__ int factor_y(int k) {  // -1: one
    if (k == 1 || k == 2) return kG;
    if (MODEL == kModelTranslation) return -1;
    return k == 4 || k == 7 ? kLx : k == 5 || k == 8 ? kLy : -1;
}

template <int MODEL, int INTERP, int LANES, bool GAUSS, bool PART>
__global__ void __launch_bounds__(kPartialThreads) window_block_kernel(SolveArgs a) {
    constexpr int N = SumCount<MODEL>::value, PARTS = kPartialThreads / LANES, PER = (N + PARTS - 1) / PARTS;
    constexpr int n = parameter_count(MODEL), META = meta_stride(MODEL);
    __shared__ float factors[kFactors * kPartialPitch];
    __shared__ float red[N * LANES];
    __shared__ float md[META], hi[n * n];
    __shared__ float update[8];
    const int tid = threadIdx.x, lane = tid % LANES, part = tid / LANES;
    const int group = blockIdx.x, idx = PART ? __ldg(a.partial_index + group) : group;
    const uint32_t *support = PART ? a.support + (size_t)group * a.support_words : nullptr;
    const float4 box = PART ? __ldg(a.support_box + group) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (int i = tid; i < META + n * n; i += kPartialThreads) {
        if (i < META) md[i] = __ldg(a.meta + (size_t)idx * META + i);
        else hi[i - META] = __ldg(a.inv + (size_t)idx * n * n + i - META);
    }
    Warp w = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    bool enabled = true;
    if (a.seed != nullptr) {
        const float4 *s = reinterpret_cast<const float4 *>(a.seed + (size_t)idx * state_stride(MODEL));
        const float4 s0 = __ldg(s), s1 = __ldg(s + 1);
        w.t0 = s0.x; w.l0 = s0.y; w.l1 = s0.z; w.t1 = s0.w;
        w.l2 = s1.x; w.l3 = s1.y;
        enabled = __ldg(a.active + idx) != 0u;
    }
    if (MODEL == kModelTranslation) { w.l0 = w.l1 = w.l2 = w.l3 = 0.0f; }
    __syncthreads();
    const bool valid = enabled && (PART ? md[1] == -4.0f : md[1] >= 0.5f);
    float status = valid ? 0.0f : !PART && a.roi_enabled ? fminf(-1.0f, md[1]) : -1.0f;
    float iters = 0.0f;
    const int S = a.S, npix = S * S, W = a.W, H = a.H;
    const int px0 = (idx % a.grid_w) * a.stride, py0 = (idx / a.grid_w) * a.stride;
    const unsigned origin = (unsigned)py0 * (unsigned)W + (unsigned)px0;
    const float half = 0.5f * ((float)S - 1.0f), ox = (float)px0 + half, oy = (float)py0 + half;
    const float ref_mean = PART || a.use_mean ? md[14] : 0.0f;
    const float wsum = PART || GAUSS ? md[3 + 2 * n] : (float)(S * S);
    float prev_change = 3.402823e38f;
    unsigned stalled = 0u;

    for (int it = 0; it < 30; ++it) {  // the block's threads hold the same state
        if (!(a.div_patience != 0 && status == 3.0f)) {
            if (!(PART ? warp_inside_box<MODEL>(w, px0, py0, half, box, W, H)
                       : warp_inside<MODEL>(w, px0, py0, S, half, W, H))) {
                if (!a.roi_enabled || status > -2.5f) status = -1.0f;
            }
        }
        if (it >= a.iterations || fabsf(status) > 0.5f) break;
        float s[PER];
#pragma unroll
        for (int k = 0; k < PER; ++k) s[k] = 0.0f;
        for (int base = 0; base < npix; base += kPartialChunk) {
            const int count = min(npix - base, kPartialChunk);
            if (base > 0) __syncthreads();
            PixelWalk<kPartialThreads> q(base + tid, S, W, origin);
#pragma unroll 2
            for (int i = tid; i < count; i += kPartialThreads, q.next()) {
                const int p = base + i;
                const float lx = q.col - half, ly = q.row - half;
                float wc = 0.0f, wf = 0.0f, gxg = 0.0f, gyg = 0.0f, g = 0.0f;
                if (!PART || ((__ldg(support + (p >> 5)) >> (p & 31)) & 1u)) {
                    const float4 rv = __ldg(a.plane + q.index);
                    const float wt = GAUSS ? __ldg(a.weights + p) : 1.0f, f = rv.x - ref_mean;
                    float dx, dy;
                    displacement<MODEL>(w, lx, ly, 0.0f, 0.0f, 0.0f, dx, dy);
                    g = sample_target<INTERP, false>(a.coef, a.img, W, H, (ox + lx) + dx, (oy + ly) + dy);
                    wc = GAUSS ? wt * g : g;
                    wf = GAUSS ? wt * f : f;
                    gxg = rv.y * wc;
                    gyg = rv.z * wc;
                }
                // Factors of zero leave a sum as it is (no sum is -0).
                float *o = factors + i;
                o[kWc * kPartialPitch] = wc;
                o[kWf * kPartialPitch] = wf;
                o[kGxg * kPartialPitch] = gxg;
                o[kGyg * kPartialPitch] = gyg;
                o[kG * kPartialPitch] = g;
                o[kLx * kPartialPitch] = lx;
                o[kLy * kPartialPitch] = ly;
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int k = part + PARTS * j;
                if (k >= N) continue;
                const int fy = factor_y<MODEL>(k);
                const float *x = factors + factor_x<MODEL>(k) * kPartialPitch;
                const float *y = factors + (fy < 0 ? 0 : fy) * kPartialPitch;
                float v = s[j];
#pragma unroll 8
                for (int i = lane; i < count; i += LANES) v = fmaf(x[i], fy < 0 ? 1.0f : y[i], v);
                s[j] = v;
            }
        }
        // The tree over the window's lanes: from shared memory down to a warp,
        // then shuffles.
        if constexpr (LANES > 32) {
#pragma unroll
            for (int j = 0; j < PER; ++j) {
                const int k = part + PARTS * j;
                if (k < N) red[k * LANES + lane] = s[j];
            }
            __syncthreads();
#pragma unroll
            for (int stride = LANES / 2; stride >= 32; stride >>= 1) {
#pragma unroll
                for (int j = 0; j < PER; ++j) {
                    const int k = part + PARTS * j;
                    if (k >= N) continue;
                    if (lane < stride) s[j] = red[k * LANES + lane] + red[k * LANES + lane + stride];
                    if (stride > 32 && lane < stride) red[k * LANES + lane] = s[j];
                }
                __syncthreads();
            }
        }
#pragma unroll
        for (int j = 0; j < PER; ++j) {
            const int k = part + PARTS * j;
#pragma unroll
            for (int off = (LANES > 32 ? 32 : LANES) / 2; off >= 1; off >>= 1)
                s[j] = s[j] + __shfl_down_sync(kFullMask, s[j], off, LANES > 32 ? 32 : LANES);
            if (lane == 0 && k < N) red[k * LANES] = s[j];
        }
        __syncthreads();
        if (tid < 32) {
            float total[N];
#pragma unroll
            for (int k = 0; k < N; ++k) total[k] = red[k * LANES];
            status = gn_update<MODEL, true>(a, total, md, hi, wsum, half, (unsigned)(it + 1), w, prev_change, stalled,
                                            0, 0u);
            if (tid == 0) {
                update[0] = w.t0; update[1] = w.l0; update[2] = w.l1; update[3] = w.t1;
                update[4] = w.l2; update[5] = w.l3; update[6] = status;
            }
        }
        __syncthreads();
        w.t0 = update[0]; w.l0 = update[1]; w.l1 = update[2]; w.t1 = update[3];
        w.l2 = update[4]; w.l3 = update[5];
        status = update[6];
        iters = (float)(it + 1);
    }
    if (tid != 0) return;
    if (a.iteration_total != nullptr && iters > 0.0f) atomicAdd(a.iteration_total, (unsigned long long)iters);
    if (enabled || !a.preserve_disabled) {
        const float final_status = (a.div_patience != 0 && status == 3.0f) ? 0.0f : status;
        float4 *o = reinterpret_cast<float4 *>(a.state + (size_t)idx * state_stride(MODEL));
        o[0] = make_float4(w.t0, w.l0, w.l1, w.t1);
        o[1] = make_float4(w.l2, w.l3, final_status, iters);
    }
}

template <int MODEL, int INTERP, int LANES, bool GAUSS>
cudaError_t go(const SolveArgs &a, cudaStream_t s) {
    if (a.partial_index != nullptr)
        window_block_kernel<MODEL, INTERP, LANES, GAUSS, true><<<a.count, kPartialThreads, 0, s>>>(a);
    else
        window_block_kernel<MODEL, INTERP, LANES, GAUSS, false><<<a.count, kPartialThreads, 0, s>>>(a);
    return cudaGetLastError();
}

template <int MODEL, int INTERP, bool GAUSS>
cudaError_t by_lanes(const SolveArgs &a, int lanes, cudaStream_t s) {
    switch (lanes) {
    case 16: return go<MODEL, INTERP, 16, GAUSS>(a, s);
    case 32: return go<MODEL, INTERP, 32, GAUSS>(a, s);
    case 64: return go<MODEL, INTERP, 64, GAUSS>(a, s);
    case 128: return go<MODEL, INTERP, 128, GAUSS>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int MODEL, bool GAUSS>
cudaError_t by_interp(const SolveArgs &a, int interp, int lanes, cudaStream_t s) {
    switch (interp) {
    case kInterpBspline: return by_lanes<MODEL, kInterpBspline, GAUSS>(a, lanes, s);
    case kInterpLinear: return by_lanes<MODEL, kInterpLinear, GAUSS>(a, lanes, s);
    case kInterpKeys: return by_lanes<MODEL, kInterpKeys, GAUSS>(a, lanes, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int MODEL>
cudaError_t by_weight(const SolveArgs &a, int interp, int lanes, bool gauss, cudaStream_t s) {
    return gauss ? by_interp<MODEL, true>(a, interp, lanes, s) : by_interp<MODEL, false>(a, interp, lanes, s);
}

}  // namespace

bool icgn_blocks_fit(const SolveArgs &a, int model, int interp, int lanes) {
    return model != kModelQuadratic && lanes <= 32 && !a.persistent && a.subset_list == nullptr &&
           a.list_count == nullptr && a.count <= (interp == kInterpBspline ? kBlockWindowsBspline : kBlockWindows);
}

cudaError_t launch_icgn_blocks(const SolveArgs &args, int model, int interp, int lanes, bool gauss, cudaStream_t stream) {
    return model == kModelAffine ? by_weight<kModelAffine>(args, interp, lanes, gauss, stream)
                                 : by_weight<kModelTranslation>(args, interp, lanes, gauss, stream);
}

cudaError_t launch_icgn_partial(const SolveArgs &args, int model, int interp, int lanes, bool gauss,
                                cudaStream_t stream) {
    if (args.count <= 0) return cudaSuccess;
    if (!args.partial_index || !args.support || !args.support_box || args.support_words <= 0)
        return cudaErrorInvalidValue;
    switch (model) {
    case kModelAffine: return by_weight<kModelAffine>(args, interp, lanes, gauss, stream);
    case kModelTranslation: return by_weight<kModelTranslation>(args, interp, lanes, gauss, stream);
    default: return cudaErrorInvalidValue;  // the ROI supports translation and affine windows only
    }
}

}  // namespace gbdic
