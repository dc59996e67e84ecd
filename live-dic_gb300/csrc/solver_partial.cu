// IC-GN over partial-support ROI windows (reference: solve_partial /
// solve_partial_seeded / retry_partial_seeded, shaders/icgn.wgsl:1042-1085):
// the complete-window solver's iteration with the window's support bits,
// support box and partial metadata (validity -4, partial mean and weight
// sum).  One launch over the partial windows, after the complete-window launch
// of the same frame.  Few windows, partial or complete, take a block each.
//
// A launch of few windows with one group of lanes to a window leaves the chip
// nearly idle and lasts as long as one window's chain: every lane takes its
// pixels one after the other, each with its taps' latency.  A block of 256
// threads to a window shortens the chain.  All of them sample the supported
// pixels and leave each pixel's factors in shared memory; then lane l of the
// reference's LANES accumulates its pixels from there in the reference's
// order, the sums dealt out over the 256 / LANES threads that share the lane,
// and one warp takes the update.  Each sum's chain and the reduction tree are
// the reference's, so the result is the same bit for bit.  Where there are
// many windows, or a lane has few pixels, the block's synchronisations cost
// more than the shorter chain gives (kBlockRule).
// 1279 x 717, S 25 / s 12 Gaussian, 349 partial windows, 16 lanes: 208 us ->
// 119 with the factors formed in the accumulation and 128 threads -> 53.
#include "gbdic_kernels.h"
#include "solver_impl.cuh"

namespace gbdic {
namespace {

constexpr int kPartialThreads = 256;
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

// Windows up to which a block each is faster than a group of lanes each: per SM
// gain * (pixels - start)^2, at most `most`, where `pixels` are a lane's (the
// chain that a block shortens) and `start` those that its synchronisations
// outweigh.  Fitted to measurements over S 5 to 81, 9 to 4,096 complete and 15 to
// 6,300 partial windows: of 5,000 frames 84 are over 3 % slower than the better
// of the two.  The measured device times of a frame (with its prefilter), a group
// of lanes each : a block each, affine, us:
//   complete, 16 lanes   B-spline S 9    196 windows  72 : 70         900  75 : 108
//                                 S 15   900         112 : 114      2,116  127 : 164
//                                 S 31   900         102 : 69       2,116  103 : 107
//                        linear   S 9    196          55 : 57       2,116  61 : 158
//                                 S 31   900          83 : 45       3,364  110 : 113
//                        cubic    S 15   900         130 : 92       4,096  218 : 227
//   complete, 32 lanes   B-spline S 15   196          75 : 70         900  88 : 113
//                                 S 31   900          80 : 73       1,444  81 : 92
//                        linear   S 15   196          58 : 65       2,116  75 : 132
//   partial, 16 lanes    B-spline S 9  1,007          95 : 135         S 15  999  161 : 113
//                        linear   S 9  1,006          68 : 111         S 15  999  107 : 89
//   partial, 32 lanes    B-spline S 9  1,007          81 : 143         S 31  988  134 : 82
//   partial, 64 lanes    B-spline S 9    391          94 : 93          S 31  988  100 : 85
//                                 S 9  1,007         109 : 155         S 31  2,268  135 : 151
// 128 lanes: partial windows 0.95 to 1.5 times as long by blocks; complete windows
// of 64 and 128 lanes have a block's loop in any case.
struct BlockRule {
    float start, gain, most;
};
enum { kComplete16, kComplete32, kPartial16, kPartial32, kPartial64, kBlockRules };
// [launch][affine, translation][B-spline, linear, cubic]
constexpr BlockRule kBlockRule[kBlockRules][2][3] = {
    {{{1.0f, 0.045f, 6.0f}, {1.0f, 0.045f, 14.0f}, {1.0f, 0.12f, 14.0f}},
     {{1.0f, 0.3f, 6.0f}, {2.0f, 0.15f, 14.0f}, {2.0f, 0.4f, 14.0f}}},
    {{{2.0f, 0.06f, 6.0f}, {6.0f, 0.06f, 7.0f}, {2.0f, 0.09f, 10.0f}},
     {{3.0f, 0.7f, 5.0f}, {2.0f, 0.09f, 10.0f}, {3.0f, 1.5f, 10.0f}}},
    {{{0.0f, 0.09f, 42.0f}, {0.0f, 0.06f, 28.0f}, {0.0f, 0.09f, 42.0f}},
     {{0.0f, 0.3f, 42.0f}, {0.0f, 0.15f, 42.0f}, {0.0f, 0.4f, 42.0f}}},
    {{{1.0f, 0.15f, 16.0f}, {2.0f, 0.09f, 16.0f}, {1.0f, 0.15f, 16.0f}},
     {{2.0f, 1.0f, 16.0f}, {2.0f, 0.3f, 16.0f}, {2.0f, 0.7f, 16.0f}}},
    {{{0.0f, 1.5f, 7.0f}, {0.0f, 1.5f, 5.0f}, {0.0f, 1.5f, 5.0f}},
     {{0.0f, 1.5f, 7.0f}, {1.0f, 1.5f, 7.0f}, {1.0f, 1.5f, 3.0f}}},
};

bool block_each(const SolveArgs &a, int model, int interp, int lanes, bool partial) {
    if (model == kModelQuadratic || lanes > (partial ? 64 : 32)) return false;
    const int launch = partial ? (lanes == 16 ? kPartial16 : lanes == 32 ? kPartial32 : kPartial64)
                               : (lanes == 16 ? kComplete16 : kComplete32);
    const BlockRule &r = kBlockRule[launch][model == kModelTranslation ? 1 : 0]
                                   [interp == kInterpBspline ? 0 : interp == kInterpLinear ? 1 : 2];
    const float excess = fmaxf((float)(a.S * a.S) / (float)lanes - r.start, 0.0f);
    return (float)a.count <= fminf(r.gain * excess * excess, r.most) * (float)a.sm_count;
}

// blocks: a block to a window; else a group of LANES lanes to a partial one.
template <int MODEL, int INTERP, int LANES, bool GAUSS>
cudaError_t go(const SolveArgs &a, bool blocks, cudaStream_t s) {
    if (a.partial_index != nullptr && !blocks) {
        icgn_kernel<MODEL, INTERP, LANES, GAUSS, true><<<icgn_grid(a.count, LANES), 128, 0, s>>>(a);
        return cudaGetLastError();
    }
    if constexpr (LANES <= 64) {
        if (a.partial_index != nullptr) {
            window_block_kernel<MODEL, INTERP, LANES, GAUSS, true><<<a.count, kPartialThreads, 0, s>>>(a);
            return cudaGetLastError();
        }
    }
    if constexpr (LANES <= 32) {
        window_block_kernel<MODEL, INTERP, LANES, GAUSS, false><<<a.count, kPartialThreads, 0, s>>>(a);
        return cudaGetLastError();
    }
    return cudaErrorInvalidValue;
}

template <int MODEL, int INTERP, bool GAUSS>
cudaError_t by_lanes(const SolveArgs &a, int lanes, bool blocks, cudaStream_t s) {
    switch (lanes) {
    case 16: return go<MODEL, INTERP, 16, GAUSS>(a, blocks, s);
    case 32: return go<MODEL, INTERP, 32, GAUSS>(a, blocks, s);
    case 64: return go<MODEL, INTERP, 64, GAUSS>(a, blocks, s);
    case 128: return go<MODEL, INTERP, 128, GAUSS>(a, blocks, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int MODEL, bool GAUSS>
cudaError_t by_interp(const SolveArgs &a, int interp, int lanes, bool blocks, cudaStream_t s) {
    switch (interp) {
    case kInterpBspline: return by_lanes<MODEL, kInterpBspline, GAUSS>(a, lanes, blocks, s);
    case kInterpLinear: return by_lanes<MODEL, kInterpLinear, GAUSS>(a, lanes, blocks, s);
    case kInterpKeys: return by_lanes<MODEL, kInterpKeys, GAUSS>(a, lanes, blocks, s);
    default: return cudaErrorInvalidValue;
    }
}

template <int MODEL>
cudaError_t by_weight(const SolveArgs &a, int interp, int lanes, bool gauss, bool blocks, cudaStream_t s) {
    return gauss ? by_interp<MODEL, true>(a, interp, lanes, blocks, s)
                 : by_interp<MODEL, false>(a, interp, lanes, blocks, s);
}

}  // namespace

bool icgn_blocks_fit(const SolveArgs &a, int model, int interp, int lanes) {
    return !a.persistent && a.subset_list == nullptr && a.list_count == nullptr &&
           block_each(a, model, interp, lanes, false);
}

cudaError_t launch_icgn_blocks(const SolveArgs &a, int model, int interp, int lanes, bool gauss, cudaStream_t stream) {
    return model == kModelAffine ? by_weight<kModelAffine>(a, interp, lanes, gauss, true, stream)
                                 : by_weight<kModelTranslation>(a, interp, lanes, gauss, true, stream);
}

cudaError_t launch_icgn_partial(const SolveArgs &args, int model, int interp, int lanes, bool gauss,
                                cudaStream_t stream) {
    if (args.count <= 0) return cudaSuccess;
    if (!args.partial_index || !args.support || !args.support_box || args.support_words <= 0)
        return cudaErrorInvalidValue;
    SolveArgs a = args;
    a.persistent = 0;
    const bool blocks = block_each(a, model, interp, lanes, true);
    switch (model) {
    case kModelAffine: return by_weight<kModelAffine>(a, interp, lanes, gauss, blocks, stream);
    case kModelTranslation: return by_weight<kModelTranslation>(a, interp, lanes, gauss, blocks, stream);
    default: return cudaErrorInvalidValue;  // the ROI supports translation and affine windows only
    }
}

}  // namespace gbdic
