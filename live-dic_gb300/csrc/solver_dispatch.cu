// Launch geometry and dispatch of the IC-GN solver variants.
#include "gbdic_kernels.h"
#include "solver_band.cuh"

namespace gbdic {

int icgn_grid(int count, int lanes) {
    if (count <= 0) return 0;
    if (lanes > 32) {
        const int groups = 128 / lanes;  // subsets per block
        return (count + groups - 1) / groups;
    }
    const int per_warp = 32 / lanes;
    const int units = (count + per_warp - 1) / per_warp;  // warps
    return (units + 3) / 4;                                // 4 warps per block
}

namespace {

// Every subset's row as the seeded solver writes it for a disabled subset
// (solver_impl.cuh solve_group: the seed's warp, status `rejected`, zero
// iterations; preserve_disabled off).  List-mode solves write this first so
// that the rows they do not list equal the full-grid solve's.
template <int MODEL>
__global__ void disabled_rows_kernel(SolveArgs a, int total) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= total) return;
    const float4 *s = reinterpret_cast<const float4 *>(a.seed + (size_t)idx * state_stride(MODEL));
    const float4 s0 = __ldg(s), s1 = __ldg(s + 1);
    const bool translation = MODEL == kModelTranslation;
    const float mvalid = __ldg(a.meta + (size_t)idx * meta_stride(MODEL) + 1);
    const bool valid = __ldg(a.active + idx) != 0u && mvalid >= 0.5f;
    const float rejected = a.roi_enabled ? fminf(-1.0f, mvalid) : -1.0f;
    const float status = valid ? 0.0f : rejected;
    float4 *o = reinterpret_cast<float4 *>(a.state + (size_t)idx * state_stride(MODEL));
    o[0] = make_float4(s0.x, translation ? 0.0f : s0.y, translation ? 0.0f : s0.z, s0.w);
    if (MODEL == kModelQuadratic) {
        const float4 s2 = __ldg(s + 2);
        o[1] = make_float4(s1.x, s1.y, s1.z, s1.w);
        o[2] = s2;
        o[3] = make_float4(status, 0.0f, 0.0f, 0.0f);
    } else {
        o[1] = make_float4(translation ? 0.0f : s1.x, translation ? 0.0f : s1.y, status, 0.0f);
    }
}

cudaError_t dispatch(const SolveArgs &a, int model, int interp, int lanes, bool gauss, int grid,
                     cudaStream_t stream, int *occupancy_only) {
    switch (model) {
    case kModelAffine:
        return launch_icgn_model<kModelAffine>(a, interp, lanes, gauss, grid, stream, occupancy_only);
    case kModelTranslation:
        return launch_icgn_model<kModelTranslation>(a, interp, lanes, gauss, grid, stream, occupancy_only);
    case kModelQuadratic:
        return launch_icgn_model<kModelQuadratic>(a, interp, lanes, gauss, grid, stream, occupancy_only);
    default:
        return cudaErrorInvalidValue;
    }
}
}  // namespace

// Run length of one band of `rows` x S pixels walked by `samplers` lanes, and
// its steps: runs are walked two to a lane, and each costs three quarters of
// a step more for its first taps.
static double band_steps(int S, int rows, int samplers, int &run, int &segments) {
    double best = 1e30;
    for (int r = 1; r <= rows; ++r) {
        const int s = (rows + r - 1) / r, phases = (S * s + 2 * samplers - 1) / (2 * samplers);
        const double cost = phases * (r + 0.75) + 0.5;
        if (cost < best) {
            best = cost;
            run = r;
            segments = s;
        }
    }
    return best;
}

BandPlan plan_bands(int S, int model, int interp, int lanes, bool gauss, int sm_count) {
    BandPlan best{};
    if (interp != kInterpBspline || lanes > 32 || S > kMaxBandFloats) return best;
    double steps = 1e30;
    for (int bands = 1; bands <= S; ++bands) {
        const int rows = (S + bands - 1) / bands;
        if (rows * S > kMaxBandFloats) continue;
        int run = 0, segments = 0;
        const double cost = (S + rows - 1) / rows * band_steps(S, rows, lanes, run, segments);
        if (cost < steps) {
            steps = cost;
            best.rows = rows;
            best.run = run;
            best.segments = segments;
        }
    }
    // Against the direct loop's S^2 / (2 lanes) steps.  Measured at 2560 x
    // 1440 (band / direct time): affine 16 lanes 0.89 at a ratio of 1.07
    // (S 31), 0.94 at 1.20 (S 41), 1.00 at 1.26 (S 51), 1.03 at 1.34 (S 33),
    // 1.08 at 1.49 (S 65); 32 lanes 0.95 at 1.31 (S 16), 1.02 at 1.35 (S 51);
    // translation and quadratic 0.82 and 0.85 at 1.49, and with 32 lanes 1.11
    // and 1.04 at 1.70.  Affine plans of several bands lose their lead sooner,
    // with Gaussian weights (which the direct loop loads beside the plane, the
    // banded one with its pixel table) later.  8,800 windows, band / direct,
    // uniform and Gaussian: 16 lanes 0.99 and 0.83 at 1.20 (S 41), 1.04 and 0.90
    // at 1.23 (S 45); 32 lanes 0.96 and 0.90 at 1.22 (S 41), 1.03 and 0.96 at 1.29
    // (S 55), 1.02 and 0.95 at 1.31 (S 45), 1.13 and 1.04 at 1.33 (S 81).
    const bool several = best.rows < S;
    const double limit = model != kModelAffine ? 1.6
                         : lanes == 16         ? (several && !gauss ? 1.21 : 1.25)
                                               : (several ? (gauss ? 1.32 : 1.25) : 1.34);
    if (steps * 2 * lanes > limit * S * S) return BandPlan{};
    band_steps(S, best.rows, 32, best.run32, best.segments32);
    best.magic = ((1u << 20) + S - 1) / S;
    best.pitch = (best.rows * S + 15) / 32 * 32 + 16;  // groups of one warp start 16 banks apart
    if (lanes == 16) best.solo_count = sm_count * 4 * (model == kModelQuadratic ? kBandQuadBlocks : kBandBlocks);
    return best;
}

// The final ZNCC samples a window once, with all lanes of a warp; its direct
// kernel is slower at every size (no limit on the steps).
BandPlan zncc_bands(int S, int interp) {
    BandPlan best{};
    if (interp != kInterpBspline || S > kMaxBandFloats) return best;
    double steps = 1e30;
    for (int bands = 1; bands <= S; ++bands) {
        const int rows = (S + bands - 1) / bands;
        if (rows * S > kMaxBandFloats) continue;
        int run = 0, segments = 0;
        const double cost = (S + rows - 1) / rows * band_steps(S, rows, 32, run, segments);
        if (cost < steps) {
            steps = cost;
            best.rows = rows;
            best.run = best.run32 = run;
            best.segments = best.segments32 = segments;
        }
    }
    best.magic = ((1u << 20) + S - 1) / S;
    best.pitch = (best.rows * S + 31) / 32 * 32;
    return best;
}

// CTAs of a non-persistent launch of the banded loop.
int icgn_band_grid(const SolveArgs &a, int lanes) {
    const int per_warp = lanes == 16 && a.count > a.band.solo_count ? 2 : 1;
    return ((a.count + per_warp - 1) / per_warp + 3) / 4;
}

int icgn_occupancy(int model, int interp, int lanes, bool gauss, int S, const BandPlan &band) {
    SolveArgs unused{};
    unused.S = S;
    unused.band = band;
    int blocks = 0;
    if (dispatch(unused, model, interp, lanes, gauss, 0, nullptr, &blocks) != cudaSuccess) return 0;
    return blocks;
}

int icgn_fast_occupancy(int model, int lanes, bool gauss) {
    SolveArgs unused{};
    int blocks = 0;
    if (launch_icgn_fast(unused, model, lanes, gauss, 0, nullptr, &blocks) != cudaSuccess) return 0;
    return blocks;
}

cudaError_t launch_disabled_rows(const SolveArgs &a, int model, int total, cudaStream_t stream) {
    if (total <= 0) return cudaSuccess;
    const int grid = (total + 255) / 256;
    switch (model) {
    case kModelAffine: disabled_rows_kernel<kModelAffine><<<grid, 256, 0, stream>>>(a, total); break;
    case kModelTranslation: disabled_rows_kernel<kModelTranslation><<<grid, 256, 0, stream>>>(a, total); break;
    case kModelQuadratic: disabled_rows_kernel<kModelQuadratic><<<grid, 256, 0, stream>>>(a, total); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t launch_icgn(const SolveArgs &a, int model, int interp, int lanes, bool gauss,
                        int persistent_grid, cudaStream_t stream) {
    if (a.count <= 0) return cudaSuccess;
    const int grid = a.persistent ? persistent_grid : icgn_grid(a.count, lanes);
    if (grid <= 0) return cudaErrorInvalidConfiguration;
    if (a.fast_segments > 0 && icgn_fast_supported(model, interp, lanes))
        return launch_icgn_fast(a, model, lanes, gauss, grid, stream, nullptr);
    if (a.staged_tile > 0 && icgn_staged_supported(model, interp, lanes, a.W))
        return launch_icgn_staged(a, model, lanes, gauss, a.staged_tile, grid, stream, nullptr);
    if (icgn_blocks_fit(a, model, interp, lanes)) return launch_icgn_blocks(a, model, interp, lanes, gauss, stream);
    return dispatch(a, model, interp, lanes, gauss, grid, stream, nullptr);
}

}  // namespace gbdic
