// Displacement outlier detection and median repair (reference:
// shaders/icgn.wgsl:1087-1605).  One thread per subset reads its own state
// and its 3x3 (or up to 9x9) neighbours and writes the filtered state.
// Neighbour warps are Taylor-recentred to the subset centre before their
// medians are taken; medians are order statistics, so any exact selection
// algorithm gives the same values (a bubble network for <= 9 values, Hoare
// quickselect for up to 81).
#include "gbdic_common.cuh"
#include "gbdic_kernels.h"

namespace gbdic {

namespace {

__device__ float median_small(float *v, int count) {
    for (int phase = 0; phase < 9; ++phase)
        for (int i = 0; i < 8; ++i)
            if (i + 1 < count && v[i] > v[i + 1]) {
                float s = v[i];
                v[i] = v[i + 1];
                v[i + 1] = s;
            }
    if (count % 2 == 1) return v[count / 2];
    return 0.5f * (v[count / 2 - 1] + v[count / 2]);
}

__device__ float select_rank(float *v, int count, int rank) {
    int low = 0, high = count - 1;
    for (int guard = 0; guard < 4096; ++guard) {
        if (low >= high) return v[rank];
        const float pivot = v[low + (high - low) / 2];
        int left = low, right = high;
        for (;;) {
            while (left <= high && v[left] < pivot) ++left;
            while (right >= low && v[right] > pivot) --right;
            if (left > right) break;
            float s = v[left];
            v[left] = v[right];
            v[right] = s;
            ++left;
            --right;
        }
        if (rank <= right) high = right;
        else if (rank >= left) low = left;
        else return v[rank];
    }
    return v[rank];
}

__device__ float median_large(float *v, int count) {
    if (count % 2 == 1) return select_rank(v, count, count / 2);
    const float lo = select_rank(v, count, count / 2 - 1);
    const float hi = select_rank(v, count, count / 2);
    return 0.5f * (lo + hi);
}

// Taylor recentring of component `comp` of state s at offset (ox, oy).
__device__ float recentered(int model, const float *s, int comp, float ox, float oy) {
    if (model == kModelQuadratic) {
        switch (comp) {
        case 0: return fmaf(s[8], 0.5f * oy * oy, fmaf(s[7], ox * oy, fmaf(s[6], 0.5f * ox * ox, fmaf(s[2], oy, fmaf(s[1], ox, s[0])))));
        case 1: return fmaf(s[7], oy, fmaf(s[6], ox, s[1]));
        case 2: return fmaf(s[8], oy, fmaf(s[7], ox, s[2]));
        case 3: return fmaf(s[11], 0.5f * oy * oy, fmaf(s[10], ox * oy, fmaf(s[9], 0.5f * ox * ox, fmaf(s[5], oy, fmaf(s[4], ox, s[3])))));
        case 4: return fmaf(s[10], oy, fmaf(s[9], ox, s[4]));
        case 5: return fmaf(s[11], oy, fmaf(s[10], ox, s[5]));
        default: return s[comp];
        }
    }
    if (comp == 0) return fmaf(s[2], oy, fmaf(s[1], ox, s[0]));
    if (comp == 3) return fmaf(s[5], oy, fmaf(s[4], ox, s[3]));
    return s[comp];
}

__device__ __constant__ int kOrder[12] = {0, 3, 1, 2, 4, 5, 6, 7, 8, 9, 10, 11};

__device__ bool allowed(const UodArgs &a, int index, int dx, int dy, bool wide) {
    if (!a.roi_enabled) return true;
    const float *perm = a.links + (size_t)index * 4;
    unsigned bit, word;
    if (wide) {
        bit = (unsigned)((dy + 4) * 9 + dx + 4);
        word = (unsigned)perm[bit / 24];
    } else {
        bit = (unsigned)((dy + 1) * 3 + dx + 1);
        word = (unsigned)perm[0];
    }
    return (word & (1u << (bit % 24))) != 0u;
}

__device__ void load_state(const float *src, int ss, float *dst) {
    const float4 *s4 = reinterpret_cast<const float4 *>(src);
    for (int k = 0; k < ss / 4; ++k) {
        float4 v = s4[k];
        dst[4 * k] = v.x; dst[4 * k + 1] = v.y; dst[4 * k + 2] = v.z; dst[4 * k + 3] = v.w;
    }
}

__device__ void store_state(float *dst, int ss, const float *src) {
    float4 *d4 = reinterpret_cast<float4 *>(dst);
    for (int k = 0; k < ss / 4; ++k) d4[k] = make_float4(src[4 * k], src[4 * k + 1], src[4 * k + 2], src[4 * k + 3]);
}

// A subset's filtered state into the field and, for a call that waits for its
// result on the host, straight into pinned host memory: the copy that followed
// the pass cost its start and end, 8 to 12 us of a small frame's call.
__device__ __forceinline__ void publish_state(const UodArgs &a, int index, int ss, const float *src) {
    store_state(a.out + (size_t)index * ss, ss, src);
    if (a.host_out != nullptr) store_state(a.host_out + (size_t)index * ss, ss, src);
}

// icgn.wgsl:1192-1323
__device__ void median_motion(const UodArgs &a, int index) {
    const int ss = state_stride(a.model);
    const int sat = status_slot(a.model);
    float own[16];
    load_state(a.state + (size_t)index * ss, ss, own);
    float out[16];
    for (int k = 0; k < ss; ++k) out[k] = own[k];
    const float own_status = own[sat];
    const float ref_status = a.meta[(size_t)index * meta_stride(a.model) + 1];
    if (!((own_status >= 0.5f && !a.scope_all) || (ref_status < 0.5f && ref_status != -4.0f))) {
        const int px = index % a.grid_w, py = index / a.grid_w;
        const int radius = a.median_size / 2;
        const int active = a.model == kModelTranslation ? 2 : (a.model == kModelQuadratic ? 12 : 6);
        float filtered[12];
        for (int k = 0; k < 12; ++k) filtered[k] = own[k];
        bool complete = true;
        float values[81];
        float nbr[16];
        for (int ai = 0; ai < active && complete; ++ai) {
            const int comp = kOrder[ai];
            int count = 0;
            if (own_status >= 0.5f) values[count++] = recentered(a.model, own, comp, 0.0f, 0.0f);
            for (int dy = -radius; dy <= radius; ++dy)
                for (int dx = -radius; dx <= radius; ++dx) {
                    if (dx == 0 && dy == 0) continue;
                    const int nx = px + dx, ny = py + dy;
                    if (nx < 0 || ny < 0 || nx >= a.grid_w || ny >= a.grid_h) continue;
                    if (!allowed(a, index, dx, dy, a.median_size > 3)) continue;
                    const float *ns = a.state + ((size_t)ny * a.grid_w + nx) * ss;
                    if (ns[sat] < 0.5f) continue;
                    load_state(ns, ss, nbr);
                    values[count++] = recentered(a.model, nbr, comp, -(float)a.subset_stride * (float)dx,
                                                 -(float)a.subset_stride * (float)dy);
                }
            const int minimum = (a.roi_enabled && a.median_size == 3 && own_status < 0.5f) ? 3 : 4;
            if (count < minimum) {
                complete = false;
                break;
            }
            filtered[comp] = median_large(values, count);
        }
        if (complete) {
            for (int k = 0; k < 12 && k < ss; ++k) out[k] = filtered[k];
            if (a.model == kModelQuadratic) {
                out[12] = (a.seed_mode && own_status < 0.5f) ? 0.0f : own[12];
                out[13] = own[13]; out[14] = own[14]; out[15] = own[15];
            } else {
                out[6] = (a.seed_mode && own_status < 0.5f) ? 0.0f : own[6];
                out[7] = own[7];
            }
        }
    }
    publish_state(a, index, ss, out);
}

// Windows of 7x7 and 9x9: too many values for registers.
__global__ void median_motion_kernel(UodArgs a) {
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index < a.count) median_motion(a, index);
}

__device__ __noinline__ void median_motion_unordered(const UodArgs &a, int index) { median_motion(a, index); }

// Ascending order of N values in registers: odd-even merge sort, every
// exchange's place known at compile time.
template <int N>
__device__ __forceinline__ void merge_sort(float (&v)[N]) {
#pragma unroll
    for (int p = 1; p < N; p *= 2) {
#pragma unroll
        for (int k = p; k >= 1; k /= 2) {
#pragma unroll
            for (int x = 0; x < N; ++x) {
                const int from = k % p;  // exchange pairs (x, x + k) of each run of 2 k from `from`
                if (x >= from && x + k < N && ((x - from) / k) % 2 == 0 && x / (2 * p) == (x + k) / (2 * p)) {
                    const float lo = v[x], hi = v[x + k];
                    v[x] = fminf(lo, hi);
                    v[x + k] = fmaxf(lo, hi);
                }
            }
        }
    }
}

// median_motion of a window of radius R (3x3 or 5x5) with the values sorted in
// registers; missing neighbours read +inf.  An order statistic does not depend
// on how it is found, except where a NaN is among the values: then the subset
// goes the general way.  With the default scope only rejected subsets are
// filtered, a few threads whose chain is the kernel's time: 5x5 of 13,818
// translations (1000 x 701, S 15 / s 7) 28.6 us by quickselect over local memory
// -> 8.9.
template <int MODEL, int R>
__global__ void __launch_bounds__(128) median_field_kernel(UodArgs a) {
    constexpr int ss = state_stride(MODEL), sat = status_slot(MODEL), nc = parameter_count(MODEL);
    constexpr int D = 2 * R + 1, N = D * D, CENTRE = N / 2;
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= a.count) return;
    float own[ss];
    load_state(a.state + (size_t)index * ss, ss, own);
    const float own_status = own[sat], ref_status = a.meta[(size_t)index * meta_stride(MODEL) + 1];
    if (!((own_status >= 0.5f && !a.scope_all) || (ref_status < 0.5f && ref_status != -4.0f))) {
        const int px = index % a.grid_w, py = index / a.grid_w;
        unsigned valid = own_status >= 0.5f ? 1u << CENTRE : 0u;
#pragma unroll
        for (int slot = 0; slot < N; ++slot) {
            const int dx = slot % D - R, dy = slot / D - R, nx = px + dx, ny = py + dy;
            if (slot != CENTRE && nx >= 0 && ny >= 0 && nx < a.grid_w && ny < a.grid_h &&
                allowed(a, index, dx, dy, R > 1) && !(a.state[((size_t)ny * a.grid_w + nx) * ss + sat] < 0.5f))
                valid |= 1u << slot;
        }
        const int count = __popc(valid);
        if (count >= (a.roi_enabled && R == 1 && own_status < 0.5f ? 3 : 4)) {
            bool unordered = false;
#pragma unroll 1
            for (int comp = 0; comp < (MODEL == kModelTranslation ? 4 : nc); comp += MODEL == kModelTranslation ? 3 : 1) {
                float v[N];
#pragma unroll
                for (int slot = 0; slot < N; ++slot) {
                    const int dx = slot % D - R, dy = slot / D - R;
                    v[slot] = __int_as_float(0x7f800000);
                    if (valid >> slot & 1u) {
                        v[slot] = recentered(MODEL, a.state + ((size_t)index + (long long)dy * a.grid_w + dx) * ss, comp,
                                             -(float)a.subset_stride * (float)dx, -(float)a.subset_stride * (float)dy);
                        unordered = unordered || isnan(v[slot]);
                    }
                }
                merge_sort(v);
                float lo = v[0], hi = v[0];
#pragma unroll
                for (int i = 1; i < N; ++i) {
                    if (i == (count - 1) / 2) lo = v[i];
                    if (i == count / 2) hi = v[i];
                }
                const float median = count % 2 ? hi : 0.5f * (lo + hi);
#pragma unroll
                for (int k = 0; k < nc; ++k)
                    if (k == comp) own[k] = median;
            }
            if (unordered) {
                median_motion_unordered(a, index);
                return;
            }
            if (a.seed_mode && own_status < 0.5f) own[sat] = 0.0f;
        }
    }
    publish_state(a, index, ss, own);
}

template <int MODEL>
cudaError_t launch_median(const UodArgs &a, int grid, cudaStream_t stream) {
    if (a.median_size == 3) median_field_kernel<MODEL, 1><<<grid, 128, 0, stream>>>(a);
    else if (a.median_size == 5) median_field_kernel<MODEL, 2><<<grid, 128, 0, stream>>>(a);
    else median_motion_kernel<<<grid, 128, 0, stream>>>(a);
    return cudaGetLastError();
}

// 3x3 UOD of one quadratic subset by the reference's bubble sort of the valid
// neighbours' values.  uod3_kernel comes here when a value is NaN: only then
// does the order of the comparisons show in a median.
__device__ __noinline__ void quadratic_uod_unordered(const UodArgs &a, int index) {
    const int ss = state_stride(a.model);
    const int sat = status_slot(a.model);
    float own[16];
    load_state(a.state + (size_t)index * ss, ss, own);
    float out[16];
    for (int k = 0; k < ss; ++k) out[k] = own[k];
    if (own[sat] >= 0.5f) {
        const int px = index % a.grid_w, py = index / a.grid_w;
        const int ncomp = parameter_count(a.model);
        float nb[9][12];
        float nbr[16];
        int count = 0;
        for (int dy = -1; dy <= 1; ++dy)
            for (int dx = -1; dx <= 1; ++dx) {
                if (dx == 0 && dy == 0) continue;
                const int nx = px + dx, ny = py + dy;
                if (nx < 0 || ny < 0 || nx >= a.grid_w || ny >= a.grid_h) continue;
                const float *ns = a.state + ((size_t)ny * a.grid_w + nx) * ss;
                if (ns[sat] < 0.5f) continue;
                load_state(ns, ss, nbr);
                const float ox = -(float)a.subset_stride * (float)dx, oy = -(float)a.subset_stride * (float)dy;
                for (int k = 0; k < ncomp; ++k) nb[count][k] = recentered(a.model, nbr, k, ox, oy);
                ++count;
            }
        if (count >= 4) {
            float filtered[12], medians[12], values[9];
            for (int k = 0; k < 12; ++k) filtered[k] = medians[k] = (k < ncomp) ? own[k] : 0.0f;
            const int model_components = a.model == kModelTranslation ? 2 : ncomp;
            const int median_count = a.policy == 1 ? model_components : 2;
            for (int ai = 0; ai < median_count; ++ai) {
                const int comp = kOrder[ai];
                for (int i = 0; i < count; ++i) values[i] = nb[i][comp];
                medians[comp] = median_small(values, count);
            }
            bool flagged = false;
            for (int ai = 0; ai < 2; ++ai) {
                const int comp = kOrder[ai];
                for (int i = 0; i < count; ++i) values[i] = fabsf(nb[i][comp] - medians[comp]);
                const float spread = median_small(values, count);
                const float score = fabsf(filtered[comp] - medians[comp]) / (spread + 0.1f);
                if (score > 2.0f) flagged = true;
            }
            if (flagged) {
                if (a.policy == 1)
                    for (int ai = 0; ai < model_components; ++ai) filtered[kOrder[ai]] = medians[kOrder[ai]];
                for (int k = 0; k < ncomp; ++k) out[k] = filtered[k];
                if (a.model == kModelQuadratic) {
                    out[12] = 2.0f; out[13] = own[13]; out[14] = 0.0f; out[15] = 0.0f;
                } else {
                    out[6] = 2.0f; out[7] = own[7];
                }
            }
        }
    }
    publish_state(a, index, ss, out);
}

// Stable sort of 8 values (odd-even transposition, swap only when strictly
// greater): the same arrangement as a bubble sort of the compacted values,
// with the +inf padding of missing neighbours at the end.
__device__ __forceinline__ void sort8(float (&v)[8]) {
#pragma unroll
    for (int round = 0; round < 8; ++round) {
#pragma unroll
        for (int i = round & 1; i + 1 < 8; i += 2) {
            const float lo = v[i], hi = v[i + 1];
            const bool swap = lo > hi;
            v[i] = swap ? hi : lo;
            v[i + 1] = swap ? lo : hi;
        }
    }
}

// median_small() of the first `count` (4..8) sorted values.
__device__ __forceinline__ float median_sorted8(const float (&v)[8], int count) {
    switch (count) {
    case 4: return 0.5f * (v[1] + v[2]);
    case 5: return v[2];
    case 6: return 0.5f * (v[2] + v[3]);
    case 7: return v[3];
    default: return 0.5f * (v[3] + v[4]);
    }
}

// Component `comp` of the neighbours in the slots set in `valid`, recentred on
// this subset; +inf in the others.
template <int MODEL>
__device__ __forceinline__ void neighbour_values(const UodArgs &a, int index, unsigned valid, int comp, float (&v)[8]) {
    constexpr int ss = state_stride(MODEL);
#pragma unroll
    for (int slot = 0; slot < 8; ++slot) {
        const int cell = slot < 4 ? slot : slot + 1;  // 3x3 scan order without the centre
        const int dx = cell % 3 - 1, dy = cell / 3 - 1;
        v[slot] = __int_as_float(0x7f800000);
        if (valid >> slot & 1u) {
            float nbr[ss];
            load_state(a.state + ((size_t)index + dy * a.grid_w + dx) * ss, ss, nbr);
            v[slot] = recentered(MODEL, nbr, comp, -(float)a.subset_stride * (float)dx, -(float)a.subset_stride * (float)dy);
        }
    }
}

// 3x3 UOD (replace / flag) with the neighbours' values in registers: the slots
// keep the scan order of the reference, missing ones read +inf, and the
// order statistics come from sort8, so the result equals its bubble sort's
// bit for bit.  Only the translations decide whether a subset is an outlier;
// the other components' medians are taken for the few that are.  Bound by
// HBM / L2 reads of the states: UHD S 41 / s 10 quadratic (80,560 subsets)
// 112 us with every component's values in local memory, 16.5 us here; UHD
// S 31 / s 8 affine (127,359 subsets) 10.8 us with every median taken, 7.5.
template <int MODEL>
__global__ void __launch_bounds__(128) uod3_kernel(UodArgs a) {
    constexpr int ss = state_stride(MODEL), sat = status_slot(MODEL), nc = parameter_count(MODEL);
    const int index = blockIdx.x * blockDim.x + threadIdx.x;
    if (index >= a.count) return;
    float own[ss];
    load_state(a.state + (size_t)index * ss, ss, own);
    if (own[sat] >= 0.5f) {
        const int px = index % a.grid_w, py = index / a.grid_w;
        const float kInf = __int_as_float(0x7f800000);
        float nb[2][8];  // tx, ty
        unsigned valid = 0u;
#pragma unroll
        for (int slot = 0; slot < 8; ++slot) {
            const int cell = slot < 4 ? slot : slot + 1;
            const int dx = cell % 3 - 1, dy = cell / 3 - 1;
            const int nx = px + dx, ny = py + dy;
            bool ok = nx >= 0 && ny >= 0 && nx < a.grid_w && ny < a.grid_h &&
                      (MODEL == kModelQuadratic || allowed(a, index, dx, dy, false));
            nb[0][slot] = nb[1][slot] = kInf;
            if (ok) {
                float nbr[ss];
                load_state(a.state + ((size_t)ny * a.grid_w + nx) * ss, ss, nbr);
                if (nbr[sat] >= 0.5f) {
                    const float ox = -(float)a.subset_stride * (float)dx, oy = -(float)a.subset_stride * (float)dy;
                    valid |= 1u << slot;
                    nb[0][slot] = recentered(MODEL, nbr, 0, ox, oy);
                    nb[1][slot] = recentered(MODEL, nbr, 3, ox, oy);
                }
            }
        }
        const int count = __popc(valid);
        if (count >= 4) {
            bool unordered = false;
            float medians[2];
            bool flagged = false;
#pragma unroll
            for (int ai = 0; ai < 2; ++ai) {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = nb[ai][i];
                sort8(v);
                medians[ai] = median_sorted8(v, count);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    v[i] = valid >> i & 1u ? fabsf(nb[ai][i] - medians[ai]) : kInf;
                    unordered = unordered || !(v[i] >= 0.0f);
                }
                sort8(v);
                const float spread = median_sorted8(v, count);
                if (fabsf(own[ai * 3] - medians[ai]) / (spread + 0.1f) > 2.0f) flagged = true;
            }
            if (MODEL == kModelQuadratic && unordered) {
                quadratic_uod_unordered(a, index);
                return;
            }
            if (flagged) {
                if (a.policy == 1) {
                    own[0] = medians[0];
                    own[3] = medians[1];
                    if (MODEL != kModelTranslation) {
#pragma unroll
                        for (int comp = 1; comp < nc; ++comp) {
                            if (comp == 3) continue;
                            float v[8];
                            neighbour_values<MODEL>(a, index, valid, comp, v);
                            if (MODEL == kModelQuadratic) {
#pragma unroll
                                for (int i = 0; i < 8; ++i) unordered = unordered || isnan(v[i]);
                            }
                            sort8(v);
                            own[comp] = median_sorted8(v, count);
                        }
                        if (MODEL == kModelQuadratic && unordered) {
                            quadratic_uod_unordered(a, index);
                            return;
                        }
                    }
                }
                own[sat] = 2.0f;
                if (MODEL == kModelQuadratic) own[14] = own[15] = 0.0f;
            }
        }
    }
    publish_state(a, index, ss, own);
}

}  // namespace

cudaError_t launch_uod(const UodArgs &a, cudaStream_t stream) {
    if (a.count <= 0) return cudaSuccess;
    const int grid = (a.count + 127) / 128;
    if (a.policy == 3) {
        switch (a.model) {
        case kModelAffine: return launch_median<kModelAffine>(a, grid, stream);
        case kModelTranslation: return launch_median<kModelTranslation>(a, grid, stream);
        default: return launch_median<kModelQuadratic>(a, grid, stream);
        }
    }
    if (a.model == kModelAffine) uod3_kernel<kModelAffine><<<grid, 128, 0, stream>>>(a);
    else if (a.model == kModelTranslation) uod3_kernel<kModelTranslation><<<grid, 128, 0, stream>>>(a);
    else uod3_kernel<kModelQuadratic><<<grid, 128, 0, stream>>>(a);
    return cudaGetLastError();
}

}  // namespace gbdic
