// Global-translation initializer by linear phase correlation on the GPU
// (reference: fourier.py:16-111, FourierInitializer, which runs it in NumPy
// float64 on the CPU).
//
// Reference side, once: the chosen size x size window (size = a power of two
// <= 1024) minus its mean over ROI-allowed pixels, zeroed outside the ROI,
// 2x2-averaged to half x half samples, Hann-tapered, zero-padded back to
// size x size and transformed.  Per target: the same window (mean over all
// pixels), the same reduction and taper, forward FFT, normalised cross power
// spectrum F_cur conj(F_ref) / max(|.|, 1e-12), inverse FFT, the peak
// (first maximum in row-major order), its score against the background
// outside the wrapped 11 x 11 neighbourhood, the even-pixel shift, the
// window overlap, and the normalised correlation of the reduced samples over
// the overlapping, ROI-allowed region.  out = {dx, dy, peak score, overlap,
// correlation, peak, target window standard deviation}.
//
// Transforms are radix-2 decimation-in-time in float64 (the reference's
// precision).  A line of n = 2^L points lies in the registers of T = n / P
// lanes, P points to a lane; every log2 P levels the lanes exchange points
// through shared memory.  What bounds them is the FP64 pipe (a warp's
// instruction takes its quarter of an SM 64 cycles), so the design spends as
// few FP64 instructions as it can: a butterfly is six or eight FMAs, four
// additions where the twiddle is 1 or -i; the zero-padded half of an input
// skips its first level; two real rows share one complex line, so the
// spectrum is the half with columns 0..n/2; a column is transformed,
// multiplied with the reference's and transformed back without leaving its
// block; and the cross power is normalised by one rsqrt.
//
// Window 1024^2, one estimate on the device (the step at a time, before ->
// after): 4,096 line transforms -> 1,794; transforms, cross power, reduction
// and peak search 480 -> 185 us (rows 39, columns with the cross power 97,
// last rows with the peak 49); whole estimate 540 -> 215 us.  256^2: 33 + 25
// -> 28 us.  Points to a lane at 1024: 190 us with 8,
// 197 with 16, 235 with 32 (fewer and longer warps leave quarters idle); at
// 256: 28 us with 4, 90 with 16.
// Sums are exact integers where the inputs are bytes and float64 elsewhere.
#include <cmath>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "engine.h"

using gbdic::check_cuda;
using gbdic::fail;
using gbdic::Failure;

namespace {

// ---------------------------------------------------------------- transforms

__host__ __device__ constexpr int bit_reverse(int i, int bits) {
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((i >> b) & 1) << (bits - 1 - b);
    return r;
}

__host__ __device__ constexpr int log2c(int n) { return n <= 1 ? 0 : 1 + log2c(n / 2); }

// cos and -sin of 2 pi k / 32, k < 8.
__device__ __forceinline__ double2 root32(int k) {
    switch (k) {
        case 1: return make_double2(0.9807852804032304, -0.19509032201612825);
        case 2: return make_double2(0.9238795325112867, -0.3826834323650898);
        case 3: return make_double2(0.8314696123025452, -0.5555702330196022);
        case 4: return make_double2(0.7071067811865476, -0.7071067811865475);
        case 5: return make_double2(0.5555702330196023, -0.8314696123025452);
        case 6: return make_double2(0.38268343236508984, -0.9238795325112867);
        case 7: return make_double2(0.19509032201612833, -0.9807852804032304);
        default: return make_double2(1.0, 0.0);
    }
}

// (u, t) -> (u + w t, u - w t), both sums as FMA chains (EXACT, eight
// instructions) or the second as 2 u - (u + w t) (six).  With EXACT in the
// second pass' levels alone a 1024-point line's error against extended
// precision is 9.36e-15 rms where separate products and sums had 9.44e-15
// (values of rms 45); six instructions everywhere would leave 9.94e-15.
template <bool EXACT>
__device__ __forceinline__ void butterfly(double2 &u, double2 &t, double2 w) {
    const double2 a = make_double2(fma(-w.y, t.y, fma(w.x, t.x, u.x)), fma(w.y, t.x, fma(w.x, t.y, u.y)));
    t = EXACT ? make_double2(fma(w.y, t.y, fma(-w.x, t.x, u.x)), fma(-w.y, t.x, fma(-w.x, t.y, u.y)))
              : make_double2(fma(2.0, u.x, -a.x), fma(2.0, u.y, -a.y));
    u = a;
}

// (u, t) -> (u - i w t, u + i w t)
template <bool EXACT>
__device__ __forceinline__ void butterfly_quarter(double2 &u, double2 &t, double2 w) {
    const double2 a = make_double2(fma(w.y, t.x, fma(w.x, t.y, u.x)), fma(w.y, t.y, fma(-w.x, t.x, u.y)));
    t = EXACT ? make_double2(fma(-w.y, t.x, fma(-w.x, t.y, u.x)), fma(-w.y, t.y, fma(w.x, t.x, u.y)))
              : make_double2(fma(2.0, u.x, -a.x), fma(2.0, u.y, -a.y));
    u = a;
}

// Forward DFT of R points held by one thread, natural order in and out.  With
// TWIST the points are partial results at bin k1 of D = 1 << LOGD: level s
// turns by exp(-2 pi i (pos D + k1) / (D 2^s)), from the table `tw` of the
// n-point roots.  HALF: the second half of the input is zero, and the first
// level a copy.
template <int R, int LOGD, bool HALF, int LOGN>
__device__ __forceinline__ void register_dft(double2 (&v)[R], const double2 *tw, int k1) {
    constexpr int B = log2c(R);
    constexpr bool TWIST = LOGD > 0;
#pragma unroll
    for (int s = 1; s <= B; ++s) {
        const int h = 1 << (s - 1);
#pragma unroll
        for (int pos = 0; pos < (h > 1 ? h / 2 : 1); ++pos) {
            double2 w = make_double2(1.0, 0.0);
            if constexpr (TWIST) {
                w = __ldg(tw + (((pos << LOGD) + k1) << (LOGN - LOGD - s)));
            } else {
                w = root32(pos * (32 >> s));
            }
#pragma unroll
            for (int g = 0; g < R / 2 / h; ++g) {
                double2 &u = v[bit_reverse(g * 2 * h + pos, B)], &t = v[bit_reverse(g * 2 * h + pos + h, B)];
                if (HALF && s == 1) {
                    t = u;
                } else if (TWIST || pos > 0) {
                    butterfly<TWIST>(u, t, w);
                } else {
                    const double2 a = make_double2(u.x + t.x, u.y + t.y);
                    t = make_double2(u.x - t.x, u.y - t.y);
                    u = a;
                }
                if (h > 1) {
                    double2 &x = v[bit_reverse(g * 2 * h + pos + h / 2, B)];
                    double2 &y = v[bit_reverse(g * 2 * h + pos + h / 2 + h, B)];
                    if (TWIST || pos > 0) {
                        butterfly_quarter<TWIST>(x, y, w);
                    } else {
                        const double2 a = make_double2(x.x + y.y, x.y - y.x);
                        y = make_double2(x.x - y.y, x.y + y.x);
                        x = a;
                    }
                }
            }
        }
    }
    double2 out[R];
#pragma unroll
    for (int k = 0; k < R; ++k) out[k] = v[bit_reverse(k, B)];
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = out[k];
}

// Shape of a line of 2^LOGN points: P points to a lane, T lanes to a line.  A
// block is one line, or LINES short ones in a warp: the FP64 pipe belongs to a
// quarter of the SM, so lines are cut into as many warps as it takes to fill
// all quarters (the times are above).
template <int LOGN>
struct Line {
    static constexpr int N = 1 << LOGN, P = LOGN >= 9 ? 8 : 4, T = N / P, LINES = T < 32 ? 32 / T : 1,
                         THREADS = T * LINES, WARPS = THREADS / 32, PITCH = N + N / 8, EXCHANGE = LINES * PITCH;

    // A pass of radix R over the partial results Y[t][K] of D bins K and N/D
    // remaining indices t, kept at t D + K: item i takes Y[i / D + N/(D R) j]
    // [i % D], which lie at i + N/R j, and leaves Y'[i / D][i % D + D k].
    // Lane t's items are t + T sub.  One gap in eight points keeps the strided
    // writes of the first pass free of bank conflicts.
    template <int LOGD, bool HALF>
    static __device__ __forceinline__ void pass(double2 (&v)[P], double2 *ex, int t, const double2 *tw) {
        constexpr int LEFT = LOGN - LOGD, LOGP = log2c(P), R = LEFT < LOGP ? 1 << LEFT : P, SUB = P / R, D = 1 << LOGD;
#pragma unroll
        for (int sub = 0; sub < SUB; ++sub) {
            const int i = t + T * sub, bin = i & (D - 1);
            double2 u[R];
#pragma unroll
            for (int j = 0; j < R; ++j) u[j] = v[sub + SUB * j];  // point i + N/R j = t + T (sub + SUB j)
            register_dft<R, LOGD, HALF, LOGN>(u, tw, bin);
            if constexpr (LEFT > LOGP) {
                const int base = (i >> LOGD) * D * R + bin;
#pragma unroll
                for (int k = 0; k < R; ++k) {
                    const int at = base + D * k;
                    ex[at + (at >> 3)] = u[k];
                }
            } else {  // the last pass: bins i + D k = t + T (sub + SUB k)
#pragma unroll
                for (int k = 0; k < R; ++k) v[sub + SUB * k] = u[k];
            }
        }
        if constexpr (LEFT > LOGP) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const int at = t + T * j;
                v[j] = ex[at + (at >> 3)];
            }
            __syncthreads();
            pass<LOGD + LOGP, false>(v, ex, t, tw);
        }
    }

    // Lane t holds points t + T j in v[j], before and after.
    template <bool HALF>
    static __device__ __forceinline__ void forward(double2 (&v)[P], double2 *ex, int t, const double2 *tw) {
        pass<0, HALF>(v, ex, t, tw);
    }
};

// The inverse transform is the forward one between two exchanges of real and
// imaginary parts.
template <int P>
__device__ __forceinline__ void swap_parts(double2 (&v)[P]) {
#pragma unroll
    for (int i = 0; i < P; ++i) v[i] = make_double2(v[i].y, v[i].x);
}

// ------------------------------------------------------------------- kernels

// Integer sum, count and sum of squares of the window bytes (allowed pixels),
// sixteen bytes to a load (the window is dense, size a multiple of 32).
__global__ void window_sum_kernel(const uint4 *win, const uint4 *allowed, int count, unsigned long long *sums) {
    unsigned s = 0, n = 0, q = 0;  // <= 2^20 * 255^2 / (64 * 256) threads each
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        uint4 v = __ldg(win + i);
        if (allowed) {
            const uint4 m = __ldg(allowed + i);
            const unsigned k[4] = {__vcmpne4(m.x, 0u), __vcmpne4(m.y, 0u), __vcmpne4(m.z, 0u), __vcmpne4(m.w, 0u)};
            v = make_uint4(v.x & k[0], v.y & k[1], v.z & k[2], v.w & k[3]);
            n += (__popc(k[0]) + __popc(k[1]) + __popc(k[2]) + __popc(k[3])) >> 3;
        } else {
            n += 16;
        }
        const unsigned w[4] = {v.x, v.y, v.z, v.w};
        for (int b = 0; b < 4; ++b) {
            s = __dp4a(w[b], 0x01010101u, s);
            q = __dp4a(w[b], w[b], q);
        }
    }
    s = __reduce_add_sync(0xffffffffu, s);
    n = __reduce_add_sync(0xffffffffu, n);
    q = __reduce_add_sync(0xffffffffu, q);
    if ((threadIdx.x & 31) == 0 && n > 0) {
        atomicAdd(&sums[0], (unsigned long long)s);
        atomicAdd(&sums[1], (unsigned long long)n);
        atomicAdd(&sums[2], (unsigned long long)q);
    }
}

// Rows of the padded, tapered input: reduced samples (2x2 means of the
// mean-free, ROI-zeroed window), kept with their allowed flags for the overlap
// correlation, and the transform of samples rows r and r + n/4 as the real and
// imaginary part of one line, halved (the exact 1/2 of separating them again).
template <int LOGN>
__global__ void __launch_bounds__(Line<LOGN>::THREADS) row_kernel(const uint8_t *win, const uint8_t *allowed,
                                                 const unsigned long long *sums, const double *taper,
                                                 const double2 *tw, double *samples, uint8_t *allowed_samples,
                                                 double2 *rows) {
    using L = Line<LOGN>;
    constexpr int N = L::N, HALF = N / 2;
    __shared__ double2 exchange[L::EXCHANGE];
    const int t = threadIdx.x % L::T, slot = threadIdx.x / L::T, line = blockIdx.x * L::LINES + slot;
    uchar2 bytes[L::P / 2][2][2];  // in flight while the table is made
#pragma unroll
    for (int j = 0; j < L::P / 2; ++j)
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const size_t at = (size_t)(2 * (line + p * (N / 4))) * N + 2 * (t + L::T * j);
            bytes[j][p][0] = *reinterpret_cast<const uchar2 *>(win + at);
            bytes[j][p][1] = *reinterpret_cast<const uchar2 *>(win + at + N);
        }
    // byte -> mean-free value, converted once per block
    __shared__ double value[256];
    const double mean = (double)sums[0] / (double)sums[1];
    for (int i = threadIdx.x; i < 256; i += L::THREADS) value[i] = (double)i - mean;
    __syncthreads();
    double2 v[L::P];
#pragma unroll
    for (int j = 0; j < L::P; ++j) v[j] = make_double2(0.0, 0.0);
#pragma unroll
    for (int j = 0; j < L::P / 2; ++j) {
        const int c = t + L::T * j;
        double part[2];
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const int r = line + p * (N / 4);
            const uchar2 a = bytes[j][p][0], b = bytes[j][p][1];
            double acc;
            uint8_t all = 1;
            if (allowed) {
                const size_t at = (size_t)(2 * r) * N + 2 * c;
                const uchar2 ma = *reinterpret_cast<const uchar2 *>(allowed + at);
                const uchar2 mb = *reinterpret_cast<const uchar2 *>(allowed + at + N);
                acc = value[a.x] * (ma.x ? 1.0 : 0.0);
                acc += value[a.y] * (ma.y ? 1.0 : 0.0);
                acc += value[b.x] * (mb.x ? 1.0 : 0.0);
                acc += value[b.y] * (mb.y ? 1.0 : 0.0);
                all = ma.x && ma.y && mb.x && mb.y;
            } else {
                acc = value[a.x];
                acc += value[a.y];
                acc += value[b.x];
                acc += value[b.y];
            }
            const double reduced = acc * 0.25;
            samples[r * HALF + c] = reduced;
            if (allowed_samples) allowed_samples[r * HALF + c] = all;
            part[p] = reduced * (0.5 * taper[r]) * taper[c];
        }
        v[j] = make_double2(part[0], part[1]);
    }
    L::template forward<true>(v, exchange + slot * L::PITCH, t, tw);
#pragma unroll
    for (int j = 0; j < L::P; ++j) rows[(size_t)line * N + t + L::T * j] = v[j];
}

// Columns 0..n/2 of the spectrum, one to T lanes.  The two real rows of each
// packed line are separated on loading.  REFERENCE: the column's spectrum is
// stored in the lanes' order.  Otherwise it is multiplied with the
// reference's conjugate, normalised by max(|.|, 1e-12) and transformed back in
// place (lane t's bins t + T j are the order the transform takes), and rows y
// and y + n/2 of the result are packed as one complex line for the last pass:
// column c of A + iB, and its mirror n - c from the conjugates.
//
// 1024^2: about 90 FP64 instructions per point, and 513 columns on 152 SMs, four
// to the busiest: 96 us at the pipe's rate, 97 measured.
template <int LOGN, bool REFERENCE>
__global__ void __launch_bounds__(Line<LOGN>::THREADS) column_kernel(const double2 *rows, double2 *ref, const double2 *tw,
                                                    double2 *out) {
    using L = Line<LOGN>;
    constexpr int N = L::N, P = L::P, T = L::T;
    __shared__ double2 exchange[L::EXCHANGE];
    const int t = threadIdx.x % T, slot = threadIdx.x / T, line = blockIdx.x * L::LINES + slot;
    const int c = line < N / 2 ? line : N / 2, mirror = (N - c) & (N - 1);
    double2 *ex = exchange + slot * L::PITCH;
    double2 v[P];
#pragma unroll
    for (int j = 0; j < P / 4; ++j) {
        const size_t row = (size_t)(t + T * j) * N;
        const double2 z = rows[row + c], m = rows[row + mirror];
        v[j] = make_double2(z.x + m.x, z.y - m.y);
        v[j + P / 4] = make_double2(z.y + m.y, m.x - z.x);
        v[j + P / 2] = make_double2(0.0, 0.0);
        v[j + 3 * P / 4] = make_double2(0.0, 0.0);
    }
    L::template forward<true>(v, ex, t, tw);
    double2 *mine = ref + (size_t)c * N + t;
    if constexpr (REFERENCE) {
        if (line > N / 2) return;
#pragma unroll
        for (int j = 0; j < P; ++j) mine[T * j] = v[j];
    } else {
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const double2 a = v[j], b = __ldg(mine + T * j);
            const double x = a.x * b.x + a.y * b.y, y = a.y * b.x - a.x * b.y;  // a conj(b)
            const double inv = fmin(rsqrt(x * x + y * y), 1e12);                // 1 / max(|.|, 1e-12)
            v[j] = make_double2(y * inv, x * inv);                              // parts exchanged: inverse
        }
        L::template forward<false>(v, ex, t, tw);
        if (line > N / 2) return;
        const bool real = mirror == c || c == N / 2;
#pragma unroll
        for (int j = 0; j < P / 2; ++j) {
            const double2 a = make_double2(v[j].y, v[j].x), b = make_double2(v[j + P / 2].y, v[j + P / 2].x);
            double2 *row = out + (size_t)(t + T * j) * N;
            if (real) {  // zero frequency and Nyquist of a real row: no imaginary part
                row[c] = make_double2(a.x, b.x);
            } else {
                row[c] = make_double2(a.x - b.y, a.y + b.x);
                row[mirror] = make_double2(a.x + b.y, b.x - a.y);
            }
        }
    }
}

// Last pass: rows y and y + n/2 of the correlation out of each packed line,
// stored without the transform's 1/n^2 (a power of two, applied to the few
// figures at the end), and per block the first maximum (lowest index on
// ties) and the sums of the values and of their squares.
template <int LOGN>
__global__ void __launch_bounds__(Line<LOGN>::THREADS) inverse_row_kernel(const double2 *lines, const double2 *tw, double *corr,
                                                         double *pbest, int *pidx, double *psum, double *psq) {
    using L = Line<LOGN>;
    constexpr int N = L::N, P = L::P, T = L::T;
    __shared__ double2 exchange[L::EXCHANGE];
    const int t = threadIdx.x % T, slot = threadIdx.x / T, line = blockIdx.x * L::LINES + slot;
    double2 v[P];
#pragma unroll
    for (int j = 0; j < P; ++j) v[j] = __ldg(lines + (size_t)line * N + t + T * j);
    swap_parts(v);
    L::template forward<false>(v, exchange + slot * L::PITCH, t, tw);
    swap_parts(v);
    double best = -1e300, s = 0.0, q = 0.0;
    int best_i = 0x7fffffff;
#pragma unroll
    for (int p = 0; p < 2; ++p)
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const double x = p ? v[j].y : v[j].x;
            const int i = (line + p * (N / 2)) * N + t + T * j;
            corr[i] = x;
            s += x;
            q += x * x;
            if (x > best) { best = x; best_i = i; }
        }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const double b2 = __shfl_down_sync(0xffffffffu, best, off);
        const int i2 = __shfl_down_sync(0xffffffffu, best_i, off);
        if (b2 > best || (b2 == best && i2 < best_i)) { best = b2; best_i = i2; }
        s += __shfl_down_sync(0xffffffffu, s, off);
        q += __shfl_down_sync(0xffffffffu, q, off);
    }
    __shared__ double block_best[L::WARPS], block_sum[L::WARPS], block_square[L::WARPS];
    __shared__ int block_i[L::WARPS];
    if ((threadIdx.x & 31) == 0) {
        const int w = threadIdx.x / 32;
        block_best[w] = best;
        block_i[w] = best_i;
        block_sum[w] = s;
        block_square[w] = q;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < L::WARPS; ++w) {
            if (block_best[w] > best || (block_best[w] == best && block_i[w] < best_i)) {
                best = block_best[w];
                best_i = block_i[w];
            }
            s += block_sum[w];
            q += block_square[w];
        }
        pbest[blockIdx.x] = best;
        pidx[blockIdx.x] = best_i;
        psum[blockIdx.x] = s;
        psq[blockIdx.x] = q;
    }
}

// Roots of an n-point transform, k < n/2: (cos, sin) of -2 pi k / n.  Level s
// uses entry pos * (n / 2^s), whose argument is the same double as
// -2 pos / 2^s, so the factors equal a per-level sincospi() bit for bit.
__global__ void twiddle_kernel(double2 *tw, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n / 2) return;
    double sn, cs;
    sincospi(-1.0 * 2.0 * (double)k / (double)n, &sn, &cs);
    tw[k] = make_double2(cs, sn);
}

constexpr int kPeakThreads = 128;

// Combines the last pass's partial results in a fixed order (one CTA), then
// the mean and deviation of the correlation outside the wrapped 11 x 11 block
// around the peak.
__global__ void __launch_bounds__(kPeakThreads) peak_final_kernel(const double *corr, int size, int partials,
                                                                  const double *pbest, const int *pidx,
                                                                  const double *psum, const double *psq, double *out) {
    __shared__ double sb[kPeakThreads], ss[kPeakThreads], sq[kPeakThreads];
    __shared__ int si[kPeakThreads];
    const int tid = threadIdx.x;
    double best = -1e300, s = 0.0, q = 0.0;
    int best_i = 0x7fffffff;
#pragma unroll 4
    for (int i = tid; i < partials; i += kPeakThreads) {
        const double b2 = pbest[i];
        const int i2 = pidx[i];
        if (b2 > best || (b2 == best && i2 < best_i)) { best = b2; best_i = i2; }
        s += psum[i];
        q += psq[i];
    }
    sb[tid] = best; si[tid] = best_i; ss[tid] = s; sq[tid] = q;
    __syncthreads();
    for (int off = kPeakThreads / 2; off > 0; off >>= 1) {
        if (tid < off) {
            const double b2 = sb[tid + off];
            const int i2 = si[tid + off];
            if (b2 > sb[tid] || (b2 == sb[tid] && i2 < si[tid])) {
                sb[tid] = b2;
                si[tid] = i2;
            }
            ss[tid] += ss[tid + off];
            sq[tid] += sq[tid + off];
        }
        __syncthreads();
    }
    const double scale = 1.0 / ((double)size * (double)size);
    const double peak = sb[0] * scale, sum = ss[0] * scale, square = sq[0] * scale * scale;
    const int py = si[0] / size, px = si[0] % size;
    __syncthreads();
    double v = 0.0;
    if (tid < 121) {
        const int r = ((py + tid / 11 - 5) % size + size) % size, c = ((px + tid % 11 - 5) % size + size) % size;
        v = corr[r * size + c] * scale;
    }
    ss[tid] = v;
    sq[tid] = v * v;
    __syncthreads();
    for (int off = kPeakThreads / 2; off > 0; off >>= 1) {
        if (tid < off) {
            ss[tid] += ss[tid + off];
            sq[tid] += sq[tid + off];
        }
        __syncthreads();
    }
    if (tid == 0) {
        const double m = (double)(size * size - 121);
        const double mean = (sum - ss[0]) / m;
        const double var = fmax((square - sq[0]) / m - mean * mean, 0.0);
        out[0] = peak;
        out[1] = (double)px;
        out[2] = (double)py;
        out[3] = mean;
        out[4] = sqrt(var);
    }
}

// Normalised correlation of reference and current reduced samples over the
// overlap for the peak's shift (in `result`), allowed reference samples only:
// per-CTA partial sums (stage 1), combined in a fixed order (stage 2).
constexpr int kCorrCtas = 256, kCorrThreads = 256;  // both sums below take eight terms
constexpr int kCorrAt = 4 * 512;  // its place behind the peak's partial results

__global__ void __launch_bounds__(kCorrThreads) overlap_partial_kernel(const double *ref, const uint8_t *allowed,
                                                                        const double *cur, int half,
                                                                        const double *result, double *partial) {
    const int px = (int)result[1], py = (int)result[2];
    const int sx = px < half ? px : px - 2 * half, sy = py < half ? py : py - 2 * half;
    const int y0 = max(0, -sy), y1 = min(half, half - sy), x0 = max(0, -sx), x1 = min(half, half - sx);
    double sa = 0, sb = 0, sab = 0, saa = 0, sbb = 0;
    int n = 0;
    for (int r = y0 + blockIdx.x; r < y1; r += gridDim.x)
#pragma unroll 2
        for (int c = x0 + threadIdx.x; c < x1; c += blockDim.x) {
            const bool ok = allowed[r * half + c];  // all three loads in flight
            double a = ref[r * half + c], b = cur[(r + sy) * half + (c + sx)];
            if (!ok) a = b = 0.0;
            sa += a; sb += b; sab += a * b; saa += a * a; sbb += b * b; n += ok;
        }
    __shared__ double red[6][kCorrThreads / 32];
    double v[6] = {sa, sb, sab, saa, sbb, (double)n};
    for (int k = 0; k < 6; ++k) {
        for (int off = 16; off > 0; off >>= 1) v[k] += __shfl_down_sync(0xffffffffu, v[k], off);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x / 32] = v[k];
    }
    __syncthreads();
    if (threadIdx.x < 6) {
        const double *w = red[threadIdx.x];
        partial[threadIdx.x * kCorrCtas + blockIdx.x] = ((w[0] + w[1]) + (w[2] + w[3])) + ((w[4] + w[5]) + (w[6] + w[7]));
    }
}

__global__ void __launch_bounds__(192) overlap_final_kernel(const double *partial, double *out) {
    __shared__ double red[6];
    const int k = threadIdx.x / 32;  // a warp to a sum
    double p[kCorrCtas / 32];
#pragma unroll
    for (int i = 0; i < 8; ++i) p[i] = partial[k * kCorrCtas + i * 32 + threadIdx.x % 32];
    double v = ((p[0] + p[1]) + (p[2] + p[3])) + ((p[4] + p[5]) + (p[6] + p[7]));
    for (int off = 16; off > 0; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
    if (threadIdx.x % 32 == 0) red[k] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        const double cnt = red[5];
        double corr = 0.0;
        if (cnt > 0) {
            const double ma = red[0] / cnt, mb = red[1] / cnt;
            const double cab = red[2] - cnt * ma * mb;
            const double caa = fmax(red[3] - cnt * ma * ma, 0.0), cbb = fmax(red[4] - cnt * mb * mb, 0.0);
            const double norm = sqrt(caa) * sqrt(cbb);
            corr = norm > 0 ? cab / norm : 0.0;
        }
        out[5] = corr;
    }
}

// Accepted shift of the last phase correlation written into rows of affine
// parameters without a host round trip: the integer peak shift (the same
// unwrapping as the host path), accepted when the target window has texture
// (standard deviation >= 1), the peak score reaches 8 and the overlap 0.25;
// rows[i * pitch] = dx * multiplier, rows[i * pitch + 3] = dy * multiplier,
// zero when rejected.  The sample-correlation test of the host path needs the
// shift on the host to launch and is not applied here.
__global__ void shift_rows_kernel(const double *result, const unsigned long long *sums, int size, float multiplier,
                                  float *rows, int count, int pitch) {
    __shared__ float su, sv;
    if (threadIdx.x == 0) {
        const double wn = (double)sums[1], wmean = wn > 0 ? (double)sums[0] / wn : 0.0;
        const double texture = wn > 0 ? sqrt(fmax((double)sums[2] / wn - wmean * wmean, 0.0)) : 0.0;
        const int half = size / 2, px = (int)result[1], py = (int)result[2];
        const int dx = 2 * (px < half ? px : px - size), dy = 2 * (py < half ? py : py - size);
        const double sd = result[4];
        const double score = (result[0] - result[3]) / (sd > 1e-12 ? sd : 1e-12);
        const double ox = (double)max(size - abs(dx), 0), oy = (double)max(size - abs(dy), 0);
        const double overlap = ox * oy / ((double)size * size);
        const bool ok = texture >= 1.0 && score >= 8.0 && overlap >= 0.25;
        su = ok ? (float)dx * multiplier : 0.0f;
        sv = ok ? (float)dy * multiplier : 0.0f;
    }
    __syncthreads();
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        rows[(size_t)i * pitch] = su;
        rows[(size_t)i * pitch + 3] = sv;
    }
}

int log2i(int n) {
    int l = 0;
    while ((1 << l) < n) ++l;
    return l;
}

thread_local std::string g_fourier_error;

}  // namespace

struct gbdic_fourier {
    int device = 0, size = 0, half = 0, logn = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    // rows: n/4 packed lines of the forward row pass; work: the n/2 packed lines
    // between the columns and the last pass; corr: the correlation.
    gbdic::DeviceBuffer window, allowed, taper, ref_spectrum, ref_samples, allowed_samples, cur_samples, rows, work,
        corr, sums, result, twiddle, partials;
    gbdic::HostBuffer host_window, host_result;
    std::string error;
    ~gbdic_fourier() {
        cudaSetDevice(device);
        if (stream) {
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
        if (fork) cudaEventDestroy(fork);
        if (join) cudaEventDestroy(join);
    }
    // window bytes (device, dense size x size) -> samples and packed row spectra
    template <int LOGN>
    void rows_of(const uint8_t *allow, double *samples, uint8_t *allowed_out, cudaStream_t st) {
        using L = Line<LOGN>;
        check_cuda(cudaMemsetAsync(sums.get(), 0, 3 * sizeof(unsigned long long), st), "clear");
        constexpr int vectors = L::N * L::N / 16;
        window_sum_kernel<<<vectors < 64 * 256 ? (vectors + 255) / 256 : 64, 256, 0, st>>>(
            window.as<uint4>(), reinterpret_cast<const uint4 *>(allow), vectors, sums.as<unsigned long long>());
        check_cuda(cudaGetLastError(), "window mean");
        row_kernel<LOGN><<<L::N / 4 / L::LINES, L::THREADS, 0, st>>>(window.as<uint8_t>(), allow,
                                                             sums.as<unsigned long long>(), taper.as<double>(),
                                                             twiddle.as<double2>(), samples, allowed_out,
                                                             rows.as<double2>());
        check_cuda(cudaGetLastError(), "reduction, taper and row transforms");
    }
    template <int LOGN>
    void reference_spectrum(const uint8_t *allow) {
        using L = Line<LOGN>;
        rows_of<LOGN>(allow, ref_samples.as<double>(), allowed_samples.as<uint8_t>(), stream);
        column_kernel<LOGN, true><<<(L::N / 2 + L::LINES) / L::LINES, L::THREADS, 0, stream>>>(
            rows.as<double2>(), ref_spectrum.as<double2>(), twiddle.as<double2>(), nullptr);
        check_cuda(cudaGetLastError(), "column transforms");
    }
    // phase correlation of the window with the reference: peak figures in `result`
    template <int LOGN>
    void correlate(cudaStream_t st) {
        using L = Line<LOGN>;
        rows_of<LOGN>(nullptr, cur_samples.as<double>(), nullptr, st);
        column_kernel<LOGN, false><<<(L::N / 2 + L::LINES) / L::LINES, L::THREADS, 0, st>>>(
            rows.as<double2>(), ref_spectrum.as<double2>(), twiddle.as<double2>(), work.as<double2>());
        check_cuda(cudaGetLastError(), "columns and cross power");
        constexpr int parts = L::N / 2 / L::LINES;
        static_assert(4 * parts <= kCorrAt, "room for the partial results");
        double *pb = partials.as<double>();
        int *pi = reinterpret_cast<int *>(pb + 3 * parts);
        inverse_row_kernel<LOGN><<<parts, L::THREADS, 0, st>>>(work.as<double2>(), twiddle.as<double2>(), corr.as<double>(),
                                                       pb, pi, pb + parts, pb + 2 * parts);
        check_cuda(cudaGetLastError(), "inverse rows");
        peak_final_kernel<<<1, kPeakThreads, 0, st>>>(corr.as<double>(), L::N, parts, pb, pi, pb + parts,
                                                      pb + 2 * parts, result.as<double>());
        check_cuda(cudaGetLastError(), "peak");
    }
    // f(integral constant log2 n) for the handle's window size (32..1024)
    template <typename F>
    void sized(F &&f) {
        switch (logn) {
            case 5: f(std::integral_constant<int, 5>()); break;
            case 6: f(std::integral_constant<int, 6>()); break;
            case 7: f(std::integral_constant<int, 7>()); break;
            case 8: f(std::integral_constant<int, 8>()); break;
            case 9: f(std::integral_constant<int, 9>()); break;
            default: f(std::integral_constant<int, 10>()); break;
        }
    }
};

namespace {

template <typename F>
int fguarded(gbdic_fourier *f, F &&fn) {
    if (!f) {
        g_fourier_error = "null handle";
        return GBDIC_EINVAL;
    }
    try {
        check_cuda(cudaSetDevice(f->device), "cudaSetDevice");
        fn();
        return GBDIC_OK;
    } catch (const Failure &x) {
        f->error = x.message;
        return x.code;
    } catch (const std::exception &x) {
        f->error = x.what();
        return GBDIC_ECUDA;
    }
}

}  // namespace

extern "C" {

const char *gbdic_fourier_last_error(const gbdic_fourier *f) { return f ? f->error.c_str() : g_fourier_error.c_str(); }

int gbdic_fourier_create(int32_t device, const uint8_t *window, const uint8_t *allowed, int32_t size,
                         gbdic_fourier **out) {
    if (!out || !window) {
        g_fourier_error = "window and output handle are required";
        return GBDIC_EINVAL;
    }
    *out = nullptr;
    if (size < 32 || size > 1024 || (size & (size - 1))) {
        g_fourier_error = "window size must be a power of two from 32 to 1024";
        return GBDIC_EINVAL;
    }
    auto *f = new gbdic_fourier();
    try {
        f->device = device;
        check_cuda(cudaSetDevice(device), "cudaSetDevice");
        check_cuda(cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking), "stream");
        check_cuda(cudaEventCreateWithFlags(&f->fork, cudaEventDisableTiming), "event");
        check_cuda(cudaEventCreateWithFlags(&f->join, cudaEventDisableTiming), "event");
        f->size = size;
        f->half = size / 2;
        f->logn = log2i(size);
        const size_t px = (size_t)size * size, hpx = (size_t)f->half * f->half;
        f->window.ensure(px);
        f->taper.ensure((size_t)f->half * sizeof(double));
        f->ref_spectrum.ensure((px / 2 + size) * sizeof(double2));
        f->rows.ensure(px / 4 * sizeof(double2));
        f->work.ensure(px / 2 * sizeof(double2));
        f->corr.ensure(px * sizeof(double));
        f->ref_samples.ensure(hpx * sizeof(double));
        f->cur_samples.ensure(hpx * sizeof(double));
        f->allowed_samples.ensure(hpx);
        f->sums.ensure(3 * sizeof(unsigned long long));
        f->result.ensure(8 * sizeof(double));
        f->twiddle.ensure((size_t)(size / 2) * sizeof(double2));
        f->partials.ensure((size_t)(kCorrAt + 6 * kCorrCtas) * sizeof(double));
        f->host_window.ensure(px);
        f->host_result.ensure(8 * sizeof(double));
        twiddle_kernel<<<(size / 2 + 255) / 256, 256, 0, f->stream>>>(f->twiddle.as<double2>(), size);
        check_cuda(cudaGetLastError(), "twiddles");
        // Hann taper of `half` points: 0.5 - 0.5 cos(2 pi k / (half - 1)).
        std::vector<double> taper((size_t)f->half);
        const double pi = 3.14159265358979323846;
        for (int k = 0; k < f->half; ++k) taper[(size_t)k] = 0.5 - 0.5 * cos(2.0 * pi * k / (double)(f->half - 1));
        check_cuda(cudaMemcpyAsync(f->taper.get(), taper.data(), taper.size() * sizeof(double), cudaMemcpyHostToDevice,
                                   f->stream), "taper");
        check_cuda(cudaMemcpyAsync(f->window.get(), window, px, cudaMemcpyHostToDevice, f->stream), "window");
        const uint8_t *allow = nullptr;
        if (allowed) {
            f->allowed.ensure(px);
            check_cuda(cudaMemcpyAsync(f->allowed.get(), allowed, px, cudaMemcpyHostToDevice, f->stream), "ROI window");
            allow = f->allowed.as<uint8_t>();
        }
        f->sized([&](auto logn) { f->reference_spectrum<decltype(logn)::value>(allow); });
        check_cuda(cudaStreamSynchronize(f->stream), "reference spectrum");
    } catch (const Failure &x) {
        g_fourier_error = x.message;
        delete f;
        return x.code;
    }
    *out = f;
    return GBDIC_OK;
}

int gbdic_fourier_destroy(gbdic_fourier *f) {
    delete f;
    return GBDIC_OK;
}

int gbdic_fourier_estimate(gbdic_fourier *f, const uint8_t *frame, int64_t row_stride, int32_t height, int32_t x,
                           int32_t y, int32_t device_frame, double *out) {
    return fguarded(f, [&] {
        if (!frame || !out) fail(GBDIC_EINVAL, "frame and output are required");
        const int n = f->size;
        if (row_stride < x + n || x < 0 || y < 0 || y + n > height) fail(GBDIC_EINVAL, "window outside the frame");
        if (device_frame) {
            check_cuda(cudaMemcpy2DAsync(f->window.get(), n, frame + (size_t)y * row_stride + x, (size_t)row_stride, n, n,
                                         cudaMemcpyDeviceToDevice, f->stream), "window copy");
        } else {
            uint8_t *dst = f->host_window.as<uint8_t>();
            for (int r = 0; r < n; ++r) std::memcpy(dst + (size_t)r * n, frame + (size_t)(y + r) * row_stride + x, n);
            check_cuda(cudaMemcpyAsync(f->window.get(), dst, (size_t)n * n, cudaMemcpyHostToDevice, f->stream),
                       "window upload");
        }
        f->sized([&](auto logn) { f->correlate<decltype(logn)::value>(f->stream); });
        double *pc = f->partials.as<double>() + kCorrAt;
        overlap_partial_kernel<<<kCorrCtas, kCorrThreads, 0, f->stream>>>(
            f->ref_samples.as<double>(), f->allowed_samples.as<uint8_t>(), f->cur_samples.as<double>(), f->half,
            f->result.as<double>(), pc);
        check_cuda(cudaGetLastError(), "overlap correlation");
        overlap_final_kernel<<<1, 192, 0, f->stream>>>(pc, f->result.as<double>());
        check_cuda(cudaGetLastError(), "overlap correlation");
        check_cuda(cudaMemcpyAsync(f->host_result.as<double>(), f->result.get(), 6 * sizeof(double), cudaMemcpyDeviceToHost,
                                   f->stream), "peak readback");
        unsigned long long window_sums[3];
        check_cuda(cudaMemcpyAsync(window_sums, f->sums.get(), sizeof(window_sums), cudaMemcpyDeviceToHost, f->stream),
                   "window statistics");
        check_cuda(cudaStreamSynchronize(f->stream), "phase correlation");
        double *r = f->host_result.as<double>();
        const double wn = (double)window_sums[1], wmean = (double)window_sums[0] / wn;
        out[6] = sqrt(fmax((double)window_sums[2] / wn - wmean * wmean, 0.0));
        const int half = f->half;
        const int px = (int)r[1], py = (int)r[2];
        const int dx = 2 * (px < half ? px : px - n), dy = 2 * (py < half ? py : py - n);
        const double peak = r[0], mean = r[3], sd = r[4];
        out[0] = dx;
        out[1] = dy;
        out[2] = (peak - mean) / (sd > 1e-12 ? sd : 1e-12);
        const double ox = (double)(n - abs(dx) > 0 ? n - abs(dx) : 0), oy = (double)(n - abs(dy) > 0 ? n - abs(dy) : 0);
        out[3] = ox * oy / ((double)n * n);
        out[4] = r[5];
        out[5] = peak;
    });
}

int gbdic_fourier_shift_device(gbdic_fourier *f, const uint8_t *frame, int64_t row_stride, int32_t height, int32_t x,
                               int32_t y, float multiplier, float *rows, int32_t count, int32_t pitch, void *stream) {
    return fguarded(f, [&] {
        if (!frame || !rows || count < 0 || pitch < 4) fail(GBDIC_EINVAL, "frame, rows (pitch >= 4) and count >= 0 are required");
        const int n = f->size;
        if (row_stride < x + n || x < 0 || y < 0 || y + n > height) fail(GBDIC_EINVAL, "window outside the frame");
        // The caller's stream orders everything: the transform buffers belong
        // to this handle, so calls on one handle must not overlap.
        cudaStream_t s = static_cast<cudaStream_t>(stream);
        // Outside a stream capture the call is ordered after the handle's own
        // stream (host-path estimates) and before its later work; inside a
        // capture (a CUDA graph of the caller's frame) the graph's launches
        // are ordered by the caller, and the handle's stream stays out of it.
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        check_cuda(cudaStreamIsCapturing(s, &capture), "capture query");
        const bool capturing = capture != cudaStreamCaptureStatusNone;
        if (!capturing) {
            check_cuda(cudaEventRecord(f->fork, f->stream), "event");
            check_cuda(cudaStreamWaitEvent(s, f->fork, 0), "event wait");
        }
        check_cuda(cudaMemcpy2DAsync(f->window.get(), n, frame + (size_t)y * row_stride + x, (size_t)row_stride, n, n,
                                     cudaMemcpyDeviceToDevice, s), "window copy");
        f->sized([&](auto logn) { f->correlate<decltype(logn)::value>(s); });
        if (count > 0) {
            const int blocks = count < 256 * 64 ? (count + 255) / 256 : 64;
            shift_rows_kernel<<<blocks, 256, 0, s>>>(f->result.as<double>(), f->sums.as<unsigned long long>(), n,
                                                     multiplier, rows, count, pitch);
            check_cuda(cudaGetLastError(), "shift rows");
        }
        // Later host-path estimates on the handle's own stream wait for this one.
        if (!capturing) {
            check_cuda(cudaEventRecord(f->join, s), "event");
            check_cuda(cudaStreamWaitEvent(f->stream, f->join, 0), "event wait");
        }
    });
}

}  // extern "C"
