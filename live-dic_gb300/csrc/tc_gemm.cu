// BF16 tensor-core GEMM for the learned seed network (sm_103a, tcgen05).
//
//   D[m, n] (+)= sum_k A[m, k] * B[n, k]   (+ bias[n], ReLU)
//
// A (M x K) and B (N x K) are row-major BF16 with K contiguous ("K-major");
// D is FP32 and/or BF16 with row stride ldd.  M is a multiple of 128, N of
// the tile width BN, K (per split) of 64; callers pad.
//
// Persistent CTAs, up to two to an SM, walk the 128 x BN output tiles (x K
// splits).  A CTA's warps have roles that run ahead of each other:
//   * one thread issues TMA loads of 128x64 A and BNx64 B tiles (128-byte
//     swizzle) into a shared-memory ring, each stage guarded by a full/empty
//     mbarrier pair;
//   * one thread issues tcgen05.mma (M=128, N=BN, K=16, FP32 accumulator in
//     tensor memory), four per 64-wide stage, releases each stage with
//     tcgen05.commit on its empty barrier, and alternates between two
//     accumulators, so that a tile's MMAs run during the last one's epilogue;
//   * four warps read a finished accumulator's lanes with tcgen05.ld, apply the
//     epilogue and release it.
// Convolution GEMMs can gather operand A in the kernel (implicit GEMM): eight
// more warps fill each stage's A tile with 16-byte cp.async copies straight
// from the NHWC tensor (an im2col row of the forward, or the data-gradient
// gather of the output gradient; zero-filled outside the image), at the
// positions the 128-byte swizzle gives them, from a table of the tile's 128 row
// origins; each thread's arrival on the stage's full barrier follows its
// copies, and the MMA issuer fences them to the async proxy that tcgen05.mma
// reads through; TMA still loads B.  The 9x-expanded im2col matrix is never
// written or read.  The data-gradient GEMM orders its rows by the input
// pixel's stride-2 parity class and skips the K blocks of the taps that are
// zero for the tile's class (9 of the 36 class-tap pairs remain).
// What bounds these shapes (K loops of 1 to 18 blocks) is not the tensor cores
// but the bytes: 3 to 5 TB/s of gathers from L2, activations and results.
// Batch 512, before (a CTA per tile, its start,
// loop and epilogue one after the other) -> here: data gradient 32 channels
// (4,096 tiles of 1 to 4 K blocks, masked) 72 -> 48 us, 64 channels 37 -> 24;
// forward 2 -> 32 channels (4,096 tiles of one) 46 -> 21, 32 -> 64 34 -> 22,
// 128 -> 64 at 2 x 2 (16 tiles of 18) 15 -> 14.
// Every mbarrier wait is bounded: on expiry the CTA records an error code and
// carries on, so a fault of the pipeline ends the kernel instead of hanging.
// Before a failed CTA frees its tensor memory and exits, it waits (bounded
// again) for the copies of every stage the producer armed but the MMA issuer
// never consumed, and for the MMAs it did issue, so no bulk copy or MMA is
// left writing into the CTA's shared or tensor memory.
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdint>

#include "gbdic_kernels.h"

namespace gbdic {
namespace {

#ifndef GBDIC_GEMM_STAGES
#define GBDIC_GEMM_STAGES 6
#endif
#ifndef GBDIC_GATHER_WARPS
#define GBDIC_GATHER_WARPS 8
#endif
constexpr int kStages = GBDIC_GEMM_STAGES;
// Warps that fill a gathered operand A.
constexpr int kGatherWarps = GBDIC_GATHER_WARPS;
constexpr int kGatherThreads = 32 * kGatherWarps;
constexpr int kMaxThreads = 64 + kGatherThreads;  // of the weight gradient's CTAs
static_assert(kGatherWarps == 2 || kGatherWarps == 4 || kGatherWarps == 8, "1024 chunks per stage split evenly");
// Weight gradient: stages of 64 pixels.
constexpr int kWgradStages = 3;
constexpr int kBM = 128;
constexpr int kBK = 64;
constexpr uint32_t kSpinLimit = 1u << 22;

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Bounded parity wait; returns false on expiry.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity) {
    const uint32_t addr = smem_u32(bar);
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        uint32_t done;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(addr), "r"(parity)
            : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Arrives (one of the barrier's expected count) once this thread's cp.async
// copies so far have landed; the thread goes on.
__device__ __forceinline__ void mbar_arrive_copies(uint64_t *bar) {
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 16 bytes from global to shared memory; src_bytes 0 writes zeros.
__device__ __forceinline__ void cp_async_16(uint32_t dst, const void *src, uint32_t src_bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(src_bytes) : "memory");
}

// Row descriptor of the gathered operand, built once per CTA: the chunk
// (8-element) offset of the row's origin in the NHWC source, and a bit per tap
// 3 ky + kx whose pixel lies in the tensor (and, for the data gradient, exists).
// Every tap's pixel is then the origin plus an offset of the tap alone
// (gather_tap), so a copy costs a bit test and an addition.
// im2col row m = (b, oy, ox): origin (2 oy - 1, 2 ox - 1) of input image b, tap
// (ky, kx) reads pixel (y + ky, x + kx).
// Data-gradient row m = (b, iy, ix): tap (ky, kx) reads output-gradient pixel
// ((iy + 1 - ky) / 2, (ix + 1 - kx) / 2) when both are whole and inside the
// OH x OW grid; with whole quotients that is ((iy + 1) >> 1) - (ky >> 1), likewise
// in x.  Same mapping as im2col_vec_kernel / dgrad_gather_vec_kernel (nn_ops.cu).
//
// Parity classes (kGatherDgradClasses, even H and W): the rows are ordered
// by class c = 2 py + px of the input pixel (iy, ix) = (2u + py, 2v + px),
// then by (b, u, v); a class holds B OH OW rows (a multiple of 128), so a
// tile never mixes classes.  In class (py, px) the tap (ky, kx) is nonzero
// only for ky = 1 (py = 0) or ky in {0, 2} (py = 1), likewise kx, and reads
// output-gradient pixel (u + dy, v + dx), dy = 1 for (py, ky) = (1, 0), else
// 0.  The other taps' K blocks are zero for every row of the tile and are
// skipped: they would add exact zeros to the accumulator.
__device__ __forceinline__ int2 gather_row(const TcGemmArgs &a, int m, int cls) {
    const NnConvShape &s = a.conv;
    int base, mask = 0;
    if (a.gather == kGatherIm2col) {
        const int ox = m % s.OW, t = m / s.OW, oy = t % s.OH, b = t / s.OH;
        const int y = 2 * oy - 1, x = 2 * ox - 1;
        base = ((b * s.H + y) * s.W + x) * (s.C / 8);
#pragma unroll
        for (int tap = 0; tap < 9; ++tap)
            mask |= ((unsigned)(y + tap / 3) < (unsigned)s.H && (unsigned)(x + tap % 3) < (unsigned)s.W) << tap;
        return make_int2(base, mask);
    }
    if (a.gather == kGatherDgradClasses) {
        const int local = m % (s.B * s.OH * s.OW);
        const int v = local % s.OW, t = local / s.OW, u = t % s.OH, b = t / s.OH;
        base = ((b * s.OH + u) * s.OW + v) * (s.Cout / 8);
#pragma unroll
        for (int tap = 0; tap < 9; ++tap)
            mask |= (u + ((cls >> 1) && tap / 3 == 0) < s.OH && v + ((cls & 1) && tap % 3 == 0) < s.OW) << tap;
        return make_int2(base, mask);
    }
    const int ix = m % s.W, t = m / s.W, iy = t % s.H, b = t / s.H;
    base = ((b * s.OH + ((iy + 1) >> 1)) * s.OW + ((ix + 1) >> 1)) * (s.Cout / 8);
#pragma unroll
    for (int tap = 0; tap < 9; ++tap) {
        const int ty = iy + 1 - tap / 3, tx = ix + 1 - tap % 3;
        mask |= (!((ty | tx) & 1) && (unsigned)ty < (unsigned)(2 * s.OH) && (unsigned)tx < (unsigned)(2 * s.OW)) << tap;
    }
    return make_int2(base, mask);
}

// Chunk offset of tap (ky, kx) from a row's origin.
__device__ __forceinline__ int gather_tap(const TcGemmArgs &a, int ky, int kx, int cls) {
    const NnConvShape &s = a.conv;
    if (a.gather == kGatherIm2col) return (ky * s.W + kx) * (s.C / 8);
    const int cell = a.gather == kGatherDgradClasses
                         ? ((cls >> 1) && ky == 0 ? s.OW : 0) + ((cls & 1) && kx == 0 ? 1 : 0)
                         : -((ky >> 1) * s.OW + (kx >> 1));
    return cell * (s.Cout / 8);
}

// Parity class of the tile starting at row m0 (class mode), else 0.
__device__ __forceinline__ int gather_class(const TcGemmArgs &a, int m0) {
    return a.gather == kGatherDgradClasses ? m0 / (a.conv.B * a.conv.OH * a.conv.OW) : 0;
}

// K blocks of one CTA: all of its split, or in class mode those of the
// class's nonzero taps (Cout / 64 blocks per tap).
__device__ __forceinline__ int kblock_count(const TcGemmArgs &a, int k_len, int cls) {
    if (a.gather != kGatherDgradClasses) return k_len / kBK;
    return ((cls >> 1) ? 2 : 1) * ((cls & 1) ? 2 : 1) * (a.conv.Cout / kBK);
}

// First K element of the CTA's kb-th K block.
__device__ __forceinline__ int kblock_offset(const TcGemmArgs &a, int kb, int k_begin, int cls) {
    if (a.gather != kGatherDgradClasses) return k_begin + kb * kBK;
    const int per_tap = a.conv.Cout / kBK, t = kb / per_tap, within = kb - t * per_tap;
    const int nx = (cls & 1) ? 2 : 1, ty = t / nx, tx = t - ty * nx;
    const int ky = (cls >> 1) ? 2 * ty : 1, kx = (cls & 1) ? 2 * tx : 1;
    return (ky * 3 + kx) * a.conv.Cout + within * kBK;
}

// Output row of accumulator row m (class mode: back to (b, iy, ix) order).
__device__ __forceinline__ int output_row(const TcGemmArgs &a, int m, int cls) {
    if (a.gather != kGatherDgradClasses) return m;
    const NnConvShape &s = a.conv;
    const int local = m - cls * (s.B * s.OH * s.OW);
    const int v = local % s.OW, t = local / s.OW, u = t % s.OH, b = t / s.OH;
    return (b * s.H + 2 * u + (cls >> 1)) * s.W + 2 * v + (cls & 1);
}

__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::
            "r"(smem_u32(dst)),
        "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}

// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups
// 1024 bytes apart (SBO), leading offset unused for swizzled K-major (1).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFFu);
    d |= (uint64_t)1u << 16;                  // LBO (unused)
    d |= (uint64_t)(1024u >> 4) << 32;        // SBO
    d |= (uint64_t)1u << 46;                  // descriptor version (sm_100 family)
    d |= (uint64_t)2u << 61;                  // 128-byte swizzle
    return d;
}

// Instruction descriptor, kind::f16: FP32 accumulator, BF16 A and B, both
// K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t instr_desc(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void named_barrier(int id, int threads) {
    __syncwarp();
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Warps of a CTA: 0 .. 3 epilogue (the quarter of tensor memory a warp may read
// goes by its index), then the gatherers, the TMA producer, the MMA issuer.
constexpr int kGatherWarp0 = 4, kTmaWarp = kGatherWarp0 + kGatherWarps, kMmaWarp = kTmaWarp + 1;
constexpr int kGemmThreads = 32 * (kMmaWarp + 1);

template <int BN>
__global__ void __launch_bounds__(kGemmThreads, 2) tc_gemm_kernel(const __grid_constant__ CUtensorMap map_a,
                                                                  const __grid_constant__ CUtensorMap map_b,
                                                                  TcGemmArgs args) {
    constexpr uint32_t kBytesA = kBM * kBK * 2;
    constexpr uint32_t kBytesB = BN * kBK * 2;
    constexpr uint32_t kStageBytes = kBytesA + kBytesB;
    constexpr uint32_t kAccCols = BN < 32 ? 32 : BN;  // columns of one of the two accumulators
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[kStages], empty_bar[kStages], acc_full[2], acc_empty[2], done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ int issued_kb, consumed_kb;  // K blocks whose loads were issued / consumed
    __shared__ int2 row_tab[2][kBM];        // gather mode: descriptors of the tile's rows
    __shared__ float column_sum[2][4][BN];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int n_tiles = args.N / BN, m_tiles = args.M / kBM, k_len = args.K / args.k_split;
    const int tiles = n_tiles * m_tiles * args.k_split;
    const int nst = args.ring;

    if (tid == 0) {
        // Full barriers: the TMA producer's arrive (with the stage's bytes),
        // plus one arrive per gathering thread in gather mode.
        const uint32_t full_count = args.gather ? 1u + (uint32_t)kGatherThreads : 1u;
        for (int s = 0; s < nst; ++s) {
            mbar_init(&full_bar[s], full_count);
            mbar_init(&empty_bar[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 4);
        }
        mbar_init(&done_bar, 1);
        failed = 0;
        issued_kb = 0;
        consumed_kb = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(2 * kAccCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    // Every role walks the CTA's tiles in the same order (n fastest, then m,
    // then the K split); K blocks are numbered through all of them, block g in
    // stage g % nst.  A role whose wait expires sets `failed` and takes no
    // further part, but goes on to meet the named barriers of its group.
    if (warp == kTmaWarp && lane == 0) {
        int g = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x) {
            const int r = t / n_tiles, z = r / m_tiles;
            const int n0 = (t - r * n_tiles) * BN, m0 = (r - z * m_tiles) * kBM, k_begin = z * k_len;
            const int cls = gather_class(args, m0), num_kb = kblock_count(args, k_len, cls);
            for (int kb = 0; kb < num_kb; ++kb, ++g) {
                const int s = g % nst;
                if (g >= nst && !mbar_wait(&empty_bar[s], ((g / nst) - 1) & 1)) {
                    atomicExch(&failed, 1);
                    ok = false;
                    break;
                }
                uint8_t *sa = smem + s * kStageBytes;
                uint8_t *sb = sa + kBytesA;
                mbar_expect_tx(&full_bar[s], args.gather ? kBytesB : kStageBytes);
                const int kx = kblock_offset(args, kb, k_begin, cls);
                if (!args.gather) tma_load_2d(sa, &map_a, &full_bar[s], kx, m0);
                tma_load_2d(sb, &map_b, &full_bar[s], kx, n0);
            }
        }
        issued_kb = g;
    } else if (warp == kMmaWarp && lane == 0) {
        constexpr uint32_t idesc = instr_desc(kBM, BN);
        int g = 0, i = 0;
        bool ok = true;
        for (int t = blockIdx.x; ok && t < tiles; t += gridDim.x, ++i) {
            const int m0 = (t / n_tiles) % m_tiles * kBM;
            const int num_kb = kblock_count(args, k_len, gather_class(args, m0));
            const int acc = i & 1;
            if (i >= 2 && !mbar_wait(&acc_empty[acc], ((i >> 1) - 1) & 1)) {
                atomicExch(&failed, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; kb < num_kb; ++kb, ++g) {
                const int s = g % nst;
                if (!mbar_wait(&full_bar[s], (g / nst) & 1)) {
                    atomicExch(&failed, 1);
                    ok = false;
                    break;
                }
                // gathered bytes (generic proxy) before the MMA's reads (async proxy)
                if (args.gather) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t a_addr = smem_u32(smem + s * kStageBytes);
                const uint32_t b_addr = a_addr + kBytesA;
#pragma unroll
                for (int kk = 0; kk < kBK / 16; ++kk) {
                    const uint64_t da = smem_desc(a_addr + kk * 32);
                    const uint64_t db = smem_desc(b_addr + kk * 32);
                    const uint32_t accumulate = (kb > 0 || kk > 0) ? 1u : 0u;
                    asm volatile(
                        "{\n\t.reg .pred p;\n\t"
                        "setp.ne.b32 p, %4, 0;\n\t"
                        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem + acc * kAccCols),
                        "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
                }
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&empty_bar[s]))
                             : "memory");
            }
            if (ok)
                asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                                 smem_u32(&acc_full[acc]))
                             : "memory");
        }
        consumed_kb = g;
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&done_bar))
                     : "memory");
    } else if (args.gather && warp >= kGatherWarp0 && warp < kTmaWarp) {
        // Operand A producers: kGatherThreads threads, thread g copies chunk
        // j = g % 8 of rows g / 8 + (kGatherThreads / 8) i of the 128 x 64
        // tile, so eight threads read one row's 128 contiguous bytes (one
        // tap, or two for C = 32).
        // Row r, chunk j lands at byte r * 128 + ((j ^ (r % 8)) * 16) of the
        // 1024-byte-aligned stage, the 128-byte swizzle of the TMA loads it
        // replaces.  Each thread's arrival on the stage's full barrier is left
        // to its copies, so the ring alone limits how far the gathering runs
        // ahead.  (Waiting for the oldest of three stages in flight and arriving
        // warp by warp: the 32-channel data gradient 48 -> 51 us, the 32 -> 64
        // channel weight gradient 26 -> 33.)
        constexpr int kRowStep = kGatherThreads / 8, kRowsPerThread = kBM / kRowStep;
        static_assert(kRowStep % 8 == 0, "a thread's rows share their swizzle phase");
        const int gt = tid - 32 * kGatherWarp0, j = gt & 7, r0 = gt >> 3;
        const uint4 *src = static_cast<const uint4 *>(args.a);
        const uint32_t place = (uint32_t)(r0 * 128 + ((j ^ (r0 & 7)) << 4));  // rows step by multiples of 8
        const bool classes = args.gather == kGatherDgradClasses;
        const int per_tap = (args.gather == kGatherIm2col ? args.conv.C : args.conv.Cout) / 8;
        int g = 0, i = 0;
        bool dead = false;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
            const int r = t / n_tiles, z = r / m_tiles;
            const int m0 = (r - z * m_tiles) * kBM, k_begin = z * k_len;
            const int cls = gather_class(args, m0), num_kb = kblock_count(args, k_len, cls);
            // The tile's row descriptors; the other table is still being read
            // at most by threads that have not passed this barrier.
            if (gt < kBM) row_tab[i & 1][gt] = gather_row(args, m0 + gt, cls);
            named_barrier(1, kGatherThreads);
            if (dead) continue;
            int base[kRowsPerThread], mask[kRowsPerThread];
#pragma unroll
            for (int k = 0; k < kRowsPerThread; ++k) {
                const int2 row = row_tab[i & 1][r0 + kRowStep * k];
                base[k] = row.x;
                mask[k] = row.y;
            }
            // The chunk's tap and its chunk within the tap, advanced by 8 chunks a K
            // block (class mode: over the class's taps).
            const int q = kblock_offset(args, 0, k_begin, cls) / 8 + j;
            const int kx_first = classes && !(cls & 1) ? 1 : 0, kx_step = classes ? 2 : 1;
            const int ky_step = classes && (cls >> 1) ? 2 : 1;
            int tap = q / per_tap, c8 = q - tap * per_tap, ky = tap / 3, kx = tap - 3 * ky;
            int delta = gather_tap(args, ky, kx, cls);
            for (int kb = 0; kb < num_kb; ++kb, ++g) {
                const int s = g % nst;
                if (g >= nst) {
                    int ok = 1;
                    if (lane == 0) ok = mbar_wait(&empty_bar[s], ((g / nst) - 1) & 1) ? 1 : 0;
                    ok = __shfl_sync(0xffffffffu, ok, 0);
                    if (!ok) {
                        if (lane == 0) atomicExch(&failed, 1);
                        dead = true;
                        break;
                    }
                }
                const uint32_t dst = smem_u32(smem + s * kStageBytes) + place;
                const int offset = delta + c8, bit = 3 * ky + kx;  // beyond the ninth tap (K padding): no bit is set
#pragma unroll
                for (int k = 0; k < kRowsPerThread; ++k) {
                    const bool in = (mask[k] >> bit) & 1;
                    cp_async_16(dst + (uint32_t)(kRowStep * k * 128), src + (in ? base[k] + offset : 0), in ? 16u : 0u);
                }
                mbar_arrive_copies(&full_bar[s]);
                c8 += 8;
                if (c8 >= per_tap) {
                    do {
                        c8 -= per_tap;
                        kx += kx_step;
                        if (kx > 2) {
                            kx = kx_first;
                            ky += ky_step;
                        }
                    } while (c8 >= per_tap);
                    delta = gather_tap(args, ky, kx, cls);
                }
            }
        }
        // Drain: every issued copy lands before the warp moves on (also after
        // a failed wait, so no copy is left writing into shared memory).
        asm volatile("cp.async.wait_all;" ::: "memory");
    } else if (warp < 4) {
        // Epilogue: warp w owns accumulator lanes (rows) 32w .. 32w + 31.
        const bool wide = args.ldd % 8 == 0 && (args.k_split == 1 || args.split_stride % 8 == 0) &&
                          (reinterpret_cast<uintptr_t>(args.d_bf16) & 15) == 0;
        int i = 0;
        bool dead = false;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++i) {
            const int rest = t / n_tiles, z = rest / m_tiles, m_tile = rest - z * m_tiles;
            const int n0 = (t - rest * n_tiles) * BN, m0 = m_tile * kBM, acc = i & 1;
            const int row = output_row(args, m0 + warp * 32 + lane, gather_class(args, m0));
            if (!dead) {
                if (args.mask != nullptr) {
                    // the row's activations, on their way while the last MMAs finish
                    const char *m = reinterpret_cast<const char *>(static_cast<const __nv_bfloat16 *>(args.mask) +
                                                                   (size_t)row * args.ldd + n0);
#pragma unroll
                    for (int b = 0; b < 2 * BN; b += 64) asm volatile("prefetch.global.L1 [%0];" ::"l"(m + b));
                }
                if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (i >> 1) & 1))) {
                    if (lane == 0) atomicExch(&failed, 1);
                    dead = true;
                }
            }
            if (!dead) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t lane_base = tmem + acc * kAccCols + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
                for (int c = 0; c < BN; c += 16) {
                    uint32_t r[16];
                    asm volatile(
                        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                        "%14, %15}, [%16];"
                        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                        : "r"(lane_base + (uint32_t)c));
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    float v[16];
#pragma unroll
                    for (int j = 0; j < 16; ++j) {
                        v[j] = __uint_as_float(r[j]);
                        if (args.bias) v[j] = v[j] + args.bias[n0 + c + j];
                        if (args.relu) v[j] = fmaxf(v[j], 0.0f);
                    }
                    if (args.mask != nullptr) {
                        // ReLU backward where the row's activation is zero, and the sums
                        // over the warp's 32 rows: halves of the columns go to halves of
                        // the lanes, until lane pair l holds column l / 2.
                        const uint4 *m = reinterpret_cast<const uint4 *>(static_cast<const __nv_bfloat16 *>(args.mask) +
                                                                         (size_t)row * args.ldd + n0 + c);
                        const uint4 m0 = __ldg(m), m1 = __ldg(m + 1);
                        const uint32_t words[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const __nv_bfloat162 y = *reinterpret_cast<const __nv_bfloat162 *>(&words[j]);
                            if (!(__bfloat162float(y.x) > 0.0f)) v[2 * j] = 0.0f;
                            if (!(__bfloat162float(y.y) > 0.0f)) v[2 * j + 1] = 0.0f;
                        }
                        float t[16];
#pragma unroll
                        for (int j = 0; j < 16; ++j) t[j] = v[j];
#pragma unroll
                        for (int half = 8; half >= 1; half >>= 1) {
                            const bool upper = lane & (2 * half);
#pragma unroll
                            for (int j = 0; j < half; ++j) {
                                const float keep = upper ? t[j + half] : t[j], send = upper ? t[j] : t[j + half];
                                t[j] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * half);
                            }
                        }
                        t[0] += __shfl_xor_sync(0xffffffffu, t[0], 1);
                        if ((lane & 1) == 0) column_sum[acc][warp][c + (lane >> 1)] = t[0];
                    }
                    const size_t base = (size_t)z * (size_t)args.split_stride + (size_t)row * args.ldd + n0 + c;
                    if (args.d_f32) {
                        float4 *o = reinterpret_cast<float4 *>(args.d_f32 + base);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            float4 x = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                            if (args.accumulate) {
                                const float4 y = o[j];
                                x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
                            }
                            o[j] = x;
                        }
                    }
                    if (args.d_bf16) {
                        // A store instruction per four bytes of a row touched 32 lines
                        // for 128 bytes and was these kernels' time: 16-byte ones
                        // where the rows allow it.
                        uint32_t w[8];
#pragma unroll
                        for (int j = 0; j < 8; ++j) {
                            const __nv_bfloat162 two = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
                            w[j] = *reinterpret_cast<const uint32_t *>(&two);
                        }
                        __nv_bfloat16 *o = static_cast<__nv_bfloat16 *>(args.d_bf16) + base;
                        if (wide) {
                            reinterpret_cast<uint4 *>(o)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                            reinterpret_cast<uint4 *>(o)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                        } else {
#pragma unroll
                            for (int j = 0; j < 8; ++j) reinterpret_cast<uint32_t *>(o)[j] = w[j];
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[acc]);
            }
            if (args.mask != nullptr) {
                named_barrier(2, 128);
                if (!dead)
                    for (int c = tid; c < BN; c += 128) {
                        const float(*sum)[BN] = column_sum[acc];
                        args.column_partial[(size_t)(n0 + c) * m_tiles + m_tile] =
                            (sum[0][c] + sum[1][c]) + (sum[2][c] + sum[3][c]);
                    }
            }
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        if (lane == 0 && failed) {
            // The producer runs at most nst K blocks ahead of the issuer,
            // so the unconsumed blocks occupy distinct stages.
            for (int kb = consumed_kb; kb < issued_kb; ++kb) mbar_wait(&full_bar[kb % nst], (kb / nst) & 1);
            mbar_wait(&done_bar, 0);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * kAccCols));
    }
    if (tid == 0 && failed && args.error) atomicExch(args.error, 1);
}

// ------------------------------------------------------- weight gradient
// dW^T[k][co] = sum_m A[m][k] dZ[m][co] over the output pixels m, A the im2col
// rows of the layer's input.  The reduction runs over the rows of both
// operands, so both are taken MN-major (a pixel's channels contiguous, as they
// lie in memory): neither A^T nor dZ^T is ever written.  What it replaced, the
// transposed im2col matrix of every layer and a K-major GEMM over it, moved 9 x
// the activations twice: batch 512, five layers, 109 us + 97 us, where this takes
// 84.
//
// One CTA per 128 k x BN co tile and split of m, 64 pixels to a stage: dZ by TMA
// (64-channel boxes, 128-byte swizzle; one 32-channel box, 64-byte swizzle, for
// the first layer), A gathered by eight warps with 16-byte copies to the places
// the 128-byte swizzle gives them (row r of a 64-channel group at 128 r, chunk j
// at (j ^ r % 8) 16), or, where a pixel's channels are fewer than a chunk (the
// two-channel input layer), by TMA from the forward's im2col matrix of 64
// columns.  Then the accumulator's rows 64 and up repeat the first 64 (both
// groups of the descriptor are the one tile) and are not written.
// Shared-memory matrix descriptor, MN-major: groups of 64 (32) channels `lead`
// bytes apart, groups of 8 pixels `stride` bytes apart.
__device__ __forceinline__ uint64_t smem_desc_mn(uint32_t addr, uint32_t lead, uint32_t stride, uint64_t swizzle) {
    return (uint64_t)((addr >> 4) & 0x3FFFu) | (uint64_t)((lead >> 4) & 0x3FFFu) << 16 |
           (uint64_t)((stride >> 4) & 0x3FFFu) << 32 | (uint64_t)1u << 46 | swizzle << 61;
}

template <int BN, bool GATHER>
__global__ void __launch_bounds__(GATHER ? kMaxThreads : 128, 1)
    tc_wgrad_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                    TcWgradArgs args) {
    constexpr int kPixels = 64;
    constexpr uint32_t kBytesA = (GATHER ? 2 : 1) * kPixels * 128;
    constexpr uint32_t kBytesB = BN * kPixels * 2;
    constexpr uint32_t kStageBytes = kBytesA + kBytesB;
    constexpr int kRing = kWgradStages;
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[kRing], empty_bar[kRing], done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int failed;
    __shared__ int issued_kb, consumed_kb;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint8_t *smem = reinterpret_cast<uint8_t *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const NnConvShape &s = args.conv;
    const int n0 = blockIdx.x * BN, k0 = blockIdx.y * kBM;
    const int pixels = s.B * s.OH * s.OW / args.splits, m_begin = blockIdx.z * pixels, num_kb = pixels / kPixels;

    if (tid == 0) {
        for (int i = 0; i < kRing; ++i) {
            mbar_init(&full_bar[i], GATHER ? 1u + (uint32_t)kGatherThreads : 1u);
            mbar_init(&empty_bar[i], 1);
        }
        mbar_init(&done_bar, 1);
        failed = 0;
        issued_kb = 0;
        consumed_kb = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"((uint32_t)BN));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot;

    if (warp == 0 && lane == 0) {
        int kb = 0;
        for (; kb < num_kb; ++kb) {
            const int st = kb % kRing;
            if (kb >= kRing && !mbar_wait(&empty_bar[st], ((kb / kRing) - 1) & 1)) {
                atomicExch(&failed, 1);
                break;
            }
            uint8_t *sa = smem + st * kStageBytes, *sb = sa + kBytesA;
            mbar_expect_tx(&full_bar[st], GATHER ? kBytesB : kStageBytes);
            const int m = m_begin + kb * kPixels;
            if (!GATHER) tma_load_2d(sa, &map_a, &full_bar[st], 0, m);
#pragma unroll
            for (int g = 0; g < (BN + 63) / 64; ++g)
                tma_load_2d(sb + g * kPixels * 128, &map_b, &full_bar[st], n0 + 64 * g, m);
        }
        issued_kb = kb;
    } else if (warp == 1 && lane == 0) {
        // kind::f16, FP32 accumulator, BF16 operands, both MN-major (bits 15, 16).
        constexpr uint32_t idesc = instr_desc(kBM, BN) | (1u << 15) | (1u << 16);
        constexpr uint32_t kRowB = BN < 64 ? 2 * BN : 128;  // bytes of a pixel in a group of B
        int kb = 0;
        for (; kb < num_kb; ++kb) {
            const int st = kb % kRing;
            if (!mbar_wait(&full_bar[st], (kb / kRing) & 1)) {
                atomicExch(&failed, 1);
                break;
            }
            if (GATHER) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t a_addr = smem_u32(smem + st * kStageBytes), b_addr = a_addr + kBytesA;
#pragma unroll
            for (int kk = 0; kk < kPixels / 16; ++kk) {
                const uint64_t da = smem_desc_mn(a_addr + kk * 16 * 128, GATHER ? kPixels * 128 : 0, 1024, 2);
                const uint64_t db = smem_desc_mn(b_addr + kk * 16 * kRowB, kPixels * kRowB, 8 * kRowB, BN < 64 ? 4 : 2);
                const uint32_t accumulate = (kb > 0 || kk > 0) ? 1u : 0u;
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "setp.ne.b32 p, %4, 0;\n\t"
                    "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem),
                    "l"(da), "l"(db), "r"(idesc), "r"(accumulate));
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                             smem_u32(&empty_bar[st]))
                         : "memory");
        }
        consumed_kb = kb;
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                         smem_u32(&done_bar))
                     : "memory");
    }
    if (GATHER && warp >= 2) {
        // Thread g copies chunk g % 16 (one tap's eight channels, the same for
        // every pixel) of pixels g / 16 + 16 i; the pixels advance by 64 a stage.
        constexpr int kRows = kPixels * 16 / kGatherThreads, kStep = kGatherThreads / 16;
        const int g = tid - 64, chunk = g & 15, r0 = g >> 4, j = chunk & 7;
        const int per_tap = s.C / 8, q = k0 / 8 + chunk, tap = q / per_tap, c8 = q - tap * per_tap;
        const int ky = tap / 3, kx = tap - 3 * ky;
        const bool used = tap < 9;
        const uint4 *x = static_cast<const uint4 *>(args.x);
        int ox[kRows], oy[kRows], b[kRows];
#pragma unroll
        for (int i = 0; i < kRows; ++i) {
            const int m = m_begin + r0 + kStep * i, t = m / s.OW;
            ox[i] = m - t * s.OW;
            b[i] = t / s.OH;
            oy[i] = t - b[i] * s.OH;
        }
        const int dx = kPixels % s.OW, dt = kPixels / s.OW, dy = dt % s.OH, dbatch = dt / s.OH;
        for (int kb = 0; kb < num_kb; ++kb) {
            const int st = kb % kRing;
            if (kb >= kRing) {
                int ok = 1;
                if (lane == 0) ok = mbar_wait(&empty_bar[st], ((kb / kRing) - 1) & 1) ? 1 : 0;
                ok = __shfl_sync(0xffffffffu, ok, 0);
                if (!ok) {
                    if (lane == 0) atomicExch(&failed, 1);
                    break;
                }
            }
            const uint32_t sa = smem_u32(smem + st * kStageBytes) + (uint32_t)((chunk >> 3) * kPixels * 128);
#pragma unroll
            for (int i = 0; i < kRows; ++i) {
                const int r = r0 + kStep * i, yy = 2 * oy[i] - 1 + ky, xx = 2 * ox[i] - 1 + kx;
                const bool in = used && (unsigned)yy < (unsigned)s.H && (unsigned)xx < (unsigned)s.W;
                const uint4 *src = in ? x + ((b[i] * s.H + yy) * s.W + xx) * per_tap + c8 : x;
                cp_async_16(sa + (uint32_t)(r * 128 + ((j ^ (r & 7)) << 4)), src, in ? 16u : 0u);
                ox[i] += dx;
                oy[i] += dy;
                b[i] += dbatch;
                if (ox[i] >= s.OW) { ox[i] -= s.OW; ++oy[i]; }
                if (oy[i] >= s.OH) { oy[i] -= s.OH; ++b[i]; }
            }
            mbar_arrive_copies(&full_bar[st]);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
    }
    __syncwarp();
    if (!mbar_wait(&done_bar, 0)) atomicExch(&failed, 1);
    __syncwarp();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    const int row = warp * 32 + lane;
#pragma unroll 1
    for (int c = 0; c < (warp < 4 ? BN : 0); c += 16) {
        uint32_t r[16];
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
            "%14, %15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c));
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        // Rows beyond Kp are not stored; their lanes stay for the next load,
        // which the whole warp issues (Kp need not be a multiple of 32).
        if (k0 + row < args.k_rows) {
            float4 *o = reinterpret_cast<float4 *>(args.partial +
                                                   ((size_t)blockIdx.z * args.k_rows + k0 + row) * s.Cout + n0 + c);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                o[j] = make_float4(__uint_as_float(r[4 * j]), __uint_as_float(r[4 * j + 1]), __uint_as_float(r[4 * j + 2]),
                                   __uint_as_float(r[4 * j + 3]));
        }
        __syncwarp();
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        if (lane == 0 && failed) {
            for (int kb = consumed_kb; kb < issued_kb; ++kb) mbar_wait(&full_bar[kb % kRing], (kb / kRing) & 1);
            mbar_wait(&done_bar, 0);
        }
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"((uint32_t)BN));
    }
    if (tid == 0 && failed && args.error) atomicExch(args.error, 1);
}

typedef CUresult (*EncodeTiled)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiled>(p);
    }
    return fn;
}

// 2-D BF16 row-major matrix rows x cols (cols contiguous), box box_rows x 64
// (128-byte swizzle), or x 32 (64-byte swizzle).
bool make_map(CUtensorMap *map, const void *ptr, int rows, int cols, int box_rows, int box_cols = kBK) {
    EncodeTiled fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
    const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
    const cuuint32_t estride[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estride,
              CU_TENSOR_MAP_INTERLEAVE_NONE, box_cols == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
              CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// CTAs walk their tiles, two CTAs to an SM where there are tiles for them.  The
// ring is as deep as their shared memory allows, whatever the length of a tile's
// K loop: it runs on into the next tile, whose gathering and MMAs overlap this
// one's epilogue.
constexpr int kRingBytes = 216 * 1024;  // of an SM's 227 KB, beside the CTAs' static arrays

template <int BN>
cudaError_t launch_bn(const CUtensorMap &ma, const CUtensorMap &mb, const TcGemmArgs &args, cudaStream_t stream) {
    TcGemmArgs a = args;
    constexpr int kStageBytes = kBM * kBK * 2 + BN * kBK * 2;
    const long long tiles = (long long)(a.N / BN) * (a.M / kBM) * a.k_split;
    const size_t smem_max = (size_t)kStages * kStageBytes + 1024;
    // The attribute is per device; set it once per device and tile width.
    static thread_local int configured_device = -1, sms = 0;
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    if (configured_device != device) {
        err = cudaFuncSetAttribute(tc_gemm_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_max);
        if (err == cudaSuccess) err = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        if (err != cudaSuccess) return err;
        configured_device = device;
    }
    const int per_sm = tiles > sms ? 2 : 1;
    a.ring = kRingBytes / per_sm / kStageBytes < kStages ? kRingBytes / per_sm / kStageBytes : kStages;
    const size_t smem = (size_t)a.ring * kStageBytes + 1024;
    const int grid = (int)(tiles < 2 * sms ? tiles : 2 * sms);
    tc_gemm_kernel<BN><<<grid, kGemmThreads, smem, stream>>>(ma, mb, a);
    return cudaGetLastError();
}

template <int BN, bool GATHER>
cudaError_t launch_wgrad(const CUtensorMap &ma, const CUtensorMap &mb, const TcWgradArgs &a, cudaStream_t stream) {
    const size_t smem = (size_t)kWgradStages * ((GATHER ? 2 : 1) * 64 * 128 + BN * 128) + 1024;
    static thread_local int configured_device = -1;
    int device = 0;
    cudaError_t err = cudaGetDevice(&device);
    if (err != cudaSuccess) return err;
    if (configured_device != device) {
        err = cudaFuncSetAttribute(tc_wgrad_kernel<BN, GATHER>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (err != cudaSuccess) return err;
        configured_device = device;
    }
    const dim3 grid(a.conv.Cout / BN, (a.k_rows + kBM - 1) / kBM, a.splits);
    tc_wgrad_kernel<BN, GATHER><<<grid, GATHER ? kMaxThreads : 128, smem, stream>>>(ma, mb, a);
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_tc_wgrad(const TcWgradArgs &a, cudaStream_t stream) {
    const NnConvShape &s = a.conv;
    const long long pixels = (long long)s.B * s.OH * s.OW;
    const bool gather = s.C % 8 == 0;
    if (s.B < 1 || s.H < 1 || s.W < 1 || s.OH != (s.H + 1) / 2 || s.OW != (s.W + 1) / 2 || !a.x || !a.dz ||
        !a.partial || a.splits < 1 || pixels >= (1ll << 31) || pixels % (64ll * a.splits) || s.Kp < 9 * s.C ||
        a.k_rows != s.Kp)
        return cudaErrorInvalidValue;
    if (gather) {
        // chunk offsets are 32-bit in the kernel
        if (s.Cout % 64 || (long long)s.B * s.H * s.W * (s.C / 8) >= (1ll << 31)) return cudaErrorInvalidValue;
    } else if (s.Kp != 64 || s.Cout != 32) {
        return cudaErrorInvalidValue;
    }
    if ((reinterpret_cast<uintptr_t>(a.x) | reinterpret_cast<uintptr_t>(a.dz) | reinterpret_cast<uintptr_t>(a.partial)) &
        15u)
        return cudaErrorMisalignedAddress;
    CUtensorMap ma, mb;
    if (!make_map(&mb, a.dz, (int)pixels, s.Cout, 64, gather ? 64 : 32)) return cudaErrorInvalidValue;
    if (!gather) {
        if (!make_map(&ma, a.x, (int)pixels, s.Kp, 64)) return cudaErrorInvalidValue;
        return launch_wgrad<32, false>(ma, mb, a, stream);
    }
    ma = mb;  // not read: A is gathered
    return s.Cout % 128 == 0 ? launch_wgrad<128, true>(ma, mb, a, stream) : launch_wgrad<64, true>(ma, mb, a, stream);
}

int tc_gemm_tile_n(int N) {
    if (N % 128 == 0) return 128;
    if (N % 64 == 0) return 64;
    if (N % 32 == 0) return 32;
    if (N % 16 == 0) return 16;
    return 0;
}

cudaError_t launch_tc_gemm(const TcGemmArgs &a, cudaStream_t stream) {
    const int bn = tc_gemm_tile_n(a.N);
    if (a.M <= 0 || a.N <= 0 || a.K <= 0 || a.k_split < 1 || a.M % kBM != 0 || bn == 0 ||
        a.K % (kBK * a.k_split) != 0 || a.ldd < a.N || a.ldd % 4 != 0 || !a.a || !a.b ||
        (!a.d_f32 && !a.d_bf16) || (a.mask && (!a.column_partial || a.k_split != 1 || a.ldd % 8)) ||
        (reinterpret_cast<uintptr_t>(a.mask) & 15u) || (a.accumulate && !a.d_f32) || (a.k_split > 1 && a.bias))
        return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(a.a) | reinterpret_cast<uintptr_t>(a.b)) & 15u) return cudaErrorMisalignedAddress;
    if (a.gather != kGatherNone) {
        // The gathered operand's rows and reduction length must be the
        // convolution's exactly (every row and chunk maps into the tensor).
        // k_split > 1 (partials per split, as for a plain GEMM) for the
        // im2col gather only.
        const NnConvShape &s = a.conv;
        if ((a.k_split != 1 && a.gather != kGatherIm2col) || s.B < 1 || s.H < 1 || s.W < 1 ||
            s.OH != (s.H + 1) / 2 || s.OW != (s.W + 1) / 2)
            return cudaErrorInvalidValue;
        // chunk offsets are 32-bit in the kernel
        if (a.gather == kGatherIm2col) {
            if (s.C < 8 || s.C % 8 || a.M != s.B * s.OH * s.OW || a.K != s.Kp || s.Kp < 9 * s.C ||
                (long long)s.B * s.H * s.W * (s.C / 8) >= (1ll << 31))
                return cudaErrorInvalidValue;
        } else if (a.gather == kGatherDgrad) {
            if (s.Cout < 8 || s.Cout % 8 || a.M != s.B * s.H * s.W || a.K != 9 * s.Cout ||
                (long long)s.B * s.OH * s.OW * (s.Cout / 8) >= (1ll << 31))
                return cudaErrorInvalidValue;
        } else {
            return cudaErrorInvalidValue;
        }
    }
    TcGemmArgs args = a;
    if (a.gather == kGatherDgrad) {
        // Rows by parity class, zero taps skipped: same sums (the skipped K
        // blocks are exact zeros), a quarter of the gathers and MMAs.
        const NnConvShape &s = a.conv;
        if (s.H == 2 * s.OH && s.W == 2 * s.OW && s.Cout % kBK == 0 && (s.B * s.OH * s.OW) % kBM == 0)
            args.gather = kGatherDgradClasses;
    } else if (a.gather != kGatherNone && a.gather != kGatherIm2col) {
        return cudaErrorInvalidValue;
    }
    CUtensorMap ma, mb;
    if (!make_map(&mb, args.b, args.N, args.K, bn)) return cudaErrorInvalidValue;
    if (args.gather == kGatherNone) {
        if (!make_map(&ma, args.a, args.M, args.K, kBM)) return cudaErrorInvalidValue;
    } else {
        ma = mb;  // not read: operand A is gathered
    }
    switch (bn) {
    case 128: return launch_bn<128>(ma, mb, args, stream);
    case 64: return launch_bn<64>(ma, mb, args, stream);
    case 32: return launch_bn<32>(ma, mb, args, stream);
    default: return launch_bn<16>(ma, mb, args, stream);
    }
}

}  // namespace gbdic
