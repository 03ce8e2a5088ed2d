// msgpu_dense.cu -- dense tensor-core form (MSGPU_PROP_DENSE).
//
// For a static H of modest dimension the reference's "normal" propagator
// (HSPropagator::Step dense branch, HSPropagator.cpp:92-100) applies
// U = expmat(dt G), G = -iH - K, to the factor block -- rebuilding U every
// step.  Here U is built once in FP64 on the device (scaling and squaring of
// a degree-18 Taylor polynomial, Horner form, FP64 complex GEMMs), written as
// the real 2D x 2D matrix of interleaved (re, im) pairs
//     A[2r+c][2s+d] = [[Re U, -Im U], [Im U, Re U]]_{rs}[c][d],
// and split into BF16 parts (x = x_0 + x_1 [+ x_2]).  Each step is then one
// real GEMM  Psi'^T = A Psi^T  with the trajectory block stored
// trajectory-major as interleaved complex (the reference's column-major
// factors), executed on the 5th-generation tensor cores:
//   * TMA (cp.async.bulk.tensor, 128-byte swizzle) stages A and B tiles in a
//     two-deep shared-memory ring guarded by mbarriers;
//   * one thread issues tcgen05.mma (kind::f16, BF16 inputs, FP32
//     accumulation in TMEM) for every product x_i y_j with i + j < parts;
//   * the four warps drain TMEM with tcgen05.ld and store Psi' (FP32).
// A fused epilogue kernel applies the singlet-triplet flips, evaluates the
// pair observables, advances the trapezoid, optionally restores the exact
// Haberkorn norm, and re-splits the state for the next step.
//
// Every mbarrier wait is bounded: after the limit the kernel records an
// error, waits (bounded) for its own copies in flight, frees its TMEM and
// returns.

#include "msgpu_dense.h"

#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "msgpu.h"
#include "msgpu_device.cuh"

namespace msgpu {
namespace {

constexpr int kGM = 128;          // rows of A per CTA (TMEM lanes)
constexpr int kGK = 64;           // K per stage: 64 BF16 = one 128-byte swizzle row
constexpr int kRing = 192 * 1024; // bytes of the operand ring, as many stages as fit
constexpr int kGThreads = 128;    // 4 warps
constexpr int kATile = kGM * kGK * 2;  // bytes of one A part tile (16 KB)
constexpr uint32_t kWaitLimit = 1u << 22;

// The FP32 accumulation of tcgen05.mma rounds towards zero: each MMA
// shrinks the accumulator by about half an ulp of its own magnitude, so the
// bias grows with the number of MMAs and with the size of the partial sums.
// The small split-correction products therefore go to their own accumulator
// (2^-8 of the main magnitude, so their bias is negligible), and with 3 parts
// the hi x hi product is spread over 3 K-range accumulators; the epilogue sums
// the accumulators with round-to-nearest FP32 adds (unbiased).  TMEM: NACC x BN columns,
// 512 with the wide tile.  kHalf: a tile of half as many trajectories, for blocks whose
// wide tiles would leave SMs idle (half_tiles).
template <int NS, bool kHalf = false>
struct GemmCfg {
    static constexpr int BN = (NS == 2 ? 256 : 128) / (kHalf ? 2 : 1);  // trajectories per CTA
    static constexpr int NHI = NS == 2 ? 1 : 3;          // hi x hi accumulators (K ranges)
    static constexpr int NACC = NHI + 1;                 // + the correction accumulator
    static constexpr int Cols = NACC * BN;               // TMEM columns (power of two, <= 512)
    static constexpr int BTile = BN * kGK * 2;           // bytes of one B part tile
    static constexpr int Stage = NS * kATile + NS * BTile;
    static constexpr int Stages = kRing / Stage;
    static constexpr int Smem = Stages * Stage + 1024 /*align*/ + 256 /*barriers*/;
    static_assert(Cols == (kHalf ? 256 : 512), "TMEM split");
};

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ bool mbar_try(uint32_t addr, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(addr), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait; sets *abort (shared) and returns false after the limit or
// when another role already aborted.
__device__ __forceinline__ bool mbar_wait(uint32_t addr, uint32_t parity, volatile int *abort)
{
    for (uint32_t it = 0; it < kWaitLimit; ++it) {
        if (mbar_try(addr, parity)) return true;
        if (*abort) return false;
    }
    *abort = 1;
    return false;
}

__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        :
        : "r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar)
        : "memory");
}

// UMMA shared-memory descriptor: K-major operand, swizzled rows of RowBytes (128
// or 64) in 8-row groups: SBO = 8 rows, LBO unused (1), version 1, layout type
// SWIZZLE_128B (2) or SWIZZLE_64B (4).
template <int RowBytes>
__device__ __forceinline__ uint64_t umma_desc(uint32_t addr)
{
    static_assert(RowBytes == 64 || RowBytes == 128, "one swizzle row");
    uint64_t d = 0;
    d |= static_cast<uint64_t>((addr >> 4) & 0x3FFF);
    d |= static_cast<uint64_t>(1) << 16;
    d |= static_cast<uint64_t>(8 * RowBytes >> 4) << 32;
    d |= static_cast<uint64_t>(1) << 46;
    d |= static_cast<uint64_t>(RowBytes == 128 ? 2 : 4) << 61;
    return d;
}

// kind::f16 instruction descriptor: D = F32, A = B = BF16, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc(int M, int N)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
           (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void umma_bf16(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// 32 TMEM lanes x 16 columns (one row per thread); the caller waits with
// tcgen05.wait::ld before reading v.
__device__ __forceinline__ void tmem_ld16_issue(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
}

__device__ __forceinline__ void umma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// C^T = sum over products (i, j), i + j < NS, of A_i B_j^T.
//   A parts: Dp x Dp BF16, row-major (K contiguous)  -> tensor maps ta[0..NS)
//   B parts: Mp x Dp BF16, row-major (K contiguous)  -> tensor maps tb[0..NS)
//   out:     Mp x Dp FP32, out[n][m] = C[m][n]
// grid = (trajectory tiles of this launch, Dp / 128), block = 128 threads;
// the launch covers the trajectory tiles from n_tile0 on.
template <int NS, bool kHalf>
__global__ void __launch_bounds__(kGThreads, 1)
k_dense_gemm(const __grid_constant__ CUtensorMap ta0, const __grid_constant__ CUtensorMap ta1,
             const __grid_constant__ CUtensorMap ta2, const __grid_constant__ CUtensorMap tb0,
             const __grid_constant__ CUtensorMap tb1, const __grid_constant__ CUtensorMap tb2, float *__restrict__ out,
             int Dp, int n_tile0, int *__restrict__ status)
{
    using Cfg = GemmCfg<NS, kHalf>;
    constexpr int BN = Cfg::BN;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;  // 1024-byte aligned ring (swizzle atoms)
    unsigned char *base_ptr = smem_raw + (base - raw);
    const uint32_t bars = base + Cfg::Stages * Cfg::Stage;  // full, empty (a pair a stage), accum
    uint64_t *bar_ptr = reinterpret_cast<uint64_t *>(base_ptr + Cfg::Stages * Cfg::Stage);
    volatile int *abort = reinterpret_cast<volatile int *>(bar_ptr + 16);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_ptr + 17);
    const uint32_t full0 = bars, empty0 = bars + 8 * Cfg::Stages, accum = bars + 16 * Cfg::Stages;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (n_tile0 + blockIdx.x) * BN, m0 = blockIdx.y * kGM;
    const int nk = Dp / kGK;
    const CUtensorMap *ta[3] = {&ta0, &ta1, &ta2};
    const CUtensorMap *tb[3] = {&tb0, &tb1, &tb2};

    if (threadIdx.x == 0) {
        *abort = 0;
        for (int s = 0; s < Cfg::Stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * s));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * s));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(accum));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(Cfg::Cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    grid_wait();  // the operands are the previous kernel's

    if (threadIdx.x == 0) {
        // TMA producer
        int issued = 0;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % Cfg::Stages, r = kb / Cfg::Stages;
            if (!mbar_wait(empty0 + 8 * s, (r & 1) ^ 1, abort)) break;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full0 + 8 * s),
                         "r"(Cfg::Stage));
            const uint32_t st = base + s * Cfg::Stage;
            for (int p = 0; p < NS; ++p) tma_load_2d(st + p * kATile, ta[p], kb * kGK, m0, full0 + 8 * s);
            for (int q = 0; q < NS; ++q)
                tma_load_2d(st + NS * kATile + q * Cfg::BTile, tb[q], kb * kGK, n0, full0 + 8 * s);
            issued = kb + 1;
        }
        // make sure every copy this CTA started has landed before it can exit
        for (int kb = max(0, issued - Cfg::Stages); kb < issued; ++kb) {
            const int s = kb % Cfg::Stages, r = kb / Cfg::Stages;
            for (uint32_t it = 0; it < kWaitLimit && !mbar_try(full0 + 8 * s, r & 1); ++it) {
            }
        }
    } else if (threadIdx.x == 32) {
        // MMA issuer
        constexpr uint32_t idesc = umma_idesc(kGM, BN);
        const uint32_t corr = tmem + Cfg::NHI * BN;  // correction accumulator
        uint32_t corr_on = 0;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % Cfg::Stages, r = kb / Cfg::Stages;
            if (!mbar_wait(full0 + 8 * s, r & 1, abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = base + s * Cfg::Stage;
            // hi x hi accumulator of this K range; its first MMA overwrites
            const int h = kb * Cfg::NHI / nk;
            const uint32_t hi = tmem + h * BN;
            const int first_kb = (h * nk + Cfg::NHI - 1) / Cfg::NHI;
#pragma unroll
            for (int kk = 0; kk < kGK / 16; ++kk) {
#pragma unroll
                for (int p = 0; p < NS; ++p)
#pragma unroll
                    for (int q = 0; q < NS; ++q) {
                        if (p + q >= NS) continue;
                        const uint64_t ad = umma_desc<kGK * 2>(st + p * kATile + kk * 32);
                        const uint64_t bd = umma_desc<kGK * 2>(st + NS * kATile + q * Cfg::BTile + kk * 32);
                        if (p + q == 0) {
                            umma_bf16(hi, ad, bd, idesc, (kb == first_kb && kk == 0) ? 0u : 1u);
                        } else {
                            umma_bf16(corr, ad, bd, idesc, corr_on);
                            corr_on = 1;
                        }
                    }
            }
            umma_commit(empty0 + 8 * s);
        }
        umma_commit(accum);  // tracks completion of every MMA issued above
    }
    __syncwarp();

    // epilogue: warp w drains TMEM lanes [32w, 32w+32) = rows m0 + 32w + lane
    bool ok = mbar_wait(accum, 0, abort);
    if (!ok) {
        // still wait (bounded) for the MMAs in flight before TMEM is freed
        for (uint32_t it = 0; it < kWaitLimit && !mbar_try(accum, 0); ++it) {
        }
    }
    grid_trigger();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok && !*abort) {
        const int row = m0 + 32 * warp + lane;
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(32 * warp) << 16);
#pragma unroll 1
        for (int c = 0; c < BN; c += 16) {
            // all accumulators of this column group in flight, one wait
            uint32_t v[Cfg::NACC][16];
#pragma unroll
            for (int a = 0; a < Cfg::NACC; ++a) tmem_ld16_issue(lane_base + static_cast<uint32_t>(a * BN + c), v[a]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                // round-to-nearest FP32 sums: correction first, then the hi
                // K ranges; a range with no k-block (nk < NHI) was never written
                float sum = __uint_as_float(v[Cfg::NACC - 1][j]);
#pragma unroll
                for (int a = Cfg::NHI - 1; a >= 0; --a)
                    if ((a * nk + Cfg::NHI - 1) / Cfg::NHI < nk) sum += __uint_as_float(v[a][j]);
                out[static_cast<size_t>(n0 + c + j) * Dp + row] = sum;
            }
        }
    }
    if (*abort && threadIdx.x == 0) atomicOr(status, 4);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::Cols));
    }
}

// ------------------------------------------------------------ int8 form
// Exact-accumulation GEMM.  Each operand is x = 2^e sum_{i<4} a_i / (127 254^i)
// with int8 slices a_i (a per-row scale for U, a per-trajectory scale for the
// state).  The products a_i b_j with i + j = L share the weight
// 1 / (127^2 254^L), so they are summed in one int32 accumulator per level L
// (exactly: |a_i b_j| <= 127^2 and at most 4 K-long products per level stay
// below 2^31 for K <= 8192), and the epilogue combines the four levels in FP64
// with the two scales.  The FP32 rounding of the BF16 forms is gone: the only
// errors are the slices' truncation (2^-31 of the scale) and the FP64 state.
constexpr int kIBN = 128;            // trajectories per CTA (half of them in the half tile)
constexpr int kIParts = 4;           // slices per operand
constexpr int kILevels = 4;
// The ring: bf16 64 K (a 128-byte row), int8 64 or, in the half tile, 128 K a stage:
// a row of 64 bytes costs TMA as much as one of 128.  int8, D = 576, 1000
// trajectories, half tiles, 50 steps: 64-byte rows 1.89 ms with 3 or 4 stages,
// 128-byte rows with 2 stages 1.85 ms.  Halved rows for bf16 with twice the stages:
// 39.0 -> 46.6 us a step at D = 1024, 1024 trajectories (half tiles).
template <bool kHalf>
struct I8Cfg {
    static constexpr int BN = kHalf ? kIBN / 2 : kIBN;
    static constexpr int K = kHalf ? 128 : 64;  // K (int8) per stage: one swizzle row
    static constexpr int ATile = kGM * K;       // bytes of one A slice tile
    static constexpr int BTile = BN * K;        // bytes of one B slice tile
    static constexpr int Stage = kIParts * (ATile + BTile);
    static constexpr int Stages = kRing / Stage;
    static constexpr int Smem = Stages * Stage + 1024 /*align*/ + 256 /*barriers*/;
    static constexpr int Cols = kILevels * BN;  // TMEM columns
};

// Half tiles while all of them fit one wave: the tile's latency is then all that
// counts.  int8, D = 576, 1000 trajectories: 72 whole or 144 half tiles, a step
// in 41.4 or 36.9 us; D = 1024, bf16x3: 16 / 32 tiles 45.8 / 34.7 us, 64 / 128
// tiles 49.5 / 39.0 us; bf16x6, 64 / 128 tiles 49.0 / 46.6 us.  Beyond one wave
// the half tiles only read more: bf16x3, 128 / 256 tiles 55.8 / 60.3 us.
inline bool half_tiles(int m_tiles, int n_tiles) { return 2 * m_tiles * n_tiles <= 148; }

// kind::i8 instruction descriptor: D = S32, A = B = signed int8, both K-major.
__host__ __device__ constexpr uint32_t umma_idesc_i8(int M, int N)
{
    return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
           (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void umma_i8(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}"
        :
        : "r"(tmem), "l"(a), "l"(b), "r"(idesc), "r"(acc));
}

// out[n][m] = sum over levels of the exact slice products, scaled:
//   A slices: Dp x Dp int8 (row-major, K contiguous) -> tensor maps ta[0..4)
//   B slices: Mp x Dp int8                          -> tensor maps tb[0..4)
//   sa[m], sb[n]: the power-of-two scales of U's row m and trajectory n
// grid = (trajectory tiles of this launch, Dp / 128), block = 128 threads.
template <bool kHalf>
__global__ void __launch_bounds__(kGThreads, 1)
k_dense_gemm_i8(const __grid_constant__ CUtensorMap ta0, const __grid_constant__ CUtensorMap ta1,
                const __grid_constant__ CUtensorMap ta2, const __grid_constant__ CUtensorMap ta3,
                const __grid_constant__ CUtensorMap tb0, const __grid_constant__ CUtensorMap tb1,
                const __grid_constant__ CUtensorMap tb2, const __grid_constant__ CUtensorMap tb3,
                const double *__restrict__ sa, const double *__restrict__ sb, double *__restrict__ out, int Dp,
                int n_tile0, int *__restrict__ status)
{
    using Cfg = I8Cfg<kHalf>;
    constexpr int BN = Cfg::BN;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    unsigned char *base_ptr = smem_raw + (base - raw);
    const uint32_t bars = base + Cfg::Stages * Cfg::Stage;  // full, empty (a pair a stage), accum
    uint64_t *bar_ptr = reinterpret_cast<uint64_t *>(base_ptr + Cfg::Stages * Cfg::Stage);
    volatile int *abort = reinterpret_cast<volatile int *>(bar_ptr + 16);
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(bar_ptr + 17);
    const uint32_t full0 = bars, empty0 = bars + 8 * Cfg::Stages, accum = bars + 16 * Cfg::Stages;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int n0 = (n_tile0 + blockIdx.x) * BN, m0 = blockIdx.y * kGM;
    const int nk = Dp / Cfg::K;
    const CUtensorMap *ta[4] = {&ta0, &ta1, &ta2, &ta3};
    const CUtensorMap *tb[4] = {&tb0, &tb1, &tb2, &tb3};

    if (threadIdx.x == 0) {
        *abort = 0;
        for (int s = 0; s < Cfg::Stages; ++s) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * s));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty0 + 8 * s));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(accum));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(Cfg::Cols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    grid_wait();  // the operands are the previous kernel's

    if (threadIdx.x == 0) {
        // TMA producer
        int issued = 0;
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % Cfg::Stages, r = kb / Cfg::Stages;
            if (!mbar_wait(empty0 + 8 * s, (r & 1) ^ 1, abort)) break;
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(full0 + 8 * s), "r"(Cfg::Stage));
            const uint32_t st = base + s * Cfg::Stage;
            for (int p = 0; p < kIParts; ++p) tma_load_2d(st + p * Cfg::ATile, ta[p], kb * Cfg::K, m0, full0 + 8 * s);
            for (int q = 0; q < kIParts; ++q)
                tma_load_2d(st + kIParts * Cfg::ATile + q * Cfg::BTile, tb[q], kb * Cfg::K, n0, full0 + 8 * s);
            issued = kb + 1;
        }
        for (int kb = max(0, issued - Cfg::Stages); kb < issued; ++kb) {
            const int s = kb % Cfg::Stages, r = kb / Cfg::Stages;
            for (uint32_t it = 0; it < kWaitLimit && !mbar_try(full0 + 8 * s, r & 1); ++it) {
            }
        }
    } else if (threadIdx.x == 32) {
        // MMA issuer: level L = i + j accumulates a_i b_j
        constexpr uint32_t idesc = umma_idesc_i8(kGM, BN);
        uint32_t on = 0;  // bit L: level L's accumulator was written
        for (int kb = 0; kb < nk; ++kb) {
            const int s = kb % Cfg::Stages, r = kb / Cfg::Stages;
            if (!mbar_wait(full0 + 8 * s, r & 1, abort)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t st = base + s * Cfg::Stage;
#pragma unroll
            for (int kk = 0; kk < Cfg::K / 32; ++kk)
#pragma unroll
                for (int i = 0; i < kIParts; ++i)
#pragma unroll
                    for (int j = 0; j < kIParts - i; ++j) {
                        const int L = i + j;
                        const uint64_t ad = umma_desc<Cfg::K>(st + i * Cfg::ATile + kk * 32);
                        const uint64_t bd = umma_desc<Cfg::K>(st + kIParts * Cfg::ATile + j * Cfg::BTile + kk * 32);
                        umma_i8(tmem + L * BN, ad, bd, idesc, (on >> L) & 1u);
                        on |= 1u << L;
                    }
            umma_commit(empty0 + 8 * s);
        }
        umma_commit(accum);
    }
    __syncwarp();

    bool ok = mbar_wait(accum, 0, abort);
    if (!ok) {
        for (uint32_t it = 0; it < kWaitLimit && !mbar_try(accum, 0); ++it) {
        }
    }
    grid_trigger();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (ok && !*abort) {
        const int row = m0 + 32 * warp + lane;
        const double s_row = sa[row];
        const uint32_t lane_base = tmem + (static_cast<uint32_t>(32 * warp) << 16);
        constexpr double w0 = 1.0 / (127.0 * 127.0), w1 = w0 / 254.0, w2 = w1 / 254.0, w3 = w2 / 254.0;
#pragma unroll 1
        for (int c = 0; c < BN; c += 16) {
            uint32_t v[kILevels][16];
#pragma unroll
            for (int L = 0; L < kILevels; ++L) tmem_ld16_issue(lane_base + static_cast<uint32_t>(L * BN + c), v[L]);
            asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const double y = static_cast<double>(static_cast<int>(v[3][j])) * w3 +
                                 static_cast<double>(static_cast<int>(v[2][j])) * w2 +
                                 static_cast<double>(static_cast<int>(v[1][j])) * w1 +
                                 static_cast<double>(static_cast<int>(v[0][j])) * w0;
                out[static_cast<size_t>(n0 + c + j) * Dp + row] = y * s_row * sb[n0 + c + j];
            }
        }
    }
    if (*abort && threadIdx.x == 0) atomicOr(status, 4);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::Cols));
    }
}

// ------------------------------------------------------------ U precompute
// C = scale * (A B) + (add_identity ? I : 0); n x n complex row-major.
__global__ void k_zgemm(const double2 *__restrict__ A, const double2 *__restrict__ B, double2 *__restrict__ C, int n,
                        double scale, int add_identity)
{
    __shared__ double2 As[16][17], Bs[16][17];
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int row = blockIdx.y * 16 + ty, col = blockIdx.x * 16 + tx;
    double2 acc = make_double2(0.0, 0.0);
    for (int k0 = 0; k0 < n; k0 += 16) {
        As[ty][tx] = (row < n && k0 + tx < n) ? A[static_cast<size_t>(row) * n + k0 + tx] : make_double2(0.0, 0.0);
        Bs[ty][tx] = (k0 + ty < n && col < n) ? B[static_cast<size_t>(k0 + ty) * n + col] : make_double2(0.0, 0.0);
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) acc = cfma(As[ty][k], Bs[k][tx], acc);
        __syncthreads();
    }
    if (row < n && col < n) {
        double2 v = cscale(acc, scale);
        if (add_identity && row == col) v.x += 1.0;
        C[static_cast<size_t>(row) * n + col] = v;
    }
}

// G = dt * (-iH - K) dense (row-major), from CSR; zero-filled first.
__global__ void k_dense_generator(const int *__restrict__ rowptr, const int *__restrict__ col,
                                  const double2 *__restrict__ val, const int *__restrict__ krow,
                                  const int *__restrict__ kcol, const double2 *__restrict__ kval, double kappa,
                                  double dt, int n, double2 *__restrict__ G)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    for (int k = rowptr[r]; k < rowptr[r + 1]; ++k) {
        const double2 h = val[k];
        G[static_cast<size_t>(r) * n + col[k]] = make_double2(dt * h.y, -dt * h.x);  // -i dt H
    }
    if (krow) {
        for (int k = krow[r]; k < krow[r + 1]; ++k) {
            double2 &g = G[static_cast<size_t>(r) * n + kcol[k]];
            g.x -= dt * kval[k].x;
            g.y -= dt * kval[k].y;
        }
    } else {
        G[static_cast<size_t>(r) * n + r].x -= dt * kappa;
    }
}

__global__ void k_row_norms(const double2 *__restrict__ A, int n, double *__restrict__ out)
{
    const int r = blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double s = 0.0;
    for (int c = 0; c < n; ++c) s += sqrt(cabs2(A[static_cast<size_t>(r) * n + c]));
    out[r] = s;
}

// Split an FP64 value into NS BF16 parts (round to nearest at each level).
__device__ __forceinline__ void split_bf16(double x, int ns, __nv_bfloat16 *p)
{
    double r = x;
    for (int i = 0; i < ns; ++i) {
        const __nv_bfloat16 h = __double2bfloat16(r);
        p[i] = h;
        r -= static_cast<double>(__bfloat162float(h));
    }
}

// U (n x n complex) -> real interleaved Dp x Dp matrix, split in parts
// (parts x Dp x Dp, padding rows/columns zero).
__global__ void k_u_split(const double2 *__restrict__ U, int n, int Dp, int ns, __nv_bfloat16 *__restrict__ parts)
{
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<size_t>(Dp) * Dp) return;
    const int i = static_cast<int>(idx / Dp), j = static_cast<int>(idx % Dp);
    double x = 0.0;
    if (i < 2 * n && j < 2 * n) {
        const double2 u = U[static_cast<size_t>(i >> 1) * n + (j >> 1)];
        const int c = i & 1, d = j & 1;
        x = (c == d) ? u.x : (c == 0 ? -u.y : u.y);
    }
    __nv_bfloat16 p[3];
    split_bf16(x, ns, p);
    for (int k = 0; k < ns; ++k) parts[static_cast<size_t>(k) * Dp * Dp + idx] = p[k];
}

// U (n x n complex) -> real interleaved Dp x Dp matrix, row r scaled by its
// power of two 2^e_r >= max_c |A[r][c]| and cut into four int8 slices (the
// operand form of k_dense_gemm_i8: r = A / 2^e, a_0 = rint(127 r), then
// a_i = rint(254 r_i) on the remainders); one block of 256 threads per row.
__global__ void __launch_bounds__(256) k_u_split_i8(const double2 *__restrict__ U, int n, int Dp,
                                                    int8_t *__restrict__ parts, double *__restrict__ scale)
{
    __shared__ double red[8];
    const int i = blockIdx.x;
    auto val = [&](int j) -> double {
        if (i >= 2 * n || j >= 2 * n) return 0.0;
        const double2 u = U[static_cast<size_t>(i >> 1) * n + (j >> 1)];
        const int c = i & 1, d = j & 1;
        return (c == d) ? u.x : (c == 0 ? -u.y : u.y);
    };
    double m = 0.0;
    for (int j = threadIdx.x; j < Dp; j += blockDim.x) m = fmax(m, fabs(val(j)));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
    __syncthreads();
    m = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
    const double s = m > 0.0 ? exp2(ceil(log2(m))) : 1.0, inv = 1.0 / s;
    if (threadIdx.x == 0) scale[i] = s;
    for (int j = threadIdx.x; j < Dp; j += blockDim.x) {
        double r = val(j) * inv;
        double q = rint(127.0 * r);
        parts[static_cast<size_t>(i) * Dp + j] = static_cast<int8_t>(q);
        r = 127.0 * r - q;
        for (int p = 1; p < 4; ++p) {
            q = rint(254.0 * r);
            parts[(static_cast<size_t>(p) * Dp + i) * Dp + j] = static_cast<int8_t>(q);
            r = 254.0 * r - q;
        }
    }
}

// context state (ldm x D interleaved complex128) <-> dense state (Mp x Dp, T = fp32 or fp64)
template <typename T>
__global__ void k_ctx_to_dense_t(const double2 *__restrict__ psi, int D, int M, int ldm, int Dp, int Mp,
                                 T *__restrict__ out)
{
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<size_t>(Mp) * Dp) return;
    const int t = static_cast<int>(idx / Dp), k = static_cast<int>(idx % Dp);
    T v = 0;
    if (t < M && k < 2 * D) {
        const double2 z = psi[static_cast<size_t>(k >> 1) * ldm + t];
        v = static_cast<T>((k & 1) ? z.y : z.x);
    }
    out[idx] = v;
}

template <typename T>
__global__ void k_dense_to_ctx_t(const T *__restrict__ in, int D, int M, int ldm, int Dp, double2 *__restrict__ psi)
{
    const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (idx >= static_cast<size_t>(D) * ldm) return;
    const int r = static_cast<int>(idx / ldm), t = static_cast<int>(idx % ldm);
    double2 z = make_double2(0.0, 0.0);
    if (t < M) z = make_double2(in[static_cast<size_t>(t) * Dp + 2 * r], in[static_cast<size_t>(t) * Dp + 2 * r + 1]);
    psi[idx] = z;
}

struct DenseEpi {
    int D, Dp, M, Mp, s1, s2, nobs, ns;
    // pair observable o as upper-triangle coefficients over the quartet's
    // (a <= c) pairs: Re <x|O|x> = sum Cr P_ac - Ci Q_ac with P = Re(x_a* x_c),
    // Q = Im(x_a* x_c), C_ac = O_ac + conj(O_ca) (a < c), C_aa = Re O_aa
    double2 obs_c[8][10];
    unsigned obs_mask[8];  // bit k: obs_c[o][k] != 0 (most pair operators are sparse)
    const double *rates;
    // noise
    int noise_mode;
    const unsigned char *bits;
    long long bits_steps;
    int bits_ntraj;
    unsigned long long seed;
    long long stepA, stepB;
    int halfA, halfB;
    double pA, pB;
    // yields
    double dt;
    int init;
    double *acc, *comp, *prev;
    int acc_ld;
    double *tvals;        // M x nobs (this time point)
    double *norm0;        // per trajectory: |psi(0)|^2 (renormalisation reference)
    double decay;         // target |psi|^2 = norm0 * exp(-decay * (t - t0))
    double elapsed;       // t - t0 of this time point
    int renormalize;
    int store_state;            // write the FP32 state back (last time point of a run)
    int t0, t1;                 // this launch's trajectories [t0, t1) (one stream group)
    const double *prev_tvals;   // previous time point's per-trajectory values, or null
    double *prev_values;        // its ensemble values (nobs doubles)
    int *status;
};

__device__ __forceinline__ int dense_flip(const DenseEpi &E, int t, long long step, int half, double p)
{
    if (step < 0) return 0;
    if (E.noise_mode == MSGPU_NOISE_REPLAY) {
        if (t >= E.bits_ntraj || step >= E.bits_steps) return 0;
        const long long bit = (step * 2 + half) * E.bits_ntraj + t;
        return (E.bits[bit >> 3] >> (bit & 7)) & 1;
    }
    if (E.noise_mode == MSGPU_NOISE_PHILOX)
        return philox_flip(E.seed, static_cast<uint32_t>(t), static_cast<uint32_t>(step), static_cast<uint32_t>(half),
                           p) ? 1 : 0;
    return 0;
}

// The smallest power of two >= m (1 for 0, the smallest normal one below it, inf for inf).
__device__ __forceinline__ double pow2_above(double m)
{
    if (!(m > 0.0)) return 1.0;
    const long long b = __double_as_longlong(m), e = b & 0x7ff0000000000000ll;
    return e == 0 ? __longlong_as_double(0x0010000000000000ll)
                  : __longlong_as_double(e + (b == e ? 0ll : 0x0010000000000000ll));
}

// Ensemble value of one observable: the sum over trajectories of tvals[t][o]
// in a fixed order (256 threads, strided partial sums, warp tree, warp order).
__device__ __forceinline__ double dense_ensemble_sum(const double *__restrict__ tvals, int t0, int t1, int nobs, int o,
                                                    double (*red)[8])
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double a = 0.0;
    for (int t = t0 + threadIdx.x; t < t1; t += blockDim.x) a += tvals[static_cast<size_t>(t) * nobs + o];
    a = warp_sum(a);
    if (lane == 0) red[0][warp] = a;
    __syncthreads();
    double v = 0.0;
    for (int w = 0; w < static_cast<int>(blockDim.x >> 5); ++w) v += red[0][w];
    return v;
}

// One CTA (128 threads; int8: 256 for few trajectories) per trajectory.  The trajectory's column (2D values,
// re/im per row) is staged in shared memory once; flips, the norm, the
// optional renormalisation, the pair observables and the split of the next
// GEMM operand all work from there, and the column is written back only at
// the last time point (the next GEMM overwrites it otherwise).  Blocks
// 0..nobs-1 also sum the previous time point's per-trajectory values into its
// ensemble values, which saves a launch per step.
//   kI8 = false: FP32 state, BF16 parts (E.ns of them) for k_dense_gemm.
//   kI8 = true:  FP64 state, four int8 slices and the column's power-of-two
//                scale for k_dense_gemm_i8 (see k_u_split_i8 for the slicing).
// The int8 form is bound by the latency of its FP64 chain (the norm, the scale, four
// slices a value), so its CTA has twice the threads while all of them are resident at
// once (wide_epilogue), the scale is read off the exponent and a slice is rounded by an
// addition instead of two conversions: D = 576, 512 trajectories 13.0 -> 10.8 us.  With
// more, 128 threads leave less of an SM waiting: 8192 trajectories of D = 64, 10 steps
// 0.82 -> 0.53 ms, 4096 of D = 576 1.01 -> 0.88, 1500 of D = 1024 0.77 -> 0.74.
constexpr int kEpiThreads = 128, kEpiThreadsI8 = 256;
inline bool wide_epilogue(int trajectories) { return trajectories <= 4 * 148; }
template <bool kI8, int kThreads = kEpiThreads>
__global__ void __launch_bounds__(kThreads, 1024 / kThreads)
k_dense_epilogue(void *__restrict__ psi_v, void *__restrict__ bparts_v, double *__restrict__ bscale, DenseEpi E)
{
    using V2 = typename std::conditional<kI8, double2, float2>::type;
    extern __shared__ float4 s_col4[];  // the 2D values of the column
    V2 *s_col = reinterpret_cast<V2 *>(s_col4);
    __shared__ double red[10][8];
    __shared__ double s_scale, s_max;
    __shared__ double2 s_obs[8][10];
    const int t = E.t0 + blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x < 80) s_obs[threadIdx.x / 10][threadIdx.x % 10] = E.obs_c[threadIdx.x / 10][threadIdx.x % 10];
    grid_wait();  // the column is the GEMM's, the rest of this step's inputs the previous epilogue's
    if constexpr (kI8) {
        const double2 *col = static_cast<const double2 *>(psi_v) + static_cast<size_t>(t) * (E.Dp / 2);
        for (int i = threadIdx.x; i < E.D; i += kThreads) s_col[i] = col[i];
    } else {
        const float *col = static_cast<const float *>(psi_v) + static_cast<size_t>(t) * E.Dp;
        const int n4 = E.D / 2;
        for (int i = threadIdx.x; i < n4; i += kThreads) s_col4[i] = reinterpret_cast<const float4 *>(col)[i];
    }
    const int Q = E.D / 4;
    int flip = 0;
    if (t < E.M) {
        flip = dense_flip(E, t, E.stepA, E.halfA, E.pA);
        if (E.stepB >= 0) flip ^= dense_flip(E, t, E.stepB, E.halfB, E.pB);
    }
    // the scalars of this trajectory, fetched while the column loads: the
    // renormalisation reference (thread 0) and, for thread o < nobs, the
    // trapezoid state of observable o
    const bool yield_thread = t < E.M && static_cast<int>(threadIdx.x) < E.nobs;
    const size_t yk = static_cast<size_t>(threadIdx.x) * E.acc_ld + t;
    double y_prev = 0.0, y_acc = 0.0, y_comp = 0.0;
    if (yield_thread && !E.init) {
        y_prev = E.prev[yk];
        y_acc = E.acc[yk];
        y_comp = E.comp[yk];
    }
    const double ref = (threadIdx.x == 0 && t < E.M && !E.init) ? E.norm0[t] : 0.0;
    __syncthreads();
    // one pass over the quartets (each belongs to one thread): flip in shared
    // memory, norm and pair observables of the unscaled state, and (int8
    // operands) the largest component.  Observables are quadratic, so the
    // renormalisation enters as sc^2 afterwards.
    double nn = 0.0, mx = 0.0;
    double obs[8] = {0, 0, 0, 0, 0, 0, 0, 0};
#pragma unroll 1
    for (int q = threadIdx.x; q < Q; q += kThreads) {
        const int b = quartet_base(q, E.s1, E.s2);
        const int r[4] = {b, b + E.s2, b + E.s1, b + E.s1 + E.s2};
        V2 x[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) x[a] = s_col[r[a]];
        if (flip) {
            const V2 c1 = x[1];
            x[0].x = -x[0].x; x[0].y = -x[0].y;
            x[1].x = -x[2].x; x[1].y = -x[2].y;
            x[2].x = -c1.x;   x[2].y = -c1.y;
            x[3].x = -x[3].x; x[3].y = -x[3].y;
#pragma unroll
            for (int a = 0; a < 4; ++a) s_col[r[a]] = x[a];
        }
        double2 v[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) v[a] = make_double2(x[a].x, x[a].y);
        if (kI8)
#pragma unroll
            for (int a = 0; a < 4; ++a) mx = fmax(mx, fmax(fabs(v[a].x), fabs(v[a].y)));
        nn += v[0].x * v[0].x + v[0].y * v[0].y + v[1].x * v[1].x + v[1].y * v[1].y + v[2].x * v[2].x +
              v[2].y * v[2].y + v[3].x * v[3].x + v[3].y * v[3].y;
        const volatile double2 *so = &s_obs[0][0];  // re-read per use: nothing is held in registers
#pragma unroll
        for (int o = 0; o < 8; ++o) {
            if (o >= E.nobs) break;
            const unsigned m = E.obs_mask[o];
            double sum = 0.0;
            int k = 0;
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int c = a; c < 4; ++c, ++k)
                    if ((m >> k) & 1u) {
                        const double cr = so[o * 10 + k].x, ci = so[o * 10 + k].y;
                        sum += cr * (v[a].x * v[c].x + v[a].y * v[c].y) - ci * (v[a].x * v[c].y - v[a].y * v[c].x);
                    }
            obs[o] += sum;
        }
    }
    nn = warp_sum(nn);
    if (lane == 0) red[8][warp] = nn;
    if (kI8) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        if (lane == 0) red[9][warp] = mx;
    }
#pragma unroll
    for (int o = 0; o < 8; ++o) {
        if (o >= E.nobs) break;
        const double w = warp_sum(obs[o]);
        if (lane == 0) red[o][warp] = w;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double cur = 0.0, m = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) {
            cur += red[8][w];
            if (kI8) m = fmax(m, red[9][w]);
        }
        double sc = 1.0;
        if (E.init) {
            if (t < E.M) E.norm0[t] = cur;
        } else if (E.renormalize && cur > 0.0) {
            sc = sqrt(ref * exp(-E.decay * E.elapsed) / cur);
        }
        s_scale = sc;
        s_max = m * sc;
    }
    __syncthreads();
    const double scd = s_scale;
    if constexpr (kI8) {
        // int8 slices of the scaled state for the next GEMM.  With the column's
        // scale 2^e >= max |x|, r = x / 2^e lies in [-1, 1]; a_0 = rint(127 r),
        // then a_i = rint(254 r_i) on the remainders r_{i+1} = 254 r_i - a_i
        // (|r_i| <= 1/2), so x = 2^e sum_i a_i / (127 254^i) to 2^-31 of 2^e.
        const double s = pow2_above(s_max);
        if (threadIdx.x == 0) bscale[t] = s;
        const double inv = 1.0 / s;  // a power of two: exact
        double *colw = static_cast<double *>(psi_v) + static_cast<size_t>(t) * E.Dp;
        int8_t *bp = static_cast<int8_t *>(bparts_v);
        for (int c = threadIdx.x; c < E.Dp / 4; c += kThreads) {
            unsigned a[4][4];  // [slice][value], in the low byte
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                double x = 0.0;
                if (c < E.D / 2) {
                    const double2 z = s_col[2 * c + (j >> 1)];
                    x = ((j & 1) ? z.y : z.x) * scd;
                    if (E.store_state) colw[4 * c + j] = x;
                }
                // the addition of 1.5 2^52 rounds to an integer and leaves it in the low bits
                double r = x * inv, f = 127.0;
#pragma unroll
                for (int i = 0; i < 4; ++i, f = 254.0) {
                    const double u = fma(f, r, 6755399441055744.0);
                    a[i][j] = static_cast<unsigned>(__double2loint(u));
                    r = fma(f, r, -(u - 6755399441055744.0));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
                *reinterpret_cast<unsigned *>(bp + (static_cast<size_t>(i) * E.Mp + t) * E.Dp + 4 * c) =
                    __byte_perm(__byte_perm(a[i][0], a[i][1], 0x0040), __byte_perm(a[i][2], a[i][3], 0x0040), 0x5410);
        }
    } else {
        const int nc = E.Dp / 8, live = E.D / 4;  // chunks of 8 values; 2D / 8 of them hold data
        const float sc = static_cast<float>(scd);
        // BF16 split of the scaled state for the next GEMM: 8 floats (two float4)
        // per thread and part, 16-byte stores, the padding beyond 2D floats zero.
        // In FP32 each residual x - bf16(x) is exact, so hi + mid + lo carries all
        // 24 bits of x; conversions are round-to-nearest, two values at a time.
        float4 *col4 = reinterpret_cast<float4 *>(static_cast<float *>(psi_v) + static_cast<size_t>(t) * E.Dp);
        __nv_bfloat16 *bparts = static_cast<__nv_bfloat16 *>(bparts_v);
        for (int c = threadIdx.x; c < nc; c += kThreads) {
            float f[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
            if (c < live) {
                float4 u = s_col4[2 * c], w = s_col4[2 * c + 1];
                if (sc != 1.f) {
                    u = make_float4(u.x * sc, u.y * sc, u.z * sc, u.w * sc);
                    w = make_float4(w.x * sc, w.y * sc, w.z * sc, w.w * sc);
                }
                if (E.store_state) {
                    col4[2 * c] = u;
                    col4[2 * c + 1] = w;
                }
                f[0] = u.x; f[1] = u.y; f[2] = u.z; f[3] = u.w;
                f[4] = w.x; f[5] = w.y; f[6] = w.z; f[7] = w.w;
            }
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                if (i >= E.ns) break;
                __align__(16) __nv_bfloat162 h[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    h[j] = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
                    f[2 * j] -= __low2float(h[j]);
                    f[2 * j + 1] -= __high2float(h[j]);
                }
                *reinterpret_cast<uint4 *>(bparts + (static_cast<size_t>(i) * E.Mp + t) * E.Dp + 8 * c) =
                    *reinterpret_cast<const uint4 *>(h);
            }
        }
    }
    grid_trigger();
    // trapezoid (compensated) and this time point's value, one thread per observable
    if (yield_thread) {
        const int o = threadIdx.x;
        double vs = 0.0;
        for (int w = 0; w < kThreads / 32; ++w) vs += red[o][w];
        const double v = vs * scd * scd * E.rates[o];
        if (!E.init) {
            const double term = 0.5 * E.dt * (y_prev + v) - y_comp;
            const double s = y_acc + term;
            E.comp[yk] = (s - y_acc) - term;
            E.acc[yk] = s;
        }
        E.prev[yk] = v;
        E.tvals[static_cast<size_t>(t) * E.nobs + o] = v;
        if (!isfinite(v)) atomicOr(E.status, 2);
    }
    if (E.prev_tvals && blockIdx.x < E.nobs) {
        __syncthreads();  // red[0] is reused below
        const double v = dense_ensemble_sum(E.prev_tvals, E.t0, min(E.t1, E.M), E.nobs, blockIdx.x, red);
        if (threadIdx.x == 0) E.prev_values[blockIdx.x] = v;
    }
}

// values[o] = one group's part of the last time point's ensemble value
// (same order as above)
__global__ void __launch_bounds__(kEpiThreads) k_dense_values(const double *__restrict__ tvals, int t0, int t1,
                                                              int nobs, double *__restrict__ values)
{
    __shared__ double red[9][8];
    const double v = dense_ensemble_sum(tvals, t0, t1, nobs, blockIdx.x, red);
    if (threadIdx.x == 0) values[blockIdx.x] = v;
}

// values[i] = sum over the stream groups of their parts, in group order
__global__ void k_dense_sum_groups(const double *__restrict__ part, int groups, size_t n, double *__restrict__ values)
{
    const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double v = 0.0;
    for (int g = 0; g < groups; ++g) v += part[static_cast<size_t>(g) * n + i];
    values[i] = v;
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                 const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encoder()
{
    // looked up once; static initialisation is thread-safe (contexts may prepare from several host threads)
    static const EncodeTiled fn = []() -> EncodeTiled {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<EncodeTiled>(p);
        return nullptr;
    }();
    return fn;
}

// 2D BF16 tensor map over a rows x cols row-major matrix, box = 64 x box_rows.
bool make_map(CUtensorMap *m, const void *ptr, int rows, int cols, int box_rows)
{
    EncodeTiled enc = encoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols) * 2};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(kGK), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void *>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// 2D int8 tensor map over a rows x cols row-major matrix, box = k x box_rows with
// swizzled rows of k bytes (the operand tiles of k_dense_gemm_i8).
bool make_map_i8(CUtensorMap *m, const void *ptr, int rows, int cols, int box_rows, int k)
{
    EncodeTiled enc = encoder();
    if (!enc) return false;
    const cuuint64_t dims[2] = {static_cast<cuuint64_t>(cols), static_cast<cuuint64_t>(rows)};
    const cuuint64_t strides[1] = {static_cast<cuuint64_t>(cols)};
    const cuuint32_t box[2] = {static_cast<cuuint32_t>(k), static_cast<cuuint32_t>(box_rows)};
    const cuuint32_t estr[2] = {1, 1};
    return enc(m, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, const_cast<void *>(ptr), dims, strides, box, estr,
               CU_TENSOR_MAP_INTERLEAVE_NONE, k == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

inline int cdiv(long long a, long long b) { return static_cast<int>((a + b - 1) / b); }

}  // namespace

int dense_prepare(DenseState &st, int D, int M, int ldm, int parts, double dt, const DenseRun &run,
                  const void *psi128, cudaStream_t stream, std::string &err,
                  int (*alloc)(void *ctx, void **p, size_t bytes, const char *what), void *actx)
{
    if (parts != 2 && parts != 3 && parts != kIParts) {
        err = "dense: split depth must be 2 or 3 (BF16) or 4 (int8)";
        return MSGPU_ERR_INVALID;
    }
    const bool i8 = parts == kIParts;
    const int BN = i8 ? kIBN : parts == 2 ? GemmCfg<2>::BN : GemmCfg<3>::BN;
    const int Dp = (2 * D + kGM - 1) / kGM * kGM;
    const int Mp = (M + BN - 1) / BN * BN;
    const bool realloc = st.D != D || st.M != M || st.parts != parts || !st.psi;
    if (realloc) {
        st = DenseState();
        int rc;
        // int8: four byte slices plus the power-of-two scales (rows of U,
        // trajectories of the state) after them; FP64 state.  BF16: parts
        // of two bytes; FP32 state.
        const size_t esz = i8 ? 1 : sizeof(__nv_bfloat16);
        const size_t u_bytes = esz * parts * static_cast<size_t>(Dp) * Dp + (i8 ? sizeof(double) * Dp : 0);
        const size_t b_bytes = esz * parts * static_cast<size_t>(Mp) * Dp + (i8 ? sizeof(double) * Mp : 0);
        if ((rc = alloc(actx, &st.u_parts, u_bytes, "dense U")) ||
            (rc = alloc(actx, &st.psi, (i8 ? sizeof(double) : sizeof(float)) * static_cast<size_t>(Mp) * Dp,
                        "dense state")) ||
            (rc = alloc(actx, &st.b_parts, b_bytes, "dense split state")) ||
            // G, T, W (+ slack) for U; row norms (8D doubles); per-trajectory
            // values (8 Mp doubles) and reference norms (Mp doubles)
            (rc = alloc(actx, &st.work,
                        sizeof(double2) * 4 * static_cast<size_t>(D) * D +
                            sizeof(double) * (8 * static_cast<size_t>(D) + 17 * static_cast<size_t>(Mp)),
                        "dense scratch")))
            return rc;
        st.D = D;
        st.Dp = Dp;
        st.M = M;
        st.Mp = Mp;
        st.parts = parts;
        st.u_scale = i8 ? static_cast<unsigned char *>(st.u_parts) + static_cast<size_t>(parts) * Dp * Dp : nullptr;
        st.b_scale = i8 ? static_cast<unsigned char *>(st.b_parts) + static_cast<size_t>(parts) * Mp * Dp : nullptr;
        st.have_u = false;
    }
    cudaError_t e;
    if (!st.have_u || st.dt != dt) {
        // U = exp(G) with G = dt(-iH - K): Taylor degree 18 on G / 2^s, then s squarings
        double2 *G = static_cast<double2 *>(st.work);
        double2 *T = G + static_cast<size_t>(D) * D, *W = T + static_cast<size_t>(D) * D;
        double *rn = reinterpret_cast<double *>(W + 2 * static_cast<size_t>(D) * D);
        cudaMemsetAsync(G, 0, sizeof(double2) * static_cast<size_t>(D) * D, stream);
        k_dense_generator<<<cdiv(D, 128), 128, 0, stream>>>(run.rowptr, run.col,
                                                             reinterpret_cast<const double2 *>(run.val), run.krow,
                                                             run.kcol, reinterpret_cast<const double2 *>(run.kval),
                                                             run.kappa, dt, D, G);
        k_row_norms<<<cdiv(D, 128), 128, 0, stream>>>(G, D, rn);
        std::vector<double> h(D);
        if ((e = cudaMemcpyAsync(h.data(), rn, sizeof(double) * D, cudaMemcpyDeviceToHost, stream)) ||
            (e = cudaStreamSynchronize(stream))) {
            err = std::string("dense: generator: ") + cudaGetErrorString(e);
            return MSGPU_ERR_CUDA;
        }
        double nrm = 0.0;
        for (double x : h) nrm = std::max(nrm, x);
        if (!std::isfinite(nrm)) { err = "dense: non-finite generator"; return MSGPU_ERR_NONFINITE; }
        int s = 0;
        while (nrm / std::ldexp(1.0, s) > 0.25) ++s;
        const double inv = std::ldexp(1.0, -s);
        dim3 gb(cdiv(D, 16), cdiv(D, 16)), tb(16, 16);
        // Horner: T = I + A/18; T = I + A T / k for k = 17..1
        cudaMemsetAsync(T, 0, sizeof(double2) * static_cast<size_t>(D) * D, stream);
        k_zgemm<<<gb, tb, 0, stream>>>(G, T, T, D, 0.0, 1);  // T = I
        for (int k = 18; k >= 1; --k) {
            k_zgemm<<<gb, tb, 0, stream>>>(G, T, W, D, inv / k, 1);
            std::swap(T, W);
        }
        for (int q = 0; q < s; ++q) {
            k_zgemm<<<gb, tb, 0, stream>>>(T, T, W, D, 1.0, 0);
            std::swap(T, W);
        }
        const size_t nu = static_cast<size_t>(Dp) * Dp;
        if (i8)
            k_u_split_i8<<<Dp, 256, 0, stream>>>(T, D, Dp, static_cast<int8_t *>(st.u_parts),
                                                 static_cast<double *>(st.u_scale));
        else
            k_u_split<<<cdiv(nu, 256), 256, 0, stream>>>(T, D, Dp, parts, static_cast<__nv_bfloat16 *>(st.u_parts));
        if ((e = cudaGetLastError())) {
            err = std::string("dense: propagator: ") + cudaGetErrorString(e);
            return MSGPU_ERR_CUDA;
        }
        st.have_u = true;
        st.dt = dt;
    }
    const size_t ns = static_cast<size_t>(Mp) * Dp;
    if (i8)
        k_ctx_to_dense_t<double><<<cdiv(ns, 256), 256, 0, stream>>>(static_cast<const double2 *>(psi128), D, M, ldm,
                                                                     Dp, Mp, static_cast<double *>(st.psi));
    else
        k_ctx_to_dense_t<float><<<cdiv(ns, 256), 256, 0, stream>>>(static_cast<const double2 *>(psi128), D, M, ldm, Dp,
                                                                    Mp, static_cast<float *>(st.psi));
    if ((e = cudaGetLastError())) {
        err = std::string("dense: state: ") + cudaGetErrorString(e);
        return MSGPU_ERR_CUDA;
    }
    return MSGPU_OK;
}

int dense_run(DenseState &st, const DenseRun &run, void *psi128, int ldm, cudaStream_t stream, std::string &err,
              float *gemm_ms, long long *gemm_launches, int gemm_every)
{
    const int D = st.D, Dp = st.Dp, M = st.M, Mp = st.Mp, ns = st.parts;
    const bool i8 = ns == kIParts;
    CUtensorMap ta[4], tb[4];
    std::memset(ta, 0, sizeof(ta));
    std::memset(tb, 0, sizeof(tb));
    const int wide = i8 ? kIBN : ns == 2 ? GemmCfg<2>::BN : GemmCfg<3>::BN;
    const bool half = half_tiles(Mp / wide, Dp / kGM);
    const int BN = half ? wide / 2 : wide;
    const int ik = half ? I8Cfg<true>::K : I8Cfg<false>::K;
    void *bp = st.b_parts;
    for (int p = 0; p < ns; ++p) {
        bool okm;
        if (i8)
            okm = make_map_i8(&ta[p], static_cast<const int8_t *>(st.u_parts) + static_cast<size_t>(p) * Dp * Dp, Dp, Dp,
                              kGM, ik) &&
                  make_map_i8(&tb[p], static_cast<const int8_t *>(st.b_parts) + static_cast<size_t>(p) * Mp * Dp, Mp, Dp,
                              BN, ik);
        else
            okm = make_map(&ta[p], static_cast<const __nv_bfloat16 *>(st.u_parts) + static_cast<size_t>(p) * Dp * Dp, Dp,
                           Dp, kGM) &&
                  make_map(&tb[p], static_cast<const __nv_bfloat16 *>(st.b_parts) + static_cast<size_t>(p) * Mp * Dp, Mp,
                           Dp, BN);
        if (!okm) {
            err = "dense: cannot encode TMA tensor maps (cuTensorMapEncodeTiled unavailable or rejected)";
            return MSGPU_ERR_CUDA;
        }
    }
    for (int p = ns; p < 4; ++p) {
        ta[p] = ta[0];
        tb[p] = tb[0];
    }
    cudaError_t e;
    const size_t epi_smem = (i8 ? sizeof(double) : sizeof(float)) * 2 * static_cast<size_t>(D);
    const auto gemm2 = half ? k_dense_gemm<2, true> : k_dense_gemm<2, false>;
    const auto gemm3 = half ? k_dense_gemm<3, true> : k_dense_gemm<3, false>;
    const auto gemm8 = half ? k_dense_gemm_i8<true> : k_dense_gemm_i8<false>;
    const int smem = i8 ? (half ? I8Cfg<true>::Smem : I8Cfg<false>::Smem)
                     : ns == 2 ? (half ? GemmCfg<2, true>::Smem : GemmCfg<2>::Smem)
                               : (half ? GemmCfg<3, true>::Smem : GemmCfg<3>::Smem);
    if ((e = raise_smem_limit(i8 ? reinterpret_cast<const void *>(gemm8)
                                 : ns == 2 ? reinterpret_cast<const void *>(gemm2) : reinterpret_cast<const void *>(gemm3),
                              smem)) ||
        (e = raise_smem_limit(i8 ? reinterpret_cast<const void *>(k_dense_epilogue<true>)
                                 : reinterpret_cast<const void *>(k_dense_epilogue<false>),
                              static_cast<int>(epi_smem))) ||
        (i8 && (e = raise_smem_limit(reinterpret_cast<const void *>(k_dense_epilogue<true, kEpiThreadsI8>),
                                     static_cast<int>(epi_smem))))) {
        err = std::string("dense: shared memory: ") + cudaGetErrorString(e);
        return MSGPU_ERR_CUDA;
    }
    double *tvals = reinterpret_cast<double *>(static_cast<double2 *>(st.work) + 4 * static_cast<size_t>(D) * D) + 8 * D;
    // per-trajectory values of the current and the previous time point
    // (8 observables at most each), then the renormalisation references
    double *tv[2] = {tvals, tvals + 8 * static_cast<size_t>(Mp)};
    double *norm0 = tvals + 16 * static_cast<size_t>(Mp);
    DenseEpi E;
    std::memset(&E, 0, sizeof(E));
    E.D = D;
    E.Dp = Dp;
    E.M = M;
    E.Mp = Mp;
    E.s1 = run.s1;
    E.s2 = run.s2;
    E.nobs = run.nobs;
    E.ns = ns;
    for (int o = 0; o < run.nobs && o < 8; ++o) {
        const double *op = run.obs_host + 32 * o;  // 16 complex, row-major
        int k = 0;
        for (int a = 0; a < 4; ++a)
            for (int c = a; c < 4; ++c, ++k) {
                const double re_ac = op[2 * (4 * a + c)], im_ac = op[2 * (4 * a + c) + 1];
                const double re_ca = op[2 * (4 * c + a)], im_ca = op[2 * (4 * c + a) + 1];
                E.obs_c[o][k] = a == c ? make_double2(re_ac, 0.0) : make_double2(re_ac + re_ca, im_ac - im_ca);
                if (E.obs_c[o][k].x != 0.0 || E.obs_c[o][k].y != 0.0) E.obs_mask[o] |= 1u << k;
            }
    }
    E.rates = run.rates;
    E.noise_mode = run.noise_mode;
    E.bits = run.bits;
    E.bits_steps = run.bits_steps;
    E.bits_ntraj = run.bits_ntraj;
    E.seed = run.seed;
    E.acc = run.acc;
    E.comp = run.comp;
    E.prev = run.prev;
    E.acc_ld = run.acc_ld;
    E.tvals = tv[0];
    E.norm0 = norm0;
    E.decay = 2.0 * run.kappa;
    E.renormalize = run.renormalize && run.krow == nullptr;
    E.status = run.status;
    const int steps = run.ntimes - 1;
    auto pstep = [&](int s) {
        return s < steps ? -0.5 * std::expm1(-2.0 * (0.5 * run.st_rate) * (0.5 * (run.times[s + 1] - run.times[s])))
                         : 0.0;
    };
    // Each kernel of a group's chain is launched before its predecessor has ended and is
    // set up by then (launch_dependent); the GEMM lets the epilogue in after its last
    // MMA, the epilogue the GEMM after its last operand.  D = 576, 1000 trajectories,
    // int8: 33.3 -> 30.4 us a step; D = 1024, 1024 trajectories, bf16x3 38.9 -> 34.2,
    // int8 49.5 -> 46.4 us; 4096 trajectories, bf16x3: the same (100 us).
    // Two stream groups when the block has at least two trajectory tiles:
    // group g owns tiles [gt[g], gt[g+1]) and runs its GEMM -> epilogue chain
    // on its own stream, so one group's epilogue overlaps the other's GEMM
    // (the groups share no data: a GEMM tile reads only its own trajectories).
    const int Mt = Mp / BN;
    const int G = Mt >= 2 ? 2 : 1;
    const int gt[3] = {0, G == 2 ? Mt / 2 : Mt, Mt};
    if (G == 2 && !st.side) {
        if ((e = cudaStreamCreateWithFlags(&st.side, cudaStreamNonBlocking)) ||
            (e = cudaEventCreateWithFlags(&st.e_main, cudaEventDisableTiming)) ||
            (e = cudaEventCreateWithFlags(&st.e_side, cudaEventDisableTiming))) {
            err = std::string("dense: second stream: ") + cudaGetErrorString(e);
            return MSGPU_ERR_CUDA;
        }
    }
    cudaStream_t ss[2] = {stream, G == 2 ? st.side : stream};
    auto fork = [&]() {  // the side stream continues after everything issued on the main stream so far
        cudaEventRecord(st.e_main, stream);
        cudaStreamWaitEvent(st.side, st.e_main, 0);
    };
    auto join = [&]() {  // the main stream continues after everything issued on the side stream so far
        cudaEventRecord(st.e_side, st.side);
        cudaStreamWaitEvent(stream, st.e_side, 0);
    };
    const size_t nv = static_cast<size_t>(run.ntimes) * run.nobs;  // one group's partial values
    auto epilogue = [&](int g, long long point_prev) {
        DenseEpi Eg = E;
        Eg.t0 = gt[g] * BN;
        Eg.t1 = gt[g + 1] * BN;
        Eg.prev_values = point_prev >= 0 ? run.part + g * nv + static_cast<size_t>(point_prev) * run.nobs : nullptr;
        if (i8 && wide_epilogue(Eg.t1 - Eg.t0))
            launch_dependent(k_dense_epilogue<true, kEpiThreadsI8>, Eg.t1 - Eg.t0, kEpiThreadsI8, epi_smem, ss[g], st.psi, bp,
                             st.b_scale, Eg);
        else if (i8)
            launch_dependent(k_dense_epilogue<true>, Eg.t1 - Eg.t0, kEpiThreads, epi_smem, ss[g], st.psi, bp, st.b_scale, Eg);
        else
            launch_dependent(k_dense_epilogue<false>, Eg.t1 - Eg.t0, kEpiThreads, epi_smem, ss[g], st.psi, bp, nullptr, Eg);
    };
    auto gemm = [&](int g, cudaStream_t sg) {
        dim3 grid(gt[g + 1] - gt[g], Dp / kGM);
        if (i8)
            launch_dependent(gemm8, grid, kGThreads, smem, sg, ta[0], ta[1], ta[2], ta[3], tb[0], tb[1], tb[2], tb[3],
                             st.u_scale, st.b_scale, st.psi, Dp, gt[g], run.status);
        else
            launch_dependent(ns == 2 ? gemm2 : gemm3, grid, kGThreads, smem, sg, ta[0], ta[1], ta[2], tb[0], tb[1], tb[2],
                             st.psi, Dp, gt[g], run.status);
    };
    if (G == 2) fork();
    // first time point: evaluate, first half-step flip of step 0, split
    E.stepA = steps > 0 ? run.step_offset : -1;
    E.halfA = 0;
    E.pA = pstep(0);
    E.stepB = -1;
    E.init = 1;
    E.dt = 0.0;
    E.elapsed = 0.0;
    E.store_state = steps == 0;
    E.prev_tvals = nullptr;
    for (int g = 0; g < G; ++g) epilogue(g, -1);
    // GEMMs are bracketed by events only when timing was requested, every
    // gemm_every-th step (an event between two kernels costs them their
    // overlap).  On a timed step both groups' GEMMs run back to back on the
    // main stream, so a timed launch is one GEMM over the whole block; the
    // events are read after the loop so the host never waits.
    gemm_every = std::max(1, gemm_every);
    const int ntimed = gemm_ms ? (steps + gemm_every - 1) / gemm_every : 0;
    std::vector<cudaEvent_t> evs(2 * static_cast<size_t>(ntimed));
    for (auto &ev : evs) cudaEventCreate(&ev);
    for (int s = 0; s < steps; ++s) {
        const bool timed = gemm_ms && s % gemm_every == 0;
        if (timed) {
            if (G == 2) join();
            cudaEventRecord(evs[2 * (s / gemm_every)], stream);
            for (int g = 0; g < G; ++g) gemm(g, stream);
            cudaEventRecord(evs[2 * (s / gemm_every) + 1], stream);
            if (G == 2) fork();
        }
        E.stepA = run.step_offset + s;
        E.halfA = 1;
        E.pA = pstep(s);
        E.stepB = s + 1 < steps ? run.step_offset + s + 1 : -1;
        E.halfB = 0;
        E.pB = pstep(s + 1);
        E.init = 0;
        E.dt = run.times[s + 1] - run.times[s];
        E.elapsed = run.times[s + 1] - run.times[0];
        E.tvals = tv[(s + 1) & 1];
        E.prev_tvals = tv[s & 1];  // time point s, summed per group by blocks 0..nobs-1
        E.store_state = s + 1 == steps;
        for (int g = 0; g < G; ++g) {
            if (!timed) gemm(g, ss[g]);
            epilogue(g, s);
        }
        if ((e = cudaGetLastError())) {
            err = std::string("dense: step: ") + cudaGetErrorString(e);
            if (G == 2) join();
            for (auto &ev : evs) cudaEventDestroy(ev);
            return MSGPU_ERR_CUDA;
        }
    }
    // each group's part of the last time point, then the group sums
    for (int g = 0; g < G; ++g)
        k_dense_values<<<run.nobs, kEpiThreads, 0, ss[g]>>>(tv[steps & 1], gt[g] * BN, std::min(gt[g + 1] * BN, M),
                                                            run.nobs,
                                                            run.part + g * nv + static_cast<size_t>(steps) * run.nobs);
    if (G == 2) join();
    k_dense_sum_groups<<<static_cast<unsigned>((nv + 255) / 256), 256, 0, stream>>>(run.part, G, nv, run.values);
    if (gemm_ms) {
        float total = 0.f;
        if (!evs.empty()) cudaEventSynchronize(evs.back());
        for (int k = 0; k < ntimed; ++k) {
            float ms = 0.f;
            cudaEventElapsedTime(&ms, evs[2 * k], evs[2 * k + 1]);
            total += ms;
        }
        *gemm_ms = total;
    }
    for (auto &ev : evs) cudaEventDestroy(ev);
    if (gemm_launches) *gemm_launches = gemm_ms ? ntimed : steps;  // full-block GEMMs the time covers
    const size_t nc = static_cast<size_t>(D) * ldm;
    if (i8)
        k_dense_to_ctx_t<double><<<cdiv(nc, 256), 256, 0, stream>>>(static_cast<const double *>(st.psi), D, M, ldm, Dp,
                                                                     static_cast<double2 *>(psi128));
    else
        k_dense_to_ctx_t<float><<<cdiv(nc, 256), 256, 0, stream>>>(static_cast<const float *>(st.psi), D, M, ldm, Dp,
                                                                    static_cast<double2 *>(psi128));
    if ((e = cudaGetLastError())) {
        err = std::string("dense: state: ") + cudaGetErrorString(e);
        return MSGPU_ERR_CUDA;
    }
    return MSGPU_OK;
}

void dense_release(DenseState &st, void (*release)(void *ctx, void *p), void *ctx)
{
    if (st.side) {
        cudaStreamSynchronize(st.side);
        cudaStreamDestroy(st.side);
    }
    if (st.e_main) cudaEventDestroy(st.e_main);
    if (st.e_side) cudaEventDestroy(st.e_side);
    release(ctx, st.u_parts);
    release(ctx, st.psi);
    release(ctx, st.b_parts);
    release(ctx, st.work);
    st = DenseState();
}

}  // namespace msgpu
