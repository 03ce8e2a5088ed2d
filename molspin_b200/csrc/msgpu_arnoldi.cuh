// msgpu_arnoldi.cuh -- Gram-Schmidt passes of the streamed Arnoldi iteration.
//
// The basis holds w_j unnormalised with per-trajectory scales s_j = 1 / |w_j|
// (v_j = s_j w_j), in complex128 or in the pair-planar complex64 layout; dots
// and coefficients are FP64.  Per iteration
//   k_arn_dots:   h_i = <v_i, W>, i <= j, and |W|^2
//   k_arn_update: W -= sum_i h_i v_i, |W|^2, then beta_{j+1} and s_{j+1}
// and the same two again for the trajectories whose |W| fell below 0.3 of what
// it was (kReorthRatio2): one pass leaves W orthogonal to rounding / 0.3, which
// is closer than modified Gram-Schmidt keeps it, and few iterations cancel
// that much.  A second pass that no trajectory of a tile asks for returns at
// once.  Classical Gram-Schmidt applied twice always read the basis three
// times an iteration; this reads it twice.
//
// Held by load latency (16 warps an SM, 128 to 250 registers for the FP64
// accumulators): 16 loads of four vectors are issued before their FMAs.  B200,
// both passes of an iteration on average (m = 16 or 20): D = 4096, 256
// trajectories complex64 67 us (131 us for CGS2 and its reductions); D = 16384,
// 512 trajectories complex128 544 us, 5.2 TB/s.
//
// A tile's sums over its row tiles are done by the CTA that finishes last, in
// tile order (deterministic), so no reduction kernel runs between the passes.
#pragma once

#include "msgpu_arnoldi.h"
#include "msgpu_kernels.cuh"

namespace msgpu {
namespace {  // internal linkage (see msgpu_kernels.cuh)

__device__ __forceinline__ double2 arn_ld(const double2 *x, size_t row, int t) { return x[row + t]; }
__device__ __forceinline__ double2 arn_ld(const float2 *x, size_t row, int t)
{
    const float *f = reinterpret_cast<const float *>(x + row + (t & ~1)) + (t & 1);
    return make_double2(f[0], f[2]);
}
__device__ __forceinline__ void arn_st(double2 *x, size_t row, int t, double2 v) { x[row + t] = v; }
__device__ __forceinline__ void arn_st(float2 *x, size_t row, int t, double2 v)
{
    float *f = reinterpret_cast<float *>(x + row + (t & ~1)) + (t & 1);
    f[0] = static_cast<float>(v.x);
    f[2] = static_cast<float>(v.y);
}
// the value a later pass reads back
__device__ __forceinline__ double2 arn_round(const double2 *, double2 v) { return v; }
__device__ __forceinline__ double2 arn_round(const float2 *, double2 v)
{
    return make_double2(static_cast<float>(v.x), static_cast<float>(v.y));
}

// True on every thread of the last CTA of this trajectory tile to arrive; the
// partials the others wrote before are then visible.
__device__ __forceinline__ bool arn_last_cta(int *count)
{
    __shared__ int last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        last = atomicAdd(count, 1) == static_cast<int>(gridDim.x) - 1;
        if (last) *count = 0;  // for the next launch
    }
    __syncthreads();
    if (last) __threadfence();
    return last != 0;
}

// Grid (quartet tiles, ldm / 32), a warp per quartet and a lane per trajectory.
// NB >= j + 1: basis vectors with an accumulator.  kPairK: W is first formed
// from U = H v_j as -i U - K4 v_j (K on the electron pair) and stored.
template <typename T, int NB, bool kPairK>
__global__ void __launch_bounds__(kThreads)
k_arn_dots(ArnoldiVectors<T> B, ArnoldiPairK K, const T *__restrict__ U, ArnoldiScratch S, int j, int pass)
{
    grid_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.y * 32 + lane;
    if (pass == 1 && !S.tile_again[blockIdx.y]) return;
    T *W = B.slot(j + 1);
    const double sj = S.scale[static_cast<size_t>(j) * B.ldm + t];
    const int off[4] = {0, B.s2, B.s1, B.s1 + B.s2};
    double2 acc[NB];
    double nrm = 0.0;
#pragma unroll
    for (int i = 0; i < NB; ++i) acc[i] = make_double2(0.0, 0.0);
    const int q1 = min(static_cast<int>(blockIdx.x + 1) * S.QT, B.Q);
    for (int q = blockIdx.x * S.QT + warp; q < q1; q += kWarps) {
        const int base = quartet_base(q, B.s1, B.s2);
        size_t e[4];
        double2 w[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) e[a] = static_cast<size_t>(base + off[a]) * B.ldm;
        if constexpr (kPairK) {
            double2 v[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                v[a] = cscale(arn_ld(B.slot(j), e[a], t), sj);
                const double2 u = arn_ld(U, e[a], t);
                w[a] = make_double2(u.y, -u.x);  // -i U
            }
#pragma unroll
            for (int a = 0; a < 4; ++a) {
#pragma unroll
                for (int b = 0; b < 4; ++b) w[a] = cnfma(K.k[4 * a + b], v[b], w[a]);
                w[a] = arn_round(W, w[a]);
                arn_st(W, e[a], t, w[a]);
            }
        } else {
#pragma unroll
            for (int a = 0; a < 4; ++a) w[a] = arn_ld(W, e[a], t);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) nrm += cabs2(w[a]);
        // four vectors' rows in flight at a time; past j the last one again, unused
#pragma unroll
        for (int i0 = 0; i0 < NB; i0 += 4) {
            if (i0 > j) break;
            double2 v[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int a = 0; a < 4; ++a) v[k][a] = arn_ld(B.slot(min(i0 + k, j)), e[a], t);
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int a = 0; a < 4; ++a) acc[i0 + k] = cconjfma(v[k][a], w[a], acc[i0 + k]);
        }
    }
    // the CTA's sums over its warps, in batches of four vectors
    __shared__ double2 sm[4][kWarps][32];
    double2 *part = S.part + static_cast<size_t>(blockIdx.x) * (j + 2) * B.ldm;
#pragma unroll
    for (int i0 = 0; i0 < NB + 1; i0 += 4) {
        if (i0 > j + 1) break;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = i0 + k;
            if (i < NB && i <= j) sm[k][warp][lane] = acc[i < NB ? i : 0];
            else if (i == j + 1) sm[k][warp][lane] = make_double2(nrm, 0.0);
        }
        __syncthreads();
        if (warp < 4 && i0 + warp <= j + 1) {
            double2 s = sm[warp][0][lane];
#pragma unroll
            for (int w = 1; w < kWarps; ++w) s = cadd(s, sm[warp][w][lane]);
            part[static_cast<size_t>(i0 + warp) * B.ldm + t] = s;
        }
        __syncthreads();
    }
    if (!arn_last_cta(S.count + blockIdx.y)) return;
    // h_i (into H_m) and the update's coefficient of w_i, h_i s_i
    const bool active = S.mdim[t] == 0, again = pass == 0 || S.again[t];
    for (int i = warp; i <= j + 1; i += kWarps) {
        double2 s = make_double2(0.0, 0.0);
#pragma unroll 16
        for (int k = 0; k < static_cast<int>(gridDim.x); ++k)
            s = cadd(s, S.part[(static_cast<size_t>(k) * (j + 2) + i) * B.ldm + t]);
        if (i == j + 1) {
            if (pass == 0) S.before[t] = s.x;
            continue;
        }
        const double si = S.scale[static_cast<size_t>(i) * B.ldm + t];
        const double2 h = again ? cscale(s, si) : make_double2(0.0, 0.0);
        S.coef[static_cast<size_t>(i) * B.ldm + t] = cscale(h, si);
        double2 *Ht = S.hess + static_cast<size_t>(t) * S.m * S.m + i + j * S.m;
        if (active && again) *Ht = pass == 0 ? h : cadd(*Ht, h);
    }
    if (j == S.m - 1) {  // the last column: H_m is complete
        __syncthreads();  // every warp has read mdim
        if (active && warp == 0) S.mdim[t] = S.m;
    }
}

// Grid and roles as k_arn_dots.  The last CTA of a trajectory tile sets
// beta_{j+1} and s_{j+1}; a trajectory whose beta falls below 1e-14 (breakdown,
// as the reference) keeps dimension j + 1.
template <typename T, int NB>
__global__ void __launch_bounds__(kThreads)
k_arn_update(ArnoldiVectors<T> B, ArnoldiScratch S, int j, int pass)
{
    grid_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int t = blockIdx.y * 32 + lane;
    if (pass == 1 && !S.tile_again[blockIdx.y]) return;
    T *W = B.slot(j + 1);
    __shared__ double2 hc[NB][32];
    for (int i = warp; i < NB; i += kWarps)
        hc[i][lane] = i <= j ? S.coef[static_cast<size_t>(i) * B.ldm + t] : make_double2(0.0, 0.0);
    __syncthreads();
    const bool again = pass == 0 || S.again[t];
    const int off[4] = {0, B.s2, B.s1, B.s1 + B.s2};
    double n = 0.0;
    const int q1 = min(static_cast<int>(blockIdx.x + 1) * S.QT, B.Q);
    for (int q = blockIdx.x * S.QT + warp; q < q1; q += kWarps) {
        const int base = quartet_base(q, B.s1, B.s2);
        size_t e[4];
        double2 w[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            e[a] = static_cast<size_t>(base + off[a]) * B.ldm;
            w[a] = arn_ld(W, e[a], t);
        }
#pragma unroll
        for (int i0 = 0; i0 < NB; i0 += 4) {
            if (i0 > j) break;
            double2 v[4][4];
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int a = 0; a < 4; ++a) v[k][a] = arn_ld(B.slot(min(i0 + k, j)), e[a], t);
#pragma unroll
            for (int k = 0; k < 4; ++k)
#pragma unroll
                for (int a = 0; a < 4; ++a) w[a] = cnfma(hc[i0 + k][lane], v[k][a], w[a]);
        }
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const double2 r = arn_round(W, w[a]);
            if (again) arn_st(W, e[a], t, r);
            n += cabs2(r);
        }
    }
    __shared__ double sm[kWarps][32];
    sm[warp][lane] = n;
    __syncthreads();
    double *part = reinterpret_cast<double *>(S.part);
    if (warp == 0) {
        double s = sm[0][lane];
#pragma unroll
        for (int w = 1; w < kWarps; ++w) s += sm[w][lane];
        part[static_cast<size_t>(blockIdx.x) * B.ldm + t] = s;
    }
    if (!arn_last_cta(S.count + blockIdx.y) || warp != 0) return;
    double nn = 0.0;
#pragma unroll 16
    for (int k = 0; k < static_cast<int>(gridDim.x); ++k) nn += part[static_cast<size_t>(k) * B.ldm + t];
    const bool redo = pass == 0 && nn < kReorthRatio2 * S.before[t];
    if (pass == 0) {
        S.again[t] = redo;
        const unsigned any = __ballot_sync(0xffffffffu, redo);
        if (lane == 0) S.tile_again[blockIdx.y] = any != 0;
    }
    if (redo || !again) return;  // a second pass follows, or the first one settled it
    double *next = S.scale + static_cast<size_t>(j + 1) * B.ldm + t;
    if (S.mdim[t] != 0) {
        *next = 0.0;
        return;
    }
    const double beta = sqrt(nn);
    S.hess[static_cast<size_t>(t) * S.m * S.m + (j + 1) + j * S.m] = make_double2(beta, 0.0);
    if (beta < 1e-14) {
        S.mdim[t] = j + 1;
        *next = 0.0;
        return;
    }
    *next = 1.0 / beta;
}

}  // namespace
}  // namespace msgpu
