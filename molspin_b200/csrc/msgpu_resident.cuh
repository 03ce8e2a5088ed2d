// msgpu_resident.cuh -- "resident" form for small Hilbert dimensions.
//
// One CTA owns one trajectory for the whole time loop: its Krylov basis lives
// in shared memory, the trajectory is read from and written back to the state
// once per launch, and every time step (evaluation, ST flips, Krylov step,
// trapezoid) runs inside one kernel launch.  A step is a serial chain of m
// products with H and their reductions, so the chain's latency sets the time:
// rows are spread over the warps of the CTA (RPT rows a thread), a Krylov
// iteration has two barriers, and the small exponential is a Taylor series on
// a vector in one warp.
//
// What bounds it: dependent FP64 latency and, at few warps an SM, the
// instructions of a warp.  B200, us per time step of the whole block:
//   D = 64, 256 trajectories, m = 16, complex128: 14 (186 with a warp per
//     trajectory, Arnoldi and Pade); complex64: 14.3 (36), at 4096 trajectories 66;
//   D = 96, 100 trajectories, unequal sinks: 35 (220);
//   D = 1024, 256 trajectories, complex64: 280 (1570).
//
// Recurrences:
//   Lanczos on H (Hermitian, K = kappa I), complex64 or complex128 vectors,
//     FP64 dot products, norms, tridiagonal and expm;
//   Arnoldi on G = -iH - K (SpinSpace::ArnoldiProcess,
//     SpinSpace_operators.cpp:1352-1408) for any other operator, complex128,
//     with classical Gram-Schmidt applied twice; breakdown below 1e-14.
#pragma once

#include "msgpu_arnoldi.h"
#include "msgpu_kernels.cuh"

namespace msgpu {
namespace {  // internal linkage (see msgpu_kernels.cuh)

// Carves a team's shared memory (the same sequence sizes it on the host).
struct SmemCarve {
    unsigned char *p;
    size_t off;
    template <typename U>
    __host__ __device__ U *take(size_t n)
    {
        U *q = reinterpret_cast<U *>(p + off);
        off += (n * sizeof(U) + 15) / 16 * 16;
        return q;
    }
};

// Pair observables as upper-triangle coefficients over a quartet's (a <= c)
// pairs: Re <x|O|x> = sum Cr Re(x_a* x_c) - Ci Im(x_a* x_c), C_ac = O_ac +
// conj(O_ca) (a < c), C_aa = Re O_aa.  Bit k of re / im: some observable has a
// real / imaginary part in pair k (the four pair-state projectors: 5 of 10 and
// none).
struct ObsTable {
    double2 c[10][8];
    unsigned re, im;
};

template <typename T>
struct ResidentSmem {
    T *V;               // w_0 (the state) .. w_{m-1}; Arnoldi: padded columns, then the vector being orthogonalised
    double2 *Hm;        // Arnoldi: Hessenberg, column-major; Lanczos: alpha_j, beta_{j+1} in .x, .y
    double2 *A;         // 4 m^2 + m: small exponential scratch
    double *sc;         // 1 / |w_j|
    double2 *cf;        // combination coefficients
    double *red;        // 2 x W reduction buffers
    double *rede;       // W x 9 (evaluation)
    double2 *hp;        // Arnoldi: partial dots of warps 1.., W x 32; row 0: the coefficients
    ObsTable *obs;
    int *flags;         // [0] flip of the coming evaluation, [1] Krylov dimension for the combination
    size_t bytes;
};

template <typename T, bool kLanczos>
__host__ __device__ inline ResidentSmem<T> resident_carve(unsigned char *base, int D, int m, int W)
{
    SmemCarve c{base, 0};
    ResidentSmem<T> s;
    s.V = c.take<T>(kLanczos ? static_cast<size_t>(D) * m : static_cast<size_t>(D + 1) * (m + 1));
    s.Hm = c.take<double2>(kLanczos ? m : static_cast<size_t>(m) * m);
    // complex64 Lanczos has no Pade fallback
    s.A = c.take<double2>(kLanczos && sizeof(T) == 8 ? m : 4 * static_cast<size_t>(m) * m + m);
    s.sc = c.take<double>(m);
    s.cf = c.take<double2>(m);
    s.red = c.take<double>(2 * W);
    s.rede = c.take<double>(9 * W);
    s.hp = c.take<double2>(kLanczos ? 1 : 32 * W);
    s.obs = c.take<ObsTable>(1);
    s.flags = c.take<int>(2);
    s.bytes = c.off;
    return s;
}

// One CTA of W warps working on one trajectory.
template <int W>
struct Team {
    __device__ static void sync()
    {
        if constexpr (W == 1) __syncwarp();
        else __syncthreads();
    }
    // sum over the team, the same bits on every thread; also orders the team's
    // shared-memory writes before it.  red: W doubles, not reused before the
    // next team barrier.
    __device__ static double sum(double v, double *red)
    {
        v = warp_sum(v);
        if constexpr (W == 1) {
            __syncwarp();
            return v;
        } else {
            if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
            __syncthreads();
            if constexpr (W <= 8) {
                double s = red[0];
#pragma unroll
                for (int w = 1; w < W; ++w) s += red[w];
                return s;
            } else {
                const int lane = threadIdx.x & 31;
                return warp_sum(lane < W ? red[lane] : 0.0);
            }
        }
    }
};

// A thread's rows of H.  With one row a thread, the row's first kRowRegs
// entries stay in registers for the whole time loop (absent ones: value 0 on
// the row itself), so a product costs one round of shared-memory gathers;
// entries beyond them, and every entry with more rows a thread, are read again
// from the cached copy of H on each product (about 100 cycles a round).
template <typename T, int RPT>
constexpr int row_regs() { return RPT == 1 ? kRowRegs : 0; }

template <typename T, int RPT>
struct Rows {
    static constexpr int KR = row_regs<T, RPT>();
    int base[RPT], cnt[RPT], stride;
    T h[RPT][KR ? KR : 1];
    int c[RPT][KR ? KR : 1];

    __device__ static T value(const ResidentSystem &S, int e)
    {
        if constexpr (sizeof(T) == sizeof(double2)) return __ldg(S.val + e);
        else return __ldg(S.valf + e);
    }
    __device__ static T mac(T h, T x, T a)
    {
        if constexpr (sizeof(T) == sizeof(double2)) return cfma(h, x, a);
        else return cfmaf(h, x, a);
    }
    __device__ void load(const ResidentSystem &S, int tid, int nt)
    {
        stride = S.kstride > 0 ? S.kstride : 1;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + nt * i;
            const bool in = r < S.D;
            const int b = in ? (S.kstride > 0 ? r : __ldg(S.rowptr + r)) : 0;
            cnt[i] = !in ? 0 : S.kstride > 0 ? __ldg(S.rowcnt + r) : __ldg(S.rowptr + r + 1) - b;
            base[i] = b;
#pragma unroll
            for (int k = 0; k < KR; ++k) {
                h[i][k].x = h[i][k].y = 0;
                c[i][k] = in ? r : 0;
                if (k < cnt[i]) {
                    h[i][k] = value(S, base[i] + k * stride);
                    c[i][k] = __ldg(S.col + base[i] + k * stride);
                }
            }
        }
    }
    // (H v)_r of row i in the vector's own precision; kmax: the longest row
    __device__ double2 apply(const ResidentSystem &S, int i, int kmax, const T *v) const
    {
        T a0, a1;
        a0.x = a0.y = a1.x = a1.y = 0;
#pragma unroll
        for (int k = 0; k < KR; k += 4) {
            if (k >= kmax) break;
            T x[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) x[q] = v[c[i][k + q]];
            a0 = mac(h[i][k], x[0], a0);
            a1 = mac(h[i][k + 1], x[1], a1);
            a0 = mac(h[i][k + 2], x[2], a0);
            a1 = mac(h[i][k + 3], x[3], a1);
        }
        if (KR == 0 || kmax > KR) {
#pragma unroll 4
            for (int k = KR; k < cnt[i]; ++k) {
                const int e = base[i] + k * stride;
                a0 = mac(value(S, e), v[__ldg(S.col + e)], a0);
            }
        }
        a0.x += a1.x;
        a0.y += a1.y;
        return make_double2(a0.x, a0.y);
    }
};

// The observables' table, by one warp (lane o < 8: observable o).
__device__ __forceinline__ void fill_observables(const ResidentSystem &S, ObsTable &tab, int lane)
{
    unsigned mre = 0, mim = 0;
    if (lane < 8) {
        int k = 0;
        for (int a = 0; a < 4; ++a)
            for (int c = a; c < 4; ++c, ++k) {
                double2 cc = make_double2(0.0, 0.0);
                if (lane < S.nobs) {
                    const double2 p = S.obs[16 * lane + 4 * a + c], q = S.obs[16 * lane + 4 * c + a];
                    cc = a == c ? make_double2(p.x, 0.0) : make_double2(p.x + q.x, p.y - q.y);
                }
                tab.c[k][lane] = cc;
                if (cc.x != 0.0) mre |= 1u << k;
                if (cc.y != 0.0) mim |= 1u << k;
            }
    }
    mre = __reduce_or_sync(0xffffffffu, mre);
    mim = __reduce_or_sync(0xffffffffu, mim);
    if (lane == 0) {
        tab.re = mre;
        tab.im = mim;
    }
}

// Adds the quartet z's observables to v[0 .. NO) and its squared norm to v[NO].
template <int NO>
__device__ __forceinline__ void pair_observables(const ObsTable &tab, const double2 (&z)[4], double (&v)[NO + 1])
{
    const unsigned mre = tab.re, mim = tab.im;
    v[NO] += (cabs2(z[0]) + cabs2(z[1])) + (cabs2(z[2]) + cabs2(z[3]));
    int k = 0;
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int c = a; c < 4; ++c, ++k) {
            if ((mre >> k) & 1u) {
                const double p = fma(z[a].x, z[c].x, z[a].y * z[c].y);
#pragma unroll
                for (int o = 0; o < NO; ++o) v[o] = fma(tab.c[k][o].x, p, v[o]);
            }
            if ((mim >> k) & 1u) {
                const double p = fma(z[a].x, z[c].y, -z[a].y * z[c].x);
#pragma unroll
                for (int o = 0; o < NO; ++o) v[o] = fma(-tab.c[k][o].y, p, v[o]);
            }
        }
}

// Sums v over the team: val on thread o < nobs (its observable, times the
// rate), the norm on every thread.  All values go through the warp together
// (their shuffles overlap), then one barrier.
template <int W, int NO>
__device__ __forceinline__ void team_reduce_values(const ResidentSystem &S, double *rede, double (&v)[NO + 1], int lane,
                                                   int warp, double &val, double &nrm)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
#pragma unroll
        for (int o = 0; o <= NO; ++o) v[o] += __shfl_xor_sync(0xffffffffu, v[o], off);
    if (lane == 0) {
#pragma unroll
        for (int o = 0; o < NO; ++o) rede[9 * warp + o] = v[o];
        rede[9 * warp + 8] = v[NO];
    }
    Team<W>::sync();
    nrm = rede[8];
#pragma unroll
    for (int w = 1; w < W; ++w) nrm += rede[9 * w + 8];
    val = 0.0;
    if (static_cast<int>(threadIdx.x) < S.nobs) {
        for (int w = 0; w < W; ++w) val += rede[9 * w + threadIdx.x];
        val *= S.rates[threadIdx.x];
    }
}

// Flips (if set), norm and pair observables of the state x, one quartet per
// thread.  NO: 4 or 8 observable slots.
template <typename T, int W, int NO>
__device__ __forceinline__ void resident_evaluate(const ResidentSystem &S, const ResidentSmem<T> &sm, T *x, int flip,
                                                  double &val, double &nrm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, Q = S.D / 4;
    double v[NO + 1];  // observables, then the squared norm
#pragma unroll
    for (int o = 0; o <= NO; ++o) v[o] = 0.0;
    for (int q = threadIdx.x; q < Q; q += 32 * W) {
        const int base = quartet_base(q, S.s1, S.s2);
        const int r[4] = {base, base + S.s2, base + S.s1, base + S.s1 + S.s2};
        double2 z[4];
#pragma unroll
        for (int a = 0; a < 4; ++a) z[a] = ld2(x + r[a]);
        if (flip) {  // U = PS - PT on the pair
            const double2 b = z[1];
            z[0] = make_double2(-z[0].x, -z[0].y);
            z[1] = make_double2(-z[2].x, -z[2].y);
            z[2] = make_double2(-b.x, -b.y);
            z[3] = make_double2(-z[3].x, -z[3].y);
#pragma unroll
            for (int a = 0; a < 4; ++a) st2(x + r[a], z[a]);
        }
        pair_observables<NO>(*sm.obs, z, v);
    }
    team_reduce_values<W, NO>(S, sm.rede, v, lane, warp, val, nrm);
}

template <typename T, int W>
__device__ __forceinline__ void resident_epilogue(const ResidentSystem &S, const ResidentSmem<T> &sm, T *x, int flip,
                                                  double &val, double &nrm)
{
    if (S.nobs <= 4) resident_evaluate<T, W, 4>(S, sm, x, flip, val, nrm);
    else resident_evaluate<T, W, 8>(S, sm, x, flip, val, nrm);
}

// Lanczos factorisation of the state sm.V (= w_0, |w_0|^2 = nrm2): w_j
// unnormalised in slot j with scale sm.sc[j], alpha and beta in sm.Hm.
// Returns the Krylov dimension.  Two team barriers per iteration: the one of
// alpha, and the one of |w_{j+1}|^2, which also publishes w_{j+1} for the next
// product (hence stored before it is normalised).
template <typename T, int W, int RPT>
__device__ __forceinline__ int resident_lanczos(const ResidentSystem &S, const ResidentSmem<T> &sm, const Rows<T, RPT> &H,
                                                int kmax, double inv0)
{
    const int D = S.D, m = S.m, tid = threadIdx.x;
    constexpr int NT = 32 * W;
    double2 vc[RPT], vp[RPT], u[RPT];
    double s = inv0, bprev = 0.0;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        vp[i] = u[i] = make_double2(0.0, 0.0);
        const int r = tid + NT * i;
        vc[i] = r < D ? cscale(ld2(sm.V + r), s) : make_double2(0.0, 0.0);
    }
    if (tid == 0) sm.sc[0] = s;
    int n = m;
    for (int j = 0; j < m; ++j) {
        const T *wj = sm.V + static_cast<size_t>(j) * D;
        double pa = 0.0;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            if (tid + NT * i < D) {
                u[i] = cscale(H.apply(S, i, kmax, wj), s);
                pa = fma(vc[i].x, u[i].x, fma(vc[i].y, u[i].y, pa));
            }
        }
        const double alpha = Team<W>::sum(pa, sm.red);
        if (j == m - 1) {  // T_m is complete; w_m is never used
            if (tid == 0) sm.Hm[j] = make_double2(alpha, 0.0);
            break;
        }
        double pn = 0.0;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + NT * i;
            if (r < D) {
                double2 w = make_double2(fma(-bprev, vp[i].x, u[i].x), fma(-bprev, vp[i].y, u[i].y));
                w = make_double2(fma(-alpha, vc[i].x, w.x), fma(-alpha, vc[i].y, w.y));
                T wr;
                st2(&wr, w);
                sm.V[static_cast<size_t>(j + 1) * D + r] = wr;
                u[i] = ld2(&wr);  // the stored (rounded) vector is the one the norm and the next product see
                pn += cabs2(u[i]);
            }
        }
        const double nn = Team<W>::sum(pn, sm.red + W);
        s = rsqrt(nn);
        const double bn = nn > 0.0 ? nn * s : 0.0;
        if (tid == 0) {
            sm.Hm[j] = make_double2(alpha, bn);
            sm.sc[j + 1] = s;
        }
        if (__any_sync(0xffffffffu, bn < 1e-14)) { n = j + 1; break; }
        bprev = bn;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            vp[i] = vc[i];
            vc[i] = cscale(u[i], s);
        }
    }
    return n;
}

// Dots of z with the first nv basis vectors (nv <= 32), and |z|^2 when kNorm:
// a warp takes every W-th row, its lanes one basis vector each (two rows at a
// time while 16 lanes suffice), so no shuffles; then the warps' sums.  Columns
// are D + 1 apart, which keeps both this access and a thread's own rows free
// of bank conflicts.  Lane i < nv of warp 0 returns w_i^H z, lane nv |z|^2.
template <int W, bool kNorm>
__device__ __forceinline__ double2 resident_dots(const double2 *V, const double2 *z, int D, int nv, double2 *hp)
{
    const int lane = threadIdx.x & 31, warp = warp_uniform(threadIdx.x >> 5);
    const int nd = kNorm ? nv + 1 : nv;
    const bool split = nd <= 16;
    const int i = split ? (lane & 15) : lane;
    double2 a = make_double2(0.0, 0.0), b = make_double2(0.0, 0.0);
    const double2 *vi = i < nv ? V + static_cast<size_t>(i) * (D + 1) : z;  // lanes beyond nv repeat |z|^2
    const int step = split ? 2 * W : W;
    int r = split ? 2 * warp + (lane >> 4) : warp;
#pragma unroll 2
    for (; r + step < D; r += 2 * step) {
        a = cconjfma(vi[r], z[r], a);
        b = cconjfma(vi[r + step], z[r + step], b);
    }
    if (r < D) a = cconjfma(vi[r], z[r], a);
    a = cadd(a, b);
    if (split) {
        a.x += __shfl_xor_sync(0xffffffffu, a.x, 16);
        a.y += __shfl_xor_sync(0xffffffffu, a.y, 16);
    }
    if constexpr (W > 1) {
        if (warp > 0) hp[32 * warp + lane] = a;
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int w = 1; w < W; ++w) a = cadd(a, hp[32 * w + lane]);
        }
    }
    return a;
}

// Arnoldi factorisation of the state (slot 0 of sm.V) on G = -iH - K: w_j
// unnormalised in slot j with scale sm.sc[j], H_m in sm.Hm.  Classical
// Gram-Schmidt: one round of dots per iteration, where modified Gram-Schmidt
// serialises j + 1 of them; a second pass when the first cancelled
// (kReorthRatio2).  Returns the Krylov dimension.
template <int W, int RPT>
__device__ __forceinline__ int resident_arnoldi(const ResidentSystem &S, const ResidentSmem<double2> &sm,
                                                const Rows<double2, RPT> &H, int kmax, double inv0)
{
    const int D = S.D, m = S.m, tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    constexpr int NT = 32 * W;
    const size_t ld = static_cast<size_t>(D) + 1;
    double2 *V = sm.V, *z = sm.V + static_cast<size_t>(m) * ld, *h = sm.hp;  // h: coefficients of the w_i, then |z|^2
    double2 u[RPT];
    double s = inv0;
    if (tid == 0) sm.sc[0] = s;
    int n = m;
    for (int j = 0; j < m; ++j) {
        const double2 *wj = V + j * ld;
#pragma unroll
        for (int i = 0; i < RPT; ++i) {
            const int r = tid + NT * i;
            if (r >= D) continue;
            double2 g = H.apply(S, i, kmax, wj);
            if (!S.generator) {
                g = make_double2(g.y, -g.x);  // -i (H w)_r
                if (S.krow) {
                    double2 ka = make_double2(0.0, 0.0);
                    for (int k = __ldg(S.krow + r); k < __ldg(S.krow + r + 1); ++k)
                        ka = cfma(__ldg(S.kval + k), wj[__ldg(S.kcol + k)], ka);
                    g = csub(g, ka);
                } else {
                    g = csub(g, cscale(wj[r], S.kappa));
                }
            }
            u[i] = cscale(g, s);
            z[r] = u[i];
        }
        Team<W>::sync();
        double nn = 0.0;
        for (int pass = 0; pass < 2; ++pass) {
            // the column of H_m is complete after its dots when it is the last
            const bool last = j == m - 1;
            const double2 d = pass == 0 && !last ? resident_dots<W, true>(V, z, D, j + 1, sm.hp)
                                                 : resident_dots<W, false>(V, z, D, j + 1, sm.hp);
            if (warp == 0) {
                if (lane <= j) {
                    const double2 t = cscale(d, sm.sc[lane]);
                    double2 *hm = sm.Hm + lane + j * m;
                    *hm = pass ? cadd(*hm, t) : t;
                    h[lane] = cscale(t, sm.sc[lane]);
                } else if (lane == j + 1) {
                    h[lane] = d;
                }
            }
            Team<W>::sync();
            if (last) break;
            double pn = 0.0;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = tid + NT * i;
                if (r >= D) continue;
                double2 w = u[i], w2 = make_double2(0.0, 0.0);
                const double2 *col = V + r;
                int k = 0;
#pragma unroll 2
                for (; k < j; k += 2) {
                    w = cnfma(h[k], col[k * ld], w);
                    w2 = cnfma(h[k + 1], col[(k + 1) * ld], w2);
                }
                if (k <= j) w = cnfma(h[k], col[k * ld], w);
                u[i] = cadd(w, w2);
                V[(j + 1) * ld + r] = u[i];
                if (pass == 0) z[r] = u[i];
                pn += cabs2(u[i]);
            }
            const double before = h[j + 1].x;
            nn = Team<W>::sum(pn, sm.red + pass * W);
            if (pass == 0 && !__any_sync(0xffffffffu, nn < kReorthRatio2 * before)) break;
        }
        if (j == m - 1) break;
        s = rsqrt(nn);
        const double bn = nn > 0.0 ? nn * s : 0.0;
        if (tid == 0) {
            sm.Hm[(j + 1) + j * m] = make_double2(bn, 0.0);
            sm.sc[j + 1] = s;
        }
        if (__any_sync(0xffffffffu, bn < 1e-14)) { n = j + 1; break; }
    }
    return n;
}

// Whole time loop of trajectory t of system S by one CTA of W warps, RPT rows
// a thread (32 W RPT >= D).  TS: the state's type in memory.
template <typename T, typename TS, int W, int RPT, bool kLanczos>
__device__ __forceinline__ void resident_propagate(const ResidentSystem &S, int t, unsigned char *smem,
                                                   int *__restrict__ status)
{
    constexpr int NT = 32 * W;
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    const int D = S.D, m = S.m;
    const ResidentSmem<T> sm = resident_carve<T, kLanczos>(smem, D, m, W);
    T *x = sm.V;  // the state
    const size_t ld = kLanczos ? D : D + 1;
    const TS *in = static_cast<const TS *>(S.psi) + static_cast<size_t>(t) * S.ts;
    Rows<T, RPT> H;
    H.load(S, tid, NT);
    const int kmax = S.kmax;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + NT * i;
        if (r < D) st2(x + r, ld2(in + static_cast<size_t>(r) * S.rs));
    }
    if (warp == 0) fill_observables(S, *sm.obs, lane);
    const int steps = S.ntimes - 1;
    const long long g0 = S.step_offset;
    const bool noisy = S.nz.mode != 0;
    if (tid == 0) sm.flags[0] = noisy && steps > 0 ? noise_bit(S.nz, t, g0, 0, S.pflip[0]) : 0;
    // thread o < nobs keeps observable o's trapezoid
    const bool own = tid < S.nobs;
    const size_t ak = static_cast<size_t>(tid) * S.acc_ld + t;
    double acc = 0.0, comp = 0.0, prev = 0.0, val = 0.0, nrm2 = 0.0;
    if (own && S.accumulate) {
        acc = S.acc[ak];
        comp = S.comp[ak];
    }
    bool bad = false;
    Team<W>::sync();
    resident_epilogue<T, W>(S, sm, x, sm.flags[0], val, nrm2);
    prev = val;
    if (S.traj_values && own) S.traj_values[static_cast<size_t>(t) * S.nobs + tid] = val;
    if (S.check_start && !isfinite(nrm2)) bad = true;
    for (int s = 0; s < steps; ++s) {
        const double dt = S.times ? S.times[s + 1] - S.times[s] : S.dt0;
        const double inv0 = rsqrt(nrm2), beta0 = nrm2 > 0.0 ? nrm2 * inv0 : 0.0;
        // second half flip of step s and first half flip of step s + 1, by the
        // last warp while the first one exponentiates
        auto draw_flip = [&]() {
            if (warp == W - 1 && lane == 0) {
                int f = 0;
                if (noisy) {
                    f = noise_bit(S.nz, t, g0 + s, 1, S.pflip[s]);
                    if (s + 1 < steps) f ^= noise_bit(S.nz, t, g0 + s + 1, 0, S.pflip[s + 1]);
                }
                sm.flags[0] = f;
            }
        };
        if (beta0 > 0.0) {
            int n;
            if constexpr (kLanczos) n = resident_lanczos<T, W, RPT>(S, sm, H, kmax, inv0);
            else n = resident_arnoldi<W, RPT>(S, sm, H, kmax, inv0);
            if (warp == 0) {
                bool ok;
                double2 c = make_double2(0.0, 0.0);
                __syncwarp();
                if constexpr (kLanczos) {
                    const double d = lane < n ? sm.Hm[lane].x : 0.0;
                    const double lo = (lane < n && lane > 0) ? sm.Hm[lane - 1].y : 0.0;
                    const double hi = lane + 1 < n ? sm.Hm[lane].y : 0.0;
                    bool taylor = true;
                    if constexpr (sizeof(T) == sizeof(double2))
                        taylor = !__any_sync(0xffffffffu, fabs(dt) * (fabs(d) + fabs(lo) + fabs(hi)) > 256.0);
                    if (taylor) {
                        ok = warp_tridiag_expm_e1(n, d, lo, hi, S.kappa, dt, c);
                    } else {
                        // the reference's Pade form on the same matrix
                        double2 *A = sm.A, *X = A + m * m, *N = X + m * m, *Dm = N + m * m, *y = Dm + m * m;
                        if (lane < n)
                            for (int i = 0; i < n; ++i) {
                                double2 e = make_double2(0.0, 0.0);
                                if (i == lane) e = make_double2(-S.kappa, -d);
                                else if (i == lane + 1) e = make_double2(0.0, -hi);
                                else if (i + 1 == lane) e = make_double2(0.0, -lo);
                                A[i + lane * n] = cscale(e, dt);
                            }
                        __syncwarp();
                        ok = warp_expm_col0_cold(n, A, X, N, Dm, y);
                        if (lane < n) c = y[lane];
                    }
                } else {
                    double2 *A = sm.A, *X = A + m * m, *N = X + m * m, *Dm = N + m * m, *y = Dm + m * m;
                    // upper Hessenberg part only; entries below the subdiagonal are never written
                    if (lane < n)
                        for (int i = 0; i < n; ++i)
                            A[i + lane * n] = i <= lane + 1 ? cscale(sm.Hm[i + lane * m], dt) : make_double2(0.0, 0.0);
                    __syncwarp();
                    ok = warp_expm_e1(n, A, X, N, Dm, y);
                    if (lane < n) c = y[lane];
                }
                if (lane < n) c = cscale(c, beta0 * sm.sc[lane]);
                if (!ok && lane == 0) atomicOr(status, 1);
                if (lane < n) sm.cf[lane] = ok ? c : make_double2(0.0, 0.0);
            }
            draw_flip();
            Team<W>::sync();
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                const int r = tid + NT * i;
                if (r >= D) continue;
                double2 a[4];  // partial sums: the dependent FMA chain, not the loads, sets the time
#pragma unroll
                for (int k = 0; k < 4; ++k) a[k] = make_double2(0.0, 0.0);
                int j = 0;
                for (; j + 3 < n; j += 4)
#pragma unroll
                    for (int k = 0; k < 4; ++k) a[k] = cfma(sm.cf[j + k], ld2(sm.V + (j + k) * ld + r), a[k]);
                for (; j < n; ++j) a[0] = cfma(sm.cf[j], ld2(sm.V + j * ld + r), a[0]);
                st2(x + r, cadd(cadd(a[0], a[1]), cadd(a[2], a[3])));
            }
        } else {
            draw_flip();
        }
        Team<W>::sync();
        resident_epilogue<T, W>(S, sm, x, sm.flags[0], val, nrm2);
        if (own) {
            const double term = 0.5 * dt * (prev + val) - comp;
            const double sum = acc + term;
            comp = (sum - acc) - term;
            acc = sum;
            prev = val;
            if (!isfinite(val)) bad = true;
            if (S.traj_values) S.traj_values[(static_cast<size_t>(s + 1) * S.M + t) * S.nobs + tid] = val;
        }
    }
    TS *out = static_cast<TS *>(S.psi_out) + static_cast<size_t>(t) * S.ts;
    // the observables skip the pairs of rows that none of them has a coefficient
    // for: what is not finite there shows in the state, which stops evolving with it
    const bool watched = steps > 0 && S.nobs > 0;
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = tid + NT * i;
        if (r >= D) continue;
        const double2 z = ld2(x + r);
        st2(out + static_cast<size_t>(r) * S.rs, z);
        bad = bad || (watched && !(isfinite(z.x) && isfinite(z.y)));
    }
    if (own) {
        S.acc[ak] = acc;
        S.comp[ak] = comp;
        S.prev[ak] = prev;
    }
    if (bad) atomicOr(status, 2);
}

// CTAs per SM the register allocation must allow.  complex64 keeps 16 warps on
// an SM (128 registers a thread): with 133 registers a scheduler holds three
// warps, not four, and 1024 trajectories of D = 64 took 27 instead of 18 us a
// step.  So do the complex128 shapes of two rows a thread up to four warps, which
// are there for many trajectories (resident_shape_c128).
template <typename T, int RPT>
constexpr int resident_min_ctas(int W)
{
    const bool full = sizeof(T) == sizeof(float2) ? W <= 16 : RPT == 2 && W <= 4;
    return full ? 16 / W : 1;
}

// One launch = the whole time loop of every trajectory (one CTA each).
template <typename T, int W, int RPT, bool kLanczos>
__global__ void __launch_bounds__(32 * W, resident_min_ctas<T, RPT>(W))
k_resident(const __grid_constant__ ResidentSystem S, int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    resident_propagate<T, double2, W, RPT, kLanczos>(S, blockIdx.x, smem_raw, status);
}

// The system that CTA b belongs to: first[i] <= b < first[i + 1].
__device__ __forceinline__ int system_of(const int *__restrict__ first, int nsystems, int b)
{
    int lo = 0, hi = nsystems;
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (__ldg(first + mid) <= b) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Copies a system's descriptor to shared memory, where it costs no registers.
__device__ __forceinline__ void load_system(ResidentSystem *to, const ResidentSystem *from)
{
    static_assert(sizeof(ResidentSystem) % 8 == 0, "copied by 8 bytes");
    for (unsigned k = threadIdx.x; k < sizeof(ResidentSystem) / 8; k += blockDim.x)
        reinterpret_cast<unsigned long long *>(to)[k] = __ldg(reinterpret_cast<const unsigned long long *>(from) + k);
    __syncthreads();
}

// The same for the trajectories of many systems (the batching form).
template <int W>
__global__ void __launch_bounds__(32 * W, resident_min_ctas<float2, 1>(W))
k_resident_many(const ResidentSystem *__restrict__ systems, const int *__restrict__ first, int nsystems,
                int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ResidentSystem S;
    const int i = system_of(first, nsystems, blockIdx.x);
    load_system(&S, systems + i);
    resident_propagate<float2, float2, W, 1, true>(S, blockIdx.x - __ldg(first + i), smem_raw, status);
}

}  // namespace
}  // namespace msgpu
