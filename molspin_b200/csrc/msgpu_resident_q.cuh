// msgpu_resident_q.cuh -- resident form over quartets, complex64 (D > 128).
//
// As msgpu_resident.cuh (one CTA per trajectory for the whole time loop,
// three-term recurrence), with a thread per quartet instead of per row: a
// nucleus' flip block is 4 values for 16 matrix entries and one gather serves
// four rows, and a thread's whole part of H -- its own 4x4 block and up to
// eight flip blocks, one slot per nucleus -- stays in registers for the whole time loop, so a product
// reads nothing but the vector in shared memory.  At D = 1024 the row form
// reads 233 KB of H a product through L2, which sets its time: a step of 256
// trajectories takes 280 us there against 65 here (B200, m = 16; 1570 with a
// warp per trajectory).  A product is then about 1900 of an iteration's 3700
// cycles (FMA issue of two warps a scheduler), its two reductions 800.
//
// A vector is kept in two planes, re and im, of one float4 a quartet (the
// quartet's four rows): 16-byte accesses without bank conflicts.
#pragma once

#include "msgpu_quartet.h"
#include "msgpu_resident.cuh"

namespace msgpu {
namespace {  // internal linkage (see msgpu_kernels.cuh)

// Own block of quartet q to full 4 x 4, columns b: re and im of the four rows.
__device__ inline void quartet_expand(int type, const float2 *v, float4 (&re)[4], float4 (&im)[4])
{
    float r[4][4], i[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int a1 = a >> 1, a2 = a & 1, b1 = b >> 1, b2 = b & 1;
            float2 z = make_float2(0.f, 0.f);
            if (type == 0) z = v[4 * a + b];
            else if (type == 1 && a2 == b2) z = v[(2 * a2 + a1) * 2 + b1];
            else if (type == 2 && a1 == b1) z = v[(2 * a1 + a2) * 2 + b2];
            else if (type == 3 && a == b) z = v[a];
            else if (type == 4 && a2 == b2) z = v[2 * a1 + b1];
            else if (type == 5 && a1 == b1) z = v[2 * a2 + b2];
            r[a][b] = z.x;
            i[a][b] = z.y;
        }
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        re[b] = make_float4(r[0][b], r[1][b], r[2][b], r[3][b]);
        im[b] = make_float4(i[0][b], i[1][b], i[2][b], i[3][b]);
    }
}

// The resident layout from the quartet form (QuartetC).
__global__ void k_build_resident_quartets(QuartetC H, int Q, int s1, int s2, QuartetSlots S, float4 *__restrict__ own,
                                          int2 *__restrict__ slot, int2 *__restrict__ blk, int *__restrict__ nblk)
{
    const int q = blockIdx.x * blockDim.x + threadIdx.x;
    if (q >= Q) return;
    const int base = H.base[q];
    const float2 *val = reinterpret_cast<const float2 *>(H.val);
    float4 re[4], im[4];
#pragma unroll
    for (int b = 0; b < 4; ++b) re[b] = im[b] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int k = 0; k < S.n; ++k) slot[static_cast<size_t>(k) * Q + q] = make_int2(q, -1);
    int n = 0;
    for (int k = H.rowptr[q]; k < H.rowptr[q + 1]; ++k) {
        const int2 c = H.blk[k];
        const int cb = c.x >> 3, type = c.x & 7;
        if (cb == base) {
            quartet_expand(type, val + 2 * static_cast<size_t>(c.y), re, im);
            continue;
        }
        const int qn = (cb / (2 * s1)) * (s1 / 2) + ((cb / (2 * s2)) % (s1 / (2 * s2))) * s2 + cb % s2;
        int at = -1;
        for (int i = 0; i < S.n; ++i)
            if (qn - q == S.delta[i] || (((S.shared >> i) & 1u) && q - qn == S.delta[i])) at = i;
        if (at >= 0) slot[static_cast<size_t>(at) * Q + q] = make_int2(qn, c.y);
        else if (n < S.left) blk[static_cast<size_t>(n++) * Q + q] = make_int2((qn << 3) | type, c.y);
    }
    nblk[q] = n;
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        own[static_cast<size_t>(2 * b) * Q + q] = re[b];
        own[static_cast<size_t>(2 * b + 1) * Q + q] = im[b];
    }
}

// The arrays of an assembled system in its buffer.
struct AssembledQuartets {
    float4 *own;   // [8][Q]
    float4 *val;   // [kQuartetSlots][Q][2]
    int2 *slot;    // [kQuartetSlots][Q]
    int *nblk;     // [Q], zero
    __host__ __device__ AssembledQuartets(void *buf, int Q)
    {
        own = static_cast<float4 *>(buf);
        val = own + 8 * static_cast<size_t>(Q);
        slot = reinterpret_cast<int2 *>(val + 2 * kQuartetSlots * static_cast<size_t>(Q));
        nblk = reinterpret_cast<int *>(slot + kQuartetSlots * static_cast<size_t>(Q));
    }
};

// The resident layout straight from CSR rows, one CTA a system and a row a thread:
// the rules of quartet_slots on FP32 values (a block with equal halves is A (x) I),
// slots for pairs of distances +-d ahead of single ones.  Systems with more than
// kQuartetSlots slots, or a block that is of neither type, are left to the host.
// On the host it takes 0.16 ms a system of D = 1024; here about 20 us for all
// systems of a batch.
constexpr int kAssembleThreads = 512, kAssembleDist = 16;
constexpr int kAssembleD = 1536;  // what resident_q_takes
__global__ void __launch_bounds__(kAssembleThreads)
k_assemble_quartets(const QuartetJob *__restrict__ jobs, QuartetFound *__restrict__ found)
{
    const QuartetJob J = jobs[blockIdx.x];
    const int D = J.D, Q = D / 4, s1 = J.s1, s2 = J.s2, tid = threadIdx.x, lane = tid & 31;
    const int off[4] = {0, s2, s1, s1 + s2};
    const AssembledQuartets B(J.buf, Q);
    __shared__ unsigned short place[kAssembleD];     // 4 (quartet of a row) + its pair index
    __shared__ unsigned mask[kAssembleD / 2];        // by signed distance + Q: entries 4 a + b in use
    __shared__ signed char list[kAssembleD / 2];     // place in dist, or -1
    __shared__ unsigned seen[kAssembleD / 4];        // by quartet: bit i, a block at dist[i]
    __shared__ int dist[kAssembleDist], slot_of[kAssembleDist];
    __shared__ unsigned state[kAssembleDist];        // bit 0: not of the one type it can be; bit 1: -d in the same quartet
    __shared__ int ndist, nslot;
    __shared__ unsigned second;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int q = tid; q < Q; q += kAssembleThreads) {
        const int base = quartet_base(q, s1, s2);
        for (int a = 0; a < 4; ++a) place[base + off[a]] = static_cast<unsigned short>(4 * q + a);
        seen[q] = 0;
        mask[q] = mask[Q + q] = 0;
        B.nblk[q] = 0;
    }
    for (int i = tid; i < 8 * Q; i += kAssembleThreads) B.own[i] = zero;
    for (int i = tid; i < 2 * kQuartetSlots * Q; i += kAssembleThreads) B.val[i] = zero;
    for (int i = tid; i < kQuartetSlots * Q; i += kAssembleThreads) B.slot[i] = make_int2(i % Q, -1);
    if (tid < kAssembleDist) state[tid] = 0;
    __syncthreads();
    // f(q, a, nq, b, value, row, column) for every entry that is not zero
    auto entries = [&](auto f) {
        for (int r = tid; r < D; r += kAssembleThreads) {
            const int at = place[r];
            for (int k = __ldg(J.rowptr + r); k < __ldg(J.rowptr + r + 1); ++k) {
                const float2 v = __ldg(J.val + k);
                if (v.x == 0.f && v.y == 0.f) continue;
                const int c = __ldg(J.col + k), to = place[c];
                f(at >> 2, at & 3, to >> 2, to & 3, v, r, c);
            }
        }
    };
    entries([&](int q, int a, int nq, int b, float2, int, int) {
        const unsigned bit = 1u << (4 * a + b);
        if (nq != q && !(mask[Q + nq - q] & bit)) atomicOr(&mask[Q + nq - q], bit);
    });
    __syncthreads();
    if (tid < 32) {  // the distances in use, ascending
        int n = 0;
        for (int i0 = 0; i0 < 2 * Q; i0 += 32) {
            const int i = i0 + lane;
            const bool on = i < 2 * Q && mask[i] != 0;
            const unsigned all = __ballot_sync(0xffffffffu, on);
            const int at = n + __popc(all & ((1u << lane) - 1u));
            if (i < 2 * Q) list[i] = static_cast<signed char>(on && at < kAssembleDist ? at : -1);
            if (on && at < kAssembleDist) dist[at] = i - Q;
            n += __popc(all);
        }
        if (lane == 0) ndist = n;
    }
    __syncthreads();
    const bool few = ndist <= kAssembleDist;
    // entries that couple different second (first) digits of the pair
    constexpr unsigned kSecond = 0x5a5au, kFirst = 0x33ccu;
    if (few)
        entries([&](int q, int a, int nq, int b, float2 v, int r, int c) {
            if (nq == q) return;
            const int i = list[Q + nq - q];
            if (!((seen[q] >> i) & 1u)) atomicOr(&seen[q], 1u << i);
            const unsigned m = mask[Q + nq - q];
            // on the first digit alone: the same for both of the second's states, and the reverse
            const int step = !(m & kSecond) ? (a & 1 ? -s2 : s2) : !(m & kFirst) ? (a & 2 ? -s1 : s1) : 0;
            bool same = false;
            if (step != 0)
                for (int k = __ldg(J.rowptr + r + step); k < __ldg(J.rowptr + r + step + 1) && !same; ++k) {
                    const float2 w = __ldg(J.val + k);
                    same = __ldg(J.col + k) == c + step && w.x == v.x && w.y == v.y;
                }
            if (!same) atomicOr(&state[i], 1u);
        });
    __syncthreads();
    if (few)
        for (int q = tid; q < Q; q += kAssembleThreads)
            for (int i = 0; i < ndist; ++i) {
                const int j = list[Q - dist[i]];
                if (j >= 0 && ((seen[q] >> i) & 1u) && ((seen[q] >> j) & 1u)) atomicOr(&state[i], 2u);
            }
    __syncthreads();
    if (tid == 0) {
        int n = 0;
        unsigned sec = 0;
        bool ok = few;
        for (int i = 0; i < ndist && ok; ++i) {
            slot_of[i] = -1;
            ok = !(state[i] & 1u);
        }
        auto is_second = [&](int i) { return (mask[Q + dist[i]] & kSecond) != 0; };
        for (int pass = 0; pass < 2 && ok; ++pass)
            for (int i = 0; i < ndist && ok; ++i) {
                const int j = list[Q - dist[i]];
                const bool pair = j >= 0 && !(state[i] & 2u) && is_second(i) == is_second(j);
                if (slot_of[i] >= 0 || (pass == 0 && !(pair && dist[i] > 0))) continue;
                if (n == kQuartetSlots) {
                    ok = false;
                    break;
                }
                slot_of[i] = n;
                if (pair) slot_of[j] = n;
                if (is_second(i)) sec |= 1u << n;
                ++n;
            }
        nslot = ok ? n : -1;
        second = sec;
        found[blockIdx.x] = QuartetFound{nslot, sec};
    }
    __syncthreads();
    if (nslot < 0) return;
    entries([&](int q, int a, int nq, int b, float2 v, int, int) {
        if (nq == q) {
            reinterpret_cast<float *>(B.own + static_cast<size_t>(2 * b) * Q + q)[a] = v.x;
            reinterpret_cast<float *>(B.own + static_cast<size_t>(2 * b + 1) * Q + q)[a] = v.y;
            return;
        }
        const int k = slot_of[list[Q + nq - q]];
        const size_t at = static_cast<size_t>(k) * Q + q;
        B.slot[at] = make_int2(nq, static_cast<int>(2 * at));  // the same from every row of the block
        const bool sec = (second >> k) & 1u;
        if ((sec ? a >> 1 : a & 1) == 0)
            reinterpret_cast<float2 *>(B.val + 2 * at)[sec ? 2 * (a & 1) + (b & 1) : 2 * (a >> 1) + (b >> 1)] = v;
    });
}

struct QuartetAcc {
    float re[4], im[4];
};

__device__ __forceinline__ void acc_mac(QuartetAcc &o, int a, float br, float bi, float xr, float xi)
{
    o.re[a] = fmaf(br, xr, o.re[a]);
    o.re[a] = fmaf(-bi, xi, o.re[a]);
    o.im[a] = fmaf(br, xi, o.im[a]);
    o.im[a] = fmaf(bi, xr, o.im[a]);
}

// One flip block, values p = A00 A01, r = A10 A11, on the first digit (A (x) I)
// or the second (I (x) A).  Plain FMAs: packed ones need every broadcast value
// or row twice in registers, and the copies cost what they save.
__device__ __forceinline__ void flip_mac(QuartetAcc &o, bool second, float4 p, float4 r, float4 xr, float4 xi)
{
    const float x[4] = {xr.x, xr.y, xr.z, xr.w}, y[4] = {xi.x, xi.y, xi.z, xi.w};
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        if (!second) {
            acc_mac(o, h, p.x, p.y, x[h], y[h]);
            acc_mac(o, 2 + h, r.x, r.y, x[h], y[h]);
            acc_mac(o, h, p.z, p.w, x[2 + h], y[2 + h]);
            acc_mac(o, 2 + h, r.z, r.w, x[2 + h], y[2 + h]);
        } else {
            acc_mac(o, 2 * h, p.x, p.y, x[2 * h], y[2 * h]);
            acc_mac(o, 2 * h + 1, r.x, r.y, x[2 * h], y[2 * h]);
            acc_mac(o, 2 * h, p.z, p.w, x[2 * h + 1], y[2 * h + 1]);
            acc_mac(o, 2 * h + 1, r.z, r.w, x[2 * h + 1], y[2 * h + 1]);
        }
    }
}

// o += B x, B full with columns (re[b], im[b])
__device__ __forceinline__ void full_mac(QuartetAcc &o, const float4 (&re)[4], const float4 (&im)[4], float4 xr, float4 xi)
{
    const float x[4] = {xr.x, xr.y, xr.z, xr.w}, y[4] = {xi.x, xi.y, xi.z, xi.w};
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        acc_mac(o, 0, re[b].x, im[b].x, x[b], y[b]);
        acc_mac(o, 1, re[b].y, im[b].y, x[b], y[b]);
        acc_mac(o, 2, re[b].z, im[b].z, x[b], y[b]);
        acc_mac(o, 3, re[b].w, im[b].w, x[b], y[b]);
    }
}

// A thread's quartet of H: its own block and its slots' blocks in registers
// (absent ones: value 0 on the quartet itself); other blocks are read on each
// product.
struct QuartetRow {
    int q, n;           // quartet, blocks without a slot
    int nb[kQuartetSlots];
    float4 p[kQuartetSlots], r[kQuartetSlots];
    float4 ore[4], oim[4];

    __device__ void load(const ResidentQuartets &H, int q_, bool live)
    {
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        q = live ? q_ : 0;
        n = live ? __ldg(H.nblk + q) : 0;
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            ore[b] = live ? __ldg(H.own + static_cast<size_t>(2 * b) * H.Q + q) : zero;
            oim[b] = live ? __ldg(H.own + static_cast<size_t>(2 * b + 1) * H.Q + q) : zero;
        }
#pragma unroll
        for (int k = 0; k < kQuartetSlots; ++k) {
            nb[k] = q;
            p[k] = r[k] = zero;
            if (k < H.nslot && live) {
                const int2 x = __ldg(H.slot + static_cast<size_t>(k) * H.Q + q);
                nb[k] = x.x;
                if (x.y >= 0) {
                    p[k] = __ldg(H.val + x.y);
                    r[k] = __ldg(H.val + x.y + 1);
                }
            }
        }
    }
    // H x at the quartet; xr, xi: its own rows; re, im: the vector's planes
    __device__ QuartetAcc apply(const ResidentQuartets &H, const float4 *re, const float4 *im, float4 xr, float4 xi) const
    {
        QuartetAcc o;
#pragma unroll
        for (int a = 0; a < 4; ++a) o.re[a] = o.im[a] = 0.f;
#pragma unroll
        for (int k = 0; k < kQuartetSlots; ++k) {
            if (k >= H.nslot) break;
            flip_mac(o, (H.second >> k) & 1u, p[k], r[k], re[nb[k]], im[nb[k]]);
        }
        full_mac(o, ore, oim, xr, xi);
        for (int k = 0; k < n; ++k) {
            const int2 x = __ldg(H.blk + static_cast<size_t>(k) * H.Q + q);
            const int type = x.x & 7, m = x.x >> 3;
            float4 br[4], bi[4];
            quartet_expand(type, reinterpret_cast<const float2 *>(H.val) + 2 * static_cast<size_t>(x.y), br, bi);
            full_mac(o, br, bi, re[m], im[m]);
        }
        return o;
    }
};

struct QuartetSmem {
    float4 *V;          // slot j: re plane at V + 2 j Q, im plane Q further; slot 0 is the state
    double2 *Hm;        // alpha_j, beta_{j+1}
    double *sc;         // 1 / |w_j|
    double2 *cf;        // combination coefficients
    double *red, *rede;
    ObsTable *obs;
    int *flags;
    size_t bytes;
};

__host__ __device__ inline QuartetSmem quartet_carve(unsigned char *base, int Q, int m, int W)
{
    SmemCarve c{base, 0};
    QuartetSmem s;
    s.V = c.take<float4>(2 * static_cast<size_t>(Q) * m);
    s.Hm = c.take<double2>(m);
    s.sc = c.take<double>(m);
    s.cf = c.take<double2>(m);
    s.red = c.take<double>(2 * W);
    s.rede = c.take<double>(9 * W);
    s.obs = c.take<ObsTable>(1);
    s.flags = c.take<int>(2);
    s.bytes = c.off;
    return s;
}

// Flip, norm and observables of the thread's quartet z, which is written back
// to the state when it flipped.
template <int W, int NO>
__device__ __forceinline__ void quartet_evaluate(const ResidentSystem &S, const QuartetSmem &sm, bool live, int flip,
                                                 double2 (&z)[4], double &val, double &nrm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[NO + 1];
#pragma unroll
    for (int o = 0; o <= NO; ++o) v[o] = 0.0;
    if (live) {
        if (flip) {  // U = PS - PT on the pair
            const double2 b = z[1];
            z[0] = make_double2(-z[0].x, -z[0].y);
            z[1] = make_double2(-z[2].x, -z[2].y);
            z[2] = make_double2(-b.x, -b.y);
            z[3] = make_double2(-z[3].x, -z[3].y);
        }
        pair_observables<NO>(*sm.obs, z, v);
    }
    team_reduce_values<W, NO>(S, sm.rede, v, lane, warp, val, nrm);
}

template <typename TS, int W>
__device__ __forceinline__ void resident_quartet_propagate(const ResidentSystem &S, int t, unsigned char *smem,
                                                           int *__restrict__ status)
{
    const int tid = threadIdx.x, lane = tid & 31, warp = warp_uniform(tid >> 5);
    const int Q = S.D / 4, m = S.m;
    const bool live = tid < Q;
    const QuartetSmem sm = quartet_carve(smem, Q, m, W);
    float4 *Vre = sm.V, *Vim = sm.V + Q;
    QuartetRow H;
    H.load(S.rq, tid, live);
    const TS *in = static_cast<const TS *>(S.psi) + static_cast<size_t>(t) * S.ts;
    size_t row[4];
    {
        const int base = live ? quartet_base(tid, S.s1, S.s2) : 0;
        row[0] = static_cast<size_t>(base) * S.rs;
        row[1] = static_cast<size_t>(base + S.s2) * S.rs;
        row[2] = static_cast<size_t>(base + S.s1) * S.rs;
        row[3] = static_cast<size_t>(base + S.s1 + S.s2) * S.rs;
    }
    double2 z[4];
#pragma unroll
    for (int a = 0; a < 4; ++a) {
        z[a] = live ? ld2(in + row[a]) : make_double2(0.0, 0.0);
        z[a] = make_double2(static_cast<float>(z[a].x), static_cast<float>(z[a].y));
    }
    auto store = [&](int slot, const double2 (&w)[4]) {
        if (!live) return;
        Vre[2 * slot * Q + tid] = make_float4(static_cast<float>(w[0].x), static_cast<float>(w[1].x),
                                              static_cast<float>(w[2].x), static_cast<float>(w[3].x));
        Vim[2 * slot * Q + tid] = make_float4(static_cast<float>(w[0].y), static_cast<float>(w[1].y),
                                              static_cast<float>(w[2].y), static_cast<float>(w[3].y));
    };
    if (warp == 0) fill_observables(S, *sm.obs, lane);
    const int steps = S.ntimes - 1;
    const long long g0 = S.step_offset;
    const bool noisy = S.nz.mode != 0;
    if (tid == 0) sm.flags[0] = noisy && steps > 0 ? noise_bit(S.nz, t, g0, 0, S.pflip[0]) : 0;
    const bool own = tid < S.nobs;  // thread o < nobs keeps observable o's trapezoid
    const size_t ak = static_cast<size_t>(tid) * S.acc_ld + t;
    double acc = 0.0, comp = 0.0, prev = 0.0, val = 0.0, nrm2 = 0.0;
    if (own && S.accumulate) {
        acc = S.acc[ak];
        comp = S.comp[ak];
    }
    bool bad = false;
    Team<W>::sync();
    auto evaluate = [&]() {
        if (S.nobs <= 4) quartet_evaluate<W, 4>(S, sm, live, sm.flags[0], z, val, nrm2);
        else quartet_evaluate<W, 8>(S, sm, live, sm.flags[0], z, val, nrm2);
    };
    evaluate();
    prev = val;
    if (S.traj_values && own) S.traj_values[static_cast<size_t>(t) * S.nobs + tid] = val;
    for (int s = 0; s < steps; ++s) {
        const double dt = S.times ? S.times[s + 1] - S.times[s] : S.dt0;
        const double inv0 = rsqrt(nrm2), beta0 = nrm2 > 0.0 ? nrm2 * inv0 : 0.0;
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
            // three-term recurrence, as resident_lanczos
            store(0, z);
            double sj = inv0, bprev = 0.0;
            double2 vc[4], vp[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                vc[a] = cscale(z[a], sj);
                vp[a] = make_double2(0.0, 0.0);
            }
            if (tid == 0) sm.sc[0] = sj;
            Team<W>::sync();
            int n = m;
            for (int j = 0; j < m; ++j) {
                const float4 *re = Vre + 2 * j * Q, *im = Vim + 2 * j * Q;
                double2 u[4];
                {
                    const float4 xr = re[H.q], xi = im[H.q];
                    const QuartetAcc o = H.apply(S.rq, re, im, xr, xi);
#pragma unroll
                    for (int a = 0; a < 4; ++a) u[a] = make_double2(o.re[a] * sj, o.im[a] * sj);
                }
                double pa = 0.0, pb = 0.0;
                if (live) {
                    pa = fma(vc[0].x, u[0].x, fma(vc[0].y, u[0].y, fma(vc[1].x, u[1].x, vc[1].y * u[1].y)));
                    pb = fma(vc[2].x, u[2].x, fma(vc[2].y, u[2].y, fma(vc[3].x, u[3].x, vc[3].y * u[3].y)));
                }
                const double alpha = Team<W>::sum(pa + pb, sm.red);
                if (j == m - 1) {  // T_m is complete; w_m is never used
                    if (tid == 0) sm.Hm[j] = make_double2(alpha, 0.0);
                    break;
                }
                double pn = 0.0;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    double2 w = make_double2(fma(-bprev, vp[a].x, u[a].x), fma(-bprev, vp[a].y, u[a].y));
                    w = make_double2(fma(-alpha, vc[a].x, w.x), fma(-alpha, vc[a].y, w.y));
                    // the stored (rounded) vector is the one the norm and the next product see
                    u[a] = make_double2(static_cast<float>(w.x), static_cast<float>(w.y));
                    pn += cabs2(u[a]);
                }
                store(j + 1, u);
                const double nn = Team<W>::sum(live ? pn : 0.0, sm.red + W);
                sj = rsqrt(nn);
                const double bn = nn > 0.0 ? nn * sj : 0.0;
                if (tid == 0) {
                    sm.Hm[j] = make_double2(alpha, bn);
                    sm.sc[j + 1] = sj;
                }
                if (__any_sync(0xffffffffu, bn < 1e-14)) { n = j + 1; break; }
                bprev = bn;
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    vp[a] = vc[a];
                    vc[a] = cscale(u[a], sj);
                }
            }
            if (warp == 0) {
                __syncwarp();
                const double d = lane < n ? sm.Hm[lane].x : 0.0;
                const double lo = (lane < n && lane > 0) ? sm.Hm[lane - 1].y : 0.0;
                const double hi = lane + 1 < n ? sm.Hm[lane].y : 0.0;
                double2 c;
                const bool ok = warp_tridiag_expm_e1(n, d, lo, hi, S.kappa, dt, c);
                if (!ok && lane == 0) atomicOr(status, 1);
                if (lane < n) sm.cf[lane] = ok ? cscale(c, beta0 * sm.sc[lane]) : make_double2(0.0, 0.0);
            }
            draw_flip();
            Team<W>::sync();
#pragma unroll
            for (int a = 0; a < 4; ++a) z[a] = make_double2(0.0, 0.0);
            if (live) {
#pragma unroll 2
                for (int j = 0; j < n; ++j) {
                    const double2 c = sm.cf[j];
                    const float4 xr = Vre[2 * j * Q + tid], xi = Vim[2 * j * Q + tid];
                    z[0] = cfma(c, make_double2(xr.x, xi.x), z[0]);
                    z[1] = cfma(c, make_double2(xr.y, xi.y), z[1]);
                    z[2] = cfma(c, make_double2(xr.z, xi.z), z[2]);
                    z[3] = cfma(c, make_double2(xr.w, xi.w), z[3]);
                }
#pragma unroll
                for (int a = 0; a < 4; ++a) z[a] = make_double2(static_cast<float>(z[a].x), static_cast<float>(z[a].y));
            }
        } else {
            draw_flip();
            Team<W>::sync();
        }
        evaluate();
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
    if (live)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            st2(out + row[a], z[a]);
            bad = bad || (steps > 0 && !(isfinite(z[a].x) && isfinite(z[a].y)));  // as resident_propagate
        }
    if (own) {
        S.acc[ak] = acc;
        S.comp[ak] = comp;
        S.prev[ak] = prev;
    }
    if (bad) atomicOr(status, 2);
}

}  // namespace
}  // namespace msgpu
