// msgpu_resident.h -- descriptors of the resident form (msgpu_resident.cuh) and
// its launch table (msgpu_resident.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

namespace msgpu {

// Flip bit for trajectory t at (global step, half): replay bits (layout
// ((step*2+half)*M + t)) or Philox.
struct Noise {
    int mode;                // 0 none, 1 replay bits, 2 philox
    const uint8_t *bits;     // replay
    long long bits_steps;    // number of steps covered by bits
    int M;                   // trajectories in the bit layout
    uint64_t seed;           // philox
    uint32_t traj_offset;    // added to the launch's trajectory index (a trajectory group's first)
    double p_full;           // flip probability for a half step of the current step
};

// Entries of a row of H that a one-row thread of the resident form keeps in registers.
constexpr int kRowRegs = 16;

// H by quartets (msgpu_resident_q.cuh), or null pointers.
struct ResidentQuartets {
    const float4 *own;   // [8][Q]: own block, columns b as re, im of the four rows
    const int2 *slot;    // [nslot][Q]: {neighbour quartet, value offset; the quartet itself and -1 if absent}
    const int2 *blk;     // [left][Q]: blocks without a slot, {neighbour quartet << 3 | type, value offset}
    const int *nblk;     // [Q]: their number
    const float4 *val;   // the quartet form's values
    int Q, nslot;
    unsigned second;     // bit k: slot k acts on the second digit
};

struct ResidentSystem {
    // H (rad/ns): row r has rowptr[r + 1] - rowptr[r] entries at rowptr[r] + k
    // (CSR); with kstride > 0 it has rowcnt[r] entries at r + k * kstride (the
    // padded, column-major ELL copy that a warp of consecutive rows reads
    // coalesced), and with generator set they are those of G = -iH - K
    const int *rowptr;
    const int *rowcnt;
    const int *col;
    const double2 *val;
    const float2 *valf;
    int kstride;
    int kmax;          // longest row
    int generator;
    ResidentQuartets rq;
    // K: CSR (krow != null) or kappa * I
    const int *krow;
    const int *kcol;
    const double2 *kval;
    double kappa;
    int D, M, m;       // dimension, trajectories, Krylov dimension
    int acc_ld;        // stride of acc/comp/prev (>= M)
    int s1, s2;        // electron-pair strides (s1 > s2)
    int nobs;
    const double2 *obs;   // nobs x 16 (row-major 4x4, kernel pair basis)
    const double *rates;  // nobs
    Noise nz;             // flip stream (replay bits indexed by this system's M)
    // state: element (row r, trajectory t) is read at psi[r * rs + t * ts] and
    // written to psi_out at the same place (double2; the batch form: float2,
    // column-major)
    const void *psi;
    void *psi_out;
    size_t rs, ts;
    double *acc, *comp, *prev;  // nobs x M (observable-major)
    double *traj_values;        // (ntimes) x M x nobs, or null
    const double *times;        // ntimes; null: every step is dt0 long
    const double *pflip;        // per step flip probability of a half step (may be null without noise)
    double dt0;
    int ntimes;
    long long step_offset;
    int accumulate;
    int check_start;            // flag a non-finite norm of the initial state
};

struct ResidentWork {
    int sys;
    int traj;
};

// Shared memory that decides whether a trajectory's basis fits one CTA: basis
// and state (D (m + 1) elements), Hessenberg matrix and the scratch of the
// Pade exponential (5 m^2 + m complex).
__host__ __device__ inline size_t resident_bytes(int D, int m, int elem)
{
    size_t b = static_cast<size_t>(elem) * D * (m + 1);
    b = (b + 15) / 16 * 16;
    b += sizeof(double2) * (static_cast<size_t>(m) * m + 4 * static_cast<size_t>(m) * m + m);
    return b;
}

using ResidentFn = void (*)(ResidentSystem, int *);
struct ResidentShape {
    ResidentFn fn;   // grid: one CTA per trajectory
    int warps;       // warps per CTA
    size_t smem;     // dynamic shared memory
};

// Trajectories of many systems in one launch (the batching form; complex64 on a
// complex64 state): system i's are the CTAs from first[i] to first[i + 1].  A
// launch for a single system takes `one` where it is there: with the descriptor in
// shared memory a quartet step at D = 1024 takes 2 % longer than with it in the
// kernel's arguments (512 trajectories, 10 steps 1.23 against 1.20 ms), a row step
// at D = 64 5 % less (0.163 against 0.173 ms).
using ResidentManyFn = void (*)(const ResidentSystem *systems, const int *first, int nsystems, int *status);
struct ResidentManyShape {
    ResidentManyFn fn;
    ResidentFn one;
    int warps;
    size_t smem;
};

// Kernel and launch shape for dimension D, Krylov dimension m and M trajectories:
// complex128 (three-term recurrence or Arnoldi), complex64 (three-term).
ResidentShape resident_shape_c128(int D, int m, int M, bool lanczos);
ResidentShape resident_shape_c64(int D, int m);
// The batching form's; fn null when no shape takes it.
ResidentManyShape resident_shape_many(int D, int m);
// complex64 over quartets (msgpu_resident_q.cu): dimensions it takes, its shape,
// the device bytes of a system's ResidentQuartets and their set-up in buf from
// the quartet form's arrays.
struct QuartetSlots;
bool resident_q_takes(int D);
ResidentShape resident_shape_q(int D, int m);
ResidentManyShape resident_shape_q_many(int D, int m);
size_t resident_q_bytes(int Q, const QuartetSlots &slots);
ResidentQuartets resident_q_build(void *buf, int Q, int s1, int s2, const QuartetSlots &slots, const int *rowptr,
                                  const int2 *blk, const float4 *val, const int *base, cudaStream_t st);

// The same from CSR rows on the device, one CTA a system, for an H whose blocks all
// have a slot (rows of up to kAssembleRow entries, one a column).  buf:
// resident_q_assembled_bytes; the view is that of a found.nslot >= 0.
constexpr int kAssembleRow = 64;
struct QuartetJob {
    const int *rowptr, *col;
    const float2 *val;
    void *buf;
    int D, s1, s2;
};
struct QuartetFound {
    int nslot;  // -1: some block has none
    unsigned second;
};
size_t resident_q_assembled_bytes(int Q);
void resident_q_assemble(const QuartetJob *jobs, int n, QuartetFound *found, cudaStream_t st);
ResidentQuartets resident_q_assembled(void *buf, int Q, const QuartetFound &found);

}  // namespace msgpu
