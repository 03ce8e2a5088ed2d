// msgpu_arnoldi.h -- interface of the streamed Arnoldi Gram-Schmidt passes
// (msgpu_arnoldi.cuh, msgpu_arnoldi.cu).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

namespace msgpu {

// Second Gram-Schmidt pass below this ratio of |w|^2 after to before (the
// resident and the streamed Arnoldi forms).
constexpr double kReorthRatio2 = 0.3 * 0.3;

struct ArnoldiPairK {
    double2 k[16];  // K4, row-major in the pair index a = 2 a1 + a2
};

// The basis: w_0 at w0, w_j (j >= 1) at w1 + (j - 1) stride.
template <typename T>
struct ArnoldiVectors {
    T *w0, *w1;
    size_t stride;
    int Q, s1, s2, ldm;
    __host__ __device__ T *slot(int j) const { return j == 0 ? w0 : w1 + static_cast<size_t>(j - 1) * stride; }
};

struct ArnoldiScratch {
    int m, QT;          // Krylov dimension, quartets per CTA
    double *scale;      // [m + 1][ldm]; row 0 given
    double2 *part;      // tiles x (m + 1) x ldm
    double2 *coef;      // [m][ldm]
    double *before;     // [ldm]: |W|^2 ahead of the first pass
    int *again;         // [ldm]: second pass wanted
    int *tile_again;    // [ldm / 32]
    int *count;         // [ldm / 32], zero between launches
    double2 *hess;      // [ldm][m][m], column-major
    int *mdim;          // [ldm]; 0 while a trajectory's factorisation goes on
};

// Lays the small arrays of S out in buf (3 (m + 1) ldm double2 of device
// memory) and clears the counters on the stream.
cudaError_t arnoldi_scratch(ArnoldiScratch &S, void *buf, int m, int ldm, cudaStream_t st);

// Quartets per CTA so that the tiles number at most max_tiles (the partials'
// capacity) and a launch a few CTAs an SM.
int arnoldi_quartet_tile(int Q, int ldm, int max_tiles);

// Gram-Schmidt of iteration j: W = w_{j+1} (already G v_j, or formed from
// U = H v_j and K when U is not null) against w_0 .. w_j; launches queued.
int arnoldi_orthogonalise(const ArnoldiVectors<double2> &B, const ArnoldiScratch &S, int j, cudaStream_t st);
int arnoldi_orthogonalise(const ArnoldiVectors<float2> &B, const ArnoldiPairK &K, const float2 *U, const ArnoldiScratch &S,
                          int j, cudaStream_t st);

}  // namespace msgpu
