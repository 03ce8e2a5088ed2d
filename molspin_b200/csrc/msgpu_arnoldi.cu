// msgpu_arnoldi.cu -- launches of the streamed Arnoldi Gram-Schmidt passes.

#include "msgpu_arnoldi.cuh"

#include <algorithm>
#include <utility>

namespace msgpu {
namespace {

// A kernel for every four basis vectors more: the accumulators are registers.
template <typename T, bool kPairK>
struct Passes {
    using Dots = void (*)(ArnoldiVectors<T>, ArnoldiPairK, const T *, ArnoldiScratch, int, int);
    using Update = void (*)(ArnoldiVectors<T>, ArnoldiScratch, int, int);
    template <int... I>
    static Dots dots(int j, std::integer_sequence<int, I...>)
    {
        static constexpr Dots table[] = {&k_arn_dots<T, 4 * (I + 1), kPairK>...};
        return table[j / 4];
    }
    template <int... I>
    static Update update(int j, std::integer_sequence<int, I...>)
    {
        static constexpr Update table[] = {&k_arn_update<T, 4 * (I + 1)>...};
        return table[j / 4];
    }
};
constexpr auto kBatches = std::make_integer_sequence<int, kMaxKrylov / 4>{};

template <typename T, bool kPairK>
int orthogonalise(const ArnoldiVectors<T> &B, const ArnoldiPairK &K, const T *U, const ArnoldiScratch &S, int j,
                  cudaStream_t st)
{
    const dim3 grid((B.Q + S.QT - 1) / S.QT, B.ldm / 32);
    launch_dependent(Passes<T, kPairK>::dots(j, kBatches), grid, kThreads, 0, st, B, K, U, S, j, 0);
    if (j == S.m - 1) return 1;  // w_m is never used
    const auto update = Passes<T, kPairK>::update(j, kBatches);
    launch_dependent(update, grid, kThreads, 0, st, B, S, j, 0);
    launch_dependent(Passes<T, false>::dots(j, kBatches), grid, kThreads, 0, st, B, K, nullptr, S, j, 1);
    launch_dependent(update, grid, kThreads, 0, st, B, S, j, 1);
    return 4;
}

}  // namespace

cudaError_t arnoldi_scratch(ArnoldiScratch &S, void *buf, int m, int ldm, cudaStream_t st)
{
    S.m = m;
    S.coef = static_cast<double2 *>(buf);
    S.before = reinterpret_cast<double *>(S.coef + static_cast<size_t>(m) * ldm);
    S.again = reinterpret_cast<int *>(S.before + ldm);
    S.tile_again = S.again + ldm;
    S.count = S.tile_again + ldm / 32;
    return cudaMemsetAsync(S.count, 0, ldm / 32 * sizeof(int), st);
}

int arnoldi_quartet_tile(int Q, int ldm, int max_tiles)
{
    // about two CTAs an SM (the registers of the larger kernels allow two) over all
    // trajectory tiles, whole rounds of the CTA's warps
    const int want = std::max(1, 2 * 148 / (ldm / 32));
    const int tiles = std::max(1, std::min(want, max_tiles));
    const int qt = (Q + tiles - 1) / tiles;
    return (qt + kWarps - 1) / kWarps * kWarps;
}

int arnoldi_orthogonalise(const ArnoldiVectors<double2> &B, const ArnoldiScratch &S, int j, cudaStream_t st)
{
    return orthogonalise<double2, false>(B, ArnoldiPairK{}, nullptr, S, j, st);
}

int arnoldi_orthogonalise(const ArnoldiVectors<float2> &B, const ArnoldiPairK &K, const float2 *U, const ArnoldiScratch &S,
                          int j, cudaStream_t st)
{
    return orthogonalise<float2, true>(B, K, U, S, j, st);
}

}  // namespace msgpu
