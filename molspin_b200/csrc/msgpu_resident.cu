// msgpu_resident.cu -- launch table of the resident form.

#include "msgpu_resident.cuh"

namespace msgpu {
namespace {

template <typename T, bool kLanczos>
ResidentShape resident_shape(int D, int m)
{
    auto make = [&](auto fn, int w) {
        return ResidentShape{fn, w, resident_carve<T, kLanczos>(nullptr, D, m, w).bytes};
    };
    // One row a thread up to D = 256 keeps the thread's row of H in registers
    // (a step of 256 complex128 trajectories at D = 64: 14.1 us with 2 warps,
    // 15.3 with 4, 25 with one warp and two rows a thread, which is bound by its
    // own instruction count).  Beyond, two to four rows a thread.
    if (D <= 32) return make(&k_resident<T, 1, 1, kLanczos>, 1);
    if (D <= 64) return make(&k_resident<T, 2, 1, kLanczos>, 2);
    if (D <= 128) return make(&k_resident<T, 4, 1, kLanczos>, 4);
    if (D <= 256) return make(&k_resident<T, 8, 1, kLanczos>, 8);
    if (D <= 512) return make(&k_resident<T, 8, 2, kLanczos>, 8);
    if (D <= 1024) return make(&k_resident<T, 16, 2, kLanczos>, 16);
    if (D <= 2048) return make(&k_resident<T, 16, 4, kLanczos>, 16);
    return make(&k_resident<T, 32, 16, kLanczos>, 32);
}

// Many trajectories at a Krylov dimension of a few: the work outside the chain of
// products (values, exponential, barriers) counts, so half the warps with two rows a
// thread, none of them in registers, and 16 warps an SM instead of 8.
template <bool kLanczos>
ResidentShape resident_shape_short(int D, int m)
{
    auto make = [&](auto fn, int w) {
        return ResidentShape{fn, w, resident_carve<double2, kLanczos>(nullptr, D, m, w).bytes};
    };
    if (D <= 64) return make(&k_resident<double2, 1, 2, kLanczos>, 1);
    if (D <= 128) return make(&k_resident<double2, 2, 2, kLanczos>, 2);
    return make(&k_resident<double2, 4, 2, kLanczos>, 4);
}

}  // namespace

// The short shape from more trajectories than the other holds at once (8 warps an SM)
// and, with D in 33 .. 256, up to m = 6 (Arnoldi) or 2 (three-term).  B200, 16384
// trajectories, 10 steps, ms, short / other shape: Arnoldi D = 64 m = 3 1.65 / 3.11,
// m = 6 2.87 / 4.49, m = 8 4.21 / 5.63 (2048 trajectories 0.88 / 0.86); D = 128 m = 2
// 2.16 / 4.21; D = 256 m = 1 2.72 / 5.22, m = 8 23.4 / 23.6; three-term D = 256 m = 1
// 2.12 / 3.22.  256 trajectories, one wave of the other: Arnoldi D = 64 m = 3 0.23 / 0.16.
ResidentShape resident_shape_c128(int D, int m, int M, bool lanczos)
{
    const int warps = D <= 64 ? 2 : D <= 128 ? 4 : 8;
    if (D > 32 && D <= 256 && m <= (lanczos ? 2 : 6) && M > 148 * (8 / warps))
        return lanczos ? resident_shape_short<true>(D, m) : resident_shape_short<false>(D, m);
    return lanczos ? resident_shape<double2, true>(D, m) : resident_shape<double2, false>(D, m);
}

ResidentShape resident_shape_c64(int D, int m) { return resident_shape<float2, true>(D, m); }

ResidentManyShape resident_shape_many(int D, int m)
{
    auto make = [&](ResidentManyFn fn, int w) {
        return ResidentManyShape{fn, nullptr, w, resident_carve<float2, true>(nullptr, D, m, w).bytes};
    };
    if (D <= 32) return make(&k_resident_many<1>, 1);
    if (D <= 64) return make(&k_resident_many<2>, 2);
    if (D <= 128) return make(&k_resident_many<4>, 4);
    return make(nullptr, 0);
}

}  // namespace msgpu
