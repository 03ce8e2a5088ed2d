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

}  // namespace

ResidentShape resident_shape_c128(int D, int m, bool lanczos)
{
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
