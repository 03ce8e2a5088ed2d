// msgpu_resident_q.cu -- launch table of the quartet form of the resident kernel.

#include "msgpu_resident_q.cuh"

namespace msgpu {
namespace {

template <int W, typename TS>
__global__ void __launch_bounds__(32 * W, W <= 3 ? 8 / W : W <= 6 ? 2 : 1)
k_resident_q(const __grid_constant__ ResidentSystem S, int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    resident_quartet_propagate<TS, W>(S, blockIdx.x, smem_raw, status);
}

}  // namespace

// Up to D = 128 the row form is as fast and leaves no thread idle; 12 warps (D =
// 1536) is what the registers of one SM hold.
bool resident_q_takes(int D) { return D > 128 && D <= 1536; }

namespace {

template <typename TS>
ResidentShape shape_q(int D, int m)
{
    const int Q = D / 4;
    auto make = [&](auto fn, int w) { return ResidentShape{fn, w, quartet_carve(nullptr, Q, m, w).bytes}; };
    if (Q <= 64) return make(&k_resident_q<2, TS>, 2);
    if (Q <= 96) return make(&k_resident_q<3, TS>, 3);
    if (Q <= 128) return make(&k_resident_q<4, TS>, 4);
    if (Q <= 160) return make(&k_resident_q<5, TS>, 5);
    if (Q <= 192) return make(&k_resident_q<6, TS>, 6);
    if (Q <= 256) return make(&k_resident_q<8, TS>, 8);
    return make(&k_resident_q<12, TS>, 12);
}

}  // namespace

ResidentShape resident_shape_q(int D, int m) { return shape_q<double2>(D, m); }
ResidentShape resident_shape_q_state(int D, int m) { return shape_q<float2>(D, m); }

size_t resident_q_bytes(int Q, const QuartetSlots &slots)
{
    return static_cast<size_t>(Q) * (8 * sizeof(float4) + (slots.n + slots.left) * sizeof(int2) + sizeof(int));
}

ResidentQuartets resident_q_build(void *buf, int Q, int s1, int s2, const QuartetSlots &slots, const int *rowptr,
                                  const int2 *blk, const float4 *val, const int *base, cudaStream_t st)
{
    float4 *own = static_cast<float4 *>(buf);
    int2 *slot = reinterpret_cast<int2 *>(own + 8 * static_cast<size_t>(Q));
    int2 *rest = slot + static_cast<size_t>(slots.n) * Q;
    int *nrest = reinterpret_cast<int *>(rest + static_cast<size_t>(slots.left) * Q);
    k_build_resident_quartets<<<(Q + 63) / 64, 64, 0, st>>>(QuartetC{rowptr, blk, val, base}, Q, s1, s2, slots, own, slot,
                                                            rest, nrest);
    return ResidentQuartets{own, slot, rest, nrest, val, Q, slots.n, slots.second};
}

}  // namespace msgpu
