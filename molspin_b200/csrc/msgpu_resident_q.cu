// msgpu_resident_q.cu -- launch table of the quartet form of the resident kernel.

#include "msgpu_resident_q.cuh"

#include <type_traits>

namespace msgpu {
namespace {

constexpr int quartet_min_ctas(int W) { return W <= 3 ? 8 / W : W <= 6 ? 2 : 1; }

template <int W, typename TS>
__global__ void __launch_bounds__(32 * W, quartet_min_ctas(W))
k_resident_q(const __grid_constant__ ResidentSystem S, int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    resident_quartet_propagate<TS, W>(S, blockIdx.x, smem_raw, status);
}

// The trajectories of many systems, as k_resident_many.
template <int W>
__global__ void __launch_bounds__(32 * W, quartet_min_ctas(W))
k_resident_q_many(const ResidentSystem *__restrict__ systems, const int *__restrict__ first, int nsystems,
                  int *__restrict__ status)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ ResidentSystem S;
    const int i = system_of(first, nsystems, blockIdx.x);
    load_system(&S, systems + i);
    resident_quartet_propagate<float2, W>(S, blockIdx.x - __ldg(first + i), smem_raw, status);
}

}  // namespace

// Up to D = 128 the row form is as fast and leaves no thread idle; 12 warps (D =
// 1536) is what the registers of one SM hold.  Blocks without a slot are read and
// expanded again on every product: with a dense H, where all of them are, 3 steps of
// 512 trajectories take 6.6 ms at D = 256 and 52 at D = 1024 (23.7 and 161 with a warp
// per trajectory over CSR rows).
bool resident_q_takes(int D) { return D > 128 && D <= kAssembleD; }

namespace {

// Warps a CTA: a thread per quartet.
template <typename Make>
auto shape_q(int D, int m, Make make_for)
{
    const int Q = D / 4;
    auto make = [&](auto w) { return make_for(w, quartet_carve(nullptr, Q, m, decltype(w)::value).bytes); };
    if (Q <= 64) return make(std::integral_constant<int, 2>{});
    if (Q <= 96) return make(std::integral_constant<int, 3>{});
    if (Q <= 128) return make(std::integral_constant<int, 4>{});
    if (Q <= 160) return make(std::integral_constant<int, 5>{});
    if (Q <= 192) return make(std::integral_constant<int, 6>{});
    if (Q <= 256) return make(std::integral_constant<int, 8>{});
    return make(std::integral_constant<int, 12>{});
}

}  // namespace

ResidentShape resident_shape_q(int D, int m)
{
    return shape_q(D, m, [](auto w, size_t smem) {
        constexpr int W = decltype(w)::value;
        return ResidentShape{&k_resident_q<W, double2>, W, smem};
    });
}

ResidentManyShape resident_shape_q_many(int D, int m)
{
    return shape_q(D, m, [](auto w, size_t smem) {
        constexpr int W = decltype(w)::value;
        return ResidentManyShape{&k_resident_q_many<W>, &k_resident_q<W, float2>, W, smem};
    });
}

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

size_t resident_q_assembled_bytes(int Q)
{
    return static_cast<size_t>(Q) * ((8 + 2 * kQuartetSlots) * sizeof(float4) + kQuartetSlots * sizeof(int2) + sizeof(int));
}

void resident_q_assemble(const QuartetJob *jobs, int n, QuartetFound *found, cudaStream_t st)
{
    k_assemble_quartets<<<n, kAssembleThreads, 0, st>>>(jobs, found);
}

ResidentQuartets resident_q_assembled(void *buf, int Q, const QuartetFound &found)
{
    const AssembledQuartets B(buf, Q);
    return ResidentQuartets{B.own, B.slot, nullptr, B.nblk, B.val, Q, found.nslot, found.second};
}

}  // namespace msgpu
