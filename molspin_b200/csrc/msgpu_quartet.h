// msgpu_quartet.h -- host assembly of the quartet-block form of H (QuartetC in
// msgpu_kernels.cuh) from its CSR arrays.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <map>
#include <vector>

namespace msgpu {

// Weight of Hamiltonian term t (0 to 15) in the combination that fixes the sparsity
// and block structure for every combination of the terms: 1 + the fraction of the
// square root of a prime.  Square roots of distinct primes are independent of one
// another and of 1 over the rationals, so values that agree or cancel here agree or
// cancel term by term.  (Multiples of one irrational number do not do: they are an
// arithmetic progression, up to whole numbers.)
inline double term_weight(int t)
{
    static const int primes[16] = {2, 3, 5, 7, 11, 13, 17, 19, 23, 29, 31, 37, 41, 43, 47, 53};
    const double root = std::sqrt(static_cast<double>(primes[t]));
    return 1.0 + root - std::floor(root);
}

struct QuartetForm {
    std::vector<int> rowptr;    // Q + 1
    std::vector<int2> blk;      // {neighbour base row << 3 | type, value offset in float4}
    std::vector<float> val;     // complex values by type
    std::vector<double> val64;  // the same in FP64
    std::vector<int> base;      // first row of each quartet
    std::vector<int> src;       // CSR index per value slot (want_src)
};

// Slots of the resident form: neighbour blocks by their distance in quartets,
// d and -d in one slot when no quartet has both (a spin-1/2 nucleus; a spin-1
// nucleus takes two).  Only distances whose blocks are all of type 4, or all of
// type 5, get one; `left` is the most blocks of a quartet without a slot.
constexpr int kQuartetSlots = 8;
struct QuartetSlots {
    int n = 0, left = 0;
    int delta[kQuartetSlots] = {0};    // distance of slot k
    unsigned shared = 0, second = 0;   // bit k: -delta too; type 5
};

inline QuartetSlots quartet_slots(const QuartetForm &f, int s1, int s2)
{
    const int Q = static_cast<int>(f.base.size());
    auto index = [&](int cb) { return (cb / (2 * s1)) * (s1 / 2) + ((cb / (2 * s2)) % (s1 / (2 * s2))) * s2 + cb % s2; };
    struct Seen {
        bool uniform = true, both = false;
        int type = -1;
        long long count = 0;
    };
    std::map<int, Seen> seen;  // by signed distance
    for (int q = 0; q < Q; ++q)
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k) {
            const int cb = f.blk[k].x >> 3, type = f.blk[k].x & 7;
            if (cb == f.base[q]) continue;
            Seen &s = seen[index(cb) - q];
            s.uniform = s.uniform && type >= 4 && (s.type < 0 || s.type == type);
            s.type = type;
            ++s.count;
        }
    for (int q = 0; q < Q; ++q)  // quartets with both d and -d
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k)
            for (int l = k + 1; l < f.rowptr[q + 1]; ++l) {
                const int d = index(f.blk[k].x >> 3) - q, e = index(f.blk[l].x >> 3) - q;
                if (d != 0 && d == -e) seen[d].both = seen[e].both = true;
            }
    // the most used first, should there be more than fit
    std::vector<std::pair<long long, std::pair<int, bool>>> cand;
    for (auto &x : seen) {
        auto neg = seen.find(-x.first);
        const bool pair = neg != seen.end() && !x.second.both && x.second.uniform && neg->second.uniform &&
                          x.second.type == neg->second.type;
        if (!x.second.uniform || (pair && x.first < 0)) continue;
        cand.push_back({-(x.second.count + (pair ? neg->second.count : 0)), {x.first, pair}});
    }
    std::sort(cand.begin(), cand.end());
    QuartetSlots out;
    for (auto &c : cand) {
        if (out.n == kQuartetSlots) break;
        out.delta[out.n] = c.second.first;
        if (c.second.second) out.shared |= 1u << out.n;
        if (seen[c.second.first].type == 5) out.second |= 1u << out.n;
        ++out.n;
    }
    for (int q = 0; q < Q; ++q) {
        int left = 0;
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k) {
            const int d = index(f.blk[k].x >> 3) - q;
            bool in = d == 0;
            for (int i = 0; i < out.n; ++i) in = in || d == out.delta[i] || (((out.shared >> i) & 1u) && d == -out.delta[i]);
            if (!in) ++left;
        }
        out.left = std::max(out.left, left);
    }
    return out;
}

inline QuartetForm quartet_form(int D, int s1, int s2, const int *h_rowptr, const int *h_col, const double *h_val,
                                bool want_src)
{
    const int Q = D / 4, nnz = h_rowptr[D];
    const int off[4] = {0, s2, s1, s1 + s2};
    QuartetForm f;
    std::vector<int> &rowptr = f.rowptr, &base = f.base, &src = f.src;
    std::vector<int2> &blks = f.blk;
    std::vector<float> &vals = f.val;
    std::vector<double> &vals64 = f.val64;
    rowptr.assign(Q + 1, 0);
    base.resize(Q);
    blks.reserve(nnz / 6 + Q);
    vals.reserve(2 * static_cast<size_t>(nnz));
    vals64.reserve(2 * static_cast<size_t>(nnz));
    if (want_src) src.reserve(nnz);
    struct Block {
        int base;
        double z[32];  // 16 complex, row-major in the pair index
        int src[16];   // CSR index of each entry
    };
    std::vector<Block> blocks;
    std::vector<int> ord;
    std::map<std::array<double, 9>, int> shared;  // values of a block of type 4 or 5 -> their offset
    // storage order (4 a + b) of each block type, see QuartetC
    static const int kOrder[6][16] = {{0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15},
                                      {0, 2, 8, 10, 5, 7, 13, 15},
                                      {0, 1, 4, 5, 10, 11, 14, 15},
                                      {0, 5, 10, 15},
                                      {0, 2, 8, 10},
                                      {0, 1, 4, 5}};
    static const int kCount[6] = {16, 8, 8, 4, 4, 4};
    for (int q = 0; q < Q; ++q) {
        const int lo = q % s2, mid = (q / s2) % (s1 / (2 * s2)), hi = q / (s1 / 2);
        const int b = hi * (2 * s1) + mid * (2 * s2) + lo;
        base[q] = b;
        size_t nblk = 0;
        for (int a = 0; a < 4; ++a) {
            const int r = b + off[a];
            size_t at = 0;  // rows meet their neighbours in a similar order
            for (int k = h_rowptr[r]; k < h_rowptr[r + 1]; ++k) {
                const int col = h_col[k];
                const int a1 = (col / s1) & 1, a2 = (col / s2) & 1;
                const int cb = col - a1 * s1 - a2 * s2, bi = 2 * a1 + a2;
                size_t slot = at;
                while (slot < nblk && blocks[slot].base != cb) ++slot;
                if (slot == nblk) {
                    slot = 0;
                    while (slot < at && blocks[slot].base != cb) ++slot;
                    if (slot == at) slot = nblk;
                }
                if (slot == nblk) {
                    if (blocks.size() == nblk) blocks.emplace_back();
                    Block &z = blocks[nblk++];
                    z.base = cb;
                    std::fill(z.z, z.z + 32, 0.0);
                    std::fill(z.src, z.src + 16, -1);
                }
                at = slot;
                Block &z = blocks[slot];
                z.src[a * 4 + bi] = k;
                z.z[2 * (a * 4 + bi)] += h_val[2 * static_cast<size_t>(k)];
                z.z[2 * (a * 4 + bi) + 1] += h_val[2 * static_cast<size_t>(k) + 1];
            }
        }
        // by neighbour base, the quartet's own block last (the SpMM reuses its
        // gathered rows for the alpha partial)
        ord.resize(nblk);
        for (size_t i = 0; i < nblk; ++i) ord[i] = static_cast<int>(i);
        std::sort(ord.begin(), ord.end(), [&](int x, int y) {
            const bool ox = blocks[x].base == b, oy = blocks[y].base == b;
            return ox != oy ? oy : blocks[x].base < blocks[y].base;
        });
        for (int oi : ord) {
            const Block &blk = blocks[oi];
            const double *B = blk.z;
            double bmax = 0.0;
            bool e1only = true, e2only = true;
            for (int a = 0; a < 4; ++a)
                for (int bb = 0; bb < 4; ++bb) {
                    const double re = B[2 * (a * 4 + bb)], im = B[2 * (a * 4 + bb) + 1];
                    if (re == 0.0 && im == 0.0) continue;
                    bmax = std::max(bmax, std::abs(re) + std::abs(im));
                    if ((a & 1) != (bb & 1)) e1only = false;  // couples different second digits
                    if ((a & 2) != (bb & 2)) e2only = false;  // couples different first digits
                }
            auto same = [&](int x, int y) {
                return std::abs(B[2 * x] - B[2 * y]) + std::abs(B[2 * x + 1] - B[2 * y + 1]) <= 1e-13 * bmax;
            };
            int type = 0;
            if (e1only && e2only) type = 3;
            // acts on one digit; A (x) I when both halves of the other digit agree
            else if (e1only) type = same(0, 5) && same(2, 7) && same(8, 13) && same(10, 15) ? 4 : 1;
            else if (e2only) type = same(0, 10) && same(1, 11) && same(4, 14) && same(5, 15) ? 5 : 2;
            // blocks A (x) I with the same four values share them: a nucleus' flip
            // block takes two values over all quartets, so they stay in L1 (D =
            // 16384, 1024 trajectories complex64: 101.6 to 99.2 ms for 20 steps).  With
            // Hamiltonian terms the values here are those of one combination, which can
            // agree where the terms differ, and every slot is written from its own CSR
            // entry when the coefficients change: each block keeps its own.
            if (type >= 4 && !want_src) {
                std::array<double, 9> key;
                key[8] = type;
                for (int k = 0; k < 4; ++k) {
                    key[2 * k] = B[2 * kOrder[type][k]];
                    key[2 * k + 1] = B[2 * kOrder[type][k] + 1];
                }
                const auto at = shared.emplace(key, static_cast<int>(vals.size() / 4));
                if (!at.second) {
                    blks.push_back({(blk.base << 3) | type, at.first->second});
                    continue;
                }
            }
            blks.push_back({(blk.base << 3) | type, static_cast<int>(vals.size() / 4)});
            for (int k = 0; k < kCount[type]; ++k) {
                const int x = kOrder[type][k];
                vals.push_back(static_cast<float>(B[2 * x]));
                vals.push_back(static_cast<float>(B[2 * x + 1]));
                vals64.push_back(B[2 * x]);
                vals64.push_back(B[2 * x + 1]);
                if (want_src) src.push_back(blk.src[x]);
            }
        }
        rowptr[q + 1] = static_cast<int>(blks.size());
    }
    return f;
}

}  // namespace msgpu
