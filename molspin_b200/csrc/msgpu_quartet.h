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

struct QuartetForm {
    std::vector<int> rowptr;    // Q + 1
    std::vector<int2> blk;      // {neighbour base row << 3 | type, value offset in float4}
    std::vector<float> val;     // complex values by type
    std::vector<double> val64;  // the same in FP64
    std::vector<int> base;      // first row of each quartet
    std::vector<int> src;       // CSR index per value slot (want_src)
    int neighbours = 0;         // most blocks of a quartet beside its own
};

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
            // 16384, 1024 trajectories complex64: 101.6 to 99.2 ms for 20 steps)
            if (type >= 4) {
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
        bool own = false;
        for (size_t i = 0; i < nblk; ++i) own = own || blocks[i].base == b;
        f.neighbours = std::max(f.neighbours, static_cast<int>(nblk) - (own ? 1 : 0));
    }
    return f;
}

}  // namespace msgpu
