// msgpu_quartet.h -- host assembly of the quartet-block form of H (QuartetC in
// msgpu_kernels.cuh) from its CSR arrays.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <cmath>
#include <cstring>
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
    std::vector<int> nbr;       // neighbour quartet of each block
    std::vector<float> val;     // complex values by type
    std::vector<double> val64;  // the same in FP64 (want64)
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

inline QuartetSlots quartet_slots(const QuartetForm &f)
{
    const int Q = static_cast<int>(f.base.size());
    struct Seen {
        bool uniform = true, both = false;
        int type = -1;
        int at = -1;  // last quartet with a block at this distance
        long long count = 0;
    };
    std::vector<Seen> seen(2 * static_cast<size_t>(Q));  // by signed distance + Q
    for (int q = 0; q < Q; ++q)
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k) {
            const int d = f.nbr[k] - q, type = f.blk[k].x & 7;
            if (d == 0) continue;
            Seen &s = seen[Q + d], &neg = seen[Q - d];
            s.uniform = s.uniform && type >= 4 && (s.type < 0 || s.type == type);
            s.type = type;
            s.at = q;
            ++s.count;
            if (neg.at == q) s.both = neg.both = true;
        }
    // the most used first, should there be more than fit
    std::vector<std::pair<long long, std::pair<int, bool>>> cand;
    for (int d = 1 - Q; d < Q; ++d) {
        const Seen &s = seen[Q + d], &neg = seen[Q - d];
        const bool pair = s.count && neg.count && !s.both && s.uniform && neg.uniform && s.type == neg.type;
        if (!s.count || !s.uniform || (pair && d < 0)) continue;
        cand.push_back({-(s.count + (pair ? neg.count : 0)), {d, pair}});
    }
    std::sort(cand.begin(), cand.end());
    QuartetSlots out;
    std::vector<char> in(2 * static_cast<size_t>(Q), 0);  // distances with a slot
    in[Q] = 1;                                            // the quartet itself
    for (auto &c : cand) {
        if (out.n == kQuartetSlots) break;
        const int d = c.second.first;
        out.delta[out.n] = d;
        in[Q + d] = 1;
        if (c.second.second) {
            out.shared |= 1u << out.n;
            in[Q - d] = 1;
        }
        if (seen[Q + d].type == 5) out.second |= 1u << out.n;
        ++out.n;
    }
    for (int q = 0; q < Q; ++q) {
        int left = 0;
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k) left += !in[Q + f.nbr[k] - q];
        out.left = std::max(out.left, left);
    }
    return out;
}

// Offsets of value quadruples already stored, by type and values (compared as
// numbers): open addressing, at most half full.
class SharedBlocks {
public:
    SharedBlocks() : at_(64, -1) {}
    // the offset stored for (type, 4 complex values), or -1 after storing `offset`
    int find_or_add(int type, const double (&v)[8], int offset)
    {
        if (2 * keys_.size() >= at_.size()) grow();
        size_t h = slot(type, v);
        for (; at_[h] >= 0; h = (h + 1) & (at_.size() - 1)) {
            const Key &k = keys_[at_[h]];
            if (k.type == type && std::equal(v, v + 8, k.v)) return k.offset;
        }
        at_[h] = static_cast<int>(keys_.size());
        keys_.push_back(Key{{}, type, offset});
        std::copy(v, v + 8, keys_.back().v);
        return -1;
    }

private:
    struct Key {
        double v[8];
        int type, offset;
    };
    std::vector<Key> keys_;
    std::vector<int> at_;
    size_t slot(int type, const double (&v)[8]) const
    {
        // independent products, added up: a chain of them took longer than the rest of a block
        uint64_t h = static_cast<uint64_t>(type) * 0x9E3779B97F4A7C15ull;
        for (int i = 0; i < 8; ++i) {
            const double y = v[i] + 0.0;  // -0 as 0
            uint64_t b;
            std::memcpy(&b, &y, sizeof b);
            h += (b ^ (b >> 29)) * (0x9E3779B97F4A7C15ull + 0x5851F42D4C957F2Eull * static_cast<uint64_t>(i));
        }
        h ^= h >> 32;
        return static_cast<size_t>(h) & (at_.size() - 1);
    }
    void grow()
    {
        at_.assign(2 * at_.size(), -1);
        for (size_t i = 0; i < keys_.size(); ++i) {
            size_t h = slot(keys_[i].type, keys_[i].v);
            while (at_[h] >= 0) h = (h + 1) & (at_.size() - 1);
            at_[h] = static_cast<int>(i);
        }
    }
};

// Storage order (4 a + b) of each block type, see QuartetC.
constexpr int kBlockOrder[6][16] = {{0, 1, 2, 3, 4, 5, 6, 7, 8, 9, 10, 11, 12, 13, 14, 15},
                                    {0, 2, 8, 10, 5, 7, 13, 15},
                                    {0, 1, 4, 5, 10, 11, 14, 15},
                                    {0, 5, 10, 15},
                                    {0, 2, 8, 10},
                                    {0, 1, 4, 5}};
constexpr int kBlockCount[6] = {16, 8, 8, 4, 4, 4};

// Type of the block B (4 x 4 complex, row-major; bit x of nz: entry x is not zero).
inline int block_type(const double *B, unsigned nz)
{
    // entries that couple different second (first) digits of the pair
    constexpr unsigned kSecond = 0x5a5au, kFirst = 0x33ccu;
    const bool e1only = !(nz & kSecond), e2only = !(nz & kFirst);
    if (e1only && e2only) return 3;
    if (!e1only && !e2only) return 0;
    double bmax = 0.0;
    for (int k = 0; k < 8; ++k) {
        const int x = kBlockOrder[e1only ? 1 : 2][k];
        bmax = std::max(bmax, std::abs(B[2 * x]) + std::abs(B[2 * x + 1]));
    }
    auto same = [&](int x, int y) {
        return std::abs(B[2 * x] - B[2 * y]) + std::abs(B[2 * x + 1] - B[2 * y + 1]) <= 1e-13 * bmax;
    };
    // acts on one digit; A (x) I when both halves of the other digit agree
    if (e1only) return same(0, 5) && same(2, 7) && same(8, 13) && same(10, 15) ? 4 : 1;
    return same(0, 10) && same(1, 11) && same(4, 14) && same(5, 15) ? 5 : 2;
}

// One pass over the CSR arrays: a column's quartet and its place in it come from a
// table, a quartet's blocks from a table by neighbour, and a flip block that repeats
// the last one at its distance takes that one's type and values.  Host time at D = 2048
// and 16384: 0.62 and 6.4 ms with searches and divisions per entry, 0.32 and 3.6 so
// (of which 2.7 for the entries).
inline QuartetForm quartet_form(int D, int s1, int s2, const int *h_rowptr, const int *h_col, const double *h_val,
                                bool want_src, bool want64 = true)
{
    const int Q = D / 4, nnz = h_rowptr[D];
    const int off[4] = {0, s2, s1, s1 + s2};
    QuartetForm f;
    f.rowptr.assign(Q + 1, 0);
    f.base.resize(Q);
    f.blk.reserve(nnz / 6 + Q);
    f.nbr.reserve(nnz / 6 + Q);
    f.val.reserve(2 * static_cast<size_t>(nnz));  // only what is used of it is ever touched
    if (want64) f.val64.reserve(2 * static_cast<size_t>(nnz));
    if (want_src) f.src.reserve(nnz);
    std::vector<int> place(D);  // 4 (quartet of a row) + its pair index
    for (int q = 0; q < Q; ++q) {
        const int lo = q % s2, mid = (q / s2) % (s1 / (2 * s2)), hi = q / (s1 / 2);
        f.base[q] = hi * (2 * s1) + mid * (2 * s2) + lo;
        for (int a = 0; a < 4; ++a) place[f.base[q] + off[a]] = 4 * q + a;
    }
    struct Block {
        double z[32];  // 16 complex, row-major in the pair index
        int src[16];   // CSR index of each entry
        unsigned nz;   // bit x: entry x is not zero
    };
    std::vector<Block> blocks;
    std::vector<int> order;                     // neighbour quartets of this quartet's blocks
    std::vector<int> owner(Q, -1), slot(Q, 0);  // quartet that met a neighbour last, and its block there
    SharedBlocks shared;
    // the last block at each signed distance (+ Q): a nucleus' flip block is the same
    // in every quartet with the same state of it
    struct Held {
        double z[32];
        int type, at;
    };
    std::vector<Held> held;
    std::vector<int> held_at(2 * static_cast<size_t>(Q), -1);
    // plain pointers: the loop over the entries stores through several of them
    const int *where = place.data();
    int *own_q = owner.data(), *own_at = slot.data();
    for (int q = 0; q < Q; ++q) {
        order.clear();
        Block *blk = blocks.data();
        for (int a = 0; a < 4; ++a) {
            const int r = f.base[q] + off[a], end = h_rowptr[r + 1];
            for (int k = h_rowptr[r]; k < end; ++k) {
                const int at = where[h_col[k]], nq = at >> 2, e = a * 4 + (at & 3);
                if (own_q[nq] != q) {
                    own_q[nq] = q;
                    own_at[nq] = static_cast<int>(order.size());
                    order.push_back(nq);
                    if (blocks.size() < order.size()) blocks.emplace_back();
                    blk = blocks.data();
                    Block &z = blk[order.size() - 1];
                    std::memset(z.z, 0, sizeof z.z);
                    z.nz = 0;
                    if (want_src) std::fill(z.src, z.src + 16, -1);
                }
                Block &z = blk[own_at[nq]];
                if (want_src) z.src[e] = k;
                const double re = h_val[2 * static_cast<size_t>(k)], im = h_val[2 * static_cast<size_t>(k) + 1];
                z.z[2 * e] += re;
                z.z[2 * e + 1] += im;
                z.nz |= static_cast<unsigned>((re != 0.0) | (im != 0.0)) << e;
            }
        }
        // by neighbour, the quartet's own block last (the SpMM reuses its gathered
        // rows for the alpha partial)
        std::sort(order.begin(), order.end());
        if (own_q[q] == q) {
            const auto own = std::lower_bound(order.begin(), order.end(), q);
            std::rotate(own, own + 1, order.end());
        }
        for (int nq : order) {
            const Block &z = blk[own_at[nq]];
            const double *B = z.z;
            int &known = held_at[Q + nq - q];
            const bool again = known >= 0 && std::memcmp(held[known].z, B, sizeof z.z) == 0;
            const int type = again ? held[known].type : block_type(B, z.nz);
            const int head = (f.base[nq] << 3) | type, at = static_cast<int>(f.val.size() / 4);
            f.nbr.push_back(nq);
            // blocks A (x) I with the same four values share them: a nucleus' flip
            // block takes two values over all quartets, so they stay in L1 (D =
            // 16384, 1024 trajectories complex64: 101.6 to 99.2 ms for 20 steps).  With
            // Hamiltonian terms the values here are those of one combination, which can
            // agree where the terms differ, and every slot is written from its own CSR
            // entry when the coefficients change: each block keeps its own.
            if (type >= 4 && !want_src) {
                if (again) {
                    f.blk.push_back({head, held[known].at});
                    continue;
                }
                double v[8];
                for (int k = 0; k < 4; ++k) {
                    v[2 * k] = B[2 * kBlockOrder[type][k]];
                    v[2 * k + 1] = B[2 * kBlockOrder[type][k] + 1];
                }
                const int first = shared.find_or_add(type, v, at);
                if (known < 0) {
                    known = static_cast<int>(held.size());
                    held.emplace_back();
                }
                std::memcpy(held[known].z, B, sizeof z.z);
                held[known].type = type;
                held[known].at = first >= 0 ? first : at;
                if (first >= 0) {
                    f.blk.push_back({head, first});
                    continue;
                }
            }
            f.blk.push_back({head, at});
            const int n = kBlockCount[type];
            const size_t end = f.val.size();
            f.val.resize(end + 2 * n);
            float *v32 = f.val.data() + end;
            for (int k = 0; k < n; ++k) {
                const int x = kBlockOrder[type][k];
                v32[2 * k] = static_cast<float>(B[2 * x]);
                v32[2 * k + 1] = static_cast<float>(B[2 * x + 1]);
                if (want_src) f.src.push_back(z.src[x]);
            }
            if (!want64) continue;
            f.val64.resize(end + 2 * n);
            double *v64 = f.val64.data() + end;
            for (int k = 0; k < n; ++k) {
                const int x = kBlockOrder[type][k];
                v64[2 * k] = B[2 * x];
                v64[2 * k + 1] = B[2 * x + 1];
            }
        }
        f.rowptr[q + 1] = static_cast<int>(f.blk.size());
    }
    return f;
}

}  // namespace msgpu
