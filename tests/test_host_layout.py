"""Host rules of the device layouts, compiled from their headers."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, source):
    """Compiles and runs a C++ program against the library's headers; returns its output."""
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-I", os.path.join(ROOT, "molspin_b200", "csrc"),
                    "-I", "/usr/local/cuda/include", str(src), "-o", str(exe)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout.strip()


PARTIALS = r"""
#include <stdio.h>
#include "msgpu_tiles.h"
using namespace msgpu;
int main()
{
    long bad = 0, shapes = 0;
    const int dims[] = {4, 16, 64, 1024, 2048, 2304, 4096, 6144, 8192, 9216, 12288, 16384, 18432, 24576, 32768, 65536, 131072};
    for (int D : dims)
        for (int m = 1; m <= 32; ++m)
            for (int ldm = 64; ldm <= 2048; ldm += 64)
                for (int G = 1; G <= 4; G *= 2) {
                    if (G > 1 && ldm % (128 * G)) continue;
                    const int R = pick_rows_per_tile(D), nt = (D + R - 1) / R, Q = D / 4;
                    const size_t rows = partial_rows_d(nt, m);
                    const int QT = quartet_tile_d(Q, ldm / G, rows);
                    const size_t nqt = (Q + QT - 1) / QT;
                    ++shapes;
                    // the update leaves one row a row tile
                    if (nqt > rows || static_cast<size_t>(nt) > rows || QT % 8) ++bad;
                }
    printf("%s %ld\n", shapes > 10000 ? "ok" : "few", bad);
}
"""


def test_three_term_partial_sums_fit_their_buffer(tmp_path):
    assert _run(tmp_path, PARTIALS) == "ok 0"


# Two electrons (strides 8 and 4) and nuclei a (stride 2) and b (stride 1), each flipped with a value
# of its own on the first electron: v and w.  Prints the slots the two nuclei's blocks take.
QUARTETS = r"""
#include <stdio.h>
#include "msgpu_quartet.h"
using namespace msgpu;
int main()
{
    std::vector<int> rowptr(1, 0), col;
    std::vector<double> val;
    for (int r = 0; r < 16; ++r) {  // flip-flops of the first electron (digit 8) with a nucleus (digit 2 or 1)
        for (int n = 2; n >= 1; --n)
            if (((r >> 3) & 1) != ((r & n) ? 1 : 0)) {
                col.push_back(r ^ 8 ^ n);
                val.push_back(0.5);
                val.push_back(0.0);
            }
        rowptr.push_back(static_cast<int>(col.size()));
    }
    for (bool terms : {false, true}) {
        const QuartetForm f = quartet_form(16, 8, 4, rowptr.data(), col.data(), val.data(), terms);
        // a slot's CSR entries belong to one block: as many slots as blocks of terms
        size_t own = 0;
        for (size_t k = 0; k < f.blk.size(); ++k)
            for (size_t l = 0; l < k; ++l) own += f.blk[k].y == f.blk[l].y;
        printf("%zu blocks, %s, %zu sources; ", f.blk.size(), own ? "shared" : "apart", f.src.size());
    }
    return 0;
}
"""


def test_blocks_of_hamiltonian_terms_keep_their_own_values(tmp_path):
    # equal values in one combination of the terms say nothing about the others
    assert _run(tmp_path, QUARTETS) == "8 blocks, shared, 0 sources; 8 blocks, apart, 32 sources;"


WEIGHTS = r"""
#include <stdio.h>
#include <math.h>
#include "msgpu_quartet.h"
using namespace msgpu;
int main()
{
    // whole-number relations a w_i + b w_j + c w_k + d w_l = 0, |a| .. |d| <= 2
    double least = 1.0;
    for (int i = 0; i < 16; ++i)
        for (int j = i + 1; j < 16; ++j)
            for (int k = j + 1; k < 16; ++k)
                for (int l = k + 1; l < 16; ++l)
                    for (int n = 1; n < 625; ++n) {
                        const int a = n % 5 - 2, b = n / 5 % 5 - 2, c = n / 25 % 5 - 2, d = n / 125 - 2;
                        if (!a && !b && !c && !d) continue;
                        least = fmin(least, fabs(a * term_weight(i) + b * term_weight(j) + c * term_weight(k) +
                                                 d * term_weight(l)));
                    }
    printf("%s", least > 1e-9 ? "ok" : "related");  // blocks are told apart at 1e-13 of their largest value
}
"""


def test_weights_of_the_terms_are_unrelated(tmp_path):
    assert _run(tmp_path, WEIGHTS) == "ok"


REPEATED = r"""
#include <stdio.h>
#include "msgpu_csr.h"
using namespace msgpu;
int main()
{
    // H01 = 1 + 1 against H10 = 1, then 2; rows in descending order
    const std::vector<int> p = {0, 3, 5}, c = {1, 0, 1, 1, 0};
    std::vector<double> both = {1, 0.5, 3, 0, 1, 0.5, 2, 0, 1, -0.5, 1, 0.5, 3, 0, 1, 0.5, 2, 0, 2, -1};
    const int sorted[] = {0, 2, 4}, cols[] = {0, 1, 0, 1};
    const MergedCsr m = merge_columns(2, p.data(), c.data(), both.data(), 2);
    printf("%d%d", repeated_columns(2, p.data(), c.data()), repeated_columns(2, sorted, cols));
    for (int t = 0; t < 2; ++t) printf(" %d", is_hermitian(2, m.rowptr.data(), m.col.data(), m.val.data() + 8 * t));
    for (int x : m.rowptr) printf(" %d", x);
    for (int x : m.col) printf(" %d", x);
    for (double x : m.val) printf(" %g", x);
    return 0;
}
"""


def test_repeated_columns_are_added_up(tmp_path):
    assert _run(tmp_path, REPEATED) == "10 0 1 0 2 4 1 0 1 0 2 1 3 0 2 0 1 -0.5 2 1 3 0 2 0 2 -1"


FORMS = r"""
#include <stdio.h>
#include <stdlib.h>
#include <array>
#include <map>
#include <set>
#include "msgpu_quartet.h"
using namespace msgpu;
static double rnd() { return 0.25 * (rand() % 64 - 32); }
// nuclei of the given multiplicities around electrons at the given places of the product basis
static int check(const std::vector<int> &mult, int e1, int e2, int kind, bool terms)
{
    const int n = static_cast<int>(mult.size());
    std::vector<int> stride(n, 1);
    for (int k = n - 2; k >= 0; --k) stride[k] = stride[k + 1] * mult[k + 1];
    const int D = stride[0] * mult[0], s1 = stride[e1], s2 = stride[e2], Q = D / 4;
    std::map<std::pair<int, int>, std::pair<double, double>> H;
    auto add = [&](int r, int c, double re, double im) {
        auto &h = H[{r, c}];
        h.first += re;
        h.second += im;
    };
    for (int k = 0; k < n; ++k) {
        if (k == e1 || k == e2) continue;
        const int se = k % 2 ? s1 : s2;  // each nucleus flips with one electron
        const double u = rnd() + 0.125, w = rnd() + 0.125;
        for (int r = 0; r < D; ++r) {
            const int d = r / stride[k] % mult[k];
            if (d + 1 < mult[k]) {
                const int c = r + stride[k], f = (r / se) % 2 ? -se : se;
                add(r, c + f, u, w);
                add(c + f, r, u, -w);
                if (kind != 1) {  // also without the electron's flip, signed by its state
                    const double z = (r / se) % 2 ? -w : w;
                    add(r, c, z, 0.5);
                    add(c, r, z, -0.5);
                }
            }
        }
    }
    for (int r = 0; r < D; ++r) {
        add(r, r, rnd(), 0.0);
        if (kind == 2) add(r, (r * 7 + 3) % D, rnd(), rnd());  // anywhere
        if (kind == 3) for (int c = 0; c < D; ++c) add(r, c, rnd(), rnd());
    }
    // rows in a scrambled order, some entries in two halves, an explicit zero
    std::vector<int> rowptr(1, 0), col;
    std::vector<double> val;
    auto at = H.begin();
    for (int r = 0; r < D; ++r) {
        std::vector<std::array<double, 3>> row;
        for (; at != H.end() && at->first.first == r; ++at) {
            const double c = at->first.second, x = at->second.first, y = at->second.second;
            if (!terms && rand() % 5 == 0) {
                row.push_back({c, x / 2, y / 2});
                row.push_back({c, x / 2, y / 2});
            } else {
                row.push_back({c, x, y});
            }
        }
        for (size_t i = 1; i < row.size() && r % 2; ++i) std::swap(row[i], row[rand() % (i + 1)]);
        for (auto &e : row) {
            col.push_back(static_cast<int>(e[0]));
            val.push_back(e[1]);
            val.push_back(e[2]);
        }
        rowptr.push_back(static_cast<int>(col.size()));
    }
    const QuartetForm f = quartet_form(D, s1, s2, rowptr.data(), col.data(), val.data(), terms);
    const int off[4] = {0, s2, s1, s1 + s2};
    if (static_cast<int>(f.rowptr.size()) != Q + 1 || f.nbr.size() != f.blk.size() || f.val.size() != f.val64.size()) return 1;
    std::map<std::pair<int, int>, std::pair<double, double>> got;
    for (int q = 0; q < Q; ++q)
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k) {
            const int type = f.blk[k].x & 7, cb = f.blk[k].x >> 3, voff = f.blk[k].y;
            if (cb != f.base[f.nbr[k]]) return 2;
            if (f.nbr[k] == q && k != f.rowptr[q + 1] - 1) return 3;  // own block last, the others in order
            if (k > f.rowptr[q] && f.nbr[k] != q && f.nbr[k] <= f.nbr[k - 1]) return 4;
            for (int x = 0; x < kBlockCount[type]; ++x) {
                const int e = kBlockOrder[type][x], copies = type == 4 || type == 5 ? 2 : 1;
                for (int c = 0; c < copies; ++c) {
                    const int a = (e >> 2) + (c ? (type == 4 ? 1 : 2) : 0), b = (e & 3) + (c ? (type == 4 ? 1 : 2) : 0);
                    const double re = f.val64[4 * static_cast<size_t>(voff) + 2 * x], im = f.val64[4 * static_cast<size_t>(voff) + 2 * x + 1];
                    if (static_cast<float>(re) != f.val[4 * static_cast<size_t>(voff) + 2 * x]) return 5;
                    if (re != 0.0 || im != 0.0) got[{f.base[q] + off[a], cb + off[b]}] = {re, im};
                }
                if (terms && f.src[2 * static_cast<size_t>(voff) + x] >= 0 &&
                    val[2 * f.src[2 * static_cast<size_t>(voff) + x]] != f.val64[4 * static_cast<size_t>(voff) + 2 * x])
                    return 6;
            }
        }
    for (auto &h : H)
        if (h.second.first != 0.0 || h.second.second != 0.0) {
            if (got[h.first] != h.second) return 7;
        }
    for (auto &g : got)
        if (H.count(g.first) == 0) return 8;
    // slots: their blocks are all of one type, -d with d only where no quartet has both
    const QuartetSlots s = quartet_slots(f);
    std::map<int, int> slot;
    for (int k = 0; k < s.n; ++k) {
        slot[s.delta[k]] = k;
        if ((s.shared >> k) & 1u) slot[-s.delta[k]] = k;
    }
    int left = 0;
    for (int q = 0; q < Q; ++q) {
        std::set<int> used;
        int rest = 0;
        for (int k = f.rowptr[q]; k < f.rowptr[q + 1]; ++k) {
            const int d = f.nbr[k] - q;
            if (d == 0) continue;
            if (!slot.count(d)) {
                ++rest;
                continue;
            }
            if (!used.insert(slot[d]).second) return 9;
            if ((f.blk[k].x & 7) != ((s.second >> slot[d]) & 1u ? 5 : 4)) return 10;
        }
        left = std::max(left, rest);
    }
    return left == s.left ? 0 : 11;
}
int main()
{
    const std::vector<std::vector<int>> systems = {{2, 2}, {2, 2, 2}, {2, 3, 2}, {2, 2, 3, 2, 3}, {3, 2, 2, 2, 2}, {2, 2, 2, 2, 2, 2, 2}};
    int runs = 0;
    for (auto &m : systems)
        for (int e1 = 0; e1 < static_cast<int>(m.size()); ++e1)
            for (int e2 = e1 + 1; e2 < static_cast<int>(m.size()); ++e2)
                for (int kind = 0; kind < 4; ++kind)
                    for (bool terms : {false, true}) {
                        if (m[e1] != 2 || m[e2] != 2) continue;
                        if (const int bad = check(m, e1, e2, kind, terms)) {
                            printf("case %d of %zu sites, electrons %d %d, kind %d, terms %d", bad, m.size(), e1, e2, kind, terms);
                            return 0;
                        }
                        ++runs;
                    }
    printf("%s", runs > 100 ? "ok" : "few");
}
"""


def test_quartet_form_and_its_slots_hold_the_matrix(tmp_path):
    # the quartet form expanded again is H; every slot holds blocks of one type
    assert _run(tmp_path, FORMS) == "ok"
