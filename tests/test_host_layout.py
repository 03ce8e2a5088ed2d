"""Host rules of the device layouts, compiled from their headers."""
import os
import subprocess

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _run(tmp_path, source):
    """Compiles and runs a C++ program against the library's headers; returns its output."""
    src, exe = tmp_path / "check.cpp", tmp_path / "check"
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(ROOT, "molspin_b200", "csrc"),
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
static bool hermitian(const std::vector<int> &p, const std::vector<int> &c, const std::vector<double> &v)
{
    const MergedCsr m = merge_columns(2, p.data(), c.data(), v.data(), 1);
    return is_hermitian(2, m.rowptr.data(), m.col.data(), m.val.data());
}
int main()
{
    // H01 = 1 + 1 against H10 = 1, then 2; rows in descending order
    const std::vector<int> p = {0, 3, 5}, c = {1, 0, 1, 1, 0};
    const std::vector<double> one = {1, 0.5, 3, 0, 1, 0.5, 2, 0, 1, -0.5}, two = {1, 0.5, 3, 0, 1, 0.5, 2, 0, 2, -1};
    const int sorted[] = {0, 2, 4}, cols[] = {0, 1, 0, 1};
    std::vector<double> both(one);
    both.insert(both.end(), two.begin(), two.end());
    const MergedCsr m = merge_columns(2, p.data(), c.data(), both.data(), 2);
    printf("%d%d %d%d", repeated_columns(2, p.data(), c.data()), repeated_columns(2, sorted, cols), hermitian(p, c, one),
           hermitian(p, c, two));
    for (int x : m.rowptr) printf(" %d", x);
    for (int x : m.col) printf(" %d", x);
    for (double x : m.val) printf(" %g", x);
    return 0;
}
"""


def test_repeated_columns_are_added_up(tmp_path):
    assert _run(tmp_path, REPEATED) == "10 01 0 2 4 1 0 1 0 2 1 3 0 2 0 1 -0.5 2 1 3 0 2 0 2 -1"
