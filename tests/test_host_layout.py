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
