"""Columns of the block Gauss-Seidel kernel: whatever word its loads past an
item's end find in shared memory, the row of x that it becomes lies in the
block's own rows, also in a short last block, or is the row of zeros.  The rule
is plain C++ (gs_columns.h) and runs here on the host."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

SRC = r"""
#include "gs_columns.h"
#include <cstdio>
#include <cstdlib>
int main(int, char **a) {
    const long long n = atoll(a[1]), brows = atoll(a[2]);
    const int nb = (int)((n + brows - 1) / brows);
    unsigned long long s = 1;
    for (int b = 0; b < nb; ++b) {
        const int lim = xk::gs_block_rows((int)n, (int)brows, b);
        if (lim < 1 || lim > brows || (b < nb - 1 && lim != brows)) return 1;
        for (long long k = -2; k <= brows + 2; ++k)  // stale columns of other blocks, the padding column
            if (k >= 0 && k < lim ? xk::gs_block_column((int)k, lim) != k : xk::gs_block_column((int)k, lim) != lim) return 2;
        for (int k = 0; k < 1000; ++k) {  // words of values
            s = s * 6364136223846793005ull + 1442695040888963407ull;
            const int c = xk::gs_block_column((int)(s >> 32) >> (k % 24), lim);
            if (c < 0 || (c < lim && b * brows + c >= n) || c > lim) return 3;
        }
    }
    return 0;
}
"""


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("gs_columns")
    (d / "t.cpp").write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-I", os.path.join(ROOT, "xamg-test_b200", "csrc"), "-o", str(d / "t"),
                    str(d / "t.cpp")], check=True)
    return str(d / "t")


@pytest.mark.parametrize("n,brows", [(512000, 1154), (884736, 1993), (640, 639), (4097, 64), (1, 1), (1300, 500)])
def test_columns_stay_in_the_block(program, n, brows):
    assert subprocess.run([program, str(n), str(brows)]).returncode == 0


def test_kernel_uses_the_rule():
    """The kernel clamps by this rule alone: x through the L1 is read at rows below the limit."""
    src = open(os.path.join(ROOT, "xamg-test_b200", "csrc", "gs.cu")).read()
    assert "where(gs_block_column(c[u], lim))" in src
    assert "XS ? brows : gs_block_rows(n, brows, b)" in src
    assert "xlg(w < lim ? xga + (size_t)w * RB : zga, r)" in src
