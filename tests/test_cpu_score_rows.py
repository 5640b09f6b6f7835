"""The rule that decides whether a consensus layer's score rows may be 16-bit
(racon_b200/csrc/score_rows.hpp), compiled here, against the slanted scores of
layers at its edge: the largest layer that it takes for each set of scores, as
a chain of nodes that match the layer everywhere or nowhere."""
import ctypes
import os
import shutil
import subprocess

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "racon_b200", "csrc")


@pytest.fixture(scope="module")
def fast(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ is needed to compile the rule")
    d = tmp_path_factory.mktemp("score_rows")
    src, lib = d / "rule.cpp", d / "rule.so"
    src.write_text('#include "score_rows.hpp"\n'
                   'extern "C" int fast(int m, int x, int g, int n, int L) { return rb::fast_scores(m, x, g, n, L); }\n')
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I", CSRC, str(src), "-o", str(lib)], check=True)
    f = ctypes.CDLL(str(lib)).fast
    return lambda *a: bool(f(*a))


def _extremes(s, gap, ndp, L):
    """Smallest and largest H - column * gap of ndp rows in a chain against L
    columns, every step's substitution score s."""
    row = np.zeros(L + 1, dtype=np.int64)  # slanted
    low = high = 0
    for _ in range(ndp):
        t = row + gap
        t[1:] = np.maximum(t[1:], row[:-1] + s - gap)
        row = np.maximum.accumulate(t)
        low, high = min(low, int(row.min())), max(high, int(row.max()))
    return low, high


@pytest.mark.parametrize("m,x,g", [(3, -5, -4), (5, -4, -8), (1, -1, -1), (5, 60, -60), (-1, 20, -40), (0, 100, -1),
                                   (100, -20, -27), (-128, 100, -27), (-5, -3, -2), (0, 0, 0), (2, 2, -1)])
def test_rows_taken_as_16_bit_fit(fast, m, x, g):
    longest = max((L for L in range(1, 4000) if fast(m, x, g, 10, L)), default=0)
    most = max((n for n in range(1, 4000) if fast(m, x, g, n, 10)), default=0)
    # a layer's graph has at least its backbone's nodes: long layers against few and many rows
    for L in {longest, longest // 2, 10}:
        for ndp in {most, L, 10}:
            if 0 < L and fast(m, x, g, ndp, L):
                for s in (m, x):
                    low, high = _extremes(s, g, ndp, L)
                    assert -32768 <= low and high <= 32767, (L, ndp, s, low, high)


def test_refused(fast):
    assert not fast(3, -5, 1, 10, 10)         # a gap that gains
    assert not fast(100, -100, -90, 10, 10)   # s - gap leaves a signed byte
    assert not fast(5, 60, -60, 500, 500)
    assert not fast(-1, 20, -40, 100, 100)    # mismatch above match
    assert not fast(5, -4, -8, 3100, 1000)    # the all-gap path itself, (rows + columns) x gap, leaves 16 bits
    assert not fast(-1, 20, -40, 700, 700)
    assert fast(3, -5, -4, 2000, 600)
