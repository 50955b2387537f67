"""CPU check of the columns that the engine's passes read from a column slab
(csrc/tile_cols.h, compiled here with the host compiler) against the buffers
that include/srk_b200.h declares: a slab's buffer may end a mapping, so no pass
may read a column outside it, not even for a value that is never stored."""
import ctypes
import os
import subprocess

import pytest

from shrinkage_full_tests_b200.shard import adjoint_need, forward_need

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CSRC = os.path.join(ROOT, "shrinkage_full_tests_b200", "csrc")
SRC = """
#include "tile_cols.h"
extern "C" void columns(int xg, int e, int S, int halo, int whole, int gx0, int N, int* out) {
  const srk::ColSpan need = whole ? srk::ColSpan{0, whole} : srk::window_span(xg, e, S, halo);
  const srk::ColSpan c = srk::clip_span(need, gx0, N);
  out[0] = gx0 + c.lo;
  out[1] = gx0 + c.hi;
}
"""


@pytest.fixture(scope="module")
def columns(tmp_path_factory):
    d = tmp_path_factory.mktemp("tile_cols")
    src, so = d / "c.cpp", d / "c.so"
    src.write_text(SRC)
    subprocess.run(["g++", "-std=c++17", "-shared", "-fPIC", "-I" + CSRC, str(src), "-o", str(so)], check=True)
    fn = ctypes.CDLL(str(so)).columns
    out = (ctypes.c_int * 2)()

    def call(xg, e, S, halo, gx0, N, whole=0):
        fn(xg, e, S, halo, whole, gx0, N, out)
        return out[0], out[1]  # image columns [lo, hi) that are copied

    return call


def blocks(S, off):  # P3's blocks of four columns, first valid column `off` past the first
    return (S + off + 3) // 4


def slabs(n_out, S):
    """First, inner and last slab of one or two tiles, the last one cut."""
    for c0 in range(0, n_out, S):
        for k in (1, 2):
            c1 = min(c0 + k * S, n_out)
            if (c1 - c0) % S == 0 or c1 == n_out:
                yield c0, c1


@pytest.mark.parametrize("M", [128, 256, 512])
@pytest.mark.parametrize("rotated", [False, True])
def test_windows_of_the_last_pass(columns, M, rotated):
    """Central differences of forward and tangent slabs, cotangents of the
    tangent-adjoint slab: inside the declared columns, and every column that a
    valid output reads is there."""
    for e in range(0, min(60, (M - 8) // 2) + 1):
        S = M - 2 * e
        N = 3 * S + 2 * e + max(1, S // 3)
        W = N - 2 * e
        xa = e if rotated else e & ~3
        xgs = [xa + 4 * b for b in range(blocks(S, e - xa))]
        for c0, c1 in slabs(W, S):
            for x0 in range(c0, c1, S):
                for xg in xgs:
                    lo, hi = columns(xg, e, S, 1, x0 + xg - 1, N)
                    first, last = (max(c0 - 1, 0), min(c1 + 1, N)) if e == 0 else (c0, min(c1 + 2 * e, N))
                    assert forward_need(c0, c1, N, e) == (first, last)
                    assert lo == hi or (first <= lo and hi <= last), (e, c0, c1, xg)
                    for x in range(max(xg, e), min(xg + 4, e + S)):
                        if x0 + x - e < W:
                            assert lo <= max(x0 + x - 1, 0) and min(x0 + x + 1, N - 1) < hi
        for c0, c1 in slabs(N, S):
            r0, r1 = max(c0 - e - 1, 0), min(c1 - e + 1, W)
            T = -(-(r1 - r0) // S) if r1 > r0 else 0
            rE = min(r0 + T * S, W) if T else r0
            first, last = min(max(c0 - 2 * e, 0), r0), max(min(c1, W), rE)
            for x0 in range(r0, r0 + T * S, S):
                for xg in xgs:
                    lo, hi = columns(xg, e, S, 0, x0 + xg - e, W)
                    assert lo == hi or (first <= lo and hi <= last), (e, c0, c1, xg)
                    for x in range(max(xg, e), min(xg + 4, e + S)):
                        if x0 + x - e < W:
                            assert lo <= x0 + x - e < hi


@pytest.mark.parametrize("M", [128, 256, 512])
def test_windows_of_the_adjoint(columns, M):
    """The adjoint's first pass stages six columns of I around every block of
    four: f, df (and I of the adjoint slab) columns [c0 - e - 1, c1 + e + 1)."""
    for e in range(1, min(60, (M - 8) // 2) + 1):
        S = M - 2 * e
        N = 3 * S + max(1, S // 3)
        for c0, c1 in slabs(N, S):
            for x0 in range(c0, c1, S):
                for xg in range(0, M, 4):
                    lo, hi = columns(0, 0, 0, 0, x0 + xg - e - 1, N, whole=6)
                    assert lo == hi or (max(c0 - e - 1, 0) <= lo and hi <= min(c1 + e + 1, N)), (e, c0, c1, xg)


def test_columns_of_the_stencil():
    """dL/dI of the adjoint slab [c0, c1) reads u v at the window columns
    [c0 - e - 1, c1 - e + 1); the first pass reads v at [c0 - 2 e, c1)."""
    for e in (0, 1, 2, 15, 60):
        N, S = 700, 100
        W = N - 2 * e
        for c0, c1 in slabs(N, S):
            first, last = adjoint_need(c0, c1, W, e)
            assert first <= max(c0 - e - 1, 0) and min(c1 - e + 1, W) <= last
            assert first <= max(c0 - 2 * e, 0) and min(c1, W) <= last
