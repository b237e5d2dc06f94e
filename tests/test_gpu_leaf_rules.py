"""The panel leaf's pivot rules where they depend on more than the column:
the shipped reference's search (lu2tlib.c:1052) in slabs that begin at an odd
row and with several rows per thread.

Factors come from lu2's own slab call (cm_column_decomposition_recursive); the
pivots are compared, index for index, with a plain NumPy elimination."""
import numpy as np
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu


def reference_pivots(a, start):
    """Right-looking elimination of the slab with unscaled multipliers and rows
    exchanged whole.  An odd column (counted over the whole matrix) searches the
    multipliers of the column before it; the first column of each leaf of 16 has
    none before it and searches its own values."""
    b = a.copy()
    m = a.shape[1]
    want = []
    for c in range(m):
        s = c - 1 if (c + start) & 1 and c % 16 else c
        p = c + int(np.argmax(np.abs(b[c:, s])))
        want.append(p + start)
        b[[c, p]] = b[[p, c]]
        d = b[c, c]
        b[c] = np.where(np.arange(m) == c, d, b[c] / d)
        b[c + 1:, c + 1:] -= np.outer(b[c + 1:, c], b[c, c + 1:])
    return want


def gpu_pivots(a, start):
    rows, m = a.shape
    n = rows + start
    slab = np.zeros((m, n))
    slab[:, start:] = a.T
    pv = np.zeros(m, dtype=np.int32)
    old = L.set_pivot_mode(L.PIVOT_REF)
    try:
        L.load().cm_column_decomposition_recursive(n, slab.ctypes.data, m, pv.ctypes.data, start)
    finally:
        L.set_pivot_mode(old)
    return pv


@pytest.mark.parametrize("rows,m", [(200, 64), (3000, 48), (6000, 32), (10000, 32), (200, 16), (18000, 16)])
@pytest.mark.parametrize("start", [0, 1, 33, 64])
def test_reference_search_in_slabs_at_any_row(rows, m, start):
    a = np.random.default_rng(rows + start).uniform(-0.5, 0.5, (rows, m))
    a[np.arange(m), np.arange(m)] += m  # its odd columns' pivots need not be large: keep the growth small
    np.testing.assert_array_equal(gpu_pivots(a, start), reference_pivots(a, start))


@pytest.mark.parametrize("m", [9, 15, 17, 31, 40, 41, 48, 63])
@pytest.mark.parametrize("rows", [100, 700])
def test_pivot_rows_right_of_a_block(rows, m):
    """The 8 pivot rows of a block are finished one column per thread: widths that fill
    part of the first warp, all of it, and part of the second.  Backward error as
    Higham, Theorem 9.3: |P A - L U| <= (m + 4) u |L| |U|, with as much again for the
    check's own product."""
    a = np.random.default_rng(rows + m).uniform(-0.5, 0.5, (rows, m))
    slab = np.ascontiguousarray(a.T)
    pv = np.zeros(m, dtype=np.int32)
    L.load().cm_column_decomposition_recursive(rows, slab.ctypes.data, m, pv.ctypes.data, 0)
    f = slab.T.copy()
    for k, p in enumerate(pv):
        a[[k, p]] = a[[p, k]]
    d = f[np.arange(m), np.arange(m)]
    low = np.tril(f)
    low[np.arange(m), np.arange(m)] = 1.0
    low[:m] *= d[:, None]  # pivot rows are scaled by 1/pivot as a whole
    up = np.triu(f[:m], 1) + np.eye(m)
    bar = 2 * (m + 4) * 2.0 ** -53 * (np.abs(low) @ np.abs(up))
    assert np.all(np.abs(a - low @ up) <= bar)
    assert np.all(np.abs(f[m:]) <= np.abs(d))
