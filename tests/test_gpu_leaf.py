"""The panel leaf on one cluster (cluster_leaf_kernel) at the edges of its
sizes: the rows one CTA, a cluster and each leaf width can hold, ragged widths,
both pivot searches, ties, zero and NaN columns.

The slab goes through lu2's own slab call (cm_column_decomposition_recursive,
lu2tlib.c:1095-1128).  The factors are checked by componentwise backward error:
a computed LU satisfies |P A - L U| <= g |L| |U| with g = m u / (1 - m u) for m
columns and u = 2^-53 (one rounding per multiply-add, Higham, Accuracy and
Stability, Theorem 9.3); scaling a pivot row by its reciprocal adds three
roundings (the reciprocal, the product, the product back in the check), so the
bar is (m + 4) u |L| |U|."""
import numpy as np
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def factor(a, m):
    n = a.shape[0]
    slab = np.ascontiguousarray(a.T)  # slab[j][r], as lu2tlib.c stores it
    pv = np.zeros(m, dtype=np.int32)
    L.load().cm_column_decomposition_recursive(n, slab.ctypes.data, m, pv.ctypes.data, 0)
    return np.ascontiguousarray(slab.T), pv


def swapped(a, pv):
    b = a.copy()
    for k, p in enumerate(pv):
        b[[k, p]] = b[[p, k]]
    return b


def check(a, f, pv):
    """|P A - L U| against (m + 4) u |L| |U|; rows k < m of f are scaled by 1/pivot."""
    m = a.shape[1]
    low = np.tril(f)
    low[np.arange(m), np.arange(m)] = 1.0
    low[:m] *= f[np.arange(m), np.arange(m)][:, None]  # undo the pivot rows' scaling
    up = np.triu(f[:m], 1) + np.eye(m)
    err = np.abs(swapped(a, pv) - low @ up)
    bar = (m + 4) * U * (np.abs(low) @ np.abs(up))
    worst = np.max(err - 2 * bar)  # the product of the check rounds, too
    assert worst <= 0, worst


@pytest.mark.parametrize("n,m", [(1, 1), (16, 16), (40, 37), (255, 64), (256, 64), (257, 64), (1025, 49), (4096, 64),
                                 (4097, 64), (8192, 32), (8193, 33), (16384, 16), (16385, 16), (5000, 7)])
def test_leaf_edges(n, m):
    rng = np.random.default_rng(n * 100 + m)
    a = rng.uniform(-0.5, 0.5, (n, m))
    f, pv = factor(a, m)
    check(a, f, pv)
    # every pivot is the largest of what was left in its column
    assert np.all(np.abs(f[m:]) <= np.abs(f[np.arange(m), np.arange(m)]))


@pytest.mark.parametrize("n", [200, 3000, 6000])
def test_leaf_ties_zero_and_nan_columns(n):
    rng = np.random.default_rng(n)
    a = rng.uniform(-0.5, 0.5, (n, 16))
    a[:, 0] = np.where(np.arange(n) % 3 == 2, -2.0, 1.0)  # ties: the first of the largest
    a[:, 1] = 0.0                                          # a zero column
    a[:, 15] = np.nan                                      # no candidate: the row stays
    f, pv = factor(a, 16)
    assert pv[0] == 2 and pv[1] == 1 and pv[15] == 15
    # the NaN pivot's row is scaled by 1/NaN as a whole; no other row sees it
    assert f[1, 1] == 0.0 and np.all(np.isnan(f[15:, 15])) and np.all(np.isnan(f[15, :15]))
    assert np.all(np.isfinite(np.delete(f, 15, axis=0)[:, :15]))


def test_leaf_reference_pivots_over_the_cluster(oracle):
    """The shipped search (lu2tlib.c:1052) with rows on all CTAs of a cluster."""
    n, m = 3000, 64
    old = L.set_pivot_mode(L.PIVOT_REF)
    try:
        a = np.random.default_rng(5).uniform(-0.5, 0.5, (n, m))
        _, pv = factor(a, m)
    finally:
        L.set_pivot_mode(old)
    b = a.copy()
    want = []
    for c in range(m):  # right-looking, unscaled multipliers, rows swapped whole
        s = c - 1 if c & 1 else c
        p = c + int(np.argmax(np.abs(b[c:, s])))
        want.append(p)
        b[[c, p]] = b[[p, c]]
        d = b[c, c]
        b[c] = np.where(np.arange(m) == c, d, b[c] / d)
        b[c + 1:, c + 1:] -= np.outer(b[c + 1:, c], b[c, c + 1:])
    np.testing.assert_array_equal(pv, want)


@pytest.mark.parametrize("n", [8704, 16640])
def test_fp32_leaf_with_several_rows_per_thread(ctx, n):
    """FP32 panels of more than 8192 and 16384 rows: the precision form's x on a
    diagonally dominant system against the FP64 solve.  Refined to a scaled
    residual below 16, so |x - x64| <= 2 * 16 n u cond |x|, cond < 4 here
    (each diagonal entry is the sum of its row's absolute values)."""
    import torch

    ld = L.device_ld(n, 1)
    a = torch.zeros((n, ld), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()  # the context has its own stream
    ctx.generate(a, n, ld, 3, kind=1)
    b = a[:, n].clone()
    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    got = ctx.mixed_solve(a, n, ld, b, x, 256)
    assert got["status"] == 0 and got["iterations"] <= 3
    assert ctx.lusolve(a, n, ld, 256) == 0
    x64 = a[:, n]
    assert float((x - x64).abs().max() / x64.abs().max()) <= 2 * 16 * n * U * 4


@pytest.mark.parametrize("n,m", [(8193, 32), (8200, 17), (12288, 32), (12289, 16), (16385, 16), (20480, 16),
                                 (20481, 16)])
@pytest.mark.parametrize("mode", [L.PIVOT_PARTIAL, L.PIVOT_REF])
def test_tall_leaf_edges(n, m, mode):
    """The instances with more rows per CTA, at both ends of their rows."""
    a = np.random.default_rng(n + m).uniform(-0.5, 0.5, (n, m))
    if mode == L.PIVOT_REF:  # its odd columns' pivots need not be large: keep the growth small
        a[np.arange(m), np.arange(m)] += m
    old = L.set_pivot_mode(mode)
    try:
        f, pv = factor(a, m)
    finally:
        L.set_pivot_mode(old)
    check(a, f, pv)
    if mode == L.PIVOT_PARTIAL:
        assert np.all(np.abs(f[m:]) <= np.abs(f[np.arange(m), np.arange(m)]))
    else:
        assert np.all(pv[::2] >= np.arange(0, m, 2)) and pv[0] == np.argmax(np.abs(a[:, 0]))


@pytest.mark.parametrize("n", [8193, 12288, 12289, 24576])
def test_fp32_tall_leaf_edges(ctx, n):
    """The FP32 tall instances' first and last row counts, as above."""
    test_fp32_leaf_with_several_rows_per_thread(ctx, n)
