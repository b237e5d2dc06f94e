"""The persistent triangular solves with stored factors at the edges of their
blocks: panel widths below, at and above a block, a ragged last panel and
block, one to eleven right-hand sides (padded, two passes), more than
SOLVE_FEW_RHS (the panel loop), orders with several blocks per CTA, and pivots
outside their range.

lu2gpu_solve is compared with the solution lu2gpu_lusolve carries along in its
augmented columns.  Both are backward stable solves with the same factors, so
they differ by at most twice n u |L||U| over |A| times the condition number;
that product was bounded by numpy on the same systems: the bar is
100 n u cond_inf(A)."""
import numpy as np
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def system(n, nrhs, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    ld = L.device_ld(n, nrhs)
    a = torch.rand((n, ld), dtype=torch.float64, device="cuda", generator=g) - 0.5
    # a permuted shift keeps the condition number small and the exchanges real
    i = torch.arange(n, device="cuda")
    a[i, (i + n // 3) % n] += n ** 0.5
    torch.cuda.synchronize()
    return a, ld


@pytest.mark.parametrize("n,nb,nrhs", [(1, 16, 1), (16, 16, 2), (100, 16, 1), (127, 64, 3), (129, 128, 1), (300, 48, 4),
                                       (640, 192, 5), (1000, 256, 8), (1111, 112, 11), (2000, 512, 1), (3000, 208, 2),
                                       (700, 64, 33)])
def test_resolve_edges(ctx, n, nb, nrhs):
    import torch

    a, ld = system(n, nrhs, n + nrhs)
    b = a[:, n:n + nrhs].clone().contiguous()
    cond = float(torch.linalg.cond(a[:, :n], float("inf")))
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert ctx.lusolve(a, n, ld, nb, nrhs, L.PIVOT_PARTIAL, ipiv) == 0
    want = a[:, n:n + nrhs]
    got = torch.full((n, nrhs + 1), 7.0, dtype=torch.float64, device="cuda")  # an odd stride, too
    got[:, :nrhs] = b
    torch.cuda.synchronize()
    ctx.solve(a, n, ld, nb, ipiv, got, nrhs + 1, nrhs)
    assert bool((got[:, nrhs] == 7.0).all())
    err = float((got[:, :nrhs] - want).abs().max() / want.abs().max())
    assert err <= 100 * n * U * cond, (err, cond)


def test_resolve_with_several_blocks_per_cta(ctx):
    """More than 148 blocks of 128 rows."""
    import torch

    n, nb = 19100, 256
    a, ld = system(n, 1, 3)
    b = a[:, n:n + 1].clone()
    a0 = a[:, :n].clone()
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert ctx.factor(a, n, ld, nb, 1, L.PIVOT_PARTIAL, ipiv) == 0
    x = b.clone()
    torch.cuda.synchronize()
    ctx.solve(a, n, ld, nb, ipiv, x, 1, 1)
    r = (a0 @ x - b).abs().max()
    hpl = float(r / (U * (a0.abs().sum(1).max() * x.abs().max() + b.abs().max()) * n))
    assert hpl < 16, hpl  # lu2's own acceptance


def test_resolve_refuses_pivots_out_of_range(ctx):
    import torch

    n, nb = 500, 64
    a, ld = system(n, 1, 9)
    b = a[:, n].clone()
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert ctx.factor(a, n, ld, nb, 1, L.PIVOT_PARTIAL, ipiv) == 0
    for k, bad in ((300, n), (300, 299), (10, -1)):
        piv = ipiv.clone()
        piv[k] = bad
        x = b.clone()
        torch.cuda.synchronize()
        with pytest.raises(L.Lu2GpuError) as e:
            ctx.solve(a, n, ld, nb, piv, x, 1, 1)
        assert e.value.rc == -1
        assert bool((x == b).all())  # nothing was written
    x = b.clone()
    torch.cuda.synchronize()
    ctx.solve(a, n, ld, nb, ipiv, x, 1, 1)  # and the context goes on
    assert bool(torch.isfinite(x).all())
