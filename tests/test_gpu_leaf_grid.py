"""The panel leaf over the whole grid, which takes panels of more rows than one
cluster holds: LU2GPU_LEAF_CTAS=8 gives a context whose panels all take it, at
sizes that cost little.  What it must find is what the cluster leaf finds: the
same pivots on random systems, in both searches, with ties, a zero and a NaN
column; solutions to lu2's own acceptance; and its own bounded wait."""
import pytest

import lu2_b200 as L
from test_gpu_leaf_faults import scaled_residual, system, withheld_then_solved, withheld_then_solved_fp32

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def grid():
    with pytest.MonkeyPatch.context() as m:
        m.setenv("LU2GPU_LEAF_CTAS", "8")
        c = L.Context(0)
    yield c
    c.close()


def factored(ctx, a, ld, nb, mode):
    import torch

    n = a.shape[0]
    f = a.clone()
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    status = ctx.lusolve(f, n, ld, nb, 1, mode, ipiv)
    torch.cuda.synchronize()
    return status, ipiv, f


# 512-column panels of 16-column leaves put off the longest lists of exchanges
@pytest.mark.parametrize("n,nb", [(1, 16), (17, 16), (100, 64), (129, 128), (1001, 112), (1500, 512), (3001, 256)])
def test_same_pivots_as_the_cluster_leaf(ctx, grid, n, nb):
    import torch

    a, ld = system(n, n)
    status, ipiv, f = factored(grid, a, ld, nb, L.PIVOT_PARTIAL)
    assert status == 0
    assert scaled_residual(a[:, :n], a[:, n], f[:, n]) < 16
    assert torch.equal(ipiv, factored(ctx, a, ld, nb, L.PIVOT_PARTIAL)[1])


@pytest.mark.parametrize("n,nb", [(40, 16), (300, 64)])
def test_same_pivots_by_the_reference_search(ctx, grid, n, nb):
    import torch

    a, ld = system(n, n + 1)
    i = torch.arange(n, device="cuda")
    a[i, i] += n  # its odd columns' pivots need not be large: keep the growth small
    assert torch.equal(factored(grid, a, ld, nb, L.PIVOT_REF)[1], factored(ctx, a, ld, nb, L.PIVOT_REF)[1])


@pytest.mark.parametrize("n", [100, 700, 2000])
def test_ties_zero_and_nan_columns(ctx, grid, n):
    import torch

    a, ld = system(n, n + 2)
    a[:, 0] = 1.0
    a[2::3, 0] = -2.0            # ties: the first of the largest
    a[:, 1] = 0.0                # a zero column
    a[:, n - 1] = float("nan")   # no candidate: the row stays
    status, ipiv, f = factored(grid, a, ld, 64, L.PIVOT_PARTIAL)
    want_status, want, g = factored(ctx, a, ld, 64, L.PIVOT_PARTIAL)
    assert status == want_status == 2
    assert torch.equal(ipiv, want) and int(ipiv[0]) == 2 and int(ipiv[1]) == 1 and int(ipiv[n - 1]) == n - 1
    assert torch.equal(torch.isnan(f[:, :n]), torch.isnan(g[:, :n]))
    assert bool(torch.isfinite(f[:n - 1, :n - 1]).all())


@pytest.mark.parametrize("n,nb", [(200, 64), (1500, 256)])
def test_fp32(grid, n, nb):
    import torch

    a, ld = system(n, n + 3)
    b, x = a[:, n].clone(), torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert grid.mixed_solve(a, n, ld, b, x, nb)["status"] == 0
    assert scaled_residual(a[:, :n], b, x) < 16.5  # it stops below 16 by its own sum


@pytest.mark.parametrize("cta", [0, 7])
def test_wait_gives_up_and_context_recovers(grid, cta):
    """1024 rows: 8 CTAs of 128."""
    withheld_then_solved(grid, 1024, cta)
    withheld_then_solved_fp32(grid, 1024, cta)
