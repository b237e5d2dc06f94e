"""What a re-solve from stored factors holds beside them, on both of its ways, and
the row maps of extreme exchanges."""
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def shifted_system(n, nrhs):
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    ld = L.device_ld(n, 0)
    a = torch.rand((n, ld), dtype=torch.float64, device="cuda", generator=g) - 0.5
    i = torch.arange(n, device="cuda")
    a[i, (i + n // 3) % n] += n ** 0.5  # well conditioned, with exchanges
    return a, ld, torch.rand((n, nrhs), dtype=torch.float64, device="cuda", generator=g) - 0.5


# (19000, 16): blocks of 16 rows, more of them per CTA than shared memory holds,
# so that the solve goes panel by panel and needs no row maps
@pytest.mark.parametrize("n,nb,maps", [(12000, 16, True), (19000, 16, False), (9000, 256, True)])
def test_resolve_holds_half_row_maps(n, nb, maps):
    """A re-solve keeps 4 n (n / nb + 1) bytes of row maps and the solves' slots and
    vectors (under 256 n with their reserve); the solution passes lu2's own
    acceptance."""
    import torch

    a, ld, b = shifted_system(n, 1)
    a0 = a[:, :n].clone()
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    x = b.clone()
    ctx = L.Context(0)
    try:
        torch.cuda.synchronize()
        assert ctx.factor(a, n, ld, nb, 0, L.PIVOT_PARTIAL, ipiv) == 0
        many = b.expand(n, 33).contiguous()
        torch.cuda.synchronize()
        ctx.solve(a, n, ld, nb, ipiv, many, 33, 33)  # every other buffer of a solve
        free = torch.cuda.mem_get_info()[0]
        ctx.solve(a, n, ld, nb, ipiv, x, 1, 1)
        held = free - torch.cuda.mem_get_info()[0]
    finally:
        ctx.close()
    assert held <= (4 * n * (n // nb + 1) if maps else 0) + 256 * n + (6 << 20), held
    r = (a0 @ x - b).abs().max()
    assert float(r / (U * (a0.abs().sum(1).max() * x.abs().max() + b.abs().max()) * n)) < 16


@pytest.mark.parametrize("n,nb", [(33, 16), (500, 496), (1100, 272), (1600, 512)])
@pytest.mark.parametrize("order", ["next", "last", "same"])
def test_row_maps_of_extreme_exchanges(ctx, n, nb, order):
    """Every row exchanged with the one after it, with the last, or with itself: chains
    as long as a panel, one row named by all, none; panel widths right above a power
    of two and the widest.  Identity factors turn the solve into the exchanges alone."""
    import torch

    ld = L.device_ld(n, 0)
    a = torch.eye(n, ld, dtype=torch.float64, device="cuda")
    k = torch.arange(n)
    piv = {"next": torch.clamp(k + 1, max=n - 1), "last": torch.full((n,), n - 1), "same": k}[order].int()
    want = list(range(n))
    for i, p in enumerate(piv.tolist()):
        want[i], want[p] = want[p], want[i]
    b = torch.arange(n, dtype=torch.float64, device="cuda")[:, None].repeat(1, 2).contiguous()
    torch.cuda.synchronize()
    ctx.solve(a, n, ld, nb, piv.cuda(), b, 2, 2)
    assert b[:, 0].tolist() == want and b[:, 1].tolist() == want
