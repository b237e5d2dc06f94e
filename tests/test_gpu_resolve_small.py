"""A re-solve of one panel of at most 128 rows: on which of its two ways it goes."""
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("n,nb,nrhs,persistent", [
    (1, 16, 1, False), (16, 16, 8, False), (17, 16, 8, True), (48, 64, 1, False), (64, 64, 4, False), (64, 256, 8, False),
    (65, 64, 8, True), (65, 256, 4, True), (65, 256, 5, False), (128, 128, 4, True), (128, 128, 5, False),
    (129, 256, 5, True)])
def test_one_panel(ctx, n, nb, nrhs, persistent):
    """Persistent: the diagonal's reciprocals, two launches for the row map, two solves.
    The solution passes lu2's own acceptance column by column."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n + nrhs)
    ld = L.device_ld(n, 0)
    a = torch.rand((n, ld), dtype=torch.float64, device="cuda", generator=g) - 0.5
    i = torch.arange(n, device="cuda")
    a[i, (i + n // 3) % n] += n ** 0.5
    a0 = a[:, :n].clone()
    b = torch.rand((n, nrhs), dtype=torch.float64, device="cuda", generator=g) - 0.5
    x = b.clone()
    ipiv = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert ctx.factor(a, n, ld, nb, 0, L.PIVOT_PARTIAL, ipiv) == 0
    before = L.load().lu2gpu_kernel_launches()
    ctx.solve(a, n, ld, nb, ipiv, x, nrhs, nrhs)
    assert (L.load().lu2gpu_kernel_launches() - before == 5) == persistent
    r = (a0 @ x - b).abs().amax(0)
    h = r / (U * (a0.abs().sum(1).max() * x.abs().amax(0) + b.abs().amax(0)) * n)
    assert float(h.max()) < 16
