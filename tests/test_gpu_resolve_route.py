"""A re-solve's two ways, the persistent solves and the panel loop, on both sides
of the rule that chooses between them (148 SMs)."""
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("n,nb,nrhs,persistent", [
    (128, 64, 8, True), (128, 64, 9, False), (100, 16, 16, True), (100, 16, 17, False), (129, 64, 18, True),
    (400, 128, 19, False), (300, 256, 18, True), (700, 256, 19, False), (300, 48, 16, True), (300, 48, 17, False),
    (300, 32, 24, True), (300, 32, 25, False), (300, 16, 24, True), (300, 16, 25, False), (600, 272, 32, True),
    (600, 272, 33, False), (4736, 16, 17, True), (4737, 16, 17, False), (9472, 16, 9, True), (9473, 16, 9, False)])
def test_both_sides_of_the_rule(ctx, n, nb, nrhs, persistent):
    """Persistent: the diagonal's reciprocals, two launches for the row map, two for each
    pass of eight.  The solution passes lu2's own acceptance column by column."""
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
    launches = L.load().lu2gpu_kernel_launches() - before
    assert (launches == 3 + 2 * -(-nrhs // 8)) == persistent, launches
    r = (a0 @ x - b).abs().amax(0)
    h = r / (U * (a0.abs().sum(1).max() * x.abs().amax(0) + b.abs().amax(0)) * n)
    assert float(h.max()) < 16
