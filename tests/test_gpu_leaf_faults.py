"""The panel leaf's bounded waits beyond one size: a CTA of a full cluster of 16,
first and last, FP64 and FP32, withholds what it should send.  The wait gives up
after 50 ms, the call reports LU2GPU_ERR_TIMEOUT, and the same context then
solves to lu2's own acceptance."""
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


def system(n, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    ld = L.device_ld(n, 1)
    a = torch.rand((n, ld), dtype=torch.float64, device="cuda", generator=g) - 0.5
    i = torch.arange(n, device="cuda")
    a[i, (i + n // 3) % n] += n ** 0.5
    torch.cuda.synchronize()
    return a, ld


def scaled_residual(a, b, x):
    r = (a @ x - b).abs().max()
    return float(r / (U * (a.abs().sum(1).max() * x.abs().max() + b.abs().max()) * a.shape[0]))


def withheld_then_solved(ctx, n, cta):
    import torch

    a, ld = system(n, n + cta)
    work = a.clone()
    torch.cuda.synchronize()
    ctx.test_leaf_withhold(cta, 50.0)
    with pytest.raises(L.Lu2GpuError) as e:
        ctx.lusolve(work, n, ld, 64)
    assert e.value.rc == -4 and "gave up" in str(e.value)
    ctx.test_leaf_withhold(-1, 0.0)
    work.copy_(a)
    torch.cuda.synchronize()
    assert ctx.lusolve(work, n, ld, 64) == 0
    assert scaled_residual(a[:, :n], a[:, n], work[:, n]) < 16


def withheld_then_solved_fp32(ctx, n, cta):
    import torch

    a, ld = system(n, n + cta)
    b, x = a[:, n].clone(), torch.zeros(n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.test_leaf_withhold(cta, 50.0)
    with pytest.raises(L.Lu2GpuError) as e:
        ctx.mixed_solve(a, n, ld, b, x, 64)
    assert e.value.rc == -4 and "gave up" in str(e.value)
    ctx.test_leaf_withhold(-1, 0.0)
    assert ctx.mixed_solve(a, n, ld, b, x, 64)["status"] == 0
    assert scaled_residual(a[:, :n], b, x) < 16.5  # it stops below 16 by its own sum


@pytest.mark.parametrize("cta", [0, 15])
def test_cluster_of_16(cta):
    ctx = L.Context(0)
    try:
        withheld_then_solved(ctx, 4000, cta)
        withheld_then_solved_fp32(ctx, 8000, cta)
    finally:
        ctx.close()
