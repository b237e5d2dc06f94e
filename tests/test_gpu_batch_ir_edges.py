"""FP32 factors with FP64 refinement at the edges of FP32's range, and what the
refinement's stop promises."""
import numpy as np
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


class _DeviceArray:
    def __init__(self, ptr, count):
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<f8", "data": (ptr, False), "version": 2}


def view(batch, i):
    """System i's augmented matrix, n rows of its stride."""
    import torch

    p, ld = batch.system(i)
    n = int(batch.n[i])
    return torch.as_tensor(_DeviceArray(p, n * ld), device="cuda").view(n, ld)


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 100, 400])
def test_last_pivot_whose_reciprocal_overflows_fp32(ctx, n):
    """1 / 2e-39 is beyond FP32, 2e-39 itself (subnormal, 2^-149 apart) is not: A is
    upper triangular with that last pivot and x = 1.  Rounding the pivot and the
    right-hand side to FP32 moves x_n by 2^-150 / 2e-39 = 3.5e-7 each, the
    division by 6e-8."""
    import torch

    rng = np.random.default_rng(n)
    a = np.triu(rng.uniform(-0.5, 0.5, (n, n)) / n, 1)
    a[np.arange(n), np.arange(n)] = 2.0
    a[n - 1, n - 1] = 2e-39
    batch = L.Batch(ctx, np.array([n], np.int32))
    try:
        v = view(batch, 0)
        v[:, :n] = torch.from_numpy(a).cuda()
        v[:, n] = torch.from_numpy(a.sum(1)).cuda()
        torch.cuda.synchronize()
        batch.set_mode(L.BATCH_FP32_IR)
        assert batch.solve()[0] == 0
        torch.cuda.synchronize()
        x = v[:, n].cpu().numpy()
    finally:
        batch.close()
    assert abs(x[n - 1] - 1.0) <= 1e-6, x[n - 1]
    assert np.all(np.abs(x[:-1] - 1.0) <= 1e-6)


def test_refinement_stops_below_the_bar_by_any_sum(ctx):
    """A system is done when its scaled residual is below 16 however the residual is
    summed.  Summed in n + 1 FP64 roundings, in whatever order, a residual is off
    by at most (n + 1) u (|A||x| + |b|), which is (n + 1) / n of the scaled unit;
    so the residual in 80-bit arithmetic stays below 16 - (n + 1) / n."""
    import torch

    count = 6000
    rng = np.random.default_rng(2)
    n = rng.integers(16, 97, count).astype(np.int32)
    batch = L.Batch(ctx, n)
    try:
        batch.generate(1)
        batch.snapshot()
        torch.cuda.synchronize()
        before = [view(batch, i).cpu().numpy().astype(np.longdouble) for i in range(count)]
        batch.set_mode(L.BATCH_FP32_IR)
        assert (batch.solve() == 0).all()
        torch.cuda.synchronize()
        done = batch.iterations() < 10
        assert done.mean() > 0.9
        worst = 0.0
        for i in range(count):
            if not done[i]:
                continue
            k = int(n[i])
            a, b = before[i][:, :k], before[i][:, k]
            x = view(batch, i)[:, k].cpu().numpy().astype(np.longdouble)
            norm = np.abs(a).sum(1).max() * np.abs(x).max() + np.abs(b).max()
            h = float(np.abs(b - a @ x).max() / (norm * U * k))
            worst = max(worst, h + (k + 1) / k)
    finally:
        batch.close()
    assert worst < 16, worst
