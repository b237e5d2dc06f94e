"""The strides that the device DGEMM refuses and takes."""
import pytest

import lu2_b200 as L

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lda", [62, 63, 0])
@pytest.mark.parametrize("offset", [0, 1])
def test_dgemm_refuses_rows_shorter_than_k(ctx, lda, offset):
    """Rows of A shorter than k, whatever their alignment."""
    import torch

    m, n, k = 40, 50, 64
    a = torch.zeros(m * k + 2, dtype=torch.float64, device="cuda")  # room for m rows of k
    b = torch.zeros((k, n), dtype=torch.float64, device="cuda")
    c = torch.ones((m, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    with pytest.raises(L.Lu2GpuError):
        ctx.dgemm(m, n, k, -1.0, a.data_ptr() + 8 * offset, lda, b, n, 1.0, c, n)
    torch.cuda.synchronize()
    assert bool((c == 1.0).all())


def test_dgemm_of_one_row_without_a_stride(ctx):
    import torch

    n, k = 50, 64
    g = torch.Generator(device="cuda").manual_seed(1)
    a = torch.rand(k, dtype=torch.float64, device="cuda", generator=g)
    b = torch.rand((k, n), dtype=torch.float64, device="cuda", generator=g)
    c = torch.zeros((1, n), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    ctx.dgemm(1, n, k, 1.0, a, 0, b, n, 0.0, c, n)
    # both sums of k products round k times: 2 k u |a||b|
    assert bool(((c - a @ b).abs() <= 2 * k * 2.0 ** -53 * (a.abs() @ b.abs())).all())
