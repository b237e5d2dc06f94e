"""The FP32 block-row solve of the precision forms, X := T^{-1} X with a unit
lower triangle, called as the factorization calls it."""
import ctypes

import pytest
import torch

import lu2_b200 as L

pytestmark = pytest.mark.gpu

_SYMBOL = "_ZN6lu2gpu26launch_trsm_unit_lower_f32EPKflPfliiS2_P11CUstream_st"


# one to 512 rows with remainders of the 16-row blocks and of the rows a warp
# takes; widths at both ends of one, two and four columns per lane (to 4736, to
# 9472, more; 512 rows stay at two) and of a CTA's columns; strides and an
# offset that forbid 16-byte copies
@pytest.mark.parametrize("K,ncols", [(1, 1), (15, 31), (16, 33), (17, 1), (40, 300), (64, 4736), (250, 4737),
                                     (256, 9472), (256, 9473), (264, 9600), (512, 9601), (496, 32), (100, 9599)])
@pytest.mark.parametrize("aligned,with_bt", [(True, True), (True, False), (False, True)])
def test_f32_block_row_solve(K, ncols, aligned, with_bt):
    """Blocked substitution in FP32 gives (T + E) x = b with |E| <= gamma_{K+2}
    |T| componentwise, whatever the order of its sums."""
    fn = getattr(L.load(), _SYMBOL)
    fn.restype = ctypes.c_int
    g = torch.Generator(device="cuda")
    g.manual_seed(K * 10007 + ncols)
    ldt, ldx, off = ((K + 3) & ~3, (ncols + 7) & ~3, 0) if aligned else (K + (1 - K % 2), ncols + 5, 1)
    tb = torch.empty(K * ldt + 4, device="cuda").uniform_(-1, 1, generator=g)
    xb = torch.empty(K * ldx + 4, device="cuda").uniform_(-1, 1, generator=g)
    t = tb[off:off + K * ldt].view(K, ldt)
    x = xb[off:off + K * ldx].view(K, ldx)
    t[:, :K] *= 4.0 / K ** 0.5  # solutions of moderate size
    before = x.clone()
    bt = torch.full((ncols, K), float("nan"), device="cuda")
    torch.cuda.synchronize()
    vp, cl = ctypes.c_void_p, ctypes.c_long
    rc = fn(vp(t.data_ptr()), cl(ldt), vp(x.data_ptr()), cl(ldx), K, ncols, vp(bt.data_ptr() if with_bt else None),
            vp(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    assert torch.equal(x[:, ncols:], before[:, ncols:])
    if with_bt:
        assert torch.equal(bt, x[:, :ncols].T)
    tri = torch.tril(t[:, :K].double(), -1) + torch.eye(K, device="cuda", dtype=torch.float64)
    sol = x[:, :ncols].double()
    gamma = (K + 2) * 2.0 ** -24 / (1 - (K + 2) * 2.0 ** -24)
    resid = (before[:, :ncols].double() - tri @ sol).abs()
    assert (resid <= gamma * (tri.abs() @ sol.abs()) + 1e-12).all()
