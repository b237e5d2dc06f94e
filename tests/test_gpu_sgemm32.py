"""The FP32 update inside the precision forms' panels, C -= A Bt^T, called as
the factorization calls it."""
import ctypes

import pytest
import torch

import lu2_b200 as L

pytestmark = pytest.mark.gpu

_SYMBOL = "_ZN6lu2gpu19launch_sgemm_updateEPKflS1_PfliiiP11CUstream_st"


# one element to several 64 x 64 tiles, remainders of the tiles and of the
# 32-column slabs; rows that allow 16-byte loads and rows that do not
@pytest.mark.parametrize("M,N,K", [(1, 1, 1), (63, 65, 31), (64, 64, 32), (65, 63, 33), (200, 64, 64), (129, 130, 4),
                                   (1000, 128, 128), (77, 192, 100), (64, 16, 16)])
@pytest.mark.parametrize("aligned", [True, False])
def test_f32_panel_update(M, N, K, aligned):
    """K products summed from zero and subtracted once: the error is at most
    gamma_{K+1} (|C| + |A| |Bt|^T) componentwise, for any order of the sum."""
    fn = getattr(L.load(), _SYMBOL)
    fn.restype = ctypes.c_int
    g = torch.Generator(device="cuda")
    g.manual_seed(M * 31 + N * 7 + K)
    off = 0 if aligned else 1
    lda, ldc = ((K + 7) & ~3, (N + 7) & ~3) if aligned else ((K + 4) | 1, (N + 4) | 1)
    ab = torch.empty(M * lda + 4, device="cuda").uniform_(-1, 1, generator=g)
    cb = torch.empty(M * ldc + 4, device="cuda").uniform_(-1, 1, generator=g)
    a, c = ab[off:off + M * lda].view(M, lda), cb[off:off + M * ldc].view(M, ldc)
    bt = torch.empty(N, K, device="cuda").uniform_(-1, 1, generator=g)
    before = c.clone()
    torch.cuda.synchronize()
    vp, cl = ctypes.c_void_p, ctypes.c_long
    rc = fn(vp(a.data_ptr()), cl(lda), vp(bt.data_ptr()), vp(c.data_ptr()), cl(ldc), M, N, K,
            vp(torch.cuda.current_stream().cuda_stream))
    torch.cuda.synchronize()
    assert rc == 0
    assert torch.equal(c[:, N:], before[:, N:])
    a64, b64, c64 = a[:, :K].double(), bt.double(), before[:, :N].double()
    gamma = (K + 1) * 2.0 ** -24 / (1 - (K + 1) * 2.0 ** -24)
    err = (c[:, :N].double() - (c64 - a64 @ b64.T)).abs()
    assert (err <= gamma * (c64.abs() + a64.abs() @ b64.abs().T) + 1e-12).all()
