"""Several row exchanges in one launch (launch_laswp_jobs), each with its own
pivots and columns, against the exchanges one by one: rows only move and the
pivot rows are multiplied once, so every bit agrees."""
import ctypes

import numpy as np
import pytest
import torch

import lu2_b200 as L

pytestmark = pytest.mark.gpu

_SYMBOL = {torch.float64: "_ZN6lu2gpu17launch_laswp_jobsEPdliRKNS_8SwapJobsEPKiiPKdPiP11CUstream_st",
           torch.float32: "_ZN6lu2gpu17launch_laswp_jobsEPfliRKNS_8SwapJobsEPKiiPKfPiP11CUstream_st"}


class SwapJobs(ctypes.Structure):
    _fields_ = [("n", ctypes.c_int), ("j", ctypes.c_int * 4 * 8)]


# (first pivot, past the last, first column, past the last): what a panel puts
# off and the exchange it joins; more pivots than stay in registers (256); a
# full list with empty jobs in it; columns that forbid 16-byte accesses
@pytest.mark.parametrize("n,jobs", [
    (300, [(64, 128, 0, 64), (0, 128, 128, 256)]),
    (300, [(192, 256, 128, 192), (128, 256, 0, 128), (0, 256, 256, 300)]),
    (700, [(300, 600, 0, 300), (0, 16, 600, 700)]),
    (130, [(16, 32, 0, 16), (5, 5, 16, 32), (48, 64, 32, 48), (64, 65, 48, 48), (80, 96, 64, 80), (96, 112, 80, 96),
           (112, 128, 96, 112), (0, 128, 112, 130)]),
    (90, [(10, 30, 1, 8), (20, 60, 9, 90)]),
])
@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
def test_exchanges_in_one_launch(n, jobs, dtype):
    fn = getattr(L.load(), _SYMBOL[dtype])
    fn.restype = ctypes.c_int
    rng = np.random.default_rng(n)
    goff = 3
    piv = np.array([rng.integers(k, n) for k in range(n)])
    dinv = torch.from_numpy(rng.uniform(0.5, 2, n)).to(dtype)
    ld = n + (-n) % 4
    a = torch.from_numpy(rng.uniform(-1, 1, (n, ld))).to(dtype)
    want = a.clone()
    for k0, k1, cs, ce in jobs:
        for k in range(k0, k1):
            if piv[k] != k:
                want[[k, piv[k]], cs:ce] = want[[piv[k], k], cs:ce]
        want[k0:k1, cs:ce] *= dinv[k0:k1, None]
    got, ipiv, dev = a.cuda(), torch.from_numpy(piv + goff).int().cuda(), dinv.cuda()
    status = torch.tensor([2 ** 31 - 1, 0, 0, 0], dtype=torch.int32, device="cuda")
    table = SwapJobs(n=len(jobs))
    for i, job in enumerate(jobs):
        table.j[i][:] = job
    torch.cuda.synchronize()
    vp = ctypes.c_void_p
    assert fn(vp(got.data_ptr()), ctypes.c_long(ld), n, ctypes.byref(table), vp(ipiv.data_ptr()), goff,
              vp(dev.data_ptr()), vp(status.data_ptr()), vp(torch.cuda.current_stream().cuda_stream)) == 0
    torch.cuda.synchronize()
    assert status[1] == 0
    assert torch.equal(got.cpu(), want)
