"""The precision form's operand maxima and BF16 conversion at ragged sizes and
strides: both are exact, so they agree with torch bit for bit."""
import ctypes

import pytest
import torch

import lu2_b200 as L

pytestmark = pytest.mark.gpu

_ABSMAX2 = "_ZN6lu2gpu14launch_absmax2EPKfliiS1_liiPjP11CUstream_st"
_TO_BF16 = "_ZN6lu2gpu18launch_f32_to_bf16EPKflPvliiS1_P11CUstream_st"
_vp, _cl = ctypes.c_void_p, ctypes.c_long


def _matrix(rows, cols, ld, off, seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    buf = torch.empty(rows * ld + 4, device="cuda").normal_(generator=g)
    return buf[off:off + rows * ld].view(rows, ld)


# one element, remainders of 4 and 128 columns, more pieces than the grid has
# warps; strides and offsets with and without 16-byte rows
@pytest.mark.parametrize("rows,cols,ld,off", [(1, 1, 1, 0), (3, 5, 8, 0), (7, 127, 128, 0), (64, 128, 128, 1),
                                              (33, 131, 133, 0), (256, 1000, 1000, 0), (40000, 256, 260, 0),
                                              (5, 70001, 70004, 0)])
def test_operand_maxima_and_bf16(rows, cols, ld, off):
    lib = L.load()
    x, y = _matrix(rows, cols, ld, off, 1), _matrix(cols, rows, rows + 3, off, 2) * 0.25
    x[:, cols:] = float("inf")  # past the operand
    x[rows // 2, cols - 1] = -9.0
    y[:, rows:] = float("nan")
    amax = torch.zeros(2, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    st = _vp(torch.cuda.current_stream().cuda_stream)
    fn = getattr(lib, _ABSMAX2)
    fn.restype = ctypes.c_int
    assert fn(_vp(x.data_ptr()), _cl(ld), rows, cols, _vp(y.data_ptr()), _cl(rows + 3), cols, rows,
              _vp(amax.data_ptr()), st) == 0
    want = torch.stack([x[:, :cols].abs().max(), y[:, :rows].abs().max()])
    assert torch.equal(amax.view(torch.float32), want)
    scale = torch.tensor([0.125], device="cuda")
    out = torch.full((rows, cols + 4 + off), 3.0, dtype=torch.bfloat16, device="cuda")
    fn = getattr(lib, _TO_BF16)
    fn.restype = ctypes.c_int
    assert fn(_vp(x.data_ptr()), _cl(ld), _vp(out.data_ptr()), _cl(out.shape[1]), rows, cols, _vp(scale.data_ptr()),
              st) == 0
    torch.cuda.synchronize()
    assert torch.equal(out[:, :cols], (x[:, :cols] * 0.125).to(torch.bfloat16))
    assert (out[:, cols:] == 3.0).all()
