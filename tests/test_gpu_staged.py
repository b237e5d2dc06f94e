"""lumcolumn on pageable host memory: matrices that travel through the
page-locked slots against the same matrix page-locked as a whole with one copy
each way (LU2GPU_H2D_OVERLAP=0), which runs the same kernels on the same data
in the same order, so every bit agrees."""
import numpy as np
import pytest
import torch

import lu2_b200 as L

pytestmark = pytest.mark.gpu


# row lengths around the 4 MB rule (n = 723, 724), one chunk more than the 16
# slots, a last chunk of one row, an odd row length
@pytest.mark.parametrize("n", [723, 724, 1000, 1431, 1536, 2049])
def test_lumcolumn_slots_move_every_row(monkeypatch, n):
    nb = 64
    rng = np.random.default_rng(n)
    given = np.full((n, L.rdim(n)), np.nan)
    given[:, :n + 1] = rng.random((n, n + 1)) - 0.5
    got = []
    for pinned in (True, False, False):
        a = torch.empty(given.shape, dtype=torch.float64, pin_memory=pinned).numpy()
        a[:] = given
        x, pv = np.zeros(n), np.zeros(nb, dtype=np.int32)
        monkeypatch.setenv("LU2GPU_H2D_OVERLAP", "0")
        assert L.lumcolumn(a, x, nb, pv) == 0
        got.append((a, x, pv[: n - (n - 1) // nb * nb].copy()))
    for a, x, pv in got[1:]:
        assert np.array_equal(a[:, :n + 1], got[0][0][:, :n + 1])
        assert np.isnan(a[:, n + 1:]).all()
        assert np.array_equal(x, got[0][1]) and np.array_equal(pv, got[0][2])
