"""Validation in tiles at the edges of its tiles (32 x 8 cells, 32 x 32 for large fields) against the
oracle, bit for bit, and the export of fields to device buffers of any alignment."""
import numpy as np
import pytest

from conftest import same_floats
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx", [(1, 1), (1, 40), (7, 31), (8, 32), (9, 33), (17, 65), (3, 100), (548, 557)])
def test_tiles_match_the_oracle(ny, nx):
    import piv_b200 as P
    rng = np.random.default_rng(ny * 1000 + nx)
    dx, dy = rng.normal(scale=2.0, size=(2, ny, nx)).astype(np.float32)
    dx[rng.random((ny, nx)) < 0.02] = 50.0            # out of range
    ppr = np.where(rng.random((ny, nx)) < 0.2, 1.1, 2.0).astype(np.float32)
    hole = np.zeros((ny, nx), bool)
    hole[ny // 3:ny // 3 + 6, nx // 3:nx // 3 + 7] = True  # nothing usable within radius 2 of its middle
    ppr[hole] = 1.0
    fl = (rng.random((ny, nx)) < 0.1).astype(np.uint8)
    dx[fl == 1] = dy[fl == 1] = np.nan
    ppr[fl == 1] = 0
    an = P.PivAnalyzer(P.PivConfig(windows=[64, 32]))
    ox, oy, of, s = an.validate_field(dx, dy, ppr, fl)
    wx, wy, wf, ws = O.validate(dx, dy, ppr, fl, max_displacement=32.0)
    assert np.array_equal(of, wf) and same_floats(ox, wx) and same_floats(oy, wy)
    live = (wf & 1) == 0
    want = [int((wf & 1).sum())] + [int(((wf & b) != 0)[live].sum()) for b in (2, 4, 16, 8)]
    assert list(s.as_dict().values()) == want


@pytest.mark.parametrize("shift", [0, 1])
def test_device_outputs_of_any_alignment(shift):
    import torch

    import piv_b200 as P
    rng = np.random.default_rng(7)
    a = rng.random((200, 333), dtype=np.float32)
    an = P.PivAnalyzer(P.PivConfig(windows=[16], overlap=0.75, final_iterations=1))
    fa, fb = an.prepare(a, P.RAW), an.prepare(np.roll(a, 2, 1), P.RAW)
    want = an.analyze(fa, fb)
    n = want.field.dx.size
    out = [torch.full((n + 8,), -7.0, device="cuda") for _ in range(3)]
    fl = torch.full((n + 8,), 77, device="cuda", dtype=torch.uint8)
    cnt = torch.full((6,), -1, device="cuda", dtype=torch.int64)
    an.analyze_device(fa, fb, *[t[shift:].data_ptr() for t in out], fl[shift:].data_ptr(), cnt.data_ptr())
    an.sync()
    f = want.field
    for t, w in zip(out, (f.dx, f.dy, f.peak_ratio)):
        assert same_floats(t[shift:shift + n].cpu().numpy(), w.ravel())
        assert (t[shift + n:] == -7.0).all() and (t[:shift] == -7.0).all()
    assert np.array_equal(fl[shift:shift + n].cpu().numpy(), f.flags.ravel()) and (fl[shift + n:] == 77).all()
    assert cnt.tolist() == list(want.summary.as_dict().values()) + [-1]
