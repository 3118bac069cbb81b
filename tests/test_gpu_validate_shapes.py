"""Validation in every tile shape, just past the lines between them and with ragged last tiles, against the
oracle bit for bit: fields of one to four columns or rows, of sixteen, and square ones."""
import numpy as np
import pytest

from conftest import same_floats
from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ny,nx", [(32768, 1), (32767, 1), (16411, 2), (1, 32769), (2, 16385), (10923, 3), (8193, 4), (8193, 5),
                                   (25001, 16), (23530, 17), (16, 25001), (17, 23531), (4, 100003), (632, 632), (633, 633),
                                   (1184, 1183)])
def test_tile_shapes_match_the_oracle(ny, nx):
    import piv_b200 as P
    rng = np.random.default_rng(ny + 7 * nx)
    dx, dy = rng.normal(scale=2.0, size=(2, ny, nx)).astype(np.float32)
    dx[rng.random((ny, nx)) < 0.02] = 50.0  # out of range
    ppr = np.where(rng.random((ny, nx)) < 0.3, 1.1, 2.0).astype(np.float32)
    ppr[ny // 3:ny // 3 + 7, nx // 3:nx // 3 + 7] = 1.0
    fl = (rng.random((ny, nx)) < 0.1).astype(np.uint8)
    dx[fl == 1] = dy[fl == 1] = np.nan
    an = P.PivAnalyzer(P.PivConfig(windows=[64, 32]))
    ox, oy, of, s = an.validate_field(dx, dy, ppr, fl)
    wx, wy, wf, _ = O.validate(dx, dy, ppr, fl, max_displacement=32.0)
    assert np.array_equal(of, wf) and same_floats(ox, wx) and same_floats(oy, wy)
    live = (wf & 1) == 0
    want = [int((wf & 1).sum())] + [int(((wf & b) != 0)[live].sum()) for b in (2, 4, 16, 8)]
    assert list(s.as_dict().values()) == want
