"""Local normalisation of frames without variance. A power of two is exact in every step of the window
statistics, whatever the number of pixels, so the deviation is exactly zero: 0 / 0 without an epsilon,
0 with one."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("value", [0.25, 1.0, 2.0 ** -20])
@pytest.mark.parametrize("radius", [1, 4, 9, 16])
def test_a_frame_of_one_value_has_no_deviation(value, radius):
    import piv_b200 as P
    an = P.PivAnalyzer(P.PivConfig(windows=[16]))
    x = np.full((70, 90), value, np.float32)
    got = an.frame(70, 90).prepare(x, P.PreprocessConfig(0.0, radius, 0.0, 0.0)).image
    assert np.isnan(got).all()
    got = an.frame(70, 90).prepare(x, P.PreprocessConfig(0.0, radius, 0.02, 0.0)).image
    assert (got == 0).all()
