"""Pinning a launch variant by number: every number that was ever offered for a size stays accepted and
gives the same field, the next one is refused."""
import numpy as np
import pytest

from conftest import same_floats

pytestmark = pytest.mark.gpu

OFFERED = {8: 4, 12: 3, 16: 8, 24: 3, 32: 6, 48: 3, 64: 3, 96: 2, 128: 2}
OFFERED_DEFORMED = {8: 1, 12: 1, 16: 2, 24: 1, 32: 2, 48: 1, 64: 2, 96: 1, 128: 1}


@pytest.mark.parametrize("deform", [False, True])
@pytest.mark.parametrize("n", sorted(OFFERED))
def test_numbers_that_were_offered_stay_accepted(n, deform):
    import piv_b200 as P
    rng = np.random.default_rng(n)
    a = rng.random((2 * n, 2 * n + 6), dtype=np.float32)
    an = P.PivAnalyzer(P.PivConfig(windows=[n], overlap=0.75, final_iterations=2, deform=deform))
    f = [an.prepare(i, P.RAW) for i in (a, np.roll(a, (1, 1), (0, 1)))]
    want = an.analyze(*f).field
    offered = (OFFERED_DEFORMED if deform else OFFERED)[n]
    for v in range(offered):
        an.set_variant(n, v)
        got = an.analyze(*f).field
        assert np.array_equal(got.flags, want.flags)
        assert same_floats(got.dx, want.dx) and same_floats(got.dy, want.dy) and same_floats(got.peak_ratio, want.peak_ratio)
    if deform or offered >= P.PivAnalyzer.num_variants(n):
        with pytest.raises(P.PivError):
            an.set_variant(n, offered)
    with pytest.raises(P.PivError):
        an.set_variant(n, -1)
