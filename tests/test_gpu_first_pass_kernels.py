"""First passes run copy-only correlation kernels; the general kernels, given the same whole-pixel origins,
give the same bits, for every window size, at odd cell counts, and with one frame off the pixel grid."""
import numpy as np
import pytest

from conftest import same_floats

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 12, 16, 24, 32, 48, 64, 96, 128])
@pytest.mark.parametrize("dh,dw", [(0, 0), (5, 17)])
def test_copy_kernels_match_the_general_ones(n, dh, dw):
    import piv_b200 as P
    rng = np.random.default_rng(n + dw)
    h, w = n + dh * (n // 8 + 1), n + dw * (n // 8 + 1)
    a = rng.random((h, w), dtype=np.float32)
    b = np.roll(a, (1, -2), (0, 1)) + np.float32(0.1) * rng.random((h, w), dtype=np.float32)
    an = P.PivAnalyzer(P.PivConfig(windows=[n], overlap=0.75, final_iterations=1))
    fa, fb = an.prepare(a, P.RAW), an.prepare(b, P.RAW)
    _, tr = an.analyze_traced(fa, fb)
    dx, dy, ppr, fl = an.correlate_origins(fa, fb, n, tr[0].origins)
    r = tr[0].raw
    assert np.array_equal(fl, r.flags.ravel())
    for got, want in ((dx, r.dx), (dy, r.dy), (ppr, r.peak_ratio)):
        assert same_floats(got, want.ravel())


@pytest.mark.parametrize("n", [16, 24, 64, 96])
def test_a_copied_frame_takes_no_value_from_outside_its_window(n):
    """Frame A's window on whole pixels, frame B's interpolated: a NaN beside A's window stays out of it."""
    import piv_b200 as P
    rng = np.random.default_rng(n)
    h = w = n + 8
    a = rng.random((h, w), dtype=np.float32)
    an = P.PivAnalyzer(P.PivConfig(windows=[n], final_iterations=1))
    org = np.array([[2, 3, 2.25, 3.5]], np.float32)
    fb = an.prepare(a, P.RAW)
    want = an.correlate_origins(an.prepare(a, P.RAW), fb, n, org)
    a2 = a.copy()
    a2[3 + n, :] = np.nan
    a2[:, 2 + n] = np.nan
    fa = an.frame(h, w).set_prepared(a2, np.nan_to_num(a2))
    got = an.correlate_origins(fa, fb, n, org)
    assert want[3][0] == 0
    for g, v in zip(got, want):
        assert same_floats(g.astype(np.float32), v.astype(np.float32))
