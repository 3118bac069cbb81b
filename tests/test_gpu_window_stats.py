"""Signal mask from the strip-wise integral tables against plain 64-bit window statistics, at the
sizes where the strips (8 rows) and the column chunks (512) begin and end."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("h,w", [(8, 8), (9, 17), (15, 512), (16, 513), (67, 1030), (264, 90)])
def test_mask_matches_window_statistics(h, w):
    import piv_b200 as P
    rng = np.random.default_rng(h * 10007 + w)
    img = rng.random((h, w), dtype=np.float32)
    img *= (rng.random(((h + 5) // 6, (w + 5) // 6)) < 0.4).repeat(6, 0).repeat(6, 1)[:h, :w]
    n, thr = 8, 0.2
    an = P.PivAnalyzer(P.PivConfig(windows=[n], final_iterations=1, mask=P.MaskConfig(0.0, thr)))
    fr = an.prepare(img, P.RAW)
    x, y = rng.integers(0, w - n + 1, 400), rng.integers(0, h - n + 1, 400)
    x[:4], y[:4] = [0, 0, w - n, w - n], [0, h - n, 0, h - n]
    fl = an.correlate_origins(fr, fr, n, np.stack([x, y, x, y], 1).astype(np.float32))[3]
    sd = np.array([img[j:j + n, i:i + n].astype(np.float64).std() for i, j in zip(x, y)])
    sure = np.abs(sd - thr) > 1e-6  # both sides round mean and deviation to f32 (ulp 3e-8 here)
    assert sure.sum() > 350 or h * w < 200
    assert np.array_equal((fl[sure] & P.flags.NO_SIGNAL) != 0, sd[sure] < thr)
