"""Local normalisation at the edges of its 32 x 24 tiles, for the unrolled and the general radius, against
plain 64-bit window statistics."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _want(v, r, eps):
    h, w = v.shape
    v = v.astype(np.float64)
    out = np.empty((h, w))
    for y in range(h):
        for x in range(w):
            box = v[max(y - r, 0):y + r + 1, max(x - r, 0):x + r + 1]
            out[y, x] = (v[y, x] - box.mean()) / (box.std() + eps)
    return out


@pytest.mark.parametrize("r", [1, 4, 9])
@pytest.mark.parametrize("h,w", [(8, 8), (24, 32), (25, 33), (49, 70)])
@pytest.mark.parametrize("scale", [1.0, 1e-12])
def test_normalisation(h, w, r, scale):
    import piv_b200 as P
    rng = np.random.default_rng(h * w + r)
    img = (rng.random((h, w)) * scale).astype(np.float32)
    img[: h // 2, : w // 3] = np.float32(0.25 * scale)  # flat parts: deviation 0
    eps = 0.02 * scale
    an = P.PivAnalyzer(P.PivConfig(windows=[8], final_iterations=1))
    got = an.prepare(img, P.PreprocessConfig(0.0, r, eps)).image
    # mean, deviation and their differences round to f32: 1.2e-7 of the values (at most `scale`) over a
    # divisor of at least eps, and 4 roundings of the quotient itself
    want = _want(img, r, float(np.float32(eps)))
    assert np.all(np.abs(got - want) <= 1.2e-7 * scale / eps + 2.4e-7 * np.abs(want))
