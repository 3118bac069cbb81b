"""The percentile clip's code at the edges of its counting: frames below one vector load, ragged and
unaligned sizes, one value only, the first and the last rank."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.uint8, np.uint16])
@pytest.mark.parametrize("h,w", [(8, 8), (9, 13), (97, 131), (700, 613)])
@pytest.mark.parametrize("pc", [0.001, 37.5, 99.0, 100.0])
def test_clip_code(dtype, h, w, pc):
    import torch

    import piv_b200 as P
    rng = np.random.default_rng(h + w)
    top = np.iinfo(dtype).max
    an = P.PivAnalyzer(P.PivConfig(windows=[8], final_iterations=1))
    cfg = P.PreprocessConfig(0.0, 0, 0.0, pc)
    for img in (rng.integers(0, top + 1, (h, w)).astype(dtype), np.full((h, w), top, dtype),
                np.minimum(rng.gamma(1.0, top / 40, (h, w)), top).astype(dtype)):
        code = np.sort(img, axis=None)[max(int(np.ceil(pc / 100 * img.size)), 1) - 1]
        want = (np.minimum(img, code).astype(np.float64) / top).astype(np.float32)
        for shift in (0, 1):  # an address that is not a multiple of 16 bytes
            buf = torch.zeros(img.nbytes + 64, dtype=torch.uint8, device="cuda")
            at = shift * dtype().itemsize
            buf[at:at + img.nbytes] = torch.from_numpy(img.reshape(-1).view(np.uint8)).cuda()
            torch.cuda.synchronize()
            f = an.frame(h, w).prepare_device(buf.data_ptr() + at, 0 if dtype == np.uint8 else 1, cfg)
            an.sync()
            assert np.array_equal(f.image, want)
