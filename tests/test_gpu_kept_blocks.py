"""Frames made and dropped for every pair (their device blocks are handed from frame to frame) give
the results of frames that are kept, from several threads at once and across sizes."""
import threading

import numpy as np
import pytest

from conftest import same_floats

pytestmark = pytest.mark.gpu


def _images(k):
    rng = np.random.default_rng(k)
    h, w = 96 + 17 * (k % 3), 130 + 31 * (k % 4)
    a = rng.random((h, w), dtype=np.float32)
    return a, np.roll(a, (1, 2), (0, 1))


def test_dropped_frames_leave_no_trace_in_later_ones():
    import piv_b200 as P
    cfg = P.PivConfig(windows=[32, 16], mask=P.MaskConfig(0.0, 0.01))
    pre = P.PreprocessConfig()
    keep = P.PivAnalyzer(cfg)
    want = {}
    frames = []
    for k in range(12):
        fa, fb = (keep.prepare(i, pre) for i in _images(k))
        frames.append((fa, fb))
        want[k] = keep.analyze(fa, fb).field
    bad = []

    def work(seed):
        an = P.PivAnalyzer(cfg)
        for k in np.random.default_rng(seed).permutation(24):
            a, b = _images(int(k) % 12)
            f = an.analyze(an.prepare(a, pre), an.prepare(b, pre)).field
            w = want[int(k) % 12]
            if not (np.array_equal(f.flags, w.flags) and same_floats(f.dx, w.dx) and same_floats(f.peak_ratio, w.peak_ratio)):
                bad.append(int(k))

    ts = [threading.Thread(target=work, args=(s,)) for s in range(4)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad
