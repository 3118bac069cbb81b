"""Frames, analyzers and their device blocks come and go while other work is queued or being captured:
a frame dropped by one thread never fails another's capture, and a block goes to its next user only
when the work that used it has completed."""
import threading

import numpy as np
import pytest

from conftest import same_floats

pytestmark = pytest.mark.gpu


def _images(seed, h=128, w=160):
    rng = np.random.default_rng(seed)
    a = rng.random((h, w), dtype=np.float32)
    return a, np.roll(a, (1, 2), (0, 1))


def _config():
    import piv_b200 as P
    return P.PivConfig(windows=[32], final_iterations=1, mask=P.MaskConfig(0.0, 0.01))


def _churn(stop, errors, regrow):
    """Makes, analyses and drops frames until told to stop."""
    import piv_b200 as P
    try:
        an = P.PivAnalyzer(_config())
        k = 0
        while not stop.is_set():
            k += 1
            a, b = _images(k % 7, 96 + 8 * (k % 3))
            if regrow:  # the staging block of 8-bit samples is too small for the f32 ones
                fa = an.frame(*a.shape).prepare((a * 255).astype(np.uint8))
                fa.prepare(a)
            else:
                fa = an.prepare(a)
            an.analyze(fa, an.prepare(b))
            if k % 5 == 0:
                an = P.PivAnalyzer(_config())
    except Exception as e:  # noqa: BLE001 - reported by the test
        errors.append(repr(e))


@pytest.mark.parametrize("regrow", [False, True])
def test_frames_dropped_during_another_analyzers_captures(regrow):
    """The second call on the same frames captures: two sets of frames in turn, two calls each."""
    import piv_b200 as P
    an = P.PivAnalyzer(_config())
    sets = [[an.prepare(i) for i in _images(s)] for s in (11, 12)]
    want = []
    for s in (11, 12):
        fresh = P.PivAnalyzer(_config())
        want.append(fresh.analyze(*[fresh.prepare(i) for i in _images(s)]).field)
    stop, errors = threading.Event(), []
    ts = [threading.Thread(target=_churn, args=(stop, errors, regrow)) for _ in range(2)]
    [t.start() for t in ts]
    try:
        for k in range(400):
            f = an.analyze(*sets[k // 2 % 2]).field
            w = want[k // 2 % 2]
            assert same_floats(f.dx, w.dx) and same_floats(f.dy, w.dy) and np.array_equal(f.flags, w.flags)
    finally:
        stop.set()
        [t.join() for t in ts]
    assert not errors


def test_frames_dropped_during_a_callers_relaxed_captures():
    import torch
    stop, errors = threading.Event(), []
    t = threading.Thread(target=_churn, args=(stop, errors, False))
    x = torch.zeros(1000, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    t.start()
    try:
        for _ in range(50):
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
                for _ in range(50):
                    x.add_(1.0)
            g.replay()
            s.synchronize()
    finally:
        stop.set()
        t.join()
    assert not errors
    torch.cuda.synchronize()
    assert float(x[0]) == 50 * 50


@pytest.mark.parametrize("stream", ["own", "caller's", "caller's, left"])
def test_blocks_of_dropped_frames_wait_for_queued_work(stream):
    """An analysis queued behind a long kernel gives its field although its frames are dropped, and
    others made and filled, before it has begun. Dropping the analyzer as well changes nothing."""
    import torch

    import piv_b200 as P
    h, w = 256, 320
    imgs = _images(3, h, w)
    cfg = _config()
    ref = P.PivAnalyzer(cfg)
    want = ref.analyze(*[ref.prepare(i, P.RAW) for i in imgs]).field
    raw = [torch.from_numpy(i).cuda() for i in imgs]
    other = [torch.from_numpy(i).cuda() for i in _images(4, h, w)]
    out = [torch.zeros(want.dx.shape, device="cuda") for _ in range(3)]
    fl = torch.zeros(want.dx.shape, device="cuda", dtype=torch.uint8)
    streams = [torch.cuda.Stream() for _ in range(2)]
    torch.cuda.synchronize()
    for drop_analyzer in (False, True):
        for _ in range(3):
            an = P.PivAnalyzer(cfg)
            if stream != "own":
                an.set_stream(streams[0].cuda_stream)
                with torch.cuda.stream(streams[0]):
                    torch.cuda._sleep(20_000_000)  # about 10 ms, then it ends by itself
            fa, fb = an.frame(h, w), an.frame(h, w)
            fa.prepare_device(raw[0].data_ptr(), P.api._lib.PIV_DTYPE_F32, P.RAW)
            fb.prepare_device(raw[1].data_ptr(), P.api._lib.PIV_DTYPE_F32, P.RAW)
            an.analyze_device(fa, fb, *[t.data_ptr() for t in out], fl.data_ptr())
            if stream == "caller's, left":
                an.set_stream(streams[1].cuda_stream)
            fa.close()
            fb.close()
            if drop_analyzer:
                an.close()
            an2 = P.PivAnalyzer(cfg)
            an2.set_stream(streams[1].cuda_stream)
            f2 = [an2.frame(h, w).prepare_device(o.data_ptr(), P.api._lib.PIV_DTYPE_F32, P.RAW) for o in other]
            an2.analyze(*f2)
            torch.cuda.synchronize()
            assert same_floats(out[0].cpu().numpy(), want.dx) and same_floats(out[1].cpu().numpy(), want.dy)
            assert same_floats(out[2].cpu().numpy(), want.peak_ratio)
            assert np.array_equal(fl.cpu().numpy(), want.flags)
            [t.zero_() for t in (*out, fl)]
            torch.cuda.synchronize()


def test_a_callers_captured_analysis_replays_while_frames_come_and_go():
    """Work captured by the caller may run at any later time: what it uses stays its own."""
    import torch

    import piv_b200 as P
    h, w = 192, 256
    an = P.PivAnalyzer(_config())
    s = torch.cuda.Stream()
    an.set_stream(s.cuda_stream)
    raw = [torch.from_numpy(i).cuda() for i in _images(5, h, w)]
    fa, fb = an.frame(h, w), an.frame(h, w)
    n = an.output_grid(h, w)
    out = [torch.zeros(n.ny, n.nx, device="cuda") for _ in range(3)]
    fl = torch.zeros(n.ny, n.nx, device="cuda", dtype=torch.uint8)

    def work():
        fa.prepare_device(raw[0].data_ptr(), P.api._lib.PIV_DTYPE_F32, P.PreprocessConfig())
        fb.prepare_device(raw[1].data_ptr(), P.api._lib.PIV_DTYPE_F32, P.PreprocessConfig())
        an.analyze_device(fa, fb, *[t.data_ptr() for t in out], fl.data_ptr())

    torch.cuda.synchronize()
    work()  # allocates
    an.sync()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        work()
    for seed in (5, 6, 7):
        a, b = _images(seed, h, w)
        ref = P.PivAnalyzer(_config())
        want = ref.analyze(ref.prepare(a), ref.prepare(b)).field  # its frames are dropped at once
        with torch.cuda.stream(s):
            raw[0].copy_(torch.from_numpy(a))
            raw[1].copy_(torch.from_numpy(b))
            g.replay()
        s.synchronize()
        assert same_floats(out[0].cpu().numpy(), want.dx) and same_floats(out[1].cpu().numpy(), want.dy)
        assert same_floats(out[2].cpu().numpy(), want.peak_ratio) and np.array_equal(fl.cpu().numpy(), want.flags)
