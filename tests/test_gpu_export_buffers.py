"""Device results into every kind of buffer: one kernel writes those that it can write as they are, the
copy commands serve the others (odd addresses, host memory, buffers that overlap), with the same values."""
import numpy as np
import pytest

from conftest import same_floats

pytestmark = pytest.mark.gpu

H, W = 128, 176


def _setup():
    import piv_b200 as P
    rng = np.random.default_rng(9)
    a = rng.random((H, W), dtype=np.float32)
    an = P.PivAnalyzer(P.PivConfig(windows=[32], final_iterations=1))
    frames = [an.prepare(i, P.RAW) for i in (a, np.roll(a, (1, 2), (0, 1)))]
    r = an.analyze(*frames)
    return an, frames, r


def _places(kind, bytes_each):
    """Five addresses (dx, dy, peak ratio, flags, summary), how to read them, and what keeps them alive."""
    import torch
    shift = {"aligned": 0, "by 4": 4, "by 1": 1, "by 2": 2, "flags by 3": 0, "pinned": 0, "pinned by 1": 1}[kind]
    host = kind.startswith("pinned")
    room = 512 + 256 * ((max(bytes_each) + 255) // 256)
    buf = torch.zeros(5 * room, dtype=torch.uint8, pin_memory=True) if host else torch.zeros(5 * room, dtype=torch.uint8,
                                                                                              device="cuda")
    at = [i * room + (256 - buf.data_ptr() % 256) % 256 + (3 if kind == "flags by 3" and i == 3 else shift) for i in range(5)]
    assert all(a + n <= (i + 1) * room for i, (a, n) in enumerate(zip(at, bytes_each)))

    def read():
        b = buf.cpu().numpy()
        return [b[a:a + n].tobytes() for a, n in zip(at, bytes_each)]

    return [buf.data_ptr() + a for a in at], read, buf


@pytest.mark.parametrize("kind,by_kernel", [("aligned", True), ("by 4", False), ("by 1", False), ("by 2", False),
                                            ("flags by 3", True), ("pinned", True), ("pinned by 1", False)])
def test_results_are_the_same_in_any_buffer(kind, by_kernel):
    """A shift by 4 is right for the floats but not for the 8-byte counts."""
    import torch
    an, frames, r = _setup()
    n = r.field.dx.size
    ptrs, read, _keep = _places(kind, [4 * n, 4 * n, 4 * n, n, 40])
    torch.cuda.synchronize()
    launches = []
    for _ in range(3):
        l0 = an.launches()
        an.analyze_device(*frames, *ptrs)
        an.sync()
        launches.append(an.launches() - l0)
        dx, dy, ppr, fl, counts = read()
        for got, want in ((dx, r.field.dx), (dy, r.field.dy), (ppr, r.field.peak_ratio)):
            assert same_floats(np.frombuffer(got, np.float32), want.ravel())
        assert np.array_equal(np.frombuffer(fl, np.uint8), r.field.flags.ravel())
        assert np.frombuffer(counts, np.uint64).tolist() == list(r.summary.as_dict().values())
    passes = 3  # placement, correlation, validation
    assert launches == [passes + by_kernel] * 3


def test_buffers_that_overlap_are_copied_in_order():
    """dx and dy into one place: the later one stands there, as with copy commands."""
    import torch
    an, frames, r = _setup()
    n = r.field.dx.size
    one = torch.zeros(n, device="cuda")
    ppr, fl = torch.zeros(n, device="cuda"), torch.zeros(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    an.analyze_device(*frames, one.data_ptr(), one.data_ptr(), ppr.data_ptr(), fl.data_ptr())
    an.sync()
    assert same_floats(one.cpu().numpy(), r.field.dy.ravel())
    assert same_floats(ppr.cpu().numpy(), r.field.peak_ratio.ravel())
