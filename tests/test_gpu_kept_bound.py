"""The device blocks kept for later frames: the newest sizes stay within the bound, the oldest make
room, and a block larger than the bound goes straight back."""
import pytest

pytestmark = pytest.mark.gpu

MB = 1 << 20


def _free():
    import torch
    return torch.cuda.mem_get_info()[0]


def _taken(an, h, w):
    """Device memory that making a frame takes from the device (0: it had a kept block)."""
    before = _free()
    f = an.frame(h, w)
    taken = before - _free()
    f.close()
    return taken


def test_new_sizes_displace_the_oldest_blocks():
    import torch

    import piv_b200 as P
    torch.cuda.init()
    an = P.PivAnalyzer(P.PivConfig(windows=[32]))
    widths = [4200 + 64 * i for i in range(8)]  # about 50 MB each: five of them fit
    for w in widths:
        assert _taken(an, 3000, w) > 20 * MB
    for w in widths[-4:]:
        assert _taken(an, 3000, w) < 20 * MB
    big = 8300  # 276 MB
    assert _taken(an, big, big) > 256 * MB and _taken(an, big, big) > 256 * MB
    for w in widths[-4:]:
        assert _taken(an, 3000, w) < 20 * MB
    assert _taken(an, 3000, widths[0]) > 20 * MB


def test_an_admission_short_of_memory_gets_the_kept_blocks_first():
    """The injected failure stands for the allocator's: the kept blocks go back to the device before the
    request is given up or deferred, and the server then serves it."""
    import numpy as np
    import torch

    import piv_b200 as P
    torch.cuda.init()
    an = P.PivAnalyzer(P.PivConfig(windows=[32]))
    for w in (4200, 4300):
        _taken(an, 3000, w)
    rng = np.random.default_rng(5)
    a = rng.random((96, 128), dtype=np.float32)
    b = np.roll(a, (1, 2), (0, 1))
    sv = P.PivServer(memory_budget_bytes=1 << 30, max_in_flight=4)
    sv.wait(sv.submit(a, b, P.PivConfig(windows=[32])))
    before = _free()
    sv.fail_next_allocations(1)
    with pytest.raises(P.PivError):  # nothing else is in flight: the failure is final
        sv.wait(sv.submit(a, b, P.PivConfig(windows=[32])))
    assert _free() - before > 80 * MB
    sv.wait(sv.submit(a, b, P.PivConfig(windows=[32])))
    sv.close()
