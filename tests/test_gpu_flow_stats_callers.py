"""Flow statistics from many host threads at once, each on a stream of its own, and after a call that
failed: every call has a place of its own for its sums and gives those of a call made alone."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(ny=60, nx=70, seed=0):
    import torch
    rng = np.random.default_rng(seed)
    u, v = (torch.from_numpy(rng.normal(size=(ny, nx)).astype(np.float32)).cuda() for _ in range(2))
    return u, v, torch.zeros(ny, nx, dtype=torch.uint8, device="cuda")


def test_many_callers_at_once():
    import torch
    from piv_b200 import post
    fields = [_field(30 + 9 * k, 41 + 3 * k, k) for k in range(40)]
    want = [post.flow_stats(*f, 16, 1.0) for f in fields]
    torch.cuda.synchronize()
    start, bad = threading.Barrier(len(fields)), []

    def call(k):
        s = torch.cuda.Stream()
        start.wait()
        for _ in range(20):
            if post.flow_stats(*fields[k], 16, 1.0, stream=s.cuda_stream) != want[k]:
                bad.append(k)

    ts = [threading.Thread(target=call, args=(k,)) for k in range(len(fields))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    assert not bad


def test_a_call_refused_during_a_capture_leaves_later_calls_right():
    """The call waits for its stream, which a capture does not allow."""
    import torch

    import piv_b200 as P
    from piv_b200 import post
    f = _field()
    want = post.flow_stats(*f, 16, 1.0)
    for _ in range(3):
        s = torch.cuda.Stream()
        g = torch.cuda.CUDAGraph()
        with pytest.raises(RuntimeError):  # the capture that the refused call was made in
            with torch.cuda.graph(g, stream=s, capture_error_mode="relaxed"):
                with pytest.raises(P.PivError):
                    post.flow_stats(*f, 16, 1.0, stream=s.cuda_stream)
        assert post.flow_stats(*f, 16, 1.0) == want
