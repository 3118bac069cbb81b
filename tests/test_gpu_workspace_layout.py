"""An analyzer's workspace is laid out for the pairs it was sized for, and its address comes back when
sizes fall in one class. A graph captured on one layout is never replayed on another: every call of a
mix of pair counts and frame sizes gives what an analyzer of its own gives."""
import ctypes

import numpy as np
import pytest

from conftest import same_floats

pytestmark = pytest.mark.gpu

# All workspaces below are smaller than 64 KiB, the class of a kept block.
SIZES = {"a": (256, 256), "b": (200, 232)}


def _config():
    import piv_b200 as P
    return P.PivConfig(windows=[64], final_iterations=1)


def _frames(an, size, pairs, seed):
    import piv_b200 as P
    h, w = SIZES[size]
    rng = np.random.default_rng(seed)
    out = []
    for k in range(pairs):
        a = rng.random((h, w), dtype=np.float32)
        b = np.roll(a, (1 + k % 3, 2 - k % 4), (0, 1)) + np.float32(0.2) * rng.random((h, w), dtype=np.float32)
        out.append((an.prepare(a, P.RAW), an.prepare(b, P.RAW)))
    return out


def _call(an, frames):
    """(dx, dy, peak ratio, flags, summaries) of all pairs through the batch call."""
    import torch

    import piv_b200 as P
    k = len(frames)
    g = an.output_grid(*frames[0][0].dim())
    out = [torch.full((k, g.ny, g.nx), 77.0, device="cuda") for _ in range(3)]
    fl = torch.full((k, g.ny, g.nx), 99, device="cuda", dtype=torch.uint8)
    sums = torch.full((k, 8), 5, device="cuda", dtype=torch.int64)
    torch.cuda.synchronize()
    arr = ctypes.c_void_p * k
    assert P.load_library().piv_analyze_batch_device(
        an._h, arr(*[a._h.value for a, _ in frames]), arr(*[b._h.value for _, b in frames]), k,
        *[t.data_ptr() for t in out], fl.data_ptr(), sums.data_ptr()) == 0
    an.sync()
    return [t.cpu().numpy() for t in (*out, fl, sums[:, :5])]


def _check(an, sets, steps):
    import piv_b200 as P
    want = {}
    for key in set(steps):
        fresh = P.PivAnalyzer(_config())
        size, k = key
        want[key] = _call(fresh, _frames(fresh, size, k, 100 * k + len(size)))
    for i, key in enumerate(steps):
        got = _call(an, sets[key])
        for x, y in zip(got[:3], want[key][:3]):
            assert same_floats(x, y), (i, key)
        for x, y in zip(got[3:], want[key][3:]):
            assert np.array_equal(x, y), (i, key)


def _sets(an, keys):
    return {(s, k): _frames(an, s, k, 100 * k + len(s)) for s, k in keys}


@pytest.mark.parametrize("steps", [
    [("a", 8), ("a", 1), ("a", 1), ("b", 1), ("a", 1)],
    [("a", 8), ("a", 2), ("a", 2), ("b", 1), ("a", 2)],
])
def test_a_graph_of_a_larger_workspace_is_not_replayed_in_a_smaller_one(steps):
    import piv_b200 as P
    an = P.PivAnalyzer(_config())
    _check(an, _sets(an, set(steps)), steps)


@pytest.mark.parametrize("seed", [0, 1])
def test_mixed_calls_match_analyzers_of_their_own(seed):
    import piv_b200 as P
    keys = [("a", 8), ("a", 1), ("a", 2), ("a", 5), ("b", 1), ("b", 8)]
    rng = np.random.default_rng(seed)
    steps = []
    for j in rng.integers(0, len(keys), 24):
        steps += [keys[j]] * int(rng.integers(1, 4))
    an = P.PivAnalyzer(_config())
    _check(an, _sets(an, keys), steps)
