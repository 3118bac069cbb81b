"""Flow statistics at the edges of their one-launch reduction (one block, several, looping blocks)
and from more host threads than the reduction has slots, against plain 64-bit sums."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _field(ny, nx, seed):
    rng = np.random.default_rng(seed)
    u, v = rng.normal(size=(2, ny, nx)).astype(np.float32)
    fl = (rng.random((ny, nx)) < 0.1).astype(np.uint8) * 2
    return u, v, fl


def _want(u, v, fl):
    ok = fl == 0
    e = 0.5 * (u.astype(np.float64) ** 2 + v.astype(np.float64) ** 2)[ok]
    return ok.sum(), e.mean() if ok.any() else np.nan


def _got(u, v, fl):
    import torch
    from piv_b200 import post
    d = [torch.from_numpy(a).cuda() for a in (u, v, fl)]
    w = torch.empty(u.shape, device="cuda")
    torch.cuda.synchronize()
    s = post.flow_stats(*d, 16, 1.0, vorticity=w)
    return s, w.cpu().numpy()


@pytest.mark.parametrize("ny,nx", [(1, 1), (2, 3), (16, 16), (1, 257), (257, 295), (400, 300)])
def test_sizes(ny, nx):
    f = _field(ny, nx, ny + nx)
    s, w = _got(*f)
    n, ke = _want(*f)
    fin = w[np.isfinite(w)].astype(np.float64)
    assert s.n_usable == n and s.n_vorticity == fin.size
    # the sums are in f64; the means are rounded once to f32
    assert np.isclose(s.ke_mean, ke, rtol=2e-7, equal_nan=True)
    if fin.size:
        assert np.isclose(s.vorticity_abs_mean, np.abs(fin).mean(), rtol=2e-7)


def test_more_callers_than_slots():
    fields = [_field(40 + k, 50, k) for k in range(24)]
    got = [None] * len(fields)

    def call(k):
        for _ in range(5):
            got[k] = _got(*fields[k])[0]

    ts = [threading.Thread(target=call, args=(k,)) for k in range(len(fields))]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for f, s in zip(fields, got):
        n, ke = _want(*f)
        assert s.n_usable == n and np.isclose(s.ke_mean, ke, rtol=2e-7)
