"""Performance cases of the framework: what a user has it do, through its public entry points.

Every case is one of six forms of use:

  device    frames that are already on the GPU: prepare both, analyse, field left on the GPU
            (PreparedFrame.prepare_device, PivAnalyzer.analyze_device)
  host      host frames through the plain calls, as the reference's own loop makes them
            (PivAnalyzer.prepare, PivAnalyzer.analyze)
  pipeline  a run of pinned host pairs through PivPipeline
  batch     a resident stretch of video, all its pairs in one PivBatch run
  serve     a burst of mixed requests submitted to one PivServer and collected
  series    post-processing of a series of fields: temporal median, spatial filter, flow statistics

Inputs are particle images rendered on the GPU from the seed alone (integer accumulation, so the
same seed gives the same bits): Gaussian blobs moved by a vortex with shear, noise, and clusters of
spurious particles that the validation has to find.

`exact` restates the analysis in 64 bits with plain torch.
"""
import math

import numpy as np
import torch

import piv_b200 as P
from piv_b200 import post

DEV = "cuda"
_DTYPES = {"u8": (0, torch.uint8, 255, np.uint8), "u16": (1, torch.uint16, 4095, np.uint16),
           "f32": (2, torch.float32, 1.0, np.float32)}
_state = {}


def _stream():
    """One side stream for all work, as a torch program that owns its stream has it."""
    if "stream" not in _state:
        _state["stream"] = torch.cuda.Stream()
    return _state["stream"].cuda_stream


# ------------------------------------------------------------------------------------- cases
def _device(name=None, **kw):
    c = dict(form="device", h=1024, w=1024, dtype="u16", windows="64,32", overlap=0.5, final_iterations=1, deform=False,
             precision="fp32", sigma=0.0, radius=0, clip=0.0, background=False, min_std=0.0, ppp=0.04, vmax=6.0,
             outliers=0.0)
    c.update(kw)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one 32 px pass over a small 8-bit pair (latency and launches)
        _device("pair 512 u8 one pass", h=512, w=512, dtype="u8", windows="32", ppp=0.05, vmax=2.8),
        # the default analysis of a 1080p camera pair: blur, local normalisation, 96, 64, 64 px
        _device("pair 1080p u8 default", h=1080, w=1920, dtype="u8", windows="96,64", final_iterations=2, sigma=1.0,
                radius=4, ppp=0.03),
        # background subtraction, percentile clip and deformed windows on a vortex
        _device("pair 1024 u16 deformed", windows="64,32,16", deform=True, clip=99.0, background=True, ppp=0.03,
                vmax=8.0),
        # the high-resolution analysis: four passes at 75 % overlap, spurious clusters
        _device("pair 4096 u16 four passes", h=4096, w=4096, windows="128,64,32,16", overlap=0.75, ppp=0.05, vmax=10.0,
                outliers=0.02),
        # an odd-sized float frame with a signal mask: window statistics, 48 and 24 px windows
        _device("pair 1437x1003 f32 masked", h=1003, w=1437, dtype="f32", windows="48,24", final_iterations=2,
                sigma=1.0, radius=4, min_std=0.01, ppp=0.02),
        # small windows on a dense 8-bit pair: 24 px, then 12 and 8 px
        _device("pair 2000x1501 u8 small windows", h=1501, w=2000, dtype="u8", windows="24,12,8", ppp=0.08, vmax=4.0),
        # the split-precision option, tensor cores allowed for the DFTs
        _device("pair 2048 u16 fp16x3", h=2048, w=2048, windows="64,32,16", precision="fp16x3"),
        # 64 sequential pairs of high-speed video, resident, in one run
        dict(_device("video 64 pairs", h=800, w=1280, windows="64,32"), form="batch", pairs=64, sequential=True),
        # the plain calls on host frames, new frame objects for every pair
        dict(_device("host pair 1024x768", h=768, w=1024), form="host"),
        # pinned host pairs of 1080p video with the default preprocessing, host to host
        dict(_device("pipeline 8 pairs 1080p", h=1080, w=1920, dtype="u8", windows="96,64", final_iterations=2, sigma=1.0,
                     radius=4, ppp=0.03), form="pipeline", pairs=8, depth=3),
        # a burst of requests of mixed sizes and schedules
        dict(form="serve", name="serve 24 mixed requests", requests=24, mix=0, dtype="u16", overlap=0.5, ppp=0.04,
             vmax=4.0),
        # a series of fields smoothed in time and space, statistics of every field
        dict(form="series", name="series 64 fields 118x66", nt=64, ny=66, nx=118, window=5, sigma=1.0),
    ]


_MAX_FLOPS = 9.0e10  # of the order of the largest listed case


def _odd(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    while True:
        form = rng.choice(["device"] * 5 + ["batch", "host", "pipeline", "serve", "series"])
        if form == "serve":
            return dict(form="serve", requests=rng.randint(6, 28), mix=rng.randint(1, 1000), dtype=rng.choice(["u8", "u16"]),
                        overlap=0.5, ppp=round(rng.uniform(0.03, 0.06), 3), vmax=round(rng.uniform(1.0, 5.0), 2))
        if form == "series":
            return dict(form="series", nt=rng.randint(5, 90), ny=_odd(rng, 24, 260), nx=_odd(rng, 24, 260),
                        window=rng.choice([3, 5, 7, 9]), sigma=round(rng.uniform(0.6, 2.0), 2))
        hi = {"device": 4096, "host": 2200, "pipeline": 2000, "batch": 1400}[form]
        h, w = _odd(rng, 400, hi), _odd(rng, 400, hi)
        dtype = rng.choice(["u8", "u16", "f32"])
        c = _device(h=h, w=w, dtype=dtype,
                    windows=rng.choice(["32", "64,32", "64,32,16", "96,64", "128,64,32", "48,24", "32,16", "24,12", "16,8",
                                        "96,48,24"]),
                    overlap=rng.choice([0.5, 0.5, 0.75]), final_iterations=rng.choice([1, 2]), deform=rng.random() < 0.25,
                    ppp=round(rng.uniform(0.03, 0.06), 3), vmax=round(rng.uniform(1.0, 8.0), 2),
                    outliers=rng.choice([0.0, 0.0, 0.02]))
        if rng.random() < 0.5:
            c.update(sigma=1.0, radius=4)
        if dtype != "f32" and rng.random() < 0.25:
            c.update(clip=99.0)
        if form == "device" and rng.random() < 0.25:
            c.update(background=True)
        if rng.random() < 0.2:
            c.update(min_std=0.01)
        if rng.random() < 0.1:
            c.update(precision=rng.choice(["bf16x3", "fp16x3"]))
        c["form"] = form
        if form == "batch":
            c.update(pairs=rng.randint(4, 64), sequential=rng.random() < 0.7)
        if form == "pipeline":
            c.update(pairs=rng.randint(4, 10), depth=rng.choice([2, 3]))
        if work(c)["flops"] <= _MAX_FLOPS:
            return c


# ------------------------------------------------------------------------------------- configuration
def _ints(s):
    return [int(v) for v in s.split(",")]


def _cfg(c):
    return P.PivConfig(windows=_ints(c["windows"]), overlap=c["overlap"], final_iterations=c["final_iterations"],
                       mask=P.MaskConfig(0.0, c["min_std"]), deform=c["deform"], precision=c["precision"])


def _pre(c):
    return P.PreprocessConfig(smooth_sigma=c["sigma"], normalize_radius=c["radius"], normalize_eps=0.02,
                              clip_percentile=c["clip"])


_SIZES = [(512, 512), (768, 1024), (2048, 2048)]
_SCHEDULES = ["32", "64,32", "64,32,16"]


def _requests(c):
    """The burst's requests: sizes and schedules from the mix, each of them present."""
    rnd = np.random.RandomState(c["mix"])
    out = []
    for i in range(c["requests"]):
        h, w = _SIZES[int(rnd.randint(3))]
        if c["mix"] and rnd.randint(4) == 0:  # drawn bursts hold odd sizes too
            h, w = h - int(rnd.randint(100)), w - int(rnd.randint(100))
        out.append(_device(h=h, w=w, dtype=c["dtype"], windows=_SCHEDULES[int(rnd.randint(3))], ppp=c["ppp"],
                           vmax=c["vmax"]))
    return out


# ------------------------------------------------------------------------------------- inputs
def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _render(h, w, x, y, sigma, amp):
    """Sum of Gaussian blobs, accumulated in integers of 2^-12 so that the order does not matter."""
    acc = torch.zeros(h * w, dtype=torch.int32, device=DEV)
    r = int(math.ceil(3.5 * float(sigma.max())))
    off = torch.arange(-r, r + 1, device=DEV)
    for s in range(0, x.numel(), 1 << 18):
        xs, ys, ss, am = (v[s:s + (1 << 18)] for v in (x, y, sigma, amp))
        cx, cy = torch.round(xs).long()[:, None] + off, torch.round(ys).long()[:, None] + off
        k = 0.5 / (ss * ss)
        ex = torch.exp(-((cx - xs[:, None]) ** 2) * k[:, None])
        ey = torch.exp(-((cy - ys[:, None]) ** 2) * k[:, None]) * am[:, None]
        v = (ey[:, :, None] * ex[:, None, :] * 4096.0).round().int()
        ok = ((cy >= 0) & (cy < h))[:, :, None] & ((cx >= 0) & (cx < w))[:, None, :]
        at = cy.clamp(0, h - 1)[:, :, None] * w + cx.clamp(0, w - 1)[:, None, :]
        acc.index_add_(0, at.reshape(-1), torch.where(ok, v, 0).reshape(-1))
    return acc.reshape(h, w).float() / 4096.0


def _quantise(f, dtype):
    _, tdt, full, _ = _DTYPES[dtype]
    if dtype == "f32":
        return f.clamp(0, 1).contiguous()
    v = torch.round(f * full).clamp(0, full)
    return v.to(torch.int32).to(tdt).contiguous()


def _frames(c, seed, count, h=None, w=None):
    """`count` frames of one flow: particles moved step by step by a vortex with shear."""
    h, w = h or c["h"], w or c["w"]
    g = _gen(seed)
    margin = 24.0
    n = int(c["ppp"] * (h + 2 * margin) * (w + 2 * margin))
    u = torch.rand(4, n, generator=g, device=DEV)
    q = torch.rand(4, generator=g, device=DEV).tolist()
    x, y = u[0] * (w + 2 * margin) - margin, u[1] * (h + 2 * margin) - margin
    sigma, amp = 0.5 + 0.5 * u[2], 0.45 + 0.55 * u[3]
    cx, cy = w * (0.3 + 0.4 * q[0]), h * (0.3 + 0.4 * q[1])
    rc = min(h, w) * 0.12
    a = c["vmax"] * (1.0 if q[2] < 0.5 else -1.0) * rc * 1.567
    ox, oy = 0.5 * (q[3] - 0.5) * c["vmax"], 0.3 * c["vmax"] * (q[2] - 0.5)

    def flow(px, py):
        rx, ry = px - cx, py - cy
        r2 = (rx * rx + ry * ry).clamp_min(1e-3)
        k = a * (1.0 - torch.exp(-r2 / (rc * rc))) / r2
        return ox - ry * k, oy + rx * k

    out = []
    for i in range(count):
        f = _render(h, w, x, y, sigma, amp)
        if i % 2 == 1 and c.get("outliers"):
            m = int(c["outliers"] * (h // 16) * (w // 16))
            v = torch.rand(4, m * 6, generator=g, device=DEV)
            bx, by = torch.rand(2, m, 1, generator=g, device=DEV)
            f = f + _render(h, w, ((bx * w).expand(m, 6).reshape(-1) + 16 * v[0]), (by * h).expand(m, 6).reshape(-1) + 16 * v[1],
                            0.5 + 0.5 * v[2], 0.6 + 0.4 * v[3])
        f = f + (4.0 / 255.0) * torch.randn(h, w, generator=g, device=DEV)
        if c.get("background"):
            f = f + 0.08 + 0.04 * torch.sin(torch.arange(w, device=DEV) * (2 * math.pi / w))
        out.append(_quantise(f, c["dtype"]))
        dx, dy = flow(x, y)
        for _ in range(2):
            dx, dy = flow(x + 0.5 * dx, y + 0.5 * dy)
        x, y = x + dx, y + dy
    return out


def _decode(t):
    """Samples as f32 intensities."""
    if t.dtype == torch.float32:
        return t
    return t.to(torch.int32).float() / (255.0 if t.dtype == torch.uint8 else 65535.0)


def _background(frames):
    return torch.stack([_decode(f) for f in frames]).amin(0).contiguous()


def _host(t, dtype):
    """A pinned numpy copy."""
    nd = _DTYPES[dtype][3]
    src = t.view(torch.int16) if t.dtype == torch.uint16 else t
    return src.cpu().pin_memory().numpy().view(nd)


def _pinned_out(g):
    f = [torch.empty(g.ny, g.nx).pin_memory().numpy() for _ in range(3)]
    return (*f, torch.empty(g.ny, g.nx, dtype=torch.uint8).pin_memory().numpy())


class _Device:
    """A view of device memory that the framework owns, for torch.as_tensor."""

    def __init__(self, ptr, shape, typestr, owner):
        self.__cuda_array_interface__ = {"data": (int(ptr), False), "shape": shape, "typestr": typestr, "version": 3}
        self.owner = owner


def _series(c, seed):
    """Fields of a slowly drifting vortex with noise; some vectors missing or not usable."""
    nt, ny, nx = c["nt"], c["ny"], c["nx"]
    g = _gen(seed)
    t, y, x = torch.meshgrid(*(torch.arange(n, device=DEV, dtype=torch.float32) for n in (nt, ny, nx)), indexing="ij")
    ph = 6.28 * torch.rand(2, generator=g, device=DEV)
    dx = 3 * torch.sin(x / 9 + ph[0] + 0.05 * t) * torch.cos(y / 9) + 0.2 * torch.randn(nt, ny, nx, generator=g, device=DEV)
    dy = -3 * torch.cos(x / 9 + ph[1] + 0.05 * t) * torch.sin(y / 9) + 0.2 * torch.randn(nt, ny, nx, generator=g, device=DEV)
    r = torch.rand(2, nt, ny, nx, generator=g, device=DEV)
    none = r[0] < 0.02
    dx, dy = dx.masked_fill(none, math.nan), dy.masked_fill(none, math.nan)
    flags = torch.where(none, 1, torch.where(r[1] < 0.03, 4, 0)).to(torch.uint8)
    usable = (flags == 0).to(torch.uint8)
    return dx.contiguous(), dy.contiguous(), flags, usable, (~none).to(torch.uint8)


# ------------------------------------------------------------------------------------- prepare and run
def prepare(case, seed):
    c = dict(case)
    s = {"case": c}
    if c["form"] == "series":
        dx, dy, fl, us, gate = _series(c, seed)
        s["in"] = (dx, dy, fl, us, gate)
        s["t"] = [torch.empty_like(dx) for _ in range(2)] + [torch.empty(dx.shape, dtype=torch.uint16, device=DEV)]
        s["s"] = [torch.empty_like(dx) for _ in range(2)] + [torch.empty(dx.shape, dtype=torch.uint16, device=DEV)]
        s["vort"] = torch.empty_like(dx)
        _stream()
        return s
    if c["form"] == "serve":
        reqs = _requests(c)
        srv = P.PivServer(memory_budget_bytes=8 << 30, max_in_flight=64)
        srv.reserve(2 << 30)
        cfgs = [_cfg(q) for q in reqs]
        grids = [P.Grid.new(q["h"], q["w"], f.windows[-1], f.overlap) for q, f in zip(reqs, cfgs)]
        total = sum(len(g) for g in grids)
        s["out"] = [torch.empty(total).pin_memory().numpy() for _ in range(3)] + [
            torch.empty(total, dtype=torch.uint8).pin_memory().numpy()]  # every request fills its part
        s["server"], s["work"], at = srv, [], 0
        for i, (q, cfg, g) in enumerate(zip(reqs, cfgs, grids)):
            a, b = _frames(q, seed * 1000 + i, 2)
            out = tuple(v[at:at + len(g)].reshape(g.ny, g.nx) for v in s["out"])
            s["work"].append((_host(a, q["dtype"]), _host(b, q["dtype"]), cfg, out))
            at += len(g)
        return s
    an = P.PivAnalyzer(_cfg(c))
    s["an"], s["pre"] = an, _pre(c)
    if c["form"] == "device":
        a, b = _frames(c, seed, 2)
        an.set_stream(_stream())
        g = an.output_grid(c["h"], c["w"])
        s["raw"], s["code"] = (a, b), _DTYPES[c["dtype"]][0]
        s["bg"] = _background((a, b)) if c["background"] else None
        s["frames"] = an.frame(c["h"], c["w"]), an.frame(c["h"], c["w"])
        s["out"] = [torch.empty(g.ny, g.nx, device=DEV) for _ in range(3)] + [
            torch.empty(g.ny, g.nx, dtype=torch.uint8, device=DEV), torch.zeros(5, dtype=torch.int64, device=DEV)]
    elif c["form"] == "host":
        s["raw"] = [_host(f, c["dtype"]) for f in _frames(c, seed, 2)]
    elif c["form"] == "pipeline":
        s["raw"] = [_host(f, c["dtype"]) for f in _frames(c, seed, c["pairs"] + 1)]
        s["pipe"] = P.PivPipeline(an, c["h"], c["w"], dtype=_DTYPES[c["dtype"]][3], cfg=s["pre"], depth=c["depth"])
        s["out"] = [_pinned_out(s["pipe"].grid) for _ in range(c["pairs"])]
    else:
        n = c["pairs"] + 1 if c["sequential"] else 2 * c["pairs"]
        batch = P.PivBatch(an, c["h"], c["w"], c["pairs"], sequential=c["sequential"], dtype=_DTYPES[c["dtype"]][3],
                           cfg=s["pre"])
        typestr = {"u8": "|u1", "u16": "<i2", "f32": "<f4"}[c["dtype"]]
        dst = torch.as_tensor(_Device(batch.input_device(), (n, c["h"], c["w"]), typestr, batch), device=DEV)
        for i, f in enumerate(_frames(c, seed, n)):
            dst[i].copy_(f.view(torch.int16) if f.dtype == torch.uint16 else f)
        batch.set_stream(_stream())
        g = batch.grid
        p = batch.outputs_device()
        s["batch"] = batch
        s["out"] = [torch.as_tensor(_Device(v, (c["pairs"], g.ny, g.nx), t, batch), device=DEV)
                    for v, t in zip(p, ("<f4", "<f4", "<f4", "|u1"))]
    return s


def run(s):
    c = s["case"]
    form = c["form"]
    if form == "device":
        (a, b), (fa, fb), out = s["raw"], s["frames"], s["out"]
        bg = None if s["bg"] is None else s["bg"].data_ptr()
        fa.prepare_device(a.data_ptr(), s["code"], s["pre"], bg)
        fb.prepare_device(b.data_ptr(), s["code"], s["pre"], bg)
        s["an"].analyze_device(fa, fb, *[t.data_ptr() for t in out])
        return out
    if form == "host":
        an, (a, b) = s["an"], s["raw"]
        fa, fb = an.prepare(a, s["pre"]), an.prepare(b, s["pre"])
        r = an.analyze(fa, fb)
        return [r.field.dx, r.field.dy, r.field.peak_ratio, r.field.flags, list(r.summary.as_dict().values())]
    if form == "pipeline":
        pipe, raw, got, pending = s["pipe"], s["raw"], [], []
        for i in range(c["pairs"]):
            if len(pending) == c["depth"]:
                got.append(pipe.wait(pending.pop(0)))
            pending.append(pipe.submit(raw[i], raw[i + 1], s["out"][i]))
        got += [pipe.wait(t) for t in pending]
        return [[r.field.dx, r.field.dy, r.field.peak_ratio, r.field.flags] for r in got]
    if form == "batch":
        s["batch"].run()
        return s["out"]
    if form == "serve":
        tickets = [s["server"].submit(a, b, cfg, P.RAW, out) for a, b, cfg, out in s["work"]]
        for t in tickets:
            s["server"].wait(t)
        return s["out"]
    dx, dy, fl, us, gate = s["in"]
    st = _stream()
    tx, ty, tn = s["t"]
    sx, sy, sn = s["s"]
    post.temporal_smooth(dx, dy, us, gate, tx, ty, tn, kernel="median", window=c["window"], stream=st)
    post.spatial_smooth(tx, ty, gate, sx, sy, sn, sigma=c["sigma"], stream=st)
    stats = [post.flow_stats(sx[t], sy[t], fl[t], 16, 0.01, vorticity=s["vort"][t], stream=st) for t in range(c["nt"])]
    table = np.array([[r.vorticity_mean, r.vorticity_abs_mean, r.ke_mean, r.ke_sum, r.coverage] for r in stats], np.float32)
    count = np.array([[r.n_usable, r.n_vorticity] for r in stats], np.int64)
    return [tx, ty, tn, sx, sy, sn, s["vort"], table, count]


# ------------------------------------------------------------------------------------- work
def _grid(h, w, n, overlap):
    step = max(int(np.float32(n) * (1.0 - np.float32(overlap)) + 0.5), 1)
    nx, ny = (w - n) // step + 1, (h - n) // step + 1
    return step, nx, ny, (w - n - (nx - 1) * step) // 2, (h - n - (ny - 1) * step) // 2


def _passes(c):
    v = _ints(c["windows"])
    return v + [v[-1]] * (c["final_iterations"] - 1)


def _pair_work(c):
    flops = 0.0
    for n in _passes(c):
        _, nx, ny, _, _ = _grid(c["h"], c["w"], n, c["overlap"])
        flops += nx * ny * (7.5 * n * n * math.log2(n * n) + 6 * n * (n / 2 + 1) + 2 * n * n)
    size = {"u8": 1, "u16": 2, "f32": 4}[c["dtype"]]
    return size * c["h"] * c["w"], 13 * nx * ny, flops


def work(case):
    c = dict(case)
    if c["form"] == "series":
        n = c["nt"] * c["ny"] * c["nx"]
        taps = (2 * max(math.ceil(2.5 * c["sigma"]), 1) + 1) ** 2
        return {"bytes": n * (8 + 3 + 20 + 4), "flops": n * (2.0 * c["window"] + 5.0 * taps + 20)}
    if c["form"] == "serve":
        parts = [_pair_work(q) for q in _requests(c)]
        return {"bytes": sum(2 * f + o for f, o, _ in parts), "flops": sum(p[2] for p in parts)}
    frame, out, flops = _pair_work(c)
    pairs = c.get("pairs", 1)
    frames = 2 * pairs if c["form"] in ("device", "host") or not c.get("sequential", True) else pairs + 1
    return {"bytes": frames * frame + pairs * out, "flops": pairs * flops}


# ------------------------------------------------------------------------------------- exact
_NOSIG, _LOWPPR, _OUTLIER, _REPLACED, _RANGE = 1, 2, 4, 8, 16
_INVALID = _NOSIG | _LOWPPR | _OUTLIER | _RANGE


def _x_decode(t, c):
    v = t.to(torch.int64) if t.dtype != torch.float32 else t
    if c["clip"] > 0 and t.dtype != torch.float32:
        srt = v.reshape(-1).sort().values
        v = v.clamp_max(int(srt[max(math.ceil(c["clip"] / 100 * v.numel()), 1) - 1]))
    return v.double() / (1.0 if t.dtype == torch.float32 else 255.0 if t.dtype == torch.uint8 else 65535.0)


def _x_box(v, n):
    """Sums over all n x n boxes from a 64-bit summed-area table."""
    s = torch.nn.functional.pad(v, (1, 0, 1, 0)).cumsum(0).cumsum(1)
    return s[n:, n:] - s[:-n, n:] - s[n:, :-n] + s[:-n, :-n]


def _x_prepare(t, c, bg):
    base = _x_decode(t, c)
    if bg is not None:
        base = (base - bg.double()).clamp_min(0)
    img = base
    h, w = img.shape
    if c["sigma"] > 0:
        r = max(math.ceil(3 * c["sigma"]), 1)
        k = torch.exp(-torch.arange(-r, r + 1, device=DEV).double() ** 2 / (2 * c["sigma"] ** 2))
        k = k / k.sum()
        iy = torch.arange(h, device=DEV)
        ix = torch.arange(w, device=DEV)
        img = sum(k[j + r] * img[:, (ix + j).clamp(0, w - 1)] for j in range(-r, r + 1))
        img = sum(k[j + r] * img[(iy + j).clamp(0, h - 1)] for j in range(-r, r + 1))
    if c["radius"] > 0:
        r = c["radius"]
        pad = lambda v: torch.nn.functional.pad(v, (r, r, r, r))  # noqa: E731
        n = _x_box(pad(torch.ones_like(img)), 2 * r + 1)
        mean = _x_box(pad(img), 2 * r + 1) / n
        var = _x_box(pad(img * img), 2 * r + 1) / n - mean * mean
        img = (img - mean) / (var.clamp_min(0).sqrt() + 0.02)
    return base, img


def _x_sample_field(dx, dy, grid, n, x, y):
    """The previous field at (x, y): bilinear over its finite vectors."""
    step, nx, ny, x0, y0 = grid
    fx = ((x - (x0 + (n - 1) / 2)) / step).clamp(0, nx - 1)
    fy = ((y - (y0 + (n - 1) / 2)) / step).clamp(0, ny - 1)
    ix, iy = fx.floor(), fy.floor()
    tx, ty = fx - ix, fy - iy
    ix, iy = ix.long(), iy.long()
    su = sv = sw = torch.zeros_like(fx)
    for oy, wy in ((0, 1 - ty), (1, ty)):
        for ox, wx in ((0, 1 - tx), (1, tx)):
            k = (iy + oy).clamp_max(ny - 1) * nx + (ix + ox).clamp_max(nx - 1)
            u, v, wt = dx[k], dy[k], wx * wy
            ok = (wt > 0) & u.isfinite() & v.isfinite()
            su = su + torch.where(ok, wt * u, 0.0)
            sv = sv + torch.where(ok, wt * v, 0.0)
            sw = sw + torch.where(ok, wt, 0.0)
    ok = sw > 0
    return torch.where(ok, su / sw, 0.0), torch.where(ok, sv / sw, 0.0)


def _x_place(origin, shift, mx):
    s = shift.clamp(-mx, mx)
    lo, hi = (-s).clamp_min(0), (mx - s).clamp_max(mx)
    a = torch.minimum(torch.maximum(origin - s / 2, lo), hi)
    return a, a + s


def _x_window(img, ox, oy, n):
    """Windows at (ox, oy): integer copy when both fractions are below 1e-4, else bilinear."""
    h, w = img.shape
    x0, y0 = ox.floor(), oy.floor()
    tx, ty = ox - x0, oy - y0
    whole = (tx < 1e-4) & (ty < 1e-4)
    tx, ty = torch.where(whole, 0.0, tx)[:, None, None], torch.where(whole, 0.0, ty)[:, None, None]
    r = torch.arange(n + 1, device=DEV)
    xs, ys = (x0.long()[:, None] + r).clamp(0, w - 1), (y0.long()[:, None] + r).clamp(0, h - 1)
    p = img[ys[:, :, None], xs[:, None, :]]
    top, bot = p[:, :n], p[:, 1:]
    row = top * (1 - ty) + bot * ty
    return row[:, :, :n] * (1 - tx) + row[:, :, 1:] * tx


def _x_deformed(img, gx, gy, k, n, sign):
    """Windows at (gx, gy) whose pixels are moved by half the blended corner displacements."""
    h, w = img.shape
    u = torch.arange(n, device=DEV).double() / (n - 1)
    uu, vv = u[None, None, :], u[None, :, None]
    blend = lambda d: ((1 - uu) * (1 - vv) * d[0][:, None, None] + uu * (1 - vv) * d[1][:, None, None]  # noqa: E731
                       + (1 - uu) * vv * d[2][:, None, None] + uu * vv * d[3][:, None, None])
    r = torch.arange(n, device=DEV).double()
    x = (gx[:, None, None] + r[None, None, :] + sign * 0.5 * blend([q[0] for q in k])).clamp(0, w - 1)
    y = (gy[:, None, None] + r[None, :, None] + sign * 0.5 * blend([q[1] for q in k])).clamp(0, h - 1)
    ix, iy = x.floor().long().clamp_max(w - 2), y.floor().long().clamp_max(h - 2)
    tx, ty = x - ix, y - iy
    flat, at = img.reshape(-1), iy * w + ix
    return ((1 - tx) * (1 - ty) * flat[at] + tx * (1 - ty) * flat[at + 1] + (1 - tx) * ty * flat[at + w]
            + tx * ty * flat[at + w + 1])


def _x_peaks(a, b):
    """Displacement of the correlation peak, peak ratio and whether both windows have content."""
    m, n = a.shape[0], a.shape[-1]
    a = a - a.mean((1, 2), keepdim=True)
    b = b - b.mean((1, 2), keepdim=True)
    ea, eb = (a * a).sum((1, 2)), (b * b).sum((1, 2))
    ok = (ea > 1e-12) & (eb > 1e-12)
    corr = torch.fft.irfft2(torch.fft.rfft2(a).conj() * torch.fft.rfft2(b), s=(n, n))
    corr = corr / torch.where(ok, (ea * eb).sqrt(), 1.0)[:, None, None]
    flat = corr.reshape(m, -1)
    best, at = flat.max(1)
    by, bx = at // n, at % n
    rows = torch.arange(m, device=DEV)
    hw = torch.zeros(m, dtype=torch.long, device=DEV)
    for sy, sx in ((1, 0), (-1, 0), (0, 1), (0, -1)):
        run = torch.ones(m, dtype=torch.bool, device=DEV)
        k = torch.zeros(m, dtype=torch.long, device=DEV)
        for j in range(n // 2):
            run = run & (corr[rows, (by + j * sy) % n, (bx + j * sx) % n] > 0.5 * best)
            if not bool(run.any()):
                break
            k = k + run
        hw = torch.maximum(hw, k)
    ex = torch.ceil(1.5 * hw.double()).clamp_min(2)
    ring = torch.nn.functional.max_pool2d(torch.nn.functional.pad(corr[:, None], (1, 1, 1, 1), mode="circular"), 3, 1)[:, 0]
    i = torch.arange(n, device=DEV)
    dist = lambda p: torch.minimum((i[None] - p[:, None]).abs(), n - (i[None] - p[:, None]).abs())  # noqa: E731
    far = torch.maximum(dist(by)[:, :, None], dist(bx)[:, None, :]) > ex[:, None, None]
    second = torch.where(far & (corr == ring), corr, -math.inf).amax((1, 2))
    ppr = torch.where(second > 0, (best / second).clamp_max(1000.0), 1000.0)

    def sub(lo, hi):
        pos = (lo > 0) & (best > 0) & (hi > 0)
        ll, lc, lh = (torch.where(pos, v, 1.0).log() for v in (lo, best, hi))
        d = torch.where(pos, (ll - lh) / (2 * (ll - 2 * lc + lh)), (lo - hi) / (2 * (lo - 2 * best + hi)))
        return torch.where(d.isfinite(), d.clamp(-0.5, 0.5), 0.0)

    sx = sub(corr[rows, by, (bx - 1) % n], corr[rows, by, (bx + 1) % n])
    sy = sub(corr[rows, (by - 1) % n, bx], corr[rows, (by + 1) % n, bx])
    wrap = lambda p: torch.where(p >= n // 2, p - n, p).double()  # noqa: E731
    return wrap(bx) + sx, wrap(by) + sy, ppr, ok


def _x_shifted(v, ny, nx, oy, ox, fill):
    """v[y + oy, x + ox], `fill` outside."""
    out = torch.full_like(v, fill)
    y0, y1, x0, x1 = max(0, -oy), min(ny, ny - oy), max(0, -ox), min(nx, nx - ox)
    if y0 < y1 and x0 < x1:
        out[y0:y1, x0:x1] = v[y0 + oy:y1 + oy, x0 + ox:x1 + ox]
    return out


def _x_medians(vals):
    """Median over the last axis of the finite entries (inf marks the others), and their count."""
    srt = vals.sort(-1).values
    n = vals.isfinite().sum(-1)
    lo = srt.gather(-1, ((n - 1).clamp_min(0) // 2)[..., None])[..., 0]
    hi = srt.gather(-1, (n // 2).clamp_max(vals.shape[-1] - 1)[..., None])[..., 0]
    return torch.where(n % 2 == 1, lo, 0.5 * (lo + hi)), n


def _x_validate(dx, dy, ppr, flags, ny, nx, vmax):
    sh = (ny, nx)
    u, v, p, f = dx.reshape(sh), dy.reshape(sh), ppr.reshape(sh), flags.reshape(sh)
    live = (f & _NOSIG) == 0
    f = f | torch.where(live & ((u * u + v * v).sqrt() > vmax), _RANGE, 0)
    f = f | torch.where(live & (p < 1.3), _LOWPPR, 0)

    def around(fl, radius):
        good = (fl & _INVALID) == 0
        offs = [(oy, ox) for oy in range(-radius, radius + 1) for ox in range(-radius, radius + 1) if oy or ox]
        mk = lambda q: torch.stack([_x_shifted(torch.where(good, q, math.inf), ny, nx, oy, ox, math.inf)  # noqa: E731
                                    for oy, ox in offs], -1)
        return mk(u), mk(v)

    nu, nv = around(f, 1)
    res = []
    for q, nb in ((u, nu), (v, nv)):
        med, n = _x_medians(nb)
        dev = torch.where(nb.isfinite(), (nb - med[..., None]).abs(), math.inf)
        res.append((q - med).abs() / (_x_medians(dev)[0] + 0.1))
    bad = ((f & _INVALID) == 0) & (n >= 2) & ((res[0] ** 2 + res[1] ** 2).sqrt() > 2.0)
    f = f | torch.where(bad, _OUTLIER, 0)
    need = ((f & _NOSIG) == 0) & ((f & _INVALID) != 0)
    ou, ov = torch.where(need, math.nan, u), torch.where(need, math.nan, v)
    for radius in (1, 2):
        nu, nv = around(f, radius)
        mu, n = _x_medians(nu)
        mv, _ = _x_medians(nv)
        take = need & (n > 0)
        ou, ov = torch.where(take, mu, ou), torch.where(take, mv, ov)
        f = f | torch.where(take, _REPLACED, 0)
        need = need & ~take
    return ou.reshape(-1), ov.reshape(-1), f.reshape(-1)


def _x_analyze(c, a, b, bg=None):
    """[dx, dy, peak ratio] of the pair's final field, in 64 bits."""
    (base_a, img_a), (base_b, img_b) = _x_prepare(a, c, bg), _x_prepare(b, c, bg)
    h, w = img_a.shape
    field = None
    for n in _passes(c):
        grid = _grid(h, w, n, c["overlap"])
        step, nx, ny, x0, y0 = grid
        cells = nx * ny
        k = torch.arange(cells, device=DEV)
        gx, gy = (x0 + (k % nx) * step).double(), (y0 + (k // nx) * step).double()
        mx, my = float(max(w - n - 1, 0)), float(max(h - n - 1, 0))
        at = lambda px, py: _x_sample_field(*field, px, py)  # noqa: E731
        sx, sy = at(gx + (n - 1) / 2, gy + (n - 1) / 2) if field else (torch.zeros_like(gx),) * 2
        ax, bx = _x_place(gx, sx, mx)
        ay, by = _x_place(gy, sy, my)
        signal = torch.ones(cells, dtype=torch.bool, device=DEV)
        if c["min_std"] > 0:
            for base, px, py in ((base_a, ax, ay), (base_b, bx, by)):
                qx, qy = (px + 0.5).floor().long().clamp(0, w - n), (py + 0.5).floor().long().clamp(0, h - n)
                mean = _x_box(base, n)[qy, qx] / (n * n)
                var = _x_box(base * base, n)[qy, qx] / (n * n) - mean * mean
                signal &= (mean >= 0) & (var.clamp_min(0).sqrt() >= c["min_std"])
        deform = c["deform"] and field is not None
        if deform:
            bx0, by0 = gx.clamp_max(mx), gy.clamp_max(my)
            corners = [at(bx0 + i, by0 + j) for j in (0, n - 1) for i in (0, n - 1)]
            mid = [sum(q[d] for q in corners) / 4 for d in (0, 1)]
        dx, dy, ppr = (torch.empty(cells, dtype=torch.float64, device=DEV) for _ in range(3))
        flags = torch.zeros(cells, dtype=torch.long, device=DEV)
        chunk = max(1, (1 << 24) // (n * n))
        for i in range(0, cells, chunk):
            j = slice(i, i + chunk)
            if deform:
                kk = [(q[0][j], q[1][j]) for q in corners]
                wa, wb = _x_deformed(img_a, bx0[j], by0[j], kk, n, -1.0), _x_deformed(img_b, bx0[j], by0[j], kk, n, 1.0)
                px, py = mid[0][j], mid[1][j]
            else:
                wa, wb = _x_window(img_a, ax[j], ay[j], n), _x_window(img_b, bx[j], by[j], n)
                px, py = bx[j] - ax[j], by[j] - ay[j]
            u, v, r, ok = _x_peaks(wa, wb)
            ok &= signal[j]
            dx[j], dy[j] = torch.where(ok, px + u, math.nan), torch.where(ok, py + v, math.nan)
            ppr[j] = torch.where(ok, r, 0.0)
            flags[j] = torch.where(ok, 0, _NOSIG)
        ou, ov, _ = _x_validate(dx, dy, ppr, flags, ny, nx, _passes(c)[0] / 2)
        field = (ou, ov, grid, n)
    return [v.reshape(ny, nx) for v in (ou, ov, ppr)]


def _x_series(c, seed):
    dx, dy, fl, us, gate = _series(c, seed)
    nt, ny, nx = dx.shape
    half = c["window"] // 2
    on = us.bool()

    def in_time(v):
        v = torch.where(on, v.double(), math.inf)
        st = torch.stack([torch.cat([torch.full((max(0, -k), ny, nx), math.inf, device=DEV, dtype=torch.float64),
                                     v[max(0, k):nt + min(0, k)],
                                     torch.full((max(0, k), ny, nx), math.inf, device=DEV, dtype=torch.float64)])
                          for k in range(-half, half + 1)], -1)
        med, n = _x_medians(st)
        return torch.where(gate.bool() & (n > 0), med, math.nan)

    tx, ty = in_time(dx), in_time(dy)
    r = max(math.ceil(2.5 * c["sigma"]), 1)
    i = torch.arange(-r, r + 1, device=DEV).double()
    k = torch.exp(-(i[:, None] ** 2 + i[None] ** 2) / (2 * c["sigma"] ** 2))
    ok = tx.isfinite() & ty.isfinite()
    conv = lambda v: torch.nn.functional.conv2d(v[:, None], k[None, None], padding=r)[:, 0]  # noqa: E731
    wsum = conv(ok.double())
    keep = gate.bool() & (wsum >= 0.25 * k.sum()) & (wsum > 0)
    sx, sy = (torch.where(keep, conv(torch.where(ok, v, 0.0)) / wsum, math.nan) for v in (tx, ty))
    good = sx.isfinite() & (((fl & _INVALID) == 0) | ((fl & _REPLACED) != 0))

    def slope(v, axis):
        v = torch.where(good & v.isfinite(), v * 100.0, math.nan)
        edge = torch.full_like(v.narrow(axis, 0, 1), math.nan)
        n = v.shape[axis]
        lo, hi = torch.cat([edge, v.narrow(axis, 0, n - 1)], axis), torch.cat([v.narrow(axis, 1, n - 1), edge], axis)
        d = (hi - lo) / 32.0
        d = torch.where(d.isnan() & lo.isfinite(), (v - lo) / 16.0, d)
        return torch.where(d.isnan() & hi.isfinite() & ~lo.isfinite(), (hi - v) / 16.0, torch.where(v.isnan(), math.nan, d))

    vort = slope(sx, 1) - slope(sy, 2)
    e = torch.where(good & sx.isfinite() & sy.isfinite(), 0.5 * ((sx * 100) ** 2 + (sy * 100) ** 2), 0.0)
    n = (good & sx.isfinite() & sy.isfinite()).sum((1, 2))
    nw = vort.isfinite().sum((1, 2))
    w = vort.nan_to_num()
    table = torch.stack([w.sum((1, 2)) / nw, w.abs().sum((1, 2)) / nw, e.sum((1, 2)) / n, e.sum((1, 2)) * 256.0,
                         n.double() / (ny * nx)], 1)
    return [tx, ty, None, sx, sy, None, vort, table, None]


def exact(case, seed):
    c = dict(case)
    if c["form"] == "series":
        return _x_series(c, seed)
    if c["form"] == "serve":
        got = [_x_analyze(q, *_frames(q, seed * 1000 + i, 2)) for i, q in enumerate(_requests(c))]
        return [torch.cat([g[k].reshape(-1) for g in got]) for k in range(3)] + [None]
    if c["form"] in ("device", "host"):
        a, b = _frames(c, seed, 2)
        return _x_analyze(c, a, b, _background((a, b)) if c["background"] else None) + [None, None]
    if c["form"] == "pipeline":
        f = _frames(c, seed, c["pairs"] + 1)
        return [_x_analyze(c, f[i], f[i + 1]) + [None] for i in range(c["pairs"])]
    n = c["pairs"] + 1 if c["sequential"] else 2 * c["pairs"]
    f = _frames(c, seed, n)
    pairs = [(i, i + 1) if c["sequential"] else (2 * i, 2 * i + 1) for i in range(c["pairs"])]
    got = [_x_analyze(c, f[i], f[j]) for i, j in pairs]
    return [torch.stack([g[k] for g in got]) for k in range(3)] + [None]
