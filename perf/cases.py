"""The work whose speed this repository is held to: its listed cases, more
cases of the same ranges, their inputs, one pass of each through the public
entry points, the work a pass cannot do without, and 64-bit references.

Four kinds of case:

* ``mc``     -- ``api.Pipeline``: the Monte Carlo loop on one DEM, which is
  what the ``drainage`` program and the benchmark run (single and batched
  steps, CPU-compatible and exact fill, with and without the learned start);
* ``mixed``  -- ``batch.Batch``: uneven DEMs side by side, each job with a
  filter of its own;
* ``stages`` / ``field`` -- the stage calls one after another, as a host
  application that replaces the reference's stages one by one makes them;
* ``infer`` / ``train`` -- the warm-start network on a grid, and one of its
  training steps (forward, loss, backward, update).

Terrain is seeded fractional Brownian motion with pits (and flat lakes where
a case says so), its stream raster the cells whose D8 flow accumulation
exceeds a threshold: the benchmark's recipe, made on the GPU.
"""
import math

import numpy as np
import torch

from cageo_gb300 import api, batch, learned

CELL = 10.0
NODATA = -9999.0
DRY_THRESHOLD = 0.005  # metres: the warm start's dry threshold in the benchmark


def _mc(name, w, h, count, **kw):
    c = dict(name=name, kind="mc", w=w, h=h, count=count, batch=1, mode="cpu", learned=False,
             model="gaussian", range_m=60.0, sigma=1.5, hurst=0.8, lo=0.0, hi=300.0,
             pits=max(w * h // 3400, 1), threshold=2000, plateaus=0.0, ids="ones", holes=0)
    c.update(kw)
    return c


def listed():
    return [
        # Every stage call on an odd tile of the mixed batch, with NODATA
        # holes in the DEM and a stream id per network: launch latency.
        _mc("stages 257x1013", 257, 1013, 1, kind="stages", pits=130, ids="networks", holes=40,
            threshold=500),
        # A survey strip's error field (noise, full 2D filter, realistic DEM).
        _mc("field 3001x401 exponential", 3001, 401, 1, kind="field", model="exponential",
            range_m=75.0, sigma=2.0),
        # The stage calls in the reference GPU path's semantics on a mid-size
        # tile (exact fill, GPU routing order, dead ends as errors).
        _mc("stages 1500x733 exact", 1500, 733, 1, kind="stages", mode="exact", ids="networks"),
        # A catchment study on a small map: the 512^2 workload's 20
        # realizations, one after another (latency and launches).
        _mc("mc 512x512 x20", 512, 512, 20, lo=80.0, hi=180.0, pits=200, threshold=500),
        # An ordinary map, realizations one at a time: the 4096^2 workload.
        _mc("mc 4096x4096 x4", 4096, 4096, 4, hurst=0.75, pits=2000),
        # The throughput configuration: the benchmark's 8192^2 workload in
        # batched steps.
        _mc("mc 8192x8192 batch 8", 8192, 8192, 8, batch=8, pits=20000),
        # The largest map: 16384^2 with a fifth of it in flat lakes, 90 m.
        _mc("mc 16384x16384 lakes", 16384, 16384, 1, range_m=90.0, pits=80000, plateaus=0.2),
        # The exact fill (the reference GPU path's semantics) in the loop.
        _mc("mc 4096x4096 exact x4", 4096, 4096, 4, mode="exact", hurst=0.75, pits=2000),
        # The learned warm start in the loop: inference, verified fill.
        _mc("mc 2048x2048 learned x4", 2048, 2048, 4, mode="exact", learned=True, pits=1250),
        # Jobs round-robin over a 2048^2 DEM and three uneven tiles, range
        # and standard deviation of each job drawn: the mixed batch.
        dict(name="mixed batch x16", kind="mixed", scale=1.0, jobs=16),
        # The network's depths on a map with odd sides.
        dict(name="infer 3001x2003", kind="infer", w=3001, h=2003, hurst=0.8, hi=100.0),
        # A training step at the training program's batch and crop.
        dict(name="train 16x128x128", kind="train", w=128, h=128, b=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mc", "mc", "mc", "mc", "exact", "learned", "stages", "stages", "field",
                       "mixed", "infer", "train"])
    if kind == "mixed":
        return dict(kind="mixed", scale=round(rng.uniform(0.2, 1.0), 3), jobs=rng.randint(4, 16))
    if kind == "infer":
        return dict(kind="infer", w=_log(rng, 100, 6000), h=_log(rng, 100, 6000), hurst=0.8,
                    hi=round(rng.uniform(30.0, 300.0), 1))
    if kind == "train":
        return dict(kind="train", w=rng.randint(40, 160), h=rng.randint(40, 160),
                    b=rng.randint(2, 24))
    big = {"mc": 9000, "exact": 6000, "learned": 3000}.get(kind, 4000)
    w, h = _log(rng, 128, big), _log(rng, 128, big)
    n = w * h
    c = _mc("", w, h, max(1, min(20, int(4e7 / n))), sigma=round(rng.uniform(1.0, 3.0), 2),
            hurst=round(rng.uniform(0.7, 0.85), 2), hi=round(rng.uniform(100.0, 300.0), 1),
            pits=max(n // rng.randint(1300, 8000), 1), threshold=rng.choice([500, 1000, 2000]),
            ids=rng.choice(["ones", "networks"]))
    del c["name"]
    if kind in ("stages", "field"):
        c.update(kind=kind, count=1)
    c["mode"] = {"exact": "exact", "learned": "exact"}.get(kind, "cpu")
    if kind == "stages":
        c["mode"] = rng.choice(["cpu", "exact"])
    c["learned"] = kind == "learned"
    if rng.random() < (0.5 if kind == "field" else 0.15) and n < 3e6:
        c.update(model="exponential", range_m=round(rng.uniform(30.0, 120.0), 1))
    else:
        c["range_m"] = rng.choice([60.0, 90.0, round(rng.uniform(30.0, 120.0), 1)])
    if rng.random() < 0.3:
        c["plateaus"] = 0.2
    if rng.random() < 0.3:
        c["holes"] = rng.randint(1, 200)
    if kind == "mc" and rng.random() < 0.5:
        c["batch"] = max(2, min(8, c["count"]))
        c["count"] = c["batch"] * max(1, c["count"] // c["batch"])
    return c


# ---- inputs -----------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _fbm(w, h, hurst, lo, hi, g):
    spec = torch.fft.rfft2(torch.randn((h, w), device="cuda", generator=g))
    ky = torch.fft.fftfreq(h, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(w, device="cuda")[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k.pow_(-(hurst + 1.0))
    amp[0, 0] = 0.0
    spec *= amp
    del amp, k
    z = torch.fft.irfft2(spec, s=(h, w))
    del spec
    z -= z.min()
    z *= (hi - lo) / float(z.max())
    return z.add_(lo)


def _pits(dem, count, g):
    """Cones 0.5-3 m deep, 1-4 cells wide; where they overlap, the deepest."""
    h, w = dem.shape
    y = torch.randint(1, h - 1, (count,), device="cuda", generator=g)
    x = torch.randint(1, w - 1, (count,), device="cuda", generator=g)
    depth = torch.rand(count, device="cuda", generator=g) * 2.5 + 0.5
    radius = torch.randint(1, 5, (count,), device="cuda", generator=g)
    dent = torch.zeros(h * w, device="cuda")
    for dy in range(-4, 5):
        for dx in range(-4, 5):
            dist = math.hypot(dx, dy)
            yy, xx = y + dy, x + dx
            ok = (radius >= dist) & (yy >= 0) & (yy < h) & (xx >= 0) & (xx < w)
            cone = depth * (1.0 - dist / (radius + 1.0))
            dent.scatter_reduce_(0, (yy * w + xx)[ok], cone[ok], "amax")
    dem -= dent.view(h, w)


def _lakes(dem, share, seed):
    """Discs of 50-400 cells radius (less on small grids), each at the
    elevation of its centre, covering about `share` of the grid."""
    h, w = dem.shape
    rng = np.random.default_rng(seed)
    top = min(400, max(min(w, h) // 6, 4))
    lo = min(50, max(top // 8, 2))
    mean = math.pi * (top ** 3 - lo ** 3) / (3.0 * max(top - lo, 1))
    for _ in range(max(1, int(-math.log(1.0 - share) * w * h / mean))):
        r, y, x = int(rng.integers(lo, top + 1)), int(rng.integers(h)), int(rng.integers(w))
        y0, y1, x0, x1 = max(y - r, 0), min(y + r + 1, h), max(x - r, 0), min(x + r + 1, w)
        yy = torch.arange(y0, y1, device="cuda")[:, None] - y
        xx = torch.arange(x0, x1, device="cuda")[None, :] - x
        part = dem[y0:y1, x0:x1]
        part.copy_(torch.where(yy * yy + xx * xx <= r * r, dem[y, x].clone(), part))


def _streams(dem, threshold, ids):
    """1.0 (or an id per stream network) where the D8 accumulation of the
    filled DEM exceeds `threshold` cells, NODATA elsewhere."""
    h, w = dem.shape
    n = h * w
    dirs = api.route_d8(api.pitfill(dem.clone(), mode=api.FILL_EXACT), mode=api.ROUTE_GPU_ORDER)
    step = dirs[..., 1].to(torch.int64)
    step *= w
    step += dirs[..., 0]
    y = torch.arange(h, device="cuda")[:, None] + dirs[..., 1]
    x = torch.arange(w, device="cuda")[None, :] + dirs[..., 0]
    ends = (y < 0) | (y >= h) | (x < 0) | (x >= w) | (step == 0)
    del x, y, dirs
    ptr = (torch.arange(n, device="cuda") + step.view(-1)).masked_fill_(ends.view(-1), -1)
    del step
    root = torch.where(ptr < 0, torch.arange(n, device="cuda"), ptr) if ids == "networks" else None
    acc = torch.ones(n, dtype=torch.int32, device="cuda")
    while True:  # path doubling: acc counts the cells at most 2^k steps upstream
        live = (ptr >= 0).nonzero().view(-1)
        if live.numel() == 0:
            break
        to = ptr[live]
        add = acc[live]
        acc.index_add_(0, to, add)
        ptr[live] = ptr[to]
        if root is not None:
            root = root[root]
    out = torch.full((h, w), NODATA, device="cuda")
    ids_grid = torch.ones(n, device="cuda") if root is None else (root % 1009 + 1).float()
    mask = (acc > threshold).view(h, w)
    out[mask] = ids_grid.view(h, w)[mask]
    return out


def _terrain(c, seed):
    g = _generator(seed)
    dem = _fbm(c["w"], c["h"], c["hurst"], c["lo"], c["hi"], g)
    _pits(dem, c["pits"], g)
    if c["plateaus"]:
        _lakes(dem, c["plateaus"], seed)
    streams = _streams(dem, c["threshold"], c["ids"])
    if c["holes"]:
        at = torch.randint(0, dem.numel(), (c["holes"],), device="cuda", generator=g)
        dem.view(-1)[at] = NODATA
    return dem, streams


def _model(c):
    return api.FILTER_GAUSSIAN if c["model"] == "gaussian" else api.FILTER_EXPONENTIAL


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "mixed":
        grids = []
        for k, (w, h) in enumerate([(2048, 2048), (257, 1013), (1500, 733), (3001, 401)]):
            w, h = max(int(w * c["scale"]), 64), max(int(h * c["scale"]), 64)
            grids.append(_terrain(_mc("", w, h, 1), seed * 4 + k))
        b = batch.Batch(grids, cell_size=CELL, seed=seed)
        st = dict(c=c, batch=b, jobs=batch.mixed_jobs(4, c["jobs"], seed),
                  counts=[torch.empty_like(d) for d, _ in grids])
    elif kind == "infer":
        v = _fbm(c["w"], c["h"], c["hurst"], 0.0, c["hi"], _generator(seed))
        _pits(v, max(v.numel() // 3400, 1), _generator(seed + 1))
        st = dict(c=c, v=v, params=torch.from_numpy(learned.load_params()).cuda())
    elif kind == "train":
        g = _generator(seed)
        shape = (c["b"], c["h"], c["w"])
        v = torch.stack([_fbm(c["w"], c["h"], 0.8, 0.0, 12.0, g) for _ in range(c["b"])])
        feat = api.ws_features(v.contiguous())
        target = (v.mean() - v).clamp_(0.0, 2.0)
        params = torch.from_numpy(learned.load_params()).cuda()
        n = params.numel()
        st = dict(c=c, feat=feat, target=target, params=params,
                  m=torch.randn(n, device="cuda", generator=g) * 1e-3,
                  v=torch.rand(n, device="cuda", generator=g) * 1e-4 + 1e-6,
                  dy=torch.empty(shape, device="cuda"), loss=torch.zeros(1, device="cuda"),
                  grad=torch.empty_like(params),
                  tmp1=torch.empty((c["b"], 32, c["h"], c["w"]), device="cuda"),
                  wflip=torch.empty(9216, device="cuda"))
        st["tmp2"] = torch.empty_like(st["tmp1"])
    elif kind in ("stages", "field"):
        dem, streams = _terrain(c, seed)
        r = api.filter_radius(c["range_m"], CELL)
        st = dict(c=c, dem=dem, streams=streams, r=r, seed=seed,
                  taps=api.filter_build(_model(c), c["range_m"], CELL, r),
                  noise=torch.empty_like(dem), counts=torch.empty_like(dem))
    else:
        dem, streams = _terrain(c, seed)
        p = api.Pipeline(dem, streams, cell_size=CELL, filter_model=_model(c),
                         practical_range=c["range_m"], error_stddev=c["sigma"], seed=seed,
                         fill_mode=api.FILL_EXACT if c["mode"] == "exact" else api.FILL_CPU_COMPAT)
        if c["batch"] > 1:
            p.run(0, 1)  # a program that batches has timed single steps before
            p.set_batch(c["batch"])
        if c["learned"]:
            p.set_warmstart(learned.load_params(), DRY_THRESHOLD)
        st = dict(c=c, pipe=p, counts=torch.empty_like(dem))
        del dem, streams
    torch.cuda.empty_cache()  # the generator's scratch: the pipeline allocates outside torch's pool
    return st


# ---- one pass ---------------------------------------------------------------
def run(state):
    return {"mc": _run_mc, "mixed": _run_mixed, "stages": _run_stages, "field": _run_field,
            "infer": _run_infer, "train": _run_train}[state["c"]["kind"]](state)


def _run_mc(s):
    p = s["pipe"]
    p.reset_counts()
    p.run(0, s["c"]["count"])
    return p.counts(out=s["counts"])


def _run_mixed(s):
    b = s["batch"]
    for p in b.pipes:
        p.reset_counts()
    b.run(s["jobs"])
    return [p.counts(out=t) for p, t in zip(b.pipes, s["counts"])]


def _run_field(s):
    c = s["c"]
    api.noise_philox(s["noise"], s["seed"], 0, 0.0, c["sigma"])
    v = api.convolve(s["noise"], _model(c), s["taps"], s["r"])
    api.realistic_dem(s["dem"], v)
    return {"noise": s["noise"], "v": v}


def _run_stages(s):
    exact_mode = s["c"]["mode"] == "exact"
    out = _run_field(s)
    v = out["v"]
    api.stream_burn(v, s["streams"])
    filled = api.pitfill(v, mode=api.FILL_EXACT if exact_mode else api.FILL_CPU_COMPAT)
    dirs, flat = api.route_d8(filled, with_flatdist=True,
                              mode=api.ROUTE_GPU_ORDER if exact_mode else api.ROUTE_CPU_COMPAT)
    labels = api.trace(dirs, s["streams"],
                       mode=api.TRACE_DEAD_END_ERROR if exact_mode else api.TRACE_CPU_COMPAT)
    api.border_accumulate(labels, s["counts"].zero_())
    out.update(filled=filled, dirs=dirs, flat=flat, labels=labels, counts=s["counts"])
    return out


def _run_infer(s):
    return api.ws_infer(s["params"], s["v"], DRY_THRESHOLD, want_warm=False, want_depth=True)[1]


def _run_train(s):
    p, m, v = s["params"].clone(), s["m"].clone(), s["v"].clone()
    a1, a2, out = api.ws_forward(p, s["feat"])
    api.ws_mse(out, s["target"], s["dy"], s["loss"].zero_(), margin=3)
    api.ws_backward(p, s["feat"], a1, a2, s["dy"], s["grad"].zero_(), s["tmp1"], s["tmp2"],
                    s["wflip"])
    api.ws_adam(p, s["grad"], m, v, 2e-3, 50)
    return {"a1": a1, "a2": a2, "out": out, "loss": s["loss"], "grad": s["grad"], "params": p,
            "m": m, "v": v}


# ---- the work a pass cannot do without ------------------------------------------
def _filter_flops(c):
    taps = 2 * math.ceil(c["range_m"] / CELL * 2.5) + 1
    return 4 * taps if c["model"] == "gaussian" else 2 * taps * taps


def work(case):
    """Bytes: a realization reads the DEM and the streams and adds to the
    count grid (4 + 4 + 8 a cell); a stage call reads its inputs and writes
    its outputs.  Flops: the filter's products and sums, the network's."""
    c, kind = case, case["kind"]
    if kind == "mixed":
        by = fl = 0.0
        shapes = [(2048, 2048), (257, 1013), (1500, 733), (3001, 401)]
        for j in range(c["jobs"]):
            w, h = shapes[j % 4]
            n = max(int(w * c["scale"]), 64) * max(int(h * c["scale"]), 64)
            by += 16.0 * n
            fl += n * _filter_flops(dict(model="exponential", range_m=75.0))
        return dict(bytes=by, flops=fl)
    n = float(c["w"] * c["h"])
    layers = 2.0 * 9 * (4 * 32 + 32 * 32 + 32)
    if kind == "infer":
        return dict(bytes=8.0 * n, flops=layers * n)
    if kind == "train":
        # Features, target, hidden layers and output written and read once;
        # forward, weight gradients and the input gradients of layers 2, 3.
        return dict(bytes=n * c["b"] * 4 * (4 + 1 + 2 * 64 + 2),
                    flops=n * c["b"] * (2 * layers + 2.0 * 9 * (32 * 32 + 32)))
    if kind == "field":
        return dict(bytes=n * (4 + 8 + 12), flops=n * _filter_flops(c))
    if kind == "stages":
        # noise 4, filter 8, realistic DEM 12, burning 12, fill 8, routing
        # 4 + 6, tracing 2 + 4 + 4, border 4 + 8
        return dict(bytes=n * 76, flops=n * _filter_flops(c))
    fl = _filter_flops(c) + (layers if c["learned"] else 0.0)
    return dict(bytes=16.0 * n * c["count"], flops=n * c["count"] * fl)


# ---- the same in 64 bits ----------------------------------------------------------
def _philox_normal(n, seed, realization, sd):
    """n deviates of N(0, sd): Philox4x32-10 (Salmon et al., SC'11), counter
    (cell / 4, realization, tag), 24-bit uniforms, Box-Muller."""
    g = np.arange((n + 3) // 4, dtype=np.uint64)
    mask = np.uint64(0xFFFFFFFF)
    c = [g & mask, np.full_like(g, realization), np.full_like(g, 0x63616765), g >> np.uint64(32)]
    k0, k1 = np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)
    for _ in range(10):
        p0, p1 = np.uint64(0xD2511F53) * c[0], np.uint64(0xCD9E8D57) * c[2]
        c = [(p1 >> np.uint64(32)) ^ c[1] ^ k0, p1 & mask,
             (p0 >> np.uint64(32)) ^ c[3] ^ k1, p0 & mask]
        k0 = (k0 + np.uint64(0x9E3779B9)) & mask
        k1 = (k1 + np.uint64(0xBB67AE85)) & mask
    u = [((x >> np.uint64(8)).astype(np.float64) + 0.5) / 16777216.0 for x in c]
    z = np.empty((g.size, 4))
    for j in (0, 2):
        rad = np.sqrt(-2.0 * np.log(u[j]))
        z[:, j] = rad * np.cos(2.0 * np.pi * u[j + 1])
        z[:, j + 1] = rad * np.sin(2.0 * np.pi * u[j + 1])
    return z.reshape(-1)[:n] * sd


def _field64(s):
    """The noise, and it periodically convolved, on the DEM, at least 0 -> 1."""
    c, r = s["c"], s["r"]
    h, w = s["dem"].shape
    noise = torch.from_numpy(_philox_normal(h * w, s["seed"], 0, c["sigma"])).view(h, w).cuda()
    taps = torch.from_numpy(np.asarray(s["taps"], np.float64)).cuda()
    if c["model"] == "gaussian":
        taps = taps[:, None] * taps[None, :]
    else:
        taps = taps.view(2 * r + 1, 2 * r + 1)
    kernel = torch.zeros((h, w), dtype=torch.float64, device="cuda")
    at = torch.arange(-r, r + 1, device="cuda")
    kernel[(-at % h)[:, None], (-at % w)[None, :]] = taps
    conv = torch.fft.irfft2(torch.fft.rfft2(noise) * torch.fft.rfft2(kernel), s=(h, w))
    dem = s["dem"].double()
    v = torch.where(dem != NODATA, dem + conv, conv)
    return noise, torch.where((v <= 0.0) & (v != NODATA), torch.ones_like(v), v)


def _net64(params):
    """Weights and biases as the network uses them: rounded to bfloat16."""
    q = params.bfloat16().double()
    return (q[0:1152].view(32, 4, 3, 3), q[1152:1184], q[1184:10400].view(32, 32, 3, 3),
            q[10400:10432], q[10432:10720].view(1, 32, 3, 3), q[10720:10721])


def _features64(v):
    x = v.double()[:, None]
    f = torch.nn.functional

    def low(k):
        return -f.max_pool2d(-x, k, 1, k // 2)

    ones = torch.ones_like(x)
    total = f.avg_pool2d(x, 7, 1, 3) / f.avg_pool2d(ones, 7, 1, 3)
    return torch.cat([x - low(3), x - low(7), f.max_pool2d(x, 7, 1, 3) - x, x - total], 1)


def _forward64(feat, w):
    conv = torch.nn.functional.conv2d
    a1 = torch.relu(conv(feat, w[0], w[1], padding=1))
    a2 = torch.relu(conv(a1, w[2], w[3], padding=1))
    return a1, a2, conv(a2, w[4], w[5], padding=1)[:, 0]


def _exact_infer(s):
    w, v, rows, edge = _net64(s["params"]), s["v"], 256, 6
    parts = []
    for y in range(0, v.shape[0], rows):  # in strips; the context of a cell is 6 rows
        a, b = max(y - edge, 0), min(y + rows + edge, v.shape[0])
        part = _forward64(_features64(v[a:b][None]), w)[2][0]
        parts.append(part[y - a:y - a + min(rows, v.shape[0] - y)])
    return torch.cat(parts)


def _exact_train(s):
    params = s["params"].bfloat16().double().requires_grad_()
    w = (params[0:1152].view(32, 4, 3, 3), params[1152:1184],
         params[1184:10400].view(32, 32, 3, 3), params[10400:10432],
         params[10432:10720].view(1, 32, 3, 3), params[10720:10721])
    a1, a2, out = _forward64(s["feat"].double(), w)
    inner = (out - s["target"].double())[:, 3:-3, 3:-3]
    loss = inner.square().mean()
    grad = torch.autograd.grad(loss, params)[0]
    m = 0.9 * s["m"].double() + 0.1 * grad
    v = 0.999 * s["v"].double() + 0.001 * grad * grad
    p = s["params"].double() - 2e-3 * (m / (1 - 0.9 ** 50)) / (
        torch.sqrt(v / (1 - 0.999 ** 50)) + 1e-8)
    return {"a1": a1.detach(), "a2": a2.detach(), "out": out.detach(),
            "loss": loss.detach().view(1), "grad": grad, "params": p, "m": m, "v": v}


def exact(case, seed):
    """Counts, levels, directions and labels are whole numbers or picked from
    the inputs: they have no 64-bit value of their own."""
    kind = case["kind"]
    if kind in ("mc", "mixed"):
        return None
    s = prepare(case, seed)
    if kind == "infer":
        return _exact_infer(s)
    if kind == "train":
        return _exact_train(s)
    noise, v = _field64(s)
    if kind == "field":
        return {"noise": noise, "v": v}
    return dict(noise=noise, v=None, filled=None, dirs=None, flat=None, labels=None, counts=None)
