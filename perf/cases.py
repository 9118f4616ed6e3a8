"""The work that users of this framework have it do, as cases to time.

A landscape run advances a DEM in timesteps (flow direction, accumulation,
process update) with the state resident on the GPU, reads the budget row of
every step and, at the end of an output interval, the grids that a run writes.
Cases of kind "steps" are one output interval of a single grid, "restart" the
same from a restart snapshot, "routing" is the hydrology alone (directions and
accumulation of a DEM), "ensemble" steps
many DEMs of uneven sizes together, "serve" runs scenario requests through the
continuous-batching server, and "accumulate" is the stateless accumulation on
the caller's own device arrays.  Sizes span the repository's configurations
(96 to 4096 cells a side, ensembles of 64 to 2048); all inputs are synthetic.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from parallem_gb300 import lem
from parallem_gb300 import scenario
from parallem_gb300 import serve
from parallem_gb300.packing import TilePacker

CELLSIZE = 30.0
BUDGET_SUMS = ("tot_e", "tot_i", "tot_g", "tot_d", "tot_weather_c", "tot_weather_p", "tot_bio", "fa_max")
BUDGET_COUNTS = ("sinkcount", "outlet")
GRIDS = ("fd", "fa", "dem", "soilT")  # what an output interval of a run writes
SERVED = ("dem", "fa", "soilT", "stone", "depo")  # a request's result


def listed():
    return [
        # a test-sized DEM in its run-in (constant climate): latency and launches only
        dict(name="runin_96", kind="steps", height=96, width=96, steps=10, climate=False, graphs=False, mfd="sfd"),
        # the small configuration: 512 x 512, ten run-in steps launched eagerly
        dict(name="runin_512", kind="steps", height=512, width=512, steps=10, climate=False, graphs=False, mfd="sfd"),
        # an ordinary rectangular DEM of odd sizes under a climate series, graph steps
        dict(name="series_1021x613", kind="steps", height=1021, width=613, steps=20, climate=True, graphs=True,
             mfd="sfd"),
        # the large single grid, one interval between written grids
        dict(name="series_4096", kind="steps", height=4096, width=4096, steps=40, climate=True, graphs=True,
             mfd="sfd"),
        # multiple flow directions (slope-proportional shares): three steps restarted from a snapshot of a DEM without
        # pits (one with filled pits has undefined shares, which the model carries on as NaN)
        dict(name="mfd_restart_151x203", kind="restart", height=151, width=203, steps=3, graphs=False, mfd="slope"),
        # hydrology with multiple flow directions, on a DEM without pits
        dict(name="mfd_routing_350x401", kind="routing", height=350, width=401, contrib=False, mfd="slope"),
        # hydrology of one DEM full of flats and nested depressions
        dict(name="routing_4096", kind="routing", height=4096, width=4096, contrib=False, mfd="sfd"),
        # the same on a smaller odd-sized DEM, with contributing-cell counts
        dict(name="routing_contrib_1501", kind="routing", height=1501, width=1501, contrib=True, mfd="sfd"),
        # a batched ensemble of the usual spread of sizes, each DEM with its own climate series
        dict(name="ensemble_16", kind="ensemble", count=16, low=256, high=2048, steps=40),
        # a batched ensemble of small DEMs
        dict(name="ensemble_20_small", kind="ensemble", count=20, low=64, high=256, steps=20),
        # a burst of scenario requests through the server, joining and leaving as they finish
        dict(name="serve_12", kind="serve", count=12, low=128, high=1024, steps_low=10, steps_high=40),
        # accumulation on the caller's device arrays, near the largest grid the call takes
        dict(name="accumulate_1021x1013", kind="accumulate", height=1021, width=1013),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("steps", "steps", "restart", "routing", "ensemble", "serve", "accumulate"))
    if kind == "steps":
        climate = rng.random() < 0.7
        return dict(kind="steps", height=_log(rng, 64, 4096), width=_log(rng, 64, 4096), steps=rng.randint(10, 40),
                    climate=climate, graphs=rng.random() < 0.5, mfd="sfd")
    if kind == "restart":
        return dict(kind="restart", height=_log(rng, 48, 200), width=_log(rng, 48, 200), steps=rng.randint(1, 3),
                    graphs=rng.random() < 0.5, mfd="slope")
    if kind == "routing" and rng.random() < 0.4:
        return dict(kind="routing", height=_log(rng, 64, 360), width=_log(rng, 64, 360), contrib=False, mfd="slope")
    if kind == "routing":
        return dict(kind="routing", height=_log(rng, 128, 4096), width=_log(rng, 128, 4096),
                    contrib=rng.random() < 0.4, mfd="sfd")
    if kind == "ensemble":
        low = _log(rng, 48, 256)
        return dict(kind="ensemble", count=rng.randint(3, 16), low=low, high=_log(rng, low + 16, 1600),
                    steps=rng.randint(10, 40))
    if kind == "serve":
        low = _log(rng, 64, 256)
        return dict(kind="serve", count=rng.randint(3, 12), low=low, high=_log(rng, low + 16, 1024),
                    steps_low=5, steps_high=rng.randint(10, 40))
    return dict(kind="accumulate", height=_log(rng, 32, 1020), width=_log(rng, 32, 1020))


# ---- inputs -----------------------------------------------------------------


def _surface(h, w, hurst, gen):
    """Fractional-Brownian surface by spectral synthesis, rescaled to [0, 1]."""
    ky = torch.fft.fftfreq(h, device="cuda")[:, None]
    kx = torch.fft.rfftfreq(w, device="cuda")[None, :]
    k = torch.sqrt(kx * kx + ky * ky)
    k[0, 0] = 1.0
    amp = k ** (-(hurst + 1.0))
    amp[0, 0] = 0.0
    phase = torch.rand(k.shape, generator=gen, device="cuda") * (2.0 * math.pi)
    mag = torch.randn(k.shape, generator=gen, device="cuda") * amp
    z = torch.fft.irfft2(torch.polar(mag.abs(), phase), s=(h, w))
    return (z - z.min()) / (z.max() - z.min())


def _border(h, w, fraction, gen):
    """Nodata border of uneven width, at least two cells wide."""
    y = torch.arange(h, device="cuda")
    x = torch.arange(w, device="cuda")
    dist = torch.minimum(torch.minimum(y, h - 1 - y)[:, None], torch.minimum(x, w - 1 - x)[None, :])
    base = max(2.0, fraction * min(h, w) / 4.0)
    width = 2 + torch.floor((base - 1.5) * 2.0 * _surface(h, w, 0.9, gen))
    return dist < width.clamp(min=2)


def _dem(h, w, seed, rough=False):
    """A DEM of h x w cells as a host array (float64 holding float32 values, nodata -9999): pits and plateaus at the
    density of the large configuration, or (rough) flats in a tenth of the cells and nested depressions."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    rng = np.random.default_rng(seed)
    hurst, relief, nodata = rng.uniform(0.6, 0.9), rng.uniform(200.0, 2000.0), rng.uniform(0.01, 0.05)
    z = _surface(h, w, hurst, gen) * relief
    border = _border(h, w, nodata, gen)
    per_cell = h * w / 4096.0 ** 2
    if rough:
        inside = z[~border]
        level = inside[torch.randint(inside.numel(), (4096,), generator=gen, device="cuda")].quantile(0.1)
        z = torch.where(z <= level, torch.floor(z), z)
        # bowls of radius 2-30 and depth 1-20, summed in fixed point so that their order does not matter
        n = max(1, int(12500 * per_cell))
        cy, cx, r, depth = (torch.rand(n, generator=gen, device="cuda") for _ in range(4))
        cy, cx, r, depth = (cy * (h - 1)).long(), (cx * (w - 1)).long(), 2.0 + 28.0 * r, 1.0 + 19.0 * depth
        o = torch.arange(-30, 31, device="cuda")
        low = torch.zeros(h * w, dtype=torch.int64, device="cuda")
        for part in torch.arange(n, device="cuda").split(2048):
            yy = cy[part, None, None] + o[None, :, None]
            xx = cx[part, None, None] + o[None, None, :]
            d2 = (o[None, :, None] ** 2 + o[None, None, :] ** 2) / (r[part, None, None] ** 2)
            bowl = (1.0 - d2).clamp(min=0.0) * depth[part, None, None]
            ok = (yy >= 0) & (yy < h) & (xx >= 0) & (xx < w) & (bowl > 0)
            low.index_add_(0, (yy * w + xx)[ok], (bowl[ok] * 65536.0).long())
        z = z - (low.view(h, w).double() / 65536.0).float()
    else:
        n = max(1, int(5000 * per_cell))
        at = torch.randperm(h * w, generator=gen, device="cuda")[:n]
        z.view(-1)[at] -= 0.5 + 4.5 * torch.rand(n, generator=gen, device="cuda")
        for _ in range(max(1, int(300 * per_cell))):
            r = rng.integers(8, 41) / 2.0
            cy, cx = int(rng.integers(0, h)), int(rng.integers(0, w))
            y0, y1, x0, x1 = max(0, int(cy - r)), min(h, int(cy + r) + 1), max(0, int(cx - r)), min(w, int(cx + r) + 1)
            yy = torch.arange(y0, y1, device="cuda")[:, None] - cy
            xx = torch.arange(x0, x1, device="cuda")[None, :] - cx
            z[y0:y1, x0:x1] = torch.where(yy * yy + xx * xx <= r * r, z[cy, cx].clone(), z[y0:y1, x0:x1])
    z = z.double()
    z[border] = scenario.NODATA
    return z.cpu().numpy()


def _climate(rng, steps):
    """Rain lognormal with mean 900 mm and cv 0.3, temperature N(9, 2)."""
    sigma = math.sqrt(math.log(1.09))
    return rng.lognormal(math.log(900.0) - 0.5 * sigma * sigma, sigma, steps), rng.normal(9.0, 2.0, steps)


def _sides(case):
    """The DEM sides of an ensemble or a burst of requests: spread evenly over the logarithm of [low, high]."""
    n, low, high = case["count"], case["low"], case["high"]
    return [int(round(low * (high / low) ** ((i + 0.5) / n))) for i in range(n)]


def _request_steps(case):
    lo, hi, n = case["steps_low"], case["steps_high"], case["count"]
    return [lo + (hi - lo) * ((5 * i + 2) % n) // max(1, n - 1) for i in range(n)]


def _canvas(sides, width):
    """The lowest canvas of the given width that holds square DEMs of these sides, largest first."""
    height = 256
    while True:
        p = TilePacker(width, height)
        if all(p.alloc(n, n) is not None for n in sorted(sides, reverse=True)):
            return height
        height += 256


def _params(case):
    return lem.make_params(flow_direction_type=0 if case["mfd"] == "sfd" else 1,
                           mfd_proportions=0 if case["mfd"] == "sfd" else 1)


def _valley(h, w, gen):
    """A smooth valley landscape tilted to one side, with a nodata border and no pits (on the GPU)."""
    z = _surface(h, w, 2.0, gen).double() * 200.0
    z += torch.arange(w, 0, -1, device="cuda", dtype=torch.float64)[None, :] * (1200.0 / w)
    z[_border(h, w, 0.03, gen)] = scenario.NODATA
    return z


def _drainage(case, seed):
    """Caller-made inputs of the stateless accumulation: a valley landscape, its D8 steepest-descent codes and the
    runoff weights, on the GPU."""
    h, w = case["height"], case["width"]
    gen = torch.Generator(device="cuda").manual_seed(seed)
    z = _valley(h, w, gen)
    pad = torch.nn.functional.pad(z, (1, 1, 1, 1), value=scenario.NODATA)
    best = torch.zeros_like(z)
    code = torch.zeros((h, w), dtype=torch.int32, device="cuda")
    for bit, dy, dx in ((64, -1, 0), (128, -1, 1), (1, 0, 1), (2, 1, 1), (4, 1, 0), (8, 1, -1), (16, 0, -1),
                        (32, -1, -1)):
        zn = pad[1 + dy:1 + dy + h, 1 + dx:1 + dx + w]
        slope = torch.where(zn == scenario.NODATA, 0.0, (z - zn) / math.hypot(dy, dx))
        code = torch.where(slope > best, bit, code).int()
        best = torch.maximum(best, slope)
    outside = z == scenario.NODATA
    code[outside] = -9999
    weight = 0.3 + 0.6 * torch.rand((h, w), generator=gen, device="cuda", dtype=torch.float64)
    weight[outside] = -9999.0
    return code.contiguous(), weight, z


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed + 1)
    if kind == "accumulate":
        code, weight, z = _drainage(case, seed)
        return dict(kind=kind, code=code, weight=weight, z=z, out=torch.empty_like(z))
    if kind in ("steps", "restart", "routing"):
        h, w = case["height"], case["width"]
        if case["mfd"] == "sfd":
            dem = _dem(h, w, seed, rough=kind == "routing")
        else:
            dem = _valley(h, w, torch.Generator(device="cuda").manual_seed(seed)).cpu().numpy()
        runin = kind == "steps" and not case["climate"]
        rain0, temp0 = (800.0, 10.0) if runin else (900.0, 9.0)
        m = lem.Model(dem, CELLSIZE, rain0, temp0, params=_params(case))
        m.set_state(scenario.initial_state(dem, CELLSIZE, rain0, temp0))
        st = dict(kind=kind, model=m)
        if kind == "routing":
            return dict(st, flags=lem.STEP_CONTRIB if case["contrib"] else 0)
        m.graphs(case["graphs"])
        rain, temp = ([rain0] * case["steps"], [temp0] * case["steps"]) if runin else _climate(rng, case["steps"])
        return dict(st, rain=rain, temp=temp, recompute=not runin,
                    snapshot=m.snapshot() if kind == "restart" else None)
    sides = _sides(case)
    dems = [_dem(n, n, 1000 * seed + i) for i, n in enumerate(sides)]
    states = [scenario.initial_state(z, CELLSIZE, 900.0, 9.0) for z in dems]
    width = 2 * -(-max(sides) // 1024) * 1024
    if kind == "serve":
        steps = _request_steps(case)
        reqs = []
        for i, (z, s) in enumerate(zip(dems, states)):
            rain, temp = _climate(rng, steps[i])
            reqs.append(dict(rid=i, dem=z, state=s, rain=rain, temp=temp, steps=steps[i], arrival=0.0, outputs=SERVED))
        return dict(kind=kind, requests=reqs, server=serve.Server(width, width, max_dems=64))
    b = lem.Batch(width, _canvas(sides, width), CELLSIZE, max_dems=len(sides))
    ids, climate = [], []
    for i in sorted(range(len(sides)), key=lambda i: -sides[i]):
        k = b.add(dems[i], 900.0, 9.0)
        b.set_state(k, states[i])
        ids.append(k)
        climate.append(_climate(rng, case["steps"]))
    b.graphs(True)
    return dict(kind=kind, batch=b, ids=ids, climate=climate, steps=case["steps"])


# ---- one pass ---------------------------------------------------------------


def _budgets(steps):
    """The budget rows of the steps (one list of totals per step): the sums of the fp32 fields, and the counts."""
    return {"sums": np.array([[[t[f] for f in BUDGET_SUMS] for t in s] for s in steps], np.float32),
            "counts": np.array([[[t[f] for f in BUDGET_COUNTS] for t in s] for s in steps], np.int64)}


def run(state):
    kind = state["kind"]
    if kind in ("steps", "restart"):
        m, budgets = state["model"], []
        if kind == "restart":
            m.restore(state["snapshot"])
        for rain, temp in zip(state["rain"], state["temp"]):
            m.step(float(rain), float(temp), state["recompute"])
            budgets.append([m.totals()])
        return dict({f: m.get(f) for f in GRIDS}, **_budgets(budgets))
    if kind == "routing":
        m = state["model"]
        m.flow_direction()
        m.flow_accumulation(state["flags"])
        return {f: m.get(f) for f in ("fd", "fa") + (("contrib",) if state["flags"] else ())}
    if kind == "ensemble":
        b, ids, budgets = state["batch"], state["ids"], []
        for s in range(state["steps"]):
            for k, (rain, temp) in zip(ids, state["climate"]):
                b.set_climate(k, float(rain[s]), float(temp[s]), True)
            b.step()
            budgets.append(b.totals_n(ids))
        exports = [b.export(k, ("fd", "fa", "dem")) for k in ids]
        return dict(grids=[e.wait() for e in exports], **_budgets(budgets))
    if kind == "serve":
        reqs = [serve.Request(**r) for r in state["requests"]]
        state["server"].run(reqs)
        return [r.result for r in reqs]
    h, w = state["z"].shape
    rc = lem.load().lem_accumulate_flow_noalloc(state["code"].data_ptr(), state["weight"].data_ptr(),
                                                state["z"].data_ptr(), state["out"].data_ptr(), w, h, None)
    if rc != 0:
        raise RuntimeError(f"lem_accumulate_flow_noalloc: {lem.STATUS.get(rc, rc)}")
    return state["out"]


def work(case):
    """Per cell and step: the state of record read (DEM 8 bytes, slopes 32, seven fp32 fields, mask 1) and written
    (without the mask), and the step's products written (accumulation 8, direction 1, four fp32 grids); then the grids
    that leave at the end of the interval, in the types they are handed over in."""
    kind = case["kind"]
    if kind == "accumulate":
        n = case["height"] * case["width"]
        return {"bytes": 28 * n, "flops": 2 * n}
    if kind == "routing":
        n = case["height"] * case["width"]
        return {"bytes": (8 + 32 + 1 + 1 + 12 + 8 + 12 + (8 if case["contrib"] else 0)) * n, "flops": 60 * n}
    if kind in ("steps", "restart"):
        cells, steps = [case["height"] * case["width"]], [case["steps"]]
        out = 28 if kind == "steps" else 28 + 85
    else:
        cells = [n * n for n in _sides(case)]
        steps = _request_steps(case) if kind == "serve" else [case["steps"]] * len(cells)
        out = 40 if kind == "serve" else 20
    each = sum(c * s for c, s in zip(cells, steps))
    return {"bytes": 162 * each + out * sum(cells), "flops": 400 * each}


# ---- the values in 64 bits --------------------------------------------------


def exact(case, seed):
    """The stateless accumulation by visiting the cells from the highest down; a whole timestep (routing over flats
    and depressions, then fourteen coupled fields) has no short plain form."""
    if case["kind"] != "accumulate":
        return None
    code, weight, z = (t.cpu().numpy() for t in _drainage(case, seed))
    h, w = z.shape
    step = {64: -w, 128: 1 - w, 1: 1, 2: w + 1, 4: w, 8: w - 1, 16: -1, 32: -w - 1}
    flat = z.ravel()
    fa = np.where(flat == scenario.NODATA, 0.0, weight.ravel()).tolist()
    codes = code.ravel().tolist()
    for i in np.argsort(-flat, kind="stable").tolist():
        c = codes[i]
        if c > 0:
            fa[i + step[c]] += fa[i]
    return np.array(fa).reshape(h, w)
