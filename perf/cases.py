"""Performance cases of the sweep: what a program that drives the library has it do.

One pass is what the host plugin does on every step of a simulation: one full step
(`Sweep.run_sweeps`: the level sweeps, the chemistry, the level reassignment) and the
write-back of the per-cell fields into host arrays it keeps (`Sweep.fields`).  The
simulation goes on from pass to pass, as it does in use.  A simulation with several
timestep levels opens with steps of 1, 1, 2, 4, ... level sweeps; `prepare` takes it past
those, so every pass is one of the equal steps that follow.  The grids, densities and
sources are the seeded generators of the benchmark configurations (subsweep_gb300.workloads),
scaled from a few hundred cells to 128^3.
"""
import math

import numpy as np
import torch

from subsweep_gb300 import grid as gridmod
from subsweep_gb300 import workloads
from subsweep_gb300.sweep import MEGAYEAR, PARSEC, Sweep, SweepParameters, mass_density_from_number_density

DIRECTIONS = (16, 21, 32, 64, 84)  # the direction tables (one direction: the column)
MAX_TASKS = 128 ** 3 * 84          # a drawn case costs no more than the largest listed one
EXACT_TASKS = 48 ** 3 * 84         # exact() takes about 20 s above this


def listed():
    return [
        # the reference's one-dimensional example: a column swept along one direction, a
        # single dependency chain, so latency is all there is
        dict(name="column-600-fp64", kind="column", n=600, dirs=1, levels=1, precision="fp64", graphs=False),
        # the smallest three-dimensional box (smoke tests, parameter studies)
        dict(name="box-8-d16-fp64", kind="uniform", n=8, dirs=16, levels=1, precision="fp64", graphs=False),
        # the small periodic box of the benchmark, 84 directions, one timestep level, in both
        # precisions
        dict(name="box-32-d84-fp64", kind="uniform", n=32, dirs=84, levels=1, precision="fp64", graphs=False),
        dict(name="box-32-d84-mixed", kind="uniform", n=32, dirs=84, levels=1, precision="mixed", graphs=False),
        # a lognormal density field with many sources and four timestep levels, at an
        # ordinary size: the drop-in precision, and the mixed one replayed as CUDA graphs
        dict(name="lognormal-64-fp64", kind="lognormal", n=64, dirs=84, levels=4, precision="fp64", graphs=False),
        dict(name="lognormal-64-mixed-graphs", kind="lognormal", n=64, dirs=84, levels=4, precision="mixed", graphs=True),
        # cosmological density peaks as sources; the largest grid, and one near it in FP64
        dict(name="grf-96-fp64", kind="grf", n=96, dirs=84, levels=4, precision="fp64", graphs=False),
        dict(name="grf-128-mixed", kind="grf", n=128, dirs=84, levels=4, precision="mixed", graphs=False),
        # few directions on a wide grid of odd size (a quick look before a production run)
        dict(name="grf-101-d16-mixed", kind="grf", n=101, dirs=16, levels=3, precision="mixed", graphs=False),
        # a walled box of Poisson points (no periodic faces, irregular cells, odd counts)
        dict(name="walled-20011-d21-fp64", kind="walled", n=20011, dirs=21, levels=1, precision="fp64", graphs=False),
        # a batch of small independent periodic boxes of unequal size under one handle, in
        # both precisions
        dict(name="batch-32-d32-mixed", kind="batch", n=32, dirs=32, levels=2, precision="mixed", graphs=False),
        dict(name="batch-12-d32-fp64", kind="batch", n=12, dirs=32, levels=2, precision="fp64", graphs=False),
    ]


def draw(rng):
    kind = rng.choice(("uniform", "lognormal", "lognormal", "grf", "grf", "walled", "batch"))
    precision = rng.choice(("fp64", "mixed"))
    dirs = rng.choice(DIRECTIONS)
    levels = rng.randint(1, 4)
    if kind == "walled":
        n = int(round(math.exp(rng.uniform(math.log(400), math.log(60000)))))
    elif kind == "batch":
        n = int(round(math.exp(rng.uniform(math.log(2), math.log(32)))))
    else:
        # FP64 steps cost several times the mixed ones: their largest grids are smaller
        n = int(round(math.exp(rng.uniform(math.log(7), math.log(96 if precision == "fp64" else 128)))))
    assert kind in ("walled", "batch") or n ** 3 * dirs <= MAX_TASKS
    return dict(kind=kind, n=n, dirs=dirs, levels=levels, precision=precision, graphs=rng.random() < 0.25)


def _workload(case, seed):
    """The inputs of a case: a Workload, or for a batch the list of its boxes."""
    kind, n, dirs, levels = case["kind"], case["n"], case["dirs"], case["levels"]
    if kind == "column":
        w = workloads.cartesian_column(n, 20.0 * PARSEC, 1e-3, 3e48)
        rng = np.random.default_rng(seed)
        w.density = w.density * np.exp(0.3 * rng.standard_normal(n))
        return w
    if kind == "uniform":
        w = workloads.c1_small_periodic(n, seed=seed, num_directions=dirs, grid_device="gpu")
        w.params.num_timestep_levels = levels
        return w
    if kind == "lognormal":
        w = workloads.c2_lognormal(n, seed=seed, num_directions=dirs, num_levels=levels, grid_device="gpu")
        w.source *= (n / 128.0) ** 3  # the full-size box's emission per volume
        return w
    if kind == "grf":
        return workloads.c4_grf(n, seed=seed, num_sources=max(2, n ** 3 // 16384), num_directions=dirs,
                                num_levels=levels, grid_device="gpu", total_rate=1e52 * (n / 256.0) ** 3)
    if kind == "walled":
        rng = np.random.default_rng(seed)
        box = 100.0 * PARSEC * n ** (1.0 / 3.0)
        g = gridmod.voronoi_gpu(gridmod.poisson_points(n, box, seed), box, periodic=False)
        src = gridmod.place_sources(g, rng.uniform(0.0, box, size=(4, 3)), 10.0 ** rng.uniform(48.0, 49.0, size=4))
        params = SweepParameters(directions=dirs, num_timestep_levels=levels, periodic=False,
                                 max_timestep=0.5 * MEGAYEAR, significant_rate_threshold=workloads.THRESHOLD)
        n_h = 1e-3 * np.exp(0.5 * rng.standard_normal(n))
        return workloads.Workload("walled", params, g, mass_density_from_number_density(n_h), np.full(n, 1e-10),
                                  np.full(n, 1e4), src, steps=4)
    rng = np.random.default_rng(seed)
    counts = np.round(np.exp(np.random.default_rng(n).uniform(math.log(512), math.log(16000), size=n))).astype(int)
    boxes = [workloads.c3_box(rng, seed * 1009 + b, int(m), int(m),
                              voronoi=lambda pts, box: gridmod.voronoi_gpu(pts, box, periodic=True))
             for b, m in enumerate(counts)]
    return workloads.c3_batched(boxes=boxes, num_directions=dirs, num_levels=levels), boxes


def prepare(case, seed):
    got = _workload(case, seed % 1000003)
    opts = dict(precision=case["precision"], use_graphs=case["graphs"])
    if case["kind"] == "batch":
        w, boxes = got
        parts = [(g, mass_density_from_number_density(n_h), 1e-10, 1e4, src) for g, n_h, src in boxes]
        sweep = Sweep.batch(w.params, parts, **opts)
    else:
        w = got
        sweep = Sweep(w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source, **opts)
    cells = w.grid.num_cells
    keys = ("ionized_hydrogen_fraction", "temperature", "timestep", "photon_rate")
    if case["levels"] > 1:
        for _ in range(case["levels"]):
            sweep.run_sweeps()
    return {"sweep": sweep, "fields": {k: np.empty(cells) for k in keys}}


def run(state):
    elapsed = state["sweep"].run_sweeps()
    return {"elapsed": elapsed, **state["sweep"].fields(out=state["fields"])}


def _cells(case):
    n = case["n"]
    return {"column": n, "walled": n, "batch": 4500 * n}.get(case["kind"], n ** 3)


def work(case):
    """A step's level sweeps with all cells on the deepest level (over nine tenths of
    them are, in the larger boxes after a few steps): per sweep the faces once (normal and area, neighbour), each
    (cell, direction) rate written and read once, the cell state read and written; per task
    a multiply-add per upwind face; about 160 operations of chemistry per cell."""
    cells, sweeps = _cells(case), 2 ** (case["levels"] - 1)
    rate = 4 if case["precision"] == "mixed" else 8
    faces = 2 if case["kind"] == "column" else 15.5
    tasks = cells * case["dirs"]
    return {"bytes": sweeps * (cells * (faces * (4 * rate + 4) + 12 * 8) + 2 * rate * tasks) + 32 * cells,
            "flops": sweeps * (tasks * (faces + 4) + 160 * cells)}


# ---------------------------------------------------------------------------------------
# The first step of a simulation with one timestep level in plain torch, FP64: one sweep
# of all cells.

_PROTON = 1.67262192369e-27
_BOLTZMANN = 1.380649e-23
_EV = 1.602176634e-19
_SIGMA = 2.9580524545305314e-22  # m^2
_EPS = 2.220446049250313e-16


def _transport(g, params, directions, att, source, dev):
    """(incoming, periodic) summed over directions as [cells] tensors, and the rate of
    every cell summed over the directions in order."""
    n = g.num_cells
    row = torch.repeat_interleave(torch.arange(n, device=dev), torch.from_numpy(np.diff(g.row_ptr)).to(dev))
    nbr = torch.from_numpy(g.nbr.astype(np.int64)).to(dev)
    kind = torch.from_numpy(g.kind.astype(np.int64)).to(dev)
    area = torch.from_numpy(g.area).to(dev)
    normal = torch.from_numpy(g.normal).to(dev)
    src = source / len(directions)
    incoming = torch.zeros(n, dtype=torch.float64, device=dev)
    rate = torch.zeros(n, dtype=torch.float64, device=dev)
    for d in directions:
        dot = normal[:, 0] * d[0] + normal[:, 1] * d[1] + normal[:, 2] * d[2]
        down = torch.zeros(n, dtype=torch.float64, device=dev).index_add_(0, row, area * dot.clamp(min=0.0))
        parts = []
        for k in (0, 1):
            at = torch.nonzero((dot < 0) & (kind == k)).reshape(-1)
            m, c = nbr[at], row[at]
            parts.append((m, c, (area * -dot)[at] / down[m]))
        m, c, frac = parts[0]
        # fixed point of out = att (in + src), in = sum of frac out over the upwind faces:
        # exact after as many rounds as the longest dependency chain has cells
        inc = torch.zeros(n, dtype=torch.float64, device=dev)
        while True:
            before = inc
            for _ in range(16):
                r = inc + src
                out = torch.where(r < params.significant_rate_threshold, torch.zeros_like(r), r * att)
                inc = torch.zeros_like(r).index_add_(0, c, frac * out[m])
            if bool(((inc - before).abs() <= 1e-15 * inc.abs()).all()):
                break
        r = inc + src
        out = torch.where(r < params.significant_rate_threshold, torch.zeros_like(r), r * att)
        m, c, frac = parts[1]
        per = torch.zeros_like(r).index_add_(0, c, frac * out[m])
        incoming += inc
        rate += (inc + src) + per
    return incoming, rate


def _collision(t):
    s5 = torch.sqrt(t / 1e5)
    e = torch.exp(-157809.1 / t)
    fit = torch.sqrt(t) / (1.0 + s5) * e
    slope = e * (157809.1e-5 * t + 0.5 * s5 * (2.0 * 157809.1 + t)) / (t ** 1.5 * s5 * (s5 + 1.0) ** 2)
    return s5, fit, slope


def _attempt(dt, safety, x, t, rho, vol, size, rate, a):
    """One attempt of the hydrogen solver over dt: accepted, new x, new T, timescale."""
    erg_cm3, cm3 = 1e-13, 1e-6
    n_h = rho / _PROTON
    ne, nhn, mu = n_h * x, n_h * (1.0 - x), 1.0 / (x + 1.0)
    absorbed = 1.0 - torch.exp(-nhn * _SIGMA * size)
    s5, fit, dfit = _collision(t)
    e_exc = torch.exp(-118348.0 / t)
    exc = 7.5e-19 / (1.0 + s5) * e_exc
    dexc = 7.5e-19 * e_exc * (118348.0e-5 * t - 0.5e-5 * t * t + 118348.0 * s5) / (t * t * s5 * (1.0 + s5) ** 2)
    lam = 315614.0 / t
    q = (lam / 2.25) ** 0.376
    l197, p372 = lam ** 1.97, (1.0 + q) ** 3.72
    rec = 3.435e-30 * t * l197 / p372
    drec = 3.435e-30 * l197 / (p372 * (1.0 + q)) * (1.0 - 1.97 + (1.0 - 1.97 + 0.376 * 3.72) * q)
    z = 2.727 / a
    compton = 1.017e-37 * z ** 4 * 1e-7
    cool = ((exc + 1.27e-21 * fit) * erg_cm3 * ne * nhn + (rec + 1.42e-27 * torch.sqrt(t)) * erg_cm3 * ne * ne
            + compton * (t - z) * ne)
    dcool = ((dexc + 1.27e-21 * dfit) * erg_cm3 * ne * nhn
             + (drec + 1.42e-27 / (2.0 * torch.sqrt(t))) * erg_cm3 * ne * ne + compton * ne)
    k = (5.0 / 3.0 - 1.0) * _PROTON / (rho * _BOLTZMANN)
    heat = rate * absorbed / vol * ((18.028356312818811 - 13.65693) * _EV)
    tc = k * mu * (heat - cool) * dt / (1.0 + k * mu * dcool * dt)
    change = torch.fmin((tc / t).abs(), torch.full_like(t, 1.0 / _EPS))
    ok = ~(change > safety)
    ts = dt * (safety / change)
    t = t + tc
    lam = 315614.0 / t
    p = (lam / 2.74) ** 0.407
    b = (1.0 + p) ** 2.242
    alpha = 2.753e-14 * lam ** 1.5 / b * cm3
    dalpha = -2.753e-14 * torch.sqrt(lam) / (b * (p + 1.0)) * (0.407 * 2.242 * p - 1.5 * p - 1.5) * cm3 * (-315614.0 / (t * t))
    _, fit, dfit = _collision(t)
    beta, dbeta = 5.85e-11 * fit * cm3, 5.85e-11 * dfit * cm3
    photo = rate * absorbed / (nhn * vol)
    c, d = beta * ne + photo, alpha * ne
    dc, dd = n_h * beta - ne * t * mu * dbeta, n_h * alpha - ne * t * mu * dalpha
    j = dc - (c + d) - x * (dc + dd)
    xc = dt * (c - x * (c + d)) / (1.0 - j * dt)
    change = torch.fmin((xc / x).abs(), torch.full_like(t, 1.0 / _EPS))
    ok &= ~(change > safety)
    other = dt * (safety / change)
    return ok, x + xc, t, torch.where(ts < other, ts, other)


def _chemistry(dt, params, x, t, rho, vol, size, rate, a=1.0):
    """The solver with its halving of rejected timesteps, all cells at once: (x, T, timescale)."""
    n = x.numel()
    floor_x, floor_t = x.clone(), t.clone()
    depth = torch.zeros(n, dtype=torch.int64, device=x.device)
    pending = torch.zeros(n, 101, dtype=torch.bool, device=x.device)  # second halves left at each depth
    ts = torch.zeros_like(x)
    todo = torch.arange(n, device=x.device)

    def clamp(cx, ct, at):
        low = floor_x[at] if params.prevent_cooling else torch.full_like(cx, 1e-10)
        cx = torch.clamp(torch.maximum(cx, low), max=1.0 - 1e-10)
        return cx, torch.maximum(ct, floor_t[at]) if params.prevent_cooling else ct

    while todo.numel():
        cx, ct = clamp(x[todo], t[todo], todo)
        sub = dt * torch.pow(0.5, depth[todo].double())
        ok, nx, nt, nts = _attempt(sub, params.chemistry_timestep_safety_factor, cx, ct, rho[todo], vol[todo],
                                   size[todo], rate[todo], a)
        nx, nt = clamp(nx, nt, todo)
        x[todo], t[todo] = torch.where(ok, nx, cx), torch.where(ok, nt, ct)
        ts[todo] = torch.where(ok, nts, ts[todo])
        bad = todo[~ok]
        depth[bad] += 1
        pending[bad, depth[bad]] = True
        good = todo[ok]
        deepest = torch.where(pending[good], torch.arange(101, device=x.device), -1).max(1).values
        again = good[deepest > 0]
        depth[again] = deepest[deepest > 0]
        pending[again, depth[again]] = False
        todo = torch.cat([bad, again]).sort().values
    return x, t, ts


def exact(case, seed):
    tasks = _cells(case) * case["dirs"]
    if tasks > EXACT_TASKS or case["levels"] > 1:
        return None
    got = _workload(case, seed % 1000003)
    w = got[0] if case["kind"] == "batch" else got
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    as_t = lambda v: torch.from_numpy(np.ascontiguousarray(np.broadcast_to(v, (w.grid.num_cells,)), np.float64)).to(dev)
    rho, x, t, src = as_t(w.density).clone(), as_t(w.ionized_hydrogen_fraction).clone(), as_t(w.temperature).clone(), as_t(w.source)
    vol, size = as_t(w.grid.volume), as_t(w.grid.size)
    if isinstance(w.params.directions, int):
        from subsweep_gb300 import directions_from_num
        directions = directions_from_num(w.params.directions)  # the reference's table, an input
    else:
        directions = np.asarray(w.params.directions)
    att = torch.exp(-rho / _PROTON * (1.0 - x) * _SIGMA * size)
    incoming, rate = _transport(w.grid, w.params, directions, att, src, dev)
    dt = w.params.max_timestep
    x, t, ts = _chemistry(dt, w.params, x, t, rho, vol, size, rate)
    back = lambda v: v.cpu().numpy()
    if case["kind"] == "uniform" and case["precision"] == "mixed":
        # optically very thick cells: the rates beyond the source cell (1e-80 of it) are
        # below what FP32 holds
        incoming = None
    return {"elapsed": dt, "ionized_hydrogen_fraction": back(x), "temperature": back(t), "timestep": back(ts),
            "photon_rate": None if incoming is None else back(incoming)}
