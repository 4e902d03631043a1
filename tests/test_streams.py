"""Direction streams against the transports they replace.

Mixed path: the levelled lockstep kernels solve the same tasks with the same roundings, so every
field, rate, level and time series is compared exactly; checkpoints are written in one layout and
read in the other.  FP64: the push form hands the same shares out, in an order of its own and as
corrections, so the rates agree to rounding; the forms of the streams agree exactly.
"""
import numpy as np
import pytest

from subsweep_gb300 import grid as gridmod
from subsweep_gb300 import workloads
from subsweep_gb300.sweep import MEGAYEAR, Sweep, SweepParameters, mass_density_from_number_density

pytestmark = pytest.mark.gpu


def lattice(n, dirs, levels):
    # a 6^3 grid has streams of 216 tasks: less than the 512 of a block's warps
    return workloads.c2_lognormal(n_per_side=n, num_directions=dirs, num_levels=levels, nthreads=8, thick=n > 8)


def far_words():
    # 64,000 tasks a stream, more than shared memory holds: words read back from memory
    return workloads.c4_grf(n_per_side=40, num_sources=3, num_directions=16, nthreads=8, grid_device="gpu")


def batch():
    rng = np.random.default_rng(17)
    boxes = [workloads.c3_box(rng, 50 + b, 300, 2000, nthreads=8) for b in range(4)]
    return workloads.c3_batched(boxes=boxes, num_directions=16, num_levels=3)


def walled(n=1501):
    box = 30 * 3.0857e16 * n ** (1 / 3)
    g = gridmod.voronoi(gridmod.poisson_points(n, box, 23), box, periodic=False, nthreads=8)
    source = gridmod.place_sources(g, np.array([[box * 0.3, box * 0.6, box * 0.5]]), np.array([3e49]))
    params = SweepParameters(directions=21, num_timestep_levels=3, periodic=False, max_timestep=0.5 * MEGAYEAR,
                             significant_rate_threshold=1e-5)
    return workloads.Workload("walled", params, g, np.full(g.num_cells, float(mass_density_from_number_density(1e-2))),
                              np.full(g.num_cells, 1e-10), np.full(g.num_cells, 1e4), source, steps=6)


CASES = {
    "lattice-6": lambda: lattice(6, 16, 3),
    "lattice-20": lambda: lattice(20, 21, 4),
    "far-words": far_words,
    "batch": batch,
    "walled": walled,
}


def make(w, monkeypatch, env, precision="mixed"):
    for k in ("SUBSWEEP_STREAMS", "SUBSWEEP_COMPACT", "SUBSWEEP_STREAM_WARPS", "SUBSWEEP_STREAM_PAIRS", "SUBSWEEP_GRAPH"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    return Sweep(w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source, precision=precision,
                 autotune=False)


def results(s):
    out = {**s.fields(), **s.rates(), "level": s.cell_state()["level"]}
    out.update({"series " + k: np.asarray(v) for k, v in s.time_series().items()})
    return out


def same(a, b):
    assert a.keys() == b.keys()
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("case", CASES)
def test_streams_equal_lockstep(case, monkeypatch):
    w = CASES[case]()
    steps = 5
    with make(w, monkeypatch, {"SUBSWEEP_STREAMS": "0"}) as s:
        for _ in range(steps):
            s.run_sweeps()
        expected, tasks = results(s), s.stats()["tasks"]
    forms = [{"SUBSWEEP_COMPACT": c} for c in ("never", "always")]
    forms += [{"SUBSWEEP_STREAM_WARPS": str(n)} for n in (4, 8, 16)] + [{"SUBSWEEP_GRAPH": "1"}]
    # pairs of blocks: a stream each where there are enough, or 7 pairs with streams cut between them
    forms += [{"SUBSWEEP_STREAM_PAIRS": n} for n in ("1", "7")]
    forms += [{"SUBSWEEP_STREAM_PAIRS": "7", "SUBSWEEP_GRAPH": "1"}]
    for env in forms:
        with make(w, monkeypatch, {"SUBSWEEP_STREAMS": "1", **env}) as s:
            for _ in range(steps):
                s.run_sweeps()
            same(expected, results(s))
            if "SUBSWEEP_COMPACT" not in env:
                assert s.stats()["tasks"] == tasks


@pytest.mark.parametrize("case", CASES)
def test_fp64_streams_equal_push(case, monkeypatch):
    w = CASES[case]()
    steps = 5
    got = {}
    forms = {"push": {"SUBSWEEP_STREAMS": "0"}, "streams": {"SUBSWEEP_STREAMS": "1"}}
    forms.update({c: {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_COMPACT": c} for c in ("never", "always")})
    forms.update({"4": {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_STREAM_WARPS": "4"},
                  "graph": {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_GRAPH": "1"}})
    forms.update({"pairs " + n: {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_STREAM_PAIRS": n} for n in ("1", "7")})
    for name, env in forms.items():
        with make(w, monkeypatch, env, "fp64") as s:
            for _ in range(steps):
                s.run_sweeps()
            got[name] = results(s)
            if name == "streams":
                saved = s.save_state()
    for name in forms:
        if name not in ("push", "streams"):
            same(got["streams"], got[name])
    # A rate is a chain of at most a few hundred sums of fewer than 64 products: 300 * 70 * 2^-53 is
    # 2e-12 of it, and the push form's corrections leave as much of the largest rate behind.
    # (states that agree to 1e-10 leave the timestep, a state over its change in a step of at least
    # max_timestep / 2^(levels - 1), its inverse to 1e-10 over that)
    shortest = w.params.max_timestep / 2 ** (w.params.num_timestep_levels - 1)
    for k, a in got["push"].items():
        b = got["streams"][k]
        if k == "level":
            np.testing.assert_array_equal(a, b)
            continue
        finite = np.isfinite(a)
        np.testing.assert_array_equal(finite, np.isfinite(b), err_msg=k)
        a, b = a[finite], b[finite]
        top = float(np.max(np.abs(a), initial=0.0))
        if k == "timestep":
            a, b, top = 1.0 / a, 1.0 / b, 100.0 / shortest
        np.testing.assert_allclose(b, a, rtol=1e-10, atol=1e-12 * top, err_msg=k)
    # a checkpoint of the streams goes on in both forms
    for env in (forms["push"], forms["streams"]):
        with make(w, monkeypatch, env, "fp64") as s:
            s.load_state(saved)
            after = results(s)
            for k, a in got["streams"].items():
                if k != "level":
                    np.testing.assert_allclose(after[k], a, rtol=1e-13, err_msg=k)


def everywhere_a_source(seed=1, n=400, levels=3):
    # all cells stay at the deepest level for some steps, then leave it one by one
    rng = np.random.default_rng(seed)
    box = 30 * 3.0857e16 * n ** (1 / 3)
    g = gridmod.voronoi(gridmod.poisson_points(n, box, seed), box, periodic=False, nthreads=8)
    source = 1e46 * np.exp(0.5 * rng.standard_normal(g.num_cells))
    params = SweepParameters(directions=21, num_timestep_levels=levels, periodic=False, max_timestep=0.01 * MEGAYEAR,
                             significant_rate_threshold=1e-5)
    return workloads.Workload("sources", params, g, np.full(g.num_cells, float(mass_density_from_number_density(1e-2))),
                              np.full(g.num_cells, 1e-10), np.full(g.num_cells, 1e4), source, steps=8)


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_captured_steps_follow_the_cells_that_leave_a_level(precision, monkeypatch):
    w = everywhere_a_source()
    seen = set()
    with make(w, monkeypatch, {"SUBSWEEP_STREAMS": "1"}, precision) as direct, \
            make(w, monkeypatch, {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_GRAPH": "1"}, precision) as captured:
        for _ in range(8):
            direct.run_sweeps()
            captured.run_sweeps()
            same(results(direct), results(captured))
            seen.add(int(direct.level_counts()[-1]) == w.grid.num_cells)
    assert seen == {True, False}


@pytest.mark.parametrize("case", ["lattice-20", "batch"])
def test_checkpoints_move_between_layouts(case, monkeypatch):
    w = CASES[case]()
    saved = {}
    final = {}
    for streams in ("0", "1"):
        with make(w, monkeypatch, {"SUBSWEEP_STREAMS": streams}) as s:
            for _ in range(3):
                s.run_sweeps()
            saved[streams] = s.save_state()
            s.run_sweeps()
            final[streams] = results(s)
    same(final["0"], final["1"])
    # (the bytes may differ in the stamps of kept words, which only the dense levelled sweeps renew)
    for writer in ("0", "1"):
        for reader in ("0", "1"):
            with make(w, monkeypatch, {"SUBSWEEP_STREAMS": reader}) as s:
                s.load_state(saved[writer])
                s.run_sweeps()
                same(final["0"], results(s))
