"""Grids that were to be laid out in direction streams and are not: they keep the levelled schedule,
with the results of a handle that never tried."""
import numpy as np
import pytest

from subsweep_gb300 import workloads
from subsweep_gb300.sweep import Sweep

pytestmark = pytest.mark.gpu

STEPS = 5


def make(w, monkeypatch, env, precision):
    for k in ("SUBSWEEP_STREAMS", "SUBSWEEP_STREAM_BYTES", "SUBSWEEP_STREAM_PAIRS", "SUBSWEEP_STREAM_WARPS",
              "SUBSWEEP_STREAM_ARRAYS"):
        monkeypatch.delenv(k, raising=False)
    for k, v in env.items():
        monkeypatch.setenv(k, v)
    return Sweep(w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source, precision=precision,
                 autotune=False)


def results(s):
    for _ in range(STEPS):
        s.run_sweeps()
    return {**s.fields(), **s.rates(), "level": s.cell_state()["level"]}


def same(w, precision, expected, got):
    # Mixed path: bit for bit.  FP64: the push form adds in any order, a chain of at most a few
    # hundred sums of fewer than 64 products (2e-12); the timestep is a state over its change, so
    # its inverse is compared
    shortest = w.params.max_timestep / 2 ** (w.params.num_timestep_levels - 1)
    assert expected.keys() == got.keys()
    for k, a in expected.items():
        b = got[k]
        if precision == "mixed" or k == "level":
            np.testing.assert_array_equal(a, b, err_msg=k)
            continue
        finite = np.isfinite(a)
        np.testing.assert_array_equal(finite, np.isfinite(b), err_msg=k)
        a, b = a[finite], b[finite]
        top = float(np.max(np.abs(a), initial=0.0))
        if k == "timestep":
            a, b, top = 1.0 / a, 1.0 / b, 100.0 / shortest
        np.testing.assert_allclose(b, a, rtol=1e-10, atol=1e-12 * top, err_msg=k)


def periodic():
    return workloads.c2_lognormal(n_per_side=12, num_directions=21, num_levels=4, nthreads=8, thick=True)


def streams_bytes(w, monkeypatch, capfd, precision, env):
    """Bytes of the streams' pieces by the handle's trace; None where it has no streams."""
    monkeypatch.setenv("SUBSWEEP_TRACE", "1")
    capfd.readouterr()
    with make(w, monkeypatch, env, precision):
        said = [x for x in capfd.readouterr().err.splitlines() if x.startswith("subsweep streams:")]
    monkeypatch.delenv("SUBSWEEP_TRACE")
    return int(said[0].split(", ")[-1].split()[0]) if said else None


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_grids_whose_pieces_do_not_fit(precision, monkeypatch, capfd):
    w = periodic()
    with make(w, monkeypatch, {"SUBSWEEP_STREAMS": "0"}, precision) as s:
        expected = results(s)
    on = {"SUBSWEEP_STREAMS": "1"}
    size = streams_bytes(w, monkeypatch, capfd, precision, on)
    assert size
    # given up before anything is built, and when the pieces' sizes are known
    for limit in (0, size - 1):
        env = {**on, "SUBSWEEP_STREAM_BYTES": str(limit)}
        assert streams_bytes(w, monkeypatch, capfd, precision, env) is None
        with make(w, monkeypatch, env, precision) as s:
            same(w, precision, expected, results(s))
    assert streams_bytes(w, monkeypatch, capfd, precision, {**on, "SUBSWEEP_STREAM_BYTES": str(size)}) == size


@pytest.mark.parametrize("pairs", ["0", "1"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_grids_whose_streams_run_out_of_memory(precision, pairs, monkeypatch, capfd):
    w = periodic()
    with make(w, monkeypatch, {"SUBSWEEP_STREAMS": "0"}, precision) as s:
        expected = results(s)
    env = {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_STREAM_PAIRS": pairs}
    for arrays in range(64):  # the first so many arrays are found room for
        env["SUBSWEEP_STREAM_ARRAYS"] = str(arrays)
        if streams_bytes(w, monkeypatch, capfd, precision, env) is not None:
            break
        with make(w, monkeypatch, env, precision) as s:
            same(w, precision, expected, results(s))
    assert 8 <= arrays < 63


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_pairs_that_cannot_be_resident_are_single_blocks(precision, monkeypatch, capfd):
    # (40^3: far words, whose slots go by the warps of a block)
    w = workloads.c4_grf(n_per_side=40, num_sources=3, num_directions=16, nthreads=8, grid_device="gpu")
    got = {}
    for pairs in ("0", "-1"):
        env = {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_STREAM_PAIRS": pairs}
        assert streams_bytes(w, monkeypatch, capfd, precision, env)
        with make(w, monkeypatch, env, precision) as s:
            got[pairs] = results(s)
    for k, a in got["0"].items():
        np.testing.assert_array_equal(a, got["-1"][k], err_msg=k)


def test_upwind_faces_without_a_partner_keep_the_push_form(monkeypatch, capfd):
    # A column along z, closed on itself, whose first cell has its periodic face to the last one
    # twice: the last cell hands its rate out once, so the second face stands without a partner.
    # (Against the direction both would hand out; along it only the receiving side counts them.)
    from subsweep_gb300 import grid as gridmod
    from subsweep_gb300.sweep import SweepParameters
    n = 40
    up, down = np.array([0.0, 0.0, 1.0]), np.array([0.0, 0.0, -1.0])
    row, nbr, kind, normal = [0], [], [], []
    for c in range(n):
        faces = [((c + 1) % n, 1 if c == n - 1 else 0, up)]
        faces += [((c - 1) % n, 1 if c == 0 else 0, down)] * (2 if c == 0 else 1)
        for a, k, v in faces:
            nbr.append(a)
            kind.append(k)
            normal.append(v)
        row.append(len(nbr))
    e = len(nbr)
    length = 3e17
    g = gridmod.Grid(row_ptr=np.array(row, np.int64), nbr=np.array(nbr, np.int32), kind=np.array(kind, np.uint8),
                     area=np.full(e, length ** 2), normal=np.array(normal), volume=np.full(n, length ** 3),
                     size=np.full(n, length), position=np.zeros((n, 3)), box_size=np.ones(3), periodic=True)
    params = SweepParameters(directions=[[0.0, 0.0, 1.0]], num_timestep_levels=2, periodic=True, max_timestep=1e12)
    w = workloads.Workload("ring", params, g, np.full(n, 1.67e-24), np.full(n, 0.9), np.full(n, 1e4),
                           np.full(n, 1e45), steps=4)
    got = {}
    for streams in ("0", "1"):
        with make(w, monkeypatch, {"SUBSWEEP_STREAMS": streams}, "fp64") as s:
            got[streams] = results(s)
    same(w, "fp64", got["0"], got["1"])
    assert streams_bytes(w, monkeypatch, capfd, "fp64", {"SUBSWEEP_STREAMS": "1"}) is None


@pytest.mark.parametrize("graph", ["0", "1"])
@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_sparse_sweeps_without_room_for_their_lists(precision, graph, monkeypatch, capfd):
    w = periodic()
    env = {"SUBSWEEP_STREAMS": "1", "SUBSWEEP_GRAPH": graph, "SUBSWEEP_COMPACT": "always"}
    monkeypatch.setenv("SUBSWEEP_COMPACT", "always")
    with make(w, monkeypatch, env, precision) as s:
        expected = results(s)
    for arrays in range(64):  # the first with which a handle has streams leaves none for a list
        env["SUBSWEEP_STREAM_ARRAYS"] = str(arrays)
        if streams_bytes(w, monkeypatch, capfd, precision, env) is not None:
            break
    for more in (0, 1, 2, 3, 4):  # a list takes three: the second level's finds no room, or less
        env["SUBSWEEP_STREAM_ARRAYS"] = str(arrays + more)
        with make(w, monkeypatch, env, precision) as s:
            got = results(s)
        for k, a in expected.items():
            np.testing.assert_array_equal(a, got[k], err_msg=k)
