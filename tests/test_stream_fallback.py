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
