"""A step that fails leaves undone what comes after the failing sweep: the other sweeps, the new levels
and the ionization times."""
import numpy as np
import pytest

from subsweep_gb300 import _native, workloads
from subsweep_gb300.sweep import Sweep, SweepError, SweepParameters

pytestmark = pytest.mark.gpu


def state(s):
    cells = s.cell_state()
    return {**s.fields(), "levels": cells["level"], "counts": np.asarray(s.level_counts()),
            "ionization": cells["ionization_time"]}


def same(a, b, keys):
    for k in keys:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_a_stalled_step_moves_no_level_and_no_ionization_time(precision):
    from test_abi import _cyclic_grid
    g = _cyclic_grid()
    n = g.num_cells
    p = SweepParameters(directions=[[0.0, 0.0, 1.0]], num_timestep_levels=3, periodic=False, max_timestep=1.0)
    with Sweep(p, g, density=np.full(n, 1e-24), ionized_hydrogen_fraction=np.full(n, 0.6),
               temperature=np.full(n, 1e4), source=np.full(n, 1e40), precision=precision) as s:
        before = state(s)
        with pytest.raises(SweepError) as e:
            s.run_sweeps()
        assert e.value.status == _native.SW_ERR_STALLED
        same(before, state(s), ("ionized_hydrogen_fraction", "temperature", "levels", "counts", "ionization"))


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("streams", ["0", "1"])
def test_a_refused_floor_ends_the_step_at_its_sweep(streams, precision, monkeypatch):
    w = workloads.c2_lognormal(n_per_side=12, num_directions=21, num_levels=4, nthreads=8, thick=True)
    monkeypatch.setenv("SUBSWEEP_STREAMS", streams)
    after = []
    for trace in ("0", "1"):  # a traced step looks at every sweep before it launches the next
        monkeypatch.setenv("SUBSWEEP_TRACE", trace)
        with Sweep(w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source,
                   precision=precision, autotune=False) as s:
            for _ in range(5):
                s.run_sweeps()
            x = s.fields()["ionized_hydrogen_fraction"]
            at = np.argmax(x)
            x[at] = 1.0
            s.set_fields(ionized_hydrogen_fraction=x)
            before, sweeps = state(s), s.stats()["level_sweeps"]
            with pytest.raises(SweepError) as e:
                s.run_sweeps()
            assert e.value.status == _native.SW_ERR_INVALID_ARG
            after.append(state(s))
            same(before, after[-1], ("levels", "counts", "ionization"))
            assert s.stats()["level_sweeps"] == sweeps + 1
    keys = ("ionized_hydrogen_fraction", "temperature", "timestep")
    if precision == "mixed":
        same(after[0], after[1], keys)
    else:  # (the push form adds in any order: rates to 2e-12 of themselves)
        for k in keys[:2]:
            np.testing.assert_allclose(after[1][k], after[0][k], rtol=1e-10, err_msg=k)
