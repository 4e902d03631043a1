"""FP64 streams against the push form where that one's result does not depend on the order of its
additions: along a column a task has one task upwind, which hands on all it has, so every number is
the same, whatever cells were active in which sweep."""
import numpy as np
import pytest

from subsweep_gb300 import workloads
from subsweep_gb300.sweep import PARSEC, Sweep

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("levels", [1, 4])
@pytest.mark.parametrize("compact", ["auto", "never", "always"])
def test_column_rates_keep_the_history_of_their_changes(levels, compact, monkeypatch):
    w = workloads.cartesian_column(300, 20.0 * PARSEC, 1e-3, 3e48, num_levels=levels)
    rng = np.random.default_rng(3)
    w.density = w.density * np.exp(0.5 * rng.standard_normal(300))
    monkeypatch.setenv("SUBSWEEP_COMPACT", compact)
    handles = []
    for streams in ("0", "1"):
        monkeypatch.setenv("SUBSWEEP_STREAMS", streams)
        handles.append(Sweep(w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source))
    push, stream = handles
    for _ in range(12):
        push.run_sweeps()
        stream.run_sweeps()
        a = {**push.fields(), **push.rates(), "level": push.cell_state()["level"]}
        b = {**stream.fields(), **stream.rates(), "level": stream.cell_state()["level"]}
        for k in a:
            np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    push.close()
    stream.close()
