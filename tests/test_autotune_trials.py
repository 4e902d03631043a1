"""Trials of the transport variants are the dense sweeps of an untuned handle, and no others: a sparse
sweep launched ahead of a trial in the same step is not taken for one."""
import numpy as np
import pytest

from subsweep_gb300 import workloads
from subsweep_gb300.sweep import Sweep

pytestmark = pytest.mark.gpu

CANDIDATES = (122, 143, 344)  # in the order in which they are tried


def test_sparse_sweeps_are_no_trials(monkeypatch):
    for k in ("SUBSWEEP_PULL_VARIANT", "SUBSWEEP_AUTOTUNE", "SUBSWEEP_COMPACT", "SUBSWEEP_TRACE"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("SUBSWEEP_STREAMS", "0")
    w = workloads.c2_lognormal(n_per_side=12, num_directions=16, num_levels=4, nthreads=8)
    args = (w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source)
    n = w.grid.num_cells
    with Sweep(*args, precision="mixed", autotune=False) as s:
        for _ in range(6):  # the next step has the sweeps 0, 3, 2, 3, 1, 3, 2, 3
            s.run_sweeps()
        saved = s.save_state().tobytes()
        levels = s.cell_state()["level"].astype(np.uint8).tobytes()
    # most cells at level 1 and a few at 3: only the sweeps of levels 0 and 1 are dense
    assert saved.count(levels) == 1
    new = np.ones(n, np.uint8)
    new[:n // 8] = 0
    new[::100] = 3
    state = np.frombuffer(saved.replace(levels, new.tobytes()), np.uint8).copy()
    with Sweep(*args, precision="mixed", autotune=True) as s:
        s.load_state(state)
        assert s.level_counts()[1] * 2 > n > s.level_counts()[2] * 2 > 0
        s.run_sweeps()
        assert s.stats()["pull_variant"] == CANDIDATES[1]
