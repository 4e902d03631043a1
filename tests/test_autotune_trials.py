"""Trials of the transport variants are the dense sweeps of an untuned handle, and no others: a sparse
sweep launched ahead of a trial in the same step is not taken for one."""
import ctypes

import numpy as np
import pytest

from subsweep_gb300 import _native, workloads
from subsweep_gb300.sweep import Sweep

pytestmark = pytest.mark.gpu

CANDIDATES = (122, 143, 344)  # in the order in which they are tried


def order(levels, advances):
    lib = _native.load_gpu()
    lib.sw_host_sweep_order.restype = ctypes.c_int32
    lib.sw_host_sweep_order.argtypes = [ctypes.c_int32, ctypes.c_int32, ctypes.c_void_p, ctypes.c_int32]
    out = np.zeros(1 << levels, np.int32)
    return out[:lib.sw_host_sweep_order(levels, advances, out.ctypes.data, out.size)].tolist()


def test_sparse_sweeps_are_no_trials(monkeypatch):
    for k in ("SUBSWEEP_PULL_VARIANT", "SUBSWEEP_AUTOTUNE", "SUBSWEEP_COMPACT", "SUBSWEEP_TRACE"):
        monkeypatch.delenv(k, raising=False)
    monkeypatch.setenv("SUBSWEEP_STREAMS", "0")
    w = workloads.c2_lognormal(n_per_side=16, num_directions=21, num_levels=4, nthreads=8, thick=True)
    args = (w.params, w.grid, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source)
    found = False
    with Sweep(*args, precision="mixed", autotune=False) as s:
        for steps in range(1, 40):
            s.run_sweeps()
            n_ge = np.asarray(s.level_counts())
            kinds = []  # of the next step's sweeps: dense or not
            for level in order(4, min(steps, 8)):
                if n_ge[level]:
                    kinds.append(level == 0 or 2 * n_ge[level] >= w.grid.num_cells)
            dense = sum(kinds)
            # a sparse sweep before the last trial, and too few dense ones to end the trials
            if dense < len(CANDIDATES) and False in kinds[:max((i for i, d in enumerate(kinds) if d), default=0)]:
                saved, found = s.save_state(), True
                break
    assert found
    with Sweep(*args, precision="mixed", autotune=True) as s:
        s.load_state(saved)
        s.run_sweeps()
        assert s.stats()["pull_variant"] == CANDIDATES[dense - 1]
