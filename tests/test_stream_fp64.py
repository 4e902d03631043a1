"""FP64 streams against the push form where that one's result does not depend on the order of its
additions: along a column a task has one task upwind, which hands on all it has, so every number is
the same, whatever cells were active in which sweep."""
from fractions import Fraction

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


def test_rates_are_changed_and_not_summed_anew(monkeypatch):
    # An oblique direction through a column with walls: a task has one task upwind, which hands on
    # the share of its end face.  After a sweep of every cell the incoming rate is the one before
    # plus the share of the change upwind, rounded once.
    n, steps = 60, 12
    w = workloads.cartesian_column(n, 20.0 * PARSEC, 1e-3, 3e48)
    rng = np.random.default_rng(4)
    w.density = w.density * np.exp(0.5 * rng.standard_normal(n))
    w.params.directions = [[1.0, 0.5, 0.3]]
    monkeypatch.setenv("SUBSWEEP_STREAMS", "1")
    v = np.array([1.0, 0.5, 0.3])
    d = v * (1.0 / np.sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]))
    g = w.grid
    share = np.zeros(n)  # of cell c to cell c + 1
    for c in range(n - 1):
        total, out = 0.0, 0.0
        for f in range(g.row_ptr[c], g.row_ptr[c + 1]):
            m = g.normal[f]
            dot = (m[0] * d[0] + m[1] * d[1]) + m[2] * d[2]
            eff = g.area[f] * dot if dot > 0 else 0.0
            total += eff
            if g.kind[f] == 0 and g.nbr[f] == c + 1:
                out = eff
        share[c] = out / total
    changed = 0
    with Sweep(w.params, g, w.density, w.ionized_hydrogen_fraction, w.temperature, w.source) as s:
        before = {k: a[:, 0] for k, a in s.rates().items()}
        for _ in range(steps):
            s.run_sweeps()
            after = {k: a[:, 0] for k, a in s.rates().items()}
            for c in range(1, n):
                change = after["outgoing"][c - 1] - before["outgoing"][c - 1]
                was, part = Fraction(float(before["incoming"][c])), Fraction(float(share[c - 1]))
                expected = float(was + part * Fraction(float(change)))
                assert after["incoming"][c] == expected, c
                changed += change != 0.0 and expected != share[c - 1] * after["outgoing"][c - 1]
            before = after
    assert changed > n  # (else a sum made anew would pass)
