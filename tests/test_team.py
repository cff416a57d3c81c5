"""Teams of CTAs (one cluster per group of 32 instances, small batches)
against one CTA per group, and launches of every length modulo the three
copies of the separators' numbers."""
from __future__ import annotations

import numpy as np
import pytest

from neurogpu_b200 import configs

CELLS = {"hh": lambda n, sets: configs.hh_active(n_sets=sets, t_stop=2.5, n_comp=n),
         "ttpc": lambda n, sets: configs.ttpc_like(n_sets=sets, t_stop=1.5),
         "passive": lambda n, sets: configs.passive_cable(n_sets=sets, t_stop=2.5, n_comp=n)}


def _run(w, precision, steps):
    """Traces of the soma and the last compartment, the run cut into launches of the given lengths."""
    from neurogpu_b200.sim import Simulator
    amps = configs.step_amps([0.7 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0)
    s = Simulator(w.cell, w.n_sets, w.n_stim, precision)
    s.set_params(w.params)
    s.set_stimulus(amps, w.dts, w.stim_node, w.stim_area)
    s.set_recording([0, w.cell.n_nodes - 1])
    s.init(w.v_init)
    t = 0
    while t < w.nt:
        n = min(steps[t % len(steps)], w.nt - t)
        s.advance(t, n)
        t += n
    v = s.trace()
    assert s.n_bad() == 0
    s.close()
    return v


# 160 nodes: the smallest tree with a team; 33 and 1 instances: a nearly empty
# group; 700 sets x 3: teams of two; the TTPC-like cell: teams of eight, long
# chains of separators
@pytest.mark.gpu
@pytest.mark.parametrize("cell,n,sets,precision", [
    ("passive", 160, 1, "fp32"), ("passive", 170, 70, "fp64"), ("hh", 161, 3, "fp32"), ("hh", 500, 11, "fp32"),
    ("hh", 500, 11, "fp64"), ("hh", 500, 700, "fp32"), ("ttpc", 1501, 8, "fp32"), ("ttpc", 1501, 2, "fp64")])
def test_team_matches_one_cta(ngpu_built, monkeypatch, cell, n, sets, precision):
    w = CELLS[cell](n, sets)
    team = _run(w, precision, [w.nt])
    for steps in ([1], [2], [3, 1, 4], [5, 7]):   # bitwise: a cut run performs the same operations
        np.testing.assert_array_equal(_run(w, precision, steps), team)
    monkeypatch.setenv("NGPU_TEAM", "0")
    one = _run(w, precision, [w.nt])
    # FP64: the outputs' own rounding (float32, 3.8e-6 mV at 70 mV); FP32: two
    # orders of the same sums, within the parity bound away from spikes
    np.testing.assert_allclose(team, one, rtol=0, atol=1e-5 if precision == "fp64" else 0.1)
