"""FP32 error of the HH cells' traces against the FP64 oracle, in the first
steps after a current's onset, where spikes do not yet amplify it: at most
that of rates computed with an exponential each (2.18e-7 and 2.74e-7 of V;
3.1e-7 and 3.3e-7 where a pair shares one)."""
from __future__ import annotations

import numpy as np
import pytest

from neurogpu_b200 import configs


@pytest.mark.gpu
@pytest.mark.parametrize("n,sets,t_stop,bound", [(800, 40, 2.5, 2.2e-7), (300, 24, 3.0, 2.75e-7)])
def test_error_of_the_hh_cell(ngpu_built, oracle, n, sets, t_stop, bound):
    from neurogpu_b200.sim import run
    w = configs.hh_active(n_sets=sets, t_stop=t_stop, n_comp=n)
    w.amps = configs.step_amps((0.2, 0.5, 1.0), w.nt, w.dt, 0.5, 100.0)
    want = oracle.run_workload(w)
    got = run(w.cell, w.params, w.amps, w.dts, w.stim_node, w.stim_area, w.rec_nodes, w.v_init).astype(np.float64)
    assert np.linalg.norm(got - want) / np.linalg.norm(want) <= bound
