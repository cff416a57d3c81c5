"""What a simulation says of its tree split is the split it runs, and a count
from the environment binds as one from the caller does."""
from __future__ import annotations

import numpy as np
import pytest

from neurogpu_b200 import configs

# x 3 protocols: 300 groups of 32, CTAs of 8 warps; a tree whose skeleton does
# not fit in shared memory at the default count of items
SETS, STEPS, NODES = 3200, 60, 1700


@pytest.fixture(scope="module")
def cell():
    return configs.hh_active(n_sets=1, t_stop=STEPS * 0.025, n_comp=NODES)


def _run(w, batched=False, **shape):
    from neurogpu_b200.sim import Batch, Simulator
    s = Simulator(w.cell, SETS, w.n_stim, "fp32", **shape)
    s.set_params(np.broadcast_to(w.params, (SETS,) + w.params.shape[1:]))
    s.set_stimulus(configs.step_amps([0.7 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0), w.dts,
                   w.stim_node, w.stim_area)
    s.set_recording([0, NODES // 3, NODES // 2, NODES - 1], rec_every=2)
    b = Batch([s]) if batched else s
    b.init(w.v_init)
    b.advance(0, STEPS)
    v, lay = s.trace()[:2], s.layout()
    if batched:
        b.close()
    s.close()
    return v, lay


@pytest.mark.gpu
def test_the_reported_count_is_the_one_in_use(ngpu_built, cell):
    v, lay = _run(cell)
    assert lay["cta_warps"] == 8 and lay["items"] < 3
    again, _ = _run(cell, n_warps=8, items_per_warp=lay["items"])
    np.testing.assert_array_equal(again, v)


@pytest.mark.gpu
@pytest.mark.parametrize("batched", [False, True])
def test_the_environments_count_binds(ngpu_built, cell, monkeypatch, batched):
    want, _ = _run(cell, n_warps=8, items_per_warp=4)
    monkeypatch.setenv("NGPU_ITEMS_PER_WARP", "4")
    got, lay = _run(cell, batched)
    assert lay["items"] == 4
    np.testing.assert_array_equal(got, want)
