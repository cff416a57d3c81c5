"""The autotuner's candidates hold the library's own layouts, asked for by
their numbers they are those layouts, and a batch keeps a tuned member's CTAs
as wide as its own."""
from __future__ import annotations

import numpy as np
import pytest

from neurogpu_b200 import configs

N, STEPS = 200, 60


def _inputs(sets):
    w = configs.hh_active(n_sets=1, t_stop=STEPS * 0.025, n_comp=N)
    amps = configs.step_amps([0.7 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0)
    return w, np.repeat(w.params, sets, axis=0), amps


def _sim(sets, **shape):
    from neurogpu_b200.sim import Simulator
    w, params, amps = _inputs(sets)
    s = Simulator(w.cell, sets, w.n_stim, "fp32", **shape)
    s.set_params(params)
    s.set_stimulus(amps, w.dts, w.stim_node, w.stim_area)
    s.set_recording([0, N - 1], rec_every=2)
    return s, w.v_init


# 11 sets: a team; 1,200: 113 groups, CTAs of 16 warps; 2,134: 201 groups, of 12; 3,300: 310 groups, of 8
@pytest.mark.gpu
@pytest.mark.parametrize("sets", [11, 1200, 2134, 3300])
def test_the_librarys_choice_is_a_candidate(ngpu_built, sets):
    from neurogpu_b200 import autotune
    s, v0 = _sim(sets)
    own = s.layout()
    s.init(v0)
    s.advance(0, STEPS)
    want = s.trace()
    s.close()
    w, params, amps = _inputs(sets)
    r = autotune.tune(w.cell, params, amps, w.dts, w.stim_node, w.stim_area, [0], v0, steps=20, warmup=5,
                      warp_shapes=())
    assert f"lane:{own['cta_warps']}:{own['items']}" in r["ms_per_step"]
    t = autotune.tune_warps(w.cell, params, amps, w.dts, w.stim_node, w.stim_area, [0], v0, steps=20, warmup=5)
    assert "12:2" in t["ms_per_step"] and t["n_warps"] <= 12
    s, _ = _sim(sets, n_warps=own["cta_warps"], items_per_warp=own["items"])
    assert s.layout() == own
    s.init(v0)
    s.advance(0, STEPS)
    np.testing.assert_array_equal(s.trace(), want)
    s.close()


@pytest.mark.gpu
def test_a_batch_keeps_twelve_warps(ngpu_built):
    from neurogpu_b200.sim import Batch
    sims = [_sim(1100, n_warps=12, items_per_warp=2)[0] for _ in range(2)]  # 2 x 104 groups
    b = Batch(sims)
    assert [s.layout()["cta_warps"] for s in sims] == [12, 12]
    own = [_sim(1100)[0] for _ in range(2)]
    c = Batch(own)
    assert [s.layout() for s in own] == [s.layout() for s in sims]
    for x in (b, c):
        x.init(-65.0)
        x.advance(0, STEPS)
    for s, t in zip(sims, own):
        np.testing.assert_array_equal(s.trace(), t.trace())
    b.close()
    c.close()
