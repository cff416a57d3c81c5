"""Members that are under way when their batch is made go on in it: teams of
CTAs, CTAs of 16 and 12 warps, and trees whose layout alone differs from the
batch's.  At its next initialisation a member takes the batch's split."""
from __future__ import annotations

import numpy as np
import pytest

from neurogpu_b200 import configs

STEPS, CUT = 60, 7


def _sims(shapes, precision, n_warps=0):
    from neurogpu_b200.sim import Simulator
    out = []
    for n, sets in shapes:
        w = configs.hh_active(n_sets=1, t_stop=STEPS * 0.025, n_comp=n)
        rng = np.random.default_rng(n)
        p = np.repeat(w.params, sets, axis=0)
        g = w.cell.mechset.param_index("gbar_na")
        p[:, g] *= rng.uniform(0.5, 2.0, (sets, 1)).astype(np.float32)
        s = Simulator(w.cell, sets, w.n_stim, precision, n_warps=n_warps)
        s.set_params(p)
        s.set_stimulus(configs.step_amps([0.7 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0), w.dts,
                       w.stim_node, w.stim_area)
        s.set_recording([0, n // 2, n - 1], rec_every=2)
        out.append(s)
    return out, w.v_init


# (compartments, sets) per member, three protocols: 11 sets are two groups, a
# team of 2 and of 6 CTAs; 2,134 sets 201 groups (CTAs of 12 warps) that join
# a batch of three CTAs per SM; 50 compartments beside 3,000
@pytest.mark.gpu
@pytest.mark.parametrize("shapes,precision,n_warps", [
    ([(200, 11), (500, 11)], "fp64", 0), ([(200, 11), (500, 11)], "fp32", 0), ([(200, 11), (500, 11)], "fp64", 16),
    ([(120, 2134), (160, 2134)], "fp32", 0), ([(50, 1700), (3000, 70)], "fp64", 0)])
def test_members_go_on_in_the_batch(ngpu_built, shapes, precision, n_warps):
    from neurogpu_b200.sim import Batch
    alone, v0 = _sims(shapes, precision, n_warps)
    want = []
    for s in alone:
        s.init(v0)
        s.advance(0, STEPS)
        want.append(s.trace())
        s.close()
    sims, _ = _sims(shapes, precision, n_warps)
    for s in sims:
        s.init(v0)
        s.advance(0, CUT)
    b = Batch(sims)
    sims[0].advance(CUT, 1)      # a member by itself, on the batch's kernel
    sims[1].advance(CUT, 1)
    b.advance(CUT + 1, STEPS - CUT - 1)
    for s, v in zip(sims, want):
        assert s.n_bad() == 0
        # FP64: the traces' own rounding; FP32: other orders of the same sums over 60 steps
        np.testing.assert_allclose(s.trace(), v, rtol=0, atol=1e-5 if precision == "fp64" else 0.02)
    fresh, _ = _sims(shapes, precision, n_warps)
    c = Batch(fresh)
    for x in (b, c):
        x.init(v0)
        x.advance(0, STEPS)
    for s, f in zip(sims, fresh):
        assert s.layout() == f.layout()
        np.testing.assert_array_equal(s.trace(), f.trace())
    b.close()
    c.close()
