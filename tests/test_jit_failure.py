"""Runtime compilation that is there when a simulation is laid out and fails
when its kernel is made: the library's own wide layouts (teams, CTAs of 16
and 12 warps) give way to the ahead-of-time kernels' CTAs, a layout that the
caller asked for is refused."""
from __future__ import annotations

import numpy as np
import pytest

from neurogpu_b200 import _ffi, configs

STEPS = 40


def _sim(sets, precision="fp64", n=200, **shape):
    from neurogpu_b200.sim import Simulator
    w = configs.hh_active(n_sets=1, t_stop=STEPS * 0.025, n_comp=n)
    s = Simulator(w.cell, sets, w.n_stim, precision, **shape)
    s.set_params(np.repeat(w.params, sets, axis=0))
    s.set_stimulus(configs.step_amps([0.7 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0), w.dts,
                   w.stim_node, w.stim_area)
    s.set_recording([0, n // 2, n - 1], rec_every=2)
    return s, w


# 11 sets: a team; 1,200: 113 groups, CTAs of 16 warps; 2,134: 201 groups, of 12
@pytest.mark.gpu
@pytest.mark.parametrize("sets", [11, 1200, 2134])
@pytest.mark.parametrize("under_way", [False, True])
def test_the_librarys_choice_gives_way(ngpu_built, monkeypatch, sets, under_way):
    s, w = _sim(sets)
    s.init(w.v_init)
    s.advance(0, STEPS)
    want = s.trace()
    s.close()
    s, w = _sim(sets)
    t = 0
    if under_way:  # the kernel goes when new values break one of its folds
        s.init(w.v_init)
        s.advance(0, 5)
        t = 5
    monkeypatch.setenv("NGPU_JIT", "0")
    if under_way:
        s.set_params(np.repeat(w.params, sets, axis=0))
    else:
        s.init(w.v_init)
    assert s.classes() == 0 and s.layout()["cta_warps"] <= 8
    s.advance(t, STEPS - t)
    np.testing.assert_allclose(s.trace(), want, rtol=0, atol=1e-5)  # FP64: the traces' own rounding
    assert s.n_bad() == 0
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("under_way", [False, True])
def test_a_batch_gives_way(ngpu_built, monkeypatch, under_way):
    from neurogpu_b200.sim import Batch
    alone = []
    for n in (120, 200):
        s, w = _sim(1100, n=n)
        s.init(w.v_init)
        s.advance(0, STEPS)
        alone.append(s.trace())
        s.close()
    sims = [_sim(1100, n=n)[0] for n in (120, 200)]
    if under_way:
        for s in sims:
            s.init(w.v_init)
            s.advance(0, 5)
    monkeypatch.setenv("NGPU_JIT", "1" if under_way else "0")
    b = Batch(sims)
    if under_way:
        monkeypatch.setenv("NGPU_JIT", "0")
        for n, s in zip((120, 200), sims):
            s.set_params(np.repeat(configs.hh_active(n_sets=1, t_stop=1.0, n_comp=n).params, 1100, axis=0))
    else:
        b.init(w.v_init)
    t = 5 if under_way else 0
    b.advance(t, STEPS - t)
    for s, v in zip(sims, alone):
        assert s.classes() == 0
        np.testing.assert_allclose(s.trace(), v, rtol=0, atol=1e-5)
    b.close()


@pytest.mark.gpu
def test_the_callers_choice_is_refused(ngpu_built, monkeypatch):
    s, w = _sim(11, n_warps=12)
    monkeypatch.setenv("NGPU_JIT", "0")
    with pytest.raises(_ffi.NgpuError, match="runtime compilation"):
        s.init(w.v_init)
    s.close()
