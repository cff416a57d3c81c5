"""A team's CTAs that reach a launch's start at different times: the kernel is
compiled with one CTA of each cluster held back by a quarter of a millisecond
(many skeleton solves long; another CTA in each launch) before it touches the
group's memory, and gives the bits of the kernel without the delay."""
from __future__ import annotations

import os
import shutil
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
HEADERS = ["ngpu_math.cuh", "param_fold.cuh", "node_classes.cuh", "channels_ttpc.cuh", "channels_mainen.cuh",
           "sim_kernels.cuh"]
START = "    Group<R> G = group_of(A, g);\n    const int w = threadIdx.x >> 5;\n    const NodeRec<R>* nr = stage_nodes(A, smem);\n"
DELAY = "    if (TEAM && cluster_rank() == t0 % A.team) for (int k = 0; k < 250; ++k) __nanosleep(1000);\n"

RUN = """
import sys
import numpy as np
sys.path.insert(0, {root!r})
from neurogpu_b200 import configs
from neurogpu_b200.sim import Simulator
w = configs.hh_active(n_sets=11, t_stop=2.5, n_comp=500) if {cell!r} == "hh" else configs.ttpc_like(n_sets=8, t_stop=1.5)
s = Simulator(w.cell, w.n_sets, w.n_stim, {precision!r})
s.set_params(w.params)
s.set_stimulus(configs.step_amps([0.7 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0), w.dts,
               w.stim_node, w.stim_area)
s.set_recording([0, w.cell.n_nodes // 2, w.cell.n_nodes - 1])
out = []
for steps in (1, 7, w.nt):
    s.init(w.v_init)
    for t in range(0, w.nt, steps):
        s.advance(t, min(steps, w.nt - t))
    out.append(s.trace())
    assert s.n_bad() == 0
np.save({out!r}, np.stack(out))
"""


def _run(tmp, cell, precision, cache, name, **env):
    out = tmp / f"{name}.npy"
    code = RUN.format(root=str(ROOT), cell=cell, precision=precision, out=str(out))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300,
                   env=dict(os.environ, NGPU_JIT_CACHE=str(cache), **env))
    return np.load(out)


def _kernel(tmp, unit, name, delay):
    """unit compiled against the kernel headers, with or without the delay: a cubin."""
    inc = tmp / name
    inc.mkdir()
    for h in HEADERS:
        shutil.copy(ROOT / "neurogpu_b200" / "csrc" / h, inc / h)
    text = (inc / "sim_kernels.cuh").read_text()
    assert text.count(START) == 1
    if delay:
        (inc / "sim_kernels.cuh").write_text(text.replace(START, DELAY + START))
    cubin = inc / "unit.cubin"
    subprocess.run(["nvcc", "-cubin", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-I", str(inc),
                    str(unit), "-o", str(cubin)], check=True, capture_output=True)
    return cubin


@pytest.mark.gpu
@pytest.mark.parametrize("cell,precision", [("hh", "fp32"), ("ttpc", "fp32"), ("hh", "fp64")])
def test_late_ctas_change_nothing(ngpu_built, tmp_path, cell, precision):
    dump, cache = tmp_path / "dump", tmp_path / "cache"
    dump.mkdir()
    plain = _run(tmp_path, cell, precision, cache, "plain", NGPU_JIT_DUMP=str(dump))
    np.testing.assert_array_equal(plain[0], plain[2])
    units = [u for u in dump.glob("*.cu") if "A.team" in u.read_text()]
    assert len(units) == 1
    got = {}
    for name, delay in (("level", False), ("late", True)):
        shutil.copy(_kernel(tmp_path, units[0], name + "_inc", delay), cache / (units[0].stem + ".cubin"))
        got[name] = _run(tmp_path, cell, precision, cache, name + "_out")
    np.testing.assert_array_equal(got["late"], got["level"])
    np.testing.assert_array_equal(got["level"][0], got["level"][2])


# 60 steps from rest, before any spike: each step rounds V and a node's sums a few times (4e-6 mV each), in another
# order for each split
@pytest.mark.gpu
@pytest.mark.parametrize("cell,n,sets", [("hh", 500, 11), ("hh", 161, 3), ("ttpc", 1501, 8), ("passive", 170, 70)])
def test_teams_round_as_one_cta(ngpu_built, monkeypatch, cell, n, sets):
    from neurogpu_b200 import configs
    from neurogpu_b200.sim import Simulator
    w = {"hh": lambda: configs.hh_active(n_sets=sets, t_stop=1.5, n_comp=n),
         "ttpc": lambda: configs.ttpc_like(n_sets=sets, t_stop=1.5),
         "passive": lambda: configs.passive_cable(n_sets=sets, t_stop=1.5, n_comp=n)}[cell]()
    out = []
    for team in (None, "0"):
        if team is not None:
            monkeypatch.setenv("NGPU_TEAM", team)
        s = Simulator(w.cell, w.n_sets, w.n_stim, "fp32")
        s.set_params(w.params)
        s.set_stimulus(configs.step_amps([0.1 * (k + 1) for k in range(w.n_stim)], w.nt, w.dt, 0.25, 100.0), w.dts,
                       w.stim_node, w.stim_area)
        s.set_recording([0, n // 2, n - 1])
        s.init(w.v_init)
        s.advance(0, w.nt)
        out.append(s.trace())
        s.close()
    np.testing.assert_allclose(out[0], out[1], rtol=0, atol=5e-4)
