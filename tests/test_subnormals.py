"""FP32 keeps subnormal numbers: parameters of that size act, and the forms
that skip their handling where it cannot matter give the bits of the general
ones for every float."""
from __future__ import annotations

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from helpers import numpy_cell_run

ROOT = Path(__file__).resolve().parents[1]
HEADERS = ("ngpu_math.cuh", "param_fold.cuh", "channels_ttpc.cuh")


def _probe(tmp):
    for name in ("product", "general"):
        (tmp / name).mkdir()
        for h in HEADERS:
            text = (ROOT / "neurogpu_b200" / "csrc" / h).read_text()
            if name == "general":
                head, mark, body = text.partition("struct Math<float> {")
                for special, plain in (("::ex1(", "::ex("), ("::dvn(", "::dv("), (" ex1(-z)", " ex(-z)"),
                                       ("return ex1(x) - 1.0f", "return ex(x) - 1.0f")):
                    body = body.replace(special, plain)
                text = head + mark + body if mark else head.replace("::ex1(", "::ex(").replace("::dvn(", "::dv(")
            (tmp / name / h).write_text(f"// {name}\n" + text)  # (pragma once skips a file of the same content)
    lib = tmp / "probe.so"
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3", "-Xcompiler", "-fPIC",
                    "-shared", "--expt-relaxed-constexpr", "-I", str(tmp),
                    str(ROOT / "tests" / "native" / "subnormal_probe.cu"), "-o", str(lib)], check=True,
                   capture_output=True)
    return lib


def test_the_probe_compares_two_forms(tmp_path):
    """The copies differ (ex1 and dvn only in the product's), and both compile."""
    _probe(tmp_path)
    product = (tmp_path / "product" / "channels_ttpc.cuh").read_text()
    general = (tmp_path / "general" / "channels_ttpc.cuh").read_text()
    assert "::ex1(" in product and "::dvn(" in product
    assert "::ex1(" not in general and "::dvn(" not in general


@pytest.mark.gpu
def test_the_special_forms_give_the_general_bits_for_every_float(tmp_path):
    import torch
    L = C.CDLL(str(_probe(tmp_path)))
    n = L.probe_outputs()
    differ = torch.zeros(n, dtype=torch.int64, device="cuda")
    at = torch.zeros(n, dtype=torch.int32, device="cuda")
    assert L.probe_compare(C.c_void_p(differ.data_ptr()), C.c_void_p(at.data_ptr())) == 0
    bad = {k: (int(differ[k]), hex(int(at[k]) & 0xFFFFFFFF)) for k in range(n) if differ[k]}
    assert not bad


MOD = """
NEURON {
    SUFFIX faint
    NONSPECIFIC_CURRENT i
    RANGE g, e
}
UNITS { (mV) = (millivolt) (mA) = (milliamp) (S) = (siemens) }
PARAMETER {
    g = 2e-41 (S/cm2)
    e = -40 (mV)
}
ASSIGNED { v (mV) i (mA/cm2) }
BREAKPOINT { i = g*1e37*(v - e) }
"""


def _faint(g_value, precision):
    from neurogpu_b200 import configs, nmodl
    from neurogpu_b200.model import build_model
    from neurogpu_b200.sim import Simulator
    g = nmodl.generate({"faint": MOD}, name="faint").register()
    secs = configs.hh_morphology(np.random.default_rng(1), 40)
    regions = ("soma", "dend", "axon")
    cell = build_model(secs, g, regions, {r: ("faint",) for r in regions}, ra=100.0, cm_of_region={r: 1.0 for r in regions})
    params = np.broadcast_to(np.asarray(g.param_defaults, dtype=np.float32)[None, :, None],
                             (1, g.n_params, cell.n_sections)).copy()
    params[:, g.param_index("g_faint")] = np.float32(g_value)
    amps = configs.step_amps([0.1], 200, 0.025, 1.0, 50.0)
    s = Simulator(cell, 1, 1, precision)
    s.set_params(params)
    s.set_stimulus(amps, 0.025, 0, float(cell.area[0]))
    s.set_recording([0])
    s.init(-65.0)
    s.advance(0, 200)
    v = s.trace()[0, 0]
    assert s.n_bad() == 0
    s.close()
    cond = float(np.float32(g_value)) * 1e37

    def node(i, init, v, dt, st):
        return st, cond * (v + 40.0), cond
    return v, numpy_cell_run(cell, amps[0], np.full(200, np.float32(0.025)), 0, float(np.float32(cell.area[0])), [0],
                             -65.0, node)


# 2e-41 is subnormal in float32 (its value there, 14,272 x 2^-149, is what acts); FP64 reads the same float32
# parameter.  Bounds: FP32 V to 200 steps of its rounding, FP64 the traces' own; without the current V is 10 mV off
@pytest.mark.gpu
@pytest.mark.parametrize("precision,tol", [("fp32", 5e-3), ("fp64", 1e-5)])
def test_a_subnormal_parameter_acts(ngpu_built, precision, tol):
    v, want = _faint(2e-41, precision)
    assert np.max(np.abs(want[0] + 65.0)) > 5.0
    np.testing.assert_allclose(v, want, rtol=0, atol=tol)


@pytest.mark.gpu
def test_rates_that_are_both_subnormal_keep_their_ratio(ngpu_built):
    """A gate whose opening and closing rates are 1e-40 of the usual ones stays at its initial value, their ratio."""
    from neurogpu_b200 import configs
    from neurogpu_b200.sim import Simulator
    w = configs.hh_active(n_sets=1, t_stop=5.0, n_comp=60)
    p = w.params.copy()
    for name in ("Ra_km", "Rb_km"):
        p[:, w.cell.mechset.param_index(name)] *= np.float32(1e-38) * np.float32(1e-2)
    assert 0 < p[0, w.cell.mechset.param_index("Ra_km")].max() < 1.1e-38
    out = {}
    for precision in ("fp32", "fp64"):
        s = Simulator(w.cell, 1, 1, precision)
        s.set_params(p)
        s.set_stimulus(configs.step_amps([0.1], w.nt, w.dt, 1.0, 50.0), w.dts, w.stim_node, w.stim_area)
        s.set_recording([0])
        s.init(w.v_init)
        s.advance(0, w.nt)
        out[precision] = s.trace()
        assert s.n_bad() == 0
        s.close()
    # the ratio is as good as the rates' leading bits (1e-43: six of them): a few per cent of km's conductance
    np.testing.assert_allclose(out["fp32"], out["fp64"], rtol=0, atol=0.3)
