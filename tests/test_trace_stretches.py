"""Scores and features of traces cut into stretches of time: every cut gives
the counts of the whole trace, whatever its samples; the kernels at the
edges of their stretches, batches and blocks, in both trace layouts."""
from __future__ import annotations

import ctypes as C
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]
sys.path.insert(0, str(ROOT / "oracle"))
import find_peaks_ref as fpr  # noqa: E402


def _traces(rng, n, nt):
    """Spikes on noise, with runs of equal slopes, and in every trace after
    the first third some samples that the fast comparison does not take:
    zeros, tiny, huge and subnormal values, infinities, NaN."""
    v = -70.0 + rng.normal(0.0, 1.0, (n, nt))
    v[:, ::7] = np.round(v[:, ::7])
    for k in range(n):
        for t0 in rng.integers(0, max(1, nt - 8), 1 + nt // 60):
            v[k, t0:t0 + 4] += np.linspace(0, rng.uniform(5, 100), v[k, t0:t0 + 4].size)
        if nt > 30:
            t0 = rng.integers(0, nt - 20)
            v[k, t0:t0 + 19] = -70.0 + 2.0 * np.arange(19)  # one slope across batches
    odd = [0.0, -0.0, 1e-6, -3e-8, 1e-42, 300.0, -5e8, 3e38, np.inf, -np.inf, np.nan]
    for k in range(n // 3, n):
        for t0 in rng.integers(0, nt, 1 + nt // 40):
            v[k, t0] = odd[rng.integers(0, len(odd))]
    return v.astype(np.float32)


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    lib = tmp_path_factory.mktemp("stretch") / "probe.so"
    subprocess.run(["nvcc", "-std=c++17", "-O2", "-Xcompiler", "-fPIC", "-shared", "--expt-relaxed-constexpr",
                    str(ROOT / "tests" / "native" / "stretch_probe.cu"), "-o", str(lib)], check=True,
                   capture_output=True)
    L = C.CDLL(str(lib))
    L.probe_stretches.argtypes = [C.c_void_p, C.c_int, C.c_int64, C.c_double, C.c_double, C.c_int, C.c_int]
    return L


@pytest.mark.parametrize("nt", [1, 2, 3, 4, 8, 9, 16, 17, 63, 64, 65, 200])
@pytest.mark.parametrize("dt,height,distance", [(0.1, 15.0, 5), (0.025, 0.0, 1), (0.1, -1e30, 3), (1e-120, 15.0, 5)])
def test_every_cut_gives_the_whole_traces_count(probe, nt, dt, height, distance):
    rng = np.random.default_rng(nt)
    v = _traces(rng, 12, nt)
    with np.errstate(all="ignore"):
        want = [fpr.dvdt_peak_count(x, dt, height, distance) for x in v]
    for stretch in (8, 16, 24, 64, 208):
        got = [probe.probe_stretches(x.ctypes.data, nt, 1, dt, height, distance, stretch) for x in v]
        assert got == want, stretch
    wide = np.ascontiguousarray(np.repeat(v, 3, axis=1))  # a sample every third element
    got = [probe.probe_stretches(x.ctypes.data, nt, 3, dt, height, distance, 16) for x in wide]
    assert got == want


@pytest.mark.gpu
@pytest.mark.parametrize("n,nt", [(1, 3), (1, 4000), (2, 31), (31, 257), (33, 64), (65, 1001), (700, 300)])
@pytest.mark.parametrize("layout", ["trace_major", "sample_major", "odd_rows"])
def test_counts_at_the_edges(ngpu_built, n, nt, layout):
    import torch
    from neurogpu_b200 import explore
    v = _traces(np.random.default_rng(n * nt), n, nt)
    t = torch.from_numpy(v).cuda()
    if layout == "sample_major":
        t = t.t().contiguous().t()
    elif layout == "odd_rows":  # rows that do not start on 16 bytes
        t = torch.nn.functional.pad(t, (1, 2))[:, 1:1 + nt]
    with np.errstate(all="ignore"):
        want = [fpr.dvdt_peak_count(x, 0.1, 15.0, 5) for x in v]
    assert explore.dvdt_peak_counts(t).cpu().tolist() == want


@pytest.mark.gpu
@pytest.mark.parametrize("n,nt", [(1, 64), (3, 1001), (33, 257), (300, 2000)])
@pytest.mark.parametrize("layout", ["trace_major", "sample_major", "odd_rows"])
def test_features_at_the_edges(ngpu_built, n, nt, layout):
    """Against the batched torch statement, with the bounds the whole-trace
    kernel had: counts equal, times to float32, sums to their rounding."""
    import torch
    from neurogpu_b200 import features
    rng = np.random.default_rng(nt + n)
    v = -70.0 + rng.normal(0.0, 1.0, (n, nt))
    for k in range(n):
        for t0 in rng.integers(0, nt - 6, 1 + nt // (20 + 10 * (k % 5))):
            v[k, t0:t0 + 5] += [40.0, 90.0, 100.0, 60.0, 20.0]
    t = torch.from_numpy(v.astype(np.float32)).cuda()
    if layout == "sample_major":
        t = t.t().contiguous().t()
    elif layout == "odd_rows":
        t = torch.nn.functional.pad(t, (1, 2))[:, 1:1 + nt]
    for on, off in ((0.0, 0.1 * nt), (0.3, 0.1 * nt - 0.7), (0.05 * nt, 0.09 * nt)):
        got = features.extract_device(t, 0.1, on, off).cpu().numpy()
        want = features.extract(t.contiguous(), 0.1, on, off).cpu().numpy()
        np.testing.assert_array_equal(got[:, 0], want[:, 0])
        # the statement's mean of an empty window is NaN, the kernel's 0 (a window past the trace's end)
        np.testing.assert_allclose(got, np.where(np.isnan(want), 0.0, want), rtol=2e-5, atol=2e-4)


def _near_ties(rng, n):
    """Rises past zero whose neighbouring slopes differ by less than a
    float32 keeps, next to one that ends the peak or continues the rise."""
    out = []
    for k in range(n):
        x2 = np.float32(rng.uniform(0.005, 0.02))
        x3 = np.float32(48.0 + 2.0 * float(x2))
        lead = [np.float32(-96.0)] * int(rng.integers(8, 24)) + [np.float32(-95.0 + rng.uniform(0, 1))]
        out.append(np.array(lead + [-48.0, x2, x3, x3 + np.float32(48.5 if k % 2 else 40.0)] + [60.0] * 17,
                            np.float32))
    return out


def test_slopes_that_round_alike(probe):
    seen = set()
    for x in _near_ties(np.random.default_rng(5), 400):
        d = np.diff(x.astype(np.float64))
        k = int(np.argmax(x == -48.0))
        seen.add((np.sign(d[k + 1] - d[k]), bool(np.float32(d[k + 1]) == np.float32(d[k]))))
        want = fpr.dvdt_peak_count(x, 0.1, 15.0, 1)
        for stretch in (8, 16, 64):
            assert probe.probe_stretches(x.ctypes.data, x.size, 1, 0.1, 15.0, 1, stretch) == want
    assert {(1.0, True), (-1.0, True)} <= seen  # both orders, hidden by the rounding


@pytest.mark.gpu
def test_slopes_that_round_alike_on_the_gpu(ngpu_built):
    import torch
    from neurogpu_b200 import explore
    rows = [x for x in _near_ties(np.random.default_rng(6), 400)]
    v = np.stack([np.pad(x, (0, 64 - x.size), mode="edge") for x in rows])
    want = [fpr.dvdt_peak_count(x, 0.1, 15.0, 1) for x in v]
    got = explore.dvdt_peak_counts(torch.from_numpy(v).cuda(), distance=1).cpu().tolist()
    assert got == want
