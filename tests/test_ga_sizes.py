"""GA selection at the sizes where its kernels change: tiles of the sort,
words of two ranks, blocks of the counting kernels, and the largest set the
rank-based path takes against the path above it."""
from __future__ import annotations

import sys
from pathlib import Path

import numpy as np
import pytest

sys.path.insert(0, str(Path(__file__).resolve().parents[1] / "oracle"))
import ga_numpy  # noqa: E402


def _objectives(rng, n, m):
    """Correlated objectives with ties, duplicates, NaN, infinities and signed zeros."""
    f = np.round(rng.uniform(0, 1, (n, 1)) * 2 + rng.uniform(0, 1, (n, m)), 2)
    f[rng.integers(0, n, max(1, n // 20))] = f[rng.integers(0, n, max(1, n // 20))]
    for v in (np.nan, np.inf, -np.inf, 0.0, -0.0):
        f[rng.integers(0, n, max(1, n // 50)), rng.integers(0, m, max(1, n // 50))] = v
    return f


@pytest.mark.gpu
@pytest.mark.parametrize("n,m", [(1, 1), (2, 2), (31, 3), (64, 17), (65, 2), (255, 33), (256, 65), (257, 1), (1025, 128),
                                 (2048, 3), (2049, 5), (300, 129), (300, 192)])
def test_nsga2_at_the_edges(ngpu_built, n, m):
    import torch
    from neurogpu_b200.ga_device import select_nsga2, select_truncation
    f = _objectives(np.random.default_rng(n + m), n, m)
    mu = max(1, n // 2)
    idx, rank, crowd, fronts = select_nsga2(torch.tensor(f, device="cuda"), mu)
    with np.errstate(all="ignore"):
        w_idx, w_rank, w_crowd = ga_numpy.select_nsga2(f, mu)[:3]
    np.testing.assert_array_equal(rank.cpu().numpy(), w_rank)
    np.testing.assert_array_equal(crowd.cpu().numpy(), w_crowd)
    np.testing.assert_array_equal(idx.cpu().numpy(), w_idx)
    assert int(fronts) == int(w_rank.max()) + 1
    score = f[:, 0]
    np.testing.assert_array_equal(select_truncation(torch.tensor(score, device="cuda"), mu).cpu().numpy(),
                                  ga_numpy.select_truncation(score, mu))


@pytest.mark.gpu
@pytest.mark.parametrize("m", [2, 7])
def test_both_paths_agree_at_their_border(ngpu_built, m):
    """16,384 individuals, and the same with one more that all of them
    dominate: it makes a front of its own and changes nothing else."""
    import torch
    from neurogpu_b200.ga_device import select_nsga2, select_truncation
    rng = np.random.default_rng(m)
    f = np.round(rng.uniform(0, 1, (16384, m)), 3)
    a = select_nsga2(torch.tensor(f, device="cuda"), 16384)
    b = select_nsga2(torch.tensor(np.vstack([f, np.full((1, m), 2.0)]), device="cuda"), 16385)
    assert int(b[3]) == int(a[3]) + 1 and int(b[1][-1]) == int(a[3])
    for x, y in zip(a[:3], b[:3]):
        assert torch.equal(x, y[:16384])
    s = torch.tensor(np.append(f[:, 0], 5.0), device="cuda")
    assert torch.equal(select_truncation(s[:16384], 16384), select_truncation(s, 16385)[:16384])


@pytest.mark.gpu
def test_offspring_of_one_gene_and_many(ngpu_built):
    import torch
    from neurogpu_b200.ga_device import DeviceGA
    for genes, kids in ((1, 1), (1, 129), (7, 127), (200, 3)):
        rng = np.random.default_rng(genes)
        pop, rank, crowd = rng.uniform(-1, 1, (9, genes)), rng.integers(0, 3, 9).astype(np.int32), rng.uniform(0, 1, 9)
        ga = DeviceGA(genes, eta_c=20.0, eta_m=20.0, cx_prob=0.7, p_mut=0.3, seed=5)
        got = ga.offspring(torch.tensor(pop, device="cuda"), torch.tensor(rank, device="cuda"),
                           torch.tensor(crowd, device="cuda"), kids, 4).cpu().numpy()
        want = ga_numpy.offspring(pop, rank, crowd, kids, -1.0, 1.0, 20.0, 20.0, 0.7, 0.3, 5, 4)
        np.testing.assert_allclose(got, want, rtol=1e-12, atol=1e-15)
