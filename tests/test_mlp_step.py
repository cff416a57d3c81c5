"""The surrogate network's library calls against torch: predictions in bf16
arithmetic, gradients and the Adam step, at row counts and widths around the
tiles (128 rows, 128 and 256 columns, 148 CTAs)."""
from __future__ import annotations

import numpy as np
import pytest


def _data(rows, n_in, n_out, seed):
    import torch
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(rows, n_in, generator=g, device="cuda"), torch.randn(rows, n_out, generator=g, device="cuda") * 3 + 1)


def _net(n_in, n_out, width, stats):
    import torch
    from neurogpu_b200.surrogate import SurrogateMLP
    net = SurrogateMLP(n_in, n_out, width=width, seed=2)
    g = torch.Generator(device="cuda").manual_seed(9)
    net.b = [0.1 * torch.randn(b.shape, generator=g, device="cuda") for b in net.b]
    net.b[3][n_out:] = 0.0
    if stats:
        net.fit_stats(*_data(500, n_in, n_out, 77))
    return net


def _forward(net, X):
    """The network on bf16 activations and weights, sums in FP64."""
    import torch
    x = X if net.x_mu is None else (X - net.x_mu) / net.x_sd
    h = torch.nn.functional.pad(x, (0, net.k_in - net.n_in)).bfloat16()
    hs, zs = [h], []
    for k in range(3):
        z = (h.double() @ net.Wb[k].double().t() + net.b[k].double()).float()
        h = torch.nn.functional.gelu(z, approximate="tanh").bfloat16()
        zs.append(z)
        hs.append(h)
    return (h.double() @ net.Wb[3].double().t() + net.b[3].double())[:, :net.n_out], hs, zs


@pytest.mark.gpu
@pytest.mark.parametrize("rows,width,n_in,n_out,stats", [
    (1, 64, 1, 1, False), (127, 128, 15, 20, True), (128, 192, 64, 32, True), (129, 256, 65, 33, True),
    (4700, 512, 15, 20, True), (4800, 512, 15, 20, True), (24576, 256, 15, 20, False), (300, 128, 15, 100, True)])
def test_predict(ngpu_built, rows, width, n_in, n_out, stats):
    net = _net(n_in, n_out, width, stats)
    X, _ = _data(rows, n_in, n_out, rows)
    y = _forward(net, X)[0]
    if stats:
        y = y * net.y_sd.double() + net.y_mu.double()
    got = net.predict(X)
    # a bf16 activation may round the other way where the sums or the tanh
    # (hardware approximation, 5e-4) differ: 2^-8 of a layer, through three layers
    err = float((got - y).norm() / (y - y.mean(0)).norm().clamp(min=1e-3 * y.norm()))
    assert got.shape == (rows, n_out) and err < 2e-2, err


@pytest.mark.gpu
@pytest.mark.parametrize("rows,width,n_out,weighted", [(1, 64, 1, False), (130, 128, 20, True), (1000, 192, 33, False),
                                                       (4096, 512, 20, True), (5000, 256, 64, False)])
def test_gradients_and_step(ngpu_built, rows, width, n_out, weighted):
    import torch
    net = _net(15, n_out, width, True)
    X, Y = _data(rows, 15, n_out, rows)
    wt = torch.rand(rows, device="cuda") + 0.5 if weighted else None
    loss, gW, gb = net.loss_and_grads(X, Y, wt)
    # the same network in double, differentiated by autograd (bf16 weights as they are)
    W = [w.double().requires_grad_(True) for w in net.Wb]
    b = [x.double().requires_grad_(True) for x in net.b]
    h = torch.nn.functional.pad(((X - net.x_mu) / net.x_sd).bfloat16().double(), (0, net.k_in - 15))
    for k in range(3):
        h = torch.nn.functional.gelu(h @ W[k].t() + b[k], approximate="tanh")
    diff = (h @ W[3].t() + b[3])[:, :n_out] - ((Y - net.y_mu) / net.y_sd).double()
    if weighted:
        diff = diff * wt.double()[:, None]
    ref = (diff * diff).sum() / (rows * n_out)
    assert float(loss) == pytest.approx(float(ref.detach()), rel=2e-2)
    # the library's dY leaves the weight out of the second factor: 2 diff / count
    dy = torch.nn.functional.pad(2 * diff.detach() / (rows * n_out), (0, net.n_out_p - n_out))
    out = h @ W[3].t() + b[3]
    grads = torch.autograd.grad(out, W + b, dy)
    for got, want in zip(list(gW) + list(gb), grads):
        assert got.shape == want.shape
        scale = float(want.norm())
        if scale:
            assert float((got - want).norm()) / scale < 3e-2   # the bound of the FP64 numpy test
    # Adam: exactly the update's formula on these gradients
    p0 = [x.clone().double() for x in net.W + net.b]
    net.m = [1e-2 * torch.randn_like(x) for x in net.m]
    net.v = [1e-4 * torch.rand_like(x) for x in net.v]
    m0, v0 = [x.double() for x in net.m], [x.double() for x in net.v]
    net.step_n = 41
    net.adam_step(gW, gb, lr=3e-3)
    c1, c2 = 1 - 0.9 ** 42, 1 - 0.999 ** 42
    for k, (p, g, m, v) in enumerate(zip(p0, list(gW) + list(gb), m0, v0)):
        m, v = 0.9 * m + 0.1 * g.double(), 0.999 * v + 0.001 * g.double() ** 2
        want = p - 3e-3 * (m / c1) / ((v / c2).sqrt() + 1e-8)
        if k == 0:
            want[:, 15:] = 0
        if k == 3:
            want[n_out:] = 0
        if k == 7:
            want[n_out:] = 0
        got = (net.W + net.b)[k]
        torch.testing.assert_close(got.double(), want, rtol=1e-5, atol=1e-6)
        torch.testing.assert_close(net.m[k].double(), m, rtol=1e-5, atol=1e-7)
        torch.testing.assert_close(net.v[k].double(), v, rtol=1e-5, atol=1e-9)
    for k in range(4):
        w = net.W[k].bfloat16()
        assert torch.equal(net.Wb[k], w)
        wt_ = torch.nn.functional.pad(w.t(), (0, 64 - net.n_out_p)) if k == 3 else w.t()
        assert torch.equal(net.Wtb[k], wt_)


@pytest.mark.gpu
@pytest.mark.parametrize("rows,width", [(100, 64), (4096, 512), (20000, 512)])
def test_chained_kernels_keep_their_order(ngpu_built, rows, width):
    """Calls back to back, whose workspaces are the same memory, and replayed
    from a CUDA graph give what each call gives alone (split sums of the
    weight gradients add in any order: 4,096 terms of FP32)."""
    import torch
    net = _net(15, 20, width, True)
    data = [_data(rows, 15, 20, 50 + k) for k in range(6)]

    def step(X, Y):
        loss, gW, gb = net.loss_and_grads(X, Y)
        return [net.predict(X), loss, *gb, *gW]

    alone = []
    for X, Y in data:
        alone.append([t.clone() for t in step(X, Y)])
        torch.cuda.synchronize()

    def same(got, want):
        for k, (g, w) in enumerate(zip(got, want)):
            if k < 6:
                assert torch.equal(g, w), k
            else:
                assert float((g - w).norm()) <= 1e-5 * float(w.norm()), k

    for got, want in zip([step(X, Y) for X, Y in data], alone):
        same(got, want)
    X, Y = data[0][0].clone(), data[0][1].clone()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = step(X, Y)
    for (x, y), want in zip(data, alone):
        X.copy_(x)
        Y.copy_(y)
        graph.replay()
        torch.cuda.synchronize()
        same(out, want)
