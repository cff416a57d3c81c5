"""Standardisation statistics in every form that arithmetic with the inputs
takes: numbers, one value, a row, one per row of the batch, double precision."""
from __future__ import annotations

import pytest

ROWS, N_IN, N_OUT = 130, 15, 20


def _forms(torch, mu, sd, rows):
    yield "number", float(mu.mean()), float(sd.mean())
    yield "one value", mu[:1].clone(), sd[:1].clone()
    yield "row", mu[None], sd[None]
    yield "per row", mu.expand(rows, -1) + 0.1 * torch.arange(rows, device="cuda")[:, None], sd.expand(rows, -1).clone()
    yield "double", mu.double(), sd.double()


@pytest.mark.gpu
def test_statistics_of_every_form(ngpu_built):
    import torch
    from neurogpu_b200.surrogate import SurrogateMLP
    g = torch.Generator(device="cuda").manual_seed(4)
    X = 2.0 + 3.0 * torch.randn(ROWS, N_IN, generator=g, device="cuda")
    Y = 5.0 + 2.0 * torch.randn(ROWS, N_OUT, generator=g, device="cuda")
    forms = zip(_forms(torch, X.mean(0), X.std(0), ROWS), _forms(torch, Y.mean(0), Y.std(0), ROWS))
    for (name, x_mu, x_sd), (_, y_mu, y_sd) in forms:
        net, bare = SurrogateMLP(N_IN, N_OUT, width=128), SurrogateMLP(N_IN, N_OUT, width=128)
        net.x_mu, net.x_sd, net.y_mu, net.y_sd = x_mu, x_sd, y_mu, y_sd
        xs, ys = ((X - x_mu) / x_sd).float(), ((Y - y_mu) / y_sd).float()
        got, want = net.predict(X), bare.predict(xs) * y_sd + y_mu
        # the same network on the same bf16 inputs; the outputs' own rounding (and one of a double's)
        torch.testing.assert_close(got.double(), want.double(), rtol=1e-6, atol=1e-5, msg=name)
        (l0, w0, b0), (l1, w1, b1) = net.loss_and_grads(X, Y), bare.loss_and_grads(xs, ys)
        # split-K sums are added in any order
        torch.testing.assert_close(l0, l1, rtol=1e-5, atol=0)
        for a, b in zip(w0 + b0, w1 + b1):
            torch.testing.assert_close(a, b, rtol=1e-3, atol=1e-5 * float(b.abs().max()))
