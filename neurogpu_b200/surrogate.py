"""Surrogate network: (parameters, stimulus protocol) -> trace feature vector.

A 4-layer MLP (in -> 512 -> 512 -> 512 -> out, GELU in its tanh form) whose
forward and backward products all run on the project's tcgen05 BF16 GEMM
(FP32 accumulation in tensor memory) with fused epilogues:
  forward   Z = H W^T + b, H' = gelu(Z)      (Z fp32, H' bf16 and its transpose
                                              for the weight gradients; a
                                              prediction writes H' alone)
  output    Y = H W^T + b
  backward  dZ = (dZ_next W) * gelu'(Z)      (bf16 + transpose)
            dW = dZ^T H                      (K, the batch, split over CTAs)
Operand preparation, the loss, bias gradients and the Adam step (FP32 master
weights and their bf16 copies) are kernels of their own (csrc/mlp.cuh); each
of predict, loss_and_grads and adam_step is one library call.  PyTorch holds
the buffers.

Shapes are padded for the tensor cores: the input width to a multiple of 64,
the output to 32, the batch to a multiple of 128 (padding rows carry zero
loss gradient).  Inputs and targets are standardised with statistics fixed
at the first fit.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np

from . import _ffi

def _pad(n: int, m: int) -> int:
    return (n + m - 1) // m * m


def _p(x):
    return None if x is None else C.c_void_p(x.data_ptr())


def _ptrs(xs):
    return (C.c_void_p * len(xs))(*[x.data_ptr() for x in xs])


class SurrogateMLP:
    def __init__(self, n_in: int, n_out: int, width: int = 512, seed: int = 0, lr: float = 1e-3):
        import torch
        self.torch = torch
        self.dev = torch.device("cuda")
        self.n_in, self.n_out, self.width = n_in, n_out, width
        self.k_in = _pad(n_in, 64)
        self.n_out_p = _pad(max(n_out, 16), 32)
        dims = [(width, self.k_in), (width, width), (width, width), (self.n_out_p, width)]
        g = torch.Generator(device="cpu").manual_seed(seed)
        self.W, self.b = [], []
        for k, (n, kk) in enumerate(dims):
            fan_in = n_in if k == 0 else width
            w = torch.randn(n, kk, generator=g) / math.sqrt(fan_in)
            if k == 0:
                w[:, n_in:] = 0.0
            if k == 3:
                w[n_out:, :] = 0.0
            self.W.append(w.to(self.dev).float().contiguous())
            self.b.append(torch.zeros(n, device=self.dev))
        self.m = [torch.zeros_like(w) for w in self.W] + [torch.zeros_like(b) for b in self.b]
        self.v = [torch.zeros_like(t) for t in self.m]
        self.step_n = 0
        self.lr = lr
        self.x_mu = self.x_sd = self.y_mu = self.y_sd = None
        self._refresh()

    # -------------------------------------------------------------- plumbing
    def _refresh(self):
        """bf16 copies of the weights, row-major [N][K] and transposed [K][N]
        (the backward data GEMM reads W through its transpose); the output
        layer's transpose is padded to K = 64."""
        t = self.torch
        self.Wb = [w.to(t.bfloat16).contiguous() for w in self.W]
        self.Wtb = []
        for k, w in enumerate(self.W):
            wt = w.t().contiguous()
            if k == 3:
                wt = t.nn.functional.pad(wt, (0, 64 - self.n_out_p))
            self.Wtb.append(wt.to(t.bfloat16).contiguous())

    def _f32(self, x, *shape):
        """x as a contiguous float32 tensor of this shape on the network's device (broadcast as in arithmetic)."""
        t = self.torch
        return t.as_tensor(x, dtype=t.float32, device=self.dev).expand(*shape).contiguous()

    def _stats(self, mu, sd, n):
        """Standardisation of n columns as the kernels take it: two float32 vectors (or None, None for none).
        Statistics of another type, or given per row, are None: they are applied in torch's arithmetic."""
        if mu is None:
            return None, None
        t = self.torch
        if all(type(x) is t.Tensor and x.dtype == t.float32 and x.shape == (n,) and x.is_cuda and x.is_contiguous()
               for x in (mu, sd)):
            return mu, sd  # what fit_stats makes, as it is
        mu, sd = (t.as_tensor(x, device=self.dev) for x in (mu, sd))
        if any(x.dtype != t.float32 or tuple(x.shape) not in ((), (1,), (n,), (1, 1), (1, n)) for x in (mu, sd)):
            return None
        return tuple(x.reshape(-1).expand(n).contiguous() for x in (mu, sd))

    def _standardised(self, x, mu, sd, n):
        """(x, mean, deviation): x itself with what the kernels are to apply to it, or x standardised and None, None."""
        v = self._stats(mu, sd, n)
        return ((x - mu) / sd, None, None) if v is None else (x, *v)

    def _workspace(self, M, train):
        n = int(_ffi.lib().ngpu_mlp_workspace_bytes(M, self.width, self.k_in, self.n_out_p, int(train)))
        return self.torch.empty(max(n, 1), dtype=self.torch.uint8, device=self.dev), n

    def _stream(self):
        return C.c_void_p(self.torch.cuda.current_stream().cuda_stream)

    # ------------------------------------------------------------------- API
    def fit_stats(self, X, Y):
        t = self.torch
        X = t.as_tensor(X, dtype=t.float32, device=self.dev)
        Y = t.as_tensor(Y, dtype=t.float32, device=self.dev)
        self.x_mu, self.x_sd = X.mean(0), X.std(0).clamp(min=1e-6)
        self.y_mu, self.y_sd = Y.mean(0), Y.std(0).clamp(min=1e-6)

    def predict(self, X):
        """Features (original units) for inputs X [M, n_in]."""
        t = self.torch
        X = t.as_tensor(X, dtype=t.float32, device=self.dev)
        M = X.shape[0]
        X, x_mu, x_sd = self._standardised(X, self.x_mu, self.x_sd, self.n_in)
        X = self._f32(X, M, self.n_in)
        y_stats = self._stats(self.y_mu, self.y_sd, self.n_out)
        y_mu, y_sd = y_stats or (None, None)
        out = t.empty(M, self.n_out, device=self.dev)
        ws, n = self._workspace(M, False)
        _ffi.check("ngpu_mlp_predict", _ffi.lib().ngpu_mlp_predict(
            _p(X), M, self.n_in, _p(x_mu), _p(x_sd), _ptrs(self.Wb), _ptrs(self.b), self.width, self.k_in, self.n_out,
            self.n_out_p, _p(y_mu), _p(y_sd), _p(ws), n, _p(out), self._stream()))
        return out if y_stats is not None else out * self.y_sd + self.y_mu

    def loss_and_grads(self, X, Y, weight=None):
        """Mean squared error on standardised targets and the gradients of
        every weight and bias (lists in layer order)."""
        t = self.torch
        X = t.as_tensor(X, dtype=t.float32, device=self.dev)
        M = X.shape[0]
        Y = t.as_tensor(Y, dtype=t.float32, device=self.dev)
        X, x_mu, x_sd = self._standardised(X, self.x_mu, self.x_sd, self.n_in)
        Y, y_mu, y_sd = self._standardised(Y, self.y_mu, self.y_sd, self.n_out)
        X, Y = self._f32(X, M, self.n_in), self._f32(Y, M, self.n_out)
        if weight is not None:
            weight = self._f32(weight, M)
        ws, n = self._workspace(M, True)
        loss = t.empty((), device=self.dev)
        gW, gb = [t.empty(w.shape, device=self.dev) for w in self.W], [t.empty(b.shape, device=self.dev) for b in self.b]
        _ffi.check("ngpu_mlp_grads", _ffi.lib().ngpu_mlp_grads(
            _p(X), _p(Y), _p(weight), M, self.n_in, _p(x_mu), _p(x_sd), _p(y_mu), _p(y_sd), _ptrs(self.Wb), _ptrs(self.Wtb),
            _ptrs(self.b), self.width, self.k_in, self.n_out, self.n_out_p, _p(ws), n, _p(loss), _ptrs(gW), _ptrs(gb),
            self._stream()))
        return loss, gW, gb

    def adam_step(self, gW, gb, lr=None, b1=0.9, b2=0.999, eps=1e-8):
        t = self.torch
        lr = self.lr if lr is None else lr
        self.step_n += 1
        params = self.W + self.b
        grads = [self._f32(g, *p.shape) for g, p in zip(list(gW) + list(gb), params)]
        plain = lambda x: x if x.is_cuda and x.dtype == t.float32 and x.is_contiguous() else self._f32(x, *x.shape)
        state = [[plain(x) for x in xs] for xs in (params, self.m, self.v)]
        wb = [t.empty(w.shape, device=self.dev, dtype=t.bfloat16) for w in self.W]
        wtb = [t.empty((w.shape[1], 64 if k == 3 else w.shape[0]), device=self.dev, dtype=t.bfloat16)
               for k, w in enumerate(self.W)]
        _ffi.check("ngpu_mlp_adam", _ffi.lib().ngpu_mlp_adam(
            _ptrs(state[0]), _ptrs(grads), _ptrs(state[1]), _ptrs(state[2]), _ptrs(wb), _ptrs(wtb), self.n_in,
            self.width, self.k_in, self.n_out, self.n_out_p, float(lr), float(b1), float(b2), float(eps),
            1 - b1 ** self.step_n, 1 - b2 ** self.step_n, self._stream()))
        for xs, ys in zip((params, self.m, self.v), state):
            for x, y in zip(xs, ys):
                if x is not y:
                    x.copy_(y)
        self.Wb, self.Wtb = wb, wtb

    def train(self, X, Y, epochs: int = 10, batch: int = 4096, lr: float | None = None, seed: int = 0,
              X_val=None, Y_val=None) -> list[float]:
        """Minibatch Adam; returns the mean training loss per epoch (and sets
        self.val_loss when a validation set is given)."""
        t = self.torch
        X = t.as_tensor(X, dtype=t.float32, device=self.dev)
        Y = t.as_tensor(Y, dtype=t.float32, device=self.dev)
        if self.x_mu is None:
            self.fit_stats(X, Y)
        g = t.Generator(device="cpu").manual_seed(seed)
        hist = []
        for ep in range(epochs):
            perm = t.randperm(X.shape[0], generator=g).to(self.dev)
            tot, nb = 0.0, 0
            for i in range(0, X.shape[0], batch):
                idx = perm[i:i + batch]
                loss, gW, gb = self.loss_and_grads(X[idx], Y[idx])
                self.adam_step(gW, gb, lr)
                tot += float(loss)
                nb += 1
            hist.append(tot / max(nb, 1))
        if X_val is not None:
            self.val_loss = float(self.loss_and_grads(X_val, Y_val)[0])
        return hist
