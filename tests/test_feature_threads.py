"""Features asked for by several host threads at once, each on its own stream
and with another number of stretches (14 KB to 224 KB of shared memory a
block): no call is refused, and each gives what it gives alone."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest

CALLS = 20000


@pytest.mark.gpu
def test_threads_with_different_trace_lengths(ngpu_built):
    import torch
    from neurogpu_b200 import _ffi, features
    rng = np.random.default_rng(3)
    L = _ffi.lib()
    jobs = []
    for n, nt in ((1, 64), (1, 1100), (3, 130), (2, 1024), (1, 70), (1, 2000)):
        v = (-70.0 + 90.0 * (rng.random((n, nt)) < 0.05) * rng.random((n, nt))).astype(np.float32)
        t = torch.from_numpy(v).cuda()
        want = features.extract_device(t, 0.1, 0.0, 0.1 * nt).cpu()
        jobs.append((t, torch.empty_like(want, device="cuda"), want, torch.cuda.Stream()))
    torch.cuda.synchronize()
    refused = []
    start = threading.Barrier(len(jobs))

    def work(t, out, stream):
        n, nt = t.shape
        args = (C.c_void_p(t.data_ptr()), C.c_int64(t.stride(0)), C.c_int64(t.stride(1)), C.c_int32(n), C.c_int32(nt),
                C.c_double(0.1), C.c_double(0.0), C.c_double(0.1 * nt), C.c_float(features.THRESHOLD),
                C.c_void_p(out.data_ptr()), C.c_void_p(stream.cuda_stream))
        start.wait()
        refused.append(sum(L.ngpu_trace_features(*args) != 0 for _ in range(CALLS)))

    threads = [threading.Thread(target=work, args=(t, out, stream)) for t, out, _, stream in jobs]
    for th in threads:
        th.start()
    for th in threads:
        th.join()
    torch.cuda.synchronize()
    assert sum(refused) == 0, refused
    for _, out, want, _ in jobs:
        assert torch.equal(out.cpu(), want)
