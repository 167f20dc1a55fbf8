"""Calls of several host threads on streams of their own: the cooperative launches
(plain FP32 factorisation, batched solve) beside one another and beside FP64
products, each with the result that it has alone."""
import threading

import numpy as np
import pytest
import torch

from starpu_gb300.native import check

pytestmark = pytest.mark.gpu


def spd(n, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    b = torch.randn(n, n, device="cuda", generator=g, dtype=torch.float64)
    return (b @ b.T / n + torch.eye(n, device="cuda", dtype=torch.float64)).to(dtype)


def factor(gpu, n, dtype, seed):
    a, letter = spd(n, dtype, seed), "s" if dtype == torch.float32 else "d"
    w, info = torch.empty_like(a), torch.zeros(1, dtype=torch.int32, device="cuda")

    def call(stream):
        w.copy_(a)
        check(getattr(gpu, f"starpu_gb300_{letter}potrf")(stream, n, w.data_ptr(), n, 256, info.data_ptr()))
        return torch.cat([w.reshape(-1).double(), info.double()])
    return call


def batch(gpu, sizes, seed):
    ns = np.array(sizes, np.int32)
    mats = [spd(n, torch.float64, seed + n).reshape(-1) for n in sizes]
    off = lambda c: np.concatenate([[0], np.cumsum(c)])[:-1].astype(np.int64)
    a, ao, bo = torch.cat(mats), off(ns.astype(np.int64) ** 2), off(ns.astype(np.int64) * 3)
    b = torch.ones(3 * int(ns.sum()), dtype=torch.float64, device="cuda")
    x, status = torch.empty_like(b), np.zeros(len(ns), np.int32)
    lw = gpu.starpu_gb300_dposv_batched_workspace(len(ns), ns.ctypes.data, 3)
    work = torch.empty(lw, dtype=torch.uint8, device="cuda")

    def call(stream):
        check(gpu.starpu_gb300_dposv_batched(stream, len(ns), ns.ctypes.data, a.data_ptr(), ao.ctypes.data, b.data_ptr(),
                                             bo.ctypes.data, x.data_ptr(), 3, 1e-12, 20, work.data_ptr(), lw,
                                             status.ctypes.data, None))
        assert np.all(status >= 0)
        return x.clone()
    return call


def test_cooperative_launches_on_several_streams(gpu):
    calls = [factor(gpu, 1500, torch.float32, 1), factor(gpu, 300, torch.float32, 2), batch(gpu, [1000, 300, 64] * 20, 3),
             batch(gpu, [30, 500] * 40, 4), factor(gpu, 1100, torch.float64, 5)]
    torch.cuda.synchronize()
    alone = []
    for c in calls:
        alone.append(c(torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
    wrong = []

    def worker(i):
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(8):
                out = calls[i](s.cuda_stream)
                s.synchronize()
                if not torch.equal(out, alone[i]):
                    wrong.append(i)
    threads = [threading.Thread(target=worker, args=(i,)) for i in range(len(calls))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong
