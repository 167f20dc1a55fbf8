"""Bounded waits of the plain factorisation, solve and product kernels that run
out: the launch ends, the call's status says so, and the next call is right.

The limit of a wait is set to 1 ns (starpu_gb300_set_wait_budget_ns), so that a
wait which is not satisfied at once runs out; results of those calls are
discarded.  Reference: numpy in FP64."""
import contextlib
import ctypes as C

import numpy as np
import pytest

from starpu_gb300 import DeviceBuffer
from starpu_gb300.native import IrInfo, check

pytestmark = pytest.mark.gpu

TIMEOUT_INFO = -1000
GB300_ETIMEDOUT = -110
P = {np.float32: "s", np.float64: "d"}
EPS = {np.float32: 2.0**-24, np.float64: 2.0**-53}


def up(a):
    return DeviceBuffer.from_array(np.asfortranarray(a))


@contextlib.contextmanager
def short_waits(gpu):
    prev = gpu.starpu_gb300_set_wait_budget_ns(1)
    try:
        yield
    finally:
        gpu.starpu_gb300_set_wait_budget_ns(prev)


def spd(n, seed):
    b = np.random.default_rng(seed).standard_normal((n, n))
    return b @ b.T / n + np.eye(n)


# one and several chunks of k; one and several tiles and items for a CTA
@pytest.mark.parametrize("m,n,k", [(512, 512, 64), (512, 512, 200), (2000, 1500, 130)])
def test_fp64_product_ends_when_a_wait_runs_out(gpu, m, n, k):
    rng = np.random.default_rng(k)
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((n, k)), rng.standard_normal((m, n))
    da, db = up(a), up(b)

    def product():
        dc = up(c)
        check(gpu.starpu_gb300_dgemm_nt_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
        check(gpu.starpu_gb300_stream_sync(None))
        return dc.download((m, n), np.float64)

    with short_waits(gpu):
        for _ in range(3):
            product()
            assert gpu.starpu_gb300_take_wait_status(None) == GB300_ETIMEDOUT
    assert gpu.starpu_gb300_take_wait_status(None) == 0
    bound = (k + 2) * 2.0**-53 * (np.abs(c) + np.abs(a) @ np.abs(b).T)
    assert np.all(np.abs(product() - (c - a @ b.T)) <= bound)


# FP32: the leaf, one cooperative launch, and panels; FP64: the leaf, with updates on the tensor cores
@pytest.mark.parametrize("dtype,n", [(np.float32, 64), (np.float32, 300), (np.float32, 4200), (np.float64, 64),
                                     (np.float64, 400), (np.float64, 1500)])
@pytest.mark.parametrize("has_info", [True, False])
def test_factorisation_reports_a_wait_that_runs_out(gpu, dtype, n, has_info):
    a = spd(n, n).astype(dtype)

    def factor():
        da, info = up(a), up(np.full(1, 7, np.int32))
        check(getattr(gpu, f"starpu_gb300_{P[dtype]}potrf")(None, n, da.ptr, n, 512, info.ptr if has_info else None))
        check(gpu.starpu_gb300_stream_sync(None))
        return np.tril(da.download((n, n), dtype)).astype(np.float64), int(info.download((1,), np.int32)[0])

    with short_waits(gpu):
        assert factor()[1] == (TIMEOUT_INFO if has_info else 7)
    assert gpu.starpu_gb300_take_wait_status(None) == (0 if has_info else GB300_ETIMEDOUT)
    l, info = factor()
    assert info == (0 if has_info else 7) and gpu.starpu_gb300_take_wait_status(None) == 0
    bound = 2 * (n + 1) * EPS[dtype] * np.sqrt(np.outer(np.diag(a), np.diag(a)).astype(np.float64))
    assert np.all(np.abs(a - l @ l.T) <= bound)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("has_info", [True, False])
def test_lu_leaf_reports_a_wait_that_runs_out(gpu, dtype, has_info):
    n = 200
    a = (np.random.default_rng(n).uniform(-1, 1, (n, n)) + n * np.eye(n)).astype(dtype)

    def factor():
        da, info = up(a), up(np.full(1, 7, np.int32))
        check(getattr(gpu, f"starpu_gb300_{P[dtype]}getrf_tile")(None, n, da.ptr, n, info.ptr if has_info else None))
        check(gpu.starpu_gb300_stream_sync(None))
        return da.download((n, n), dtype).astype(np.float64), int(info.download((1,), np.int32)[0])

    with short_waits(gpu):
        info = factor()[1]
    taken = gpu.starpu_gb300_take_wait_status(None)
    if dtype == np.float32:  # the FP64 leaf has CTA barriers, no waits
        assert info == (TIMEOUT_INFO if has_info else 7) and taken == (0 if has_info else GB300_ETIMEDOUT)
    out, info = factor()
    assert info == (0 if has_info else 7) and gpu.starpu_gb300_take_wait_status(None) == 0
    l, u = np.tril(out), np.triu(out, 1) + np.eye(n)
    assert np.all(np.abs(l @ u - a) <= 2 * (n + 1) * EPS[dtype] * (np.abs(l) @ np.abs(u)))


@pytest.mark.parametrize("dtype,n,nrhs", [(np.float32, 600, 3), (np.float64, 600, 3), (np.float64, 2300, 64)])
def test_solve_reports_a_wait_that_runs_out(gpu, dtype, n, nrhs):
    l = np.linalg.cholesky(spd(n, n)).astype(dtype)
    b = np.random.default_rng(n).uniform(-1, 1, (n, nrhs)).astype(dtype)
    dl = up(l)

    def solve():
        db = up(b)
        check(getattr(gpu, f"starpu_gb300_{P[dtype]}potrs")(None, n, nrhs, dl.ptr, n, db.ptr, n))
        status = gpu.starpu_gb300_take_wait_status(None)
        return db.download((n, nrhs), dtype).astype(np.float64), status

    with short_waits(gpu):
        assert solve()[1] == GB300_ETIMEDOUT
    x, status = solve()
    assert status == 0
    l64 = l.astype(np.float64)
    bound = 8 * n * EPS[dtype] * (np.abs(l64) @ (np.abs(l64.T) @ np.abs(x)) + np.abs(b))
    assert np.all(np.abs(l64 @ (l64.T @ x) - b) <= bound)


def test_batched_solve_reports_a_wait_that_runs_out(gpu):
    sizes = np.array([300, 64, 20], np.int32)
    mats = [spd(n, n) for n in sizes]
    rhs = [np.ones((n, 2)) for n in sizes]
    cat = lambda v: np.concatenate([m.ravel(order="F") for m in v])
    off = lambda v: np.concatenate([[0], np.cumsum([m.size for m in v])])[:-1].astype(np.int64)
    da, db, ao, bo = up(cat(mats)), up(cat(rhs)), off(mats), off(rhs)
    lw = gpu.starpu_gb300_dposv_batched_workspace(3, sizes.ctypes.data, 2)
    work, dx, status = DeviceBuffer(lw), up(cat(rhs)), np.zeros(3, np.int32)

    def solve():
        check(gpu.starpu_gb300_dposv_batched(None, 3, sizes.ctypes.data, da.ptr, ao.ctypes.data, db.ptr, bo.ctypes.data,
                                             dx.ptr, 2, 1e-13, 20, work.ptr, lw, status.ctypes.data, None))
        return status.copy()

    with short_waits(gpu):
        assert solve()[0] == -1000
    assert np.all(solve() >= 0)


def test_mixed_solve_does_not_take_a_wait_that_runs_out_for_a_bad_pivot(gpu):
    n, nb = 2500, 1280  # diagonal tiles above 1024: the plain factorisation, whose info is negative then
    a, b = spd(n, n), np.ones((n, 1))
    da, db, dx = up(a), up(b), up(b)
    lw = gpu.starpu_gb300_dsposv_workspace(n, 1, nb)
    work = DeviceBuffer(lw)

    def solve():
        info = IrInfo()
        rc = gpu.starpu_gb300_dsposv(None, n, 1, da.ptr, n, db.ptr, n, dx.ptr, n, nb, 3, 1e-12, 30, work.ptr, lw,
                                     C.byref(info))
        return rc, info.status, info.fallback

    with short_waits(gpu):
        assert solve() == (GB300_ETIMEDOUT, GB300_ETIMEDOUT, 0)
    assert solve() == (0, 0, 0)


def test_dposv_reports_both_phases_in_its_info(gpu):
    n = 600
    a, b = spd(n, n), np.ones((n, 3))
    da, db, info = up(a), up(b), up(np.zeros(1, np.int32))
    with short_waits(gpu):
        check(gpu.starpu_gb300_dposv(None, n, 3, da.ptr, n, db.ptr, n, 512, info.ptr))
        check(gpu.starpu_gb300_stream_sync(None))
    assert int(info.download((1,), np.int32)[0]) == TIMEOUT_INFO
    assert gpu.starpu_gb300_take_wait_status(None) == 0
