"""Bounded waits of the plain factorisation, solve and product kernels that run
out: the launch ends, the call's status says so, and the next call is right.

The limit of a wait is set to 1 ns (starpu_gb300_set_wait_budget_ns), so that a
wait which is not satisfied at once runs out; results of those calls are
discarded.  Reference: numpy in FP64."""
import contextlib

import numpy as np
import pytest

from starpu_gb300 import DeviceBuffer
from starpu_gb300.native import check

pytestmark = pytest.mark.gpu

TIMEOUT_INFO = -1000


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
    bound = (k + 2) * 2.0**-53 * (np.abs(c) + np.abs(a) @ np.abs(b).T)
    assert np.all(np.abs(product() - (c - a @ b.T)) <= bound)


@pytest.mark.parametrize("n", [400, 1500])
def test_fp64_factorisation_reports_a_wait_that_runs_out(gpu, n):
    a = spd(n, n)

    def factor():
        da, info = up(a), up(np.full(1, 7, np.int32))
        check(gpu.starpu_gb300_dpotrf(None, n, da.ptr, n, 512, info.ptr))
        check(gpu.starpu_gb300_stream_sync(None))
        return np.tril(da.download((n, n), np.float64)), int(info.download((1,), np.int32)[0])

    with short_waits(gpu):
        assert factor()[1] == TIMEOUT_INFO
    l, info = factor()
    assert info == 0
    assert np.all(np.abs(a - l @ l.T) <= 2 * (n + 1) * 2.0**-53 * np.sqrt(np.outer(np.diag(a), np.diag(a))))
