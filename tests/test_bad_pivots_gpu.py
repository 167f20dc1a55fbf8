"""Factorisations that meet bad pivots: the first one is reported, and what was
finished before it stays.  Reference: numpy in FP64."""
import numpy as np
import pytest

from starpu_gb300 import DeviceBuffer
from starpu_gb300.native import check

pytestmark = pytest.mark.gpu

P = {np.float32: "s", np.float64: "d"}
EPS = {np.float32: 2.0**-24, np.float64: 2.0**-53}
BOTH = pytest.mark.parametrize("dtype", [np.float32, np.float64])


def up(a):
    return DeviceBuffer.from_array(np.asfortranarray(a))


@BOTH
@pytest.mark.parametrize("n,z", [(64, 1), (64, 6), (64, 30), (64, 37), (64, 63), (50, 33), (130, 100)])
def test_zero_pivot_leaves_earlier_rows_as_they_are(gpu, dtype, n, z):
    a = np.random.default_rng(n + z).uniform(-1, 1, (n, n)) + n * np.eye(n)
    a[z], a[:, z] = 0, 0
    a = a.astype(dtype)
    da, info = up(a), up(np.zeros(1, np.int32))
    check(getattr(gpu, f"starpu_gb300_{P[dtype]}getrf_tile")(None, n, da.ptr, n, info.ptr))
    out = da.download((n, n), dtype).astype(np.float64)
    assert info.download((1,), np.int32)[0] == z + 1
    # rows 0 .. z - 1 of U and the columns 0 .. z - 1 of L multiply to those rows of A
    assert np.all(np.isfinite(out[:z]))
    l, u = np.tril(out[:z, :z]), np.triu(out[:z], 1) + np.eye(z, n)
    assert np.all(np.abs(l @ u - a[:z]) <= 2 * (n + 1) * EPS[dtype] * (np.abs(l) @ np.abs(u)))


@BOTH
@pytest.mark.parametrize("n", [5, 64, 200])
def test_the_first_of_many_bad_pivots_is_reported(gpu, dtype, n):
    # from pivot z on every pivot is bad, and each is known at once to the warp that owns it
    for z in (0, 1, 2, 3, 4, n // 2, n - 1):
        chol, lu = np.eye(n, dtype=dtype), np.eye(n, dtype=dtype)
        chol[range(z, n), range(z, n)] = -1
        lu[range(z, n), range(z, n)] = 0
        for _ in range(20):
            dc, dl, info = up(chol), up(lu), up(np.zeros(2, np.int32))
            check(getattr(gpu, f"starpu_gb300_{P[dtype]}potrf")(None, n, dc.ptr, n, 64, info.ptr))
            check(getattr(gpu, f"starpu_gb300_{P[dtype]}getrf_tile")(None, n, dl.ptr, n, info.ptr + 4))
            assert info.download((2,), np.int32).tolist() == [z + 1, z + 1]
