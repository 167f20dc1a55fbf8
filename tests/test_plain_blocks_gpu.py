"""Plain FP32 / FP64 factorisation and solve kernels at the sizes where their
blocking changes: leaf and panel remainders, the row counts that pick the
panel solve's slab, the product tiles, the solve's block and column groups,
and the FP64 update on the tensor cores (tile, segment and row-block edges).
Reference: numpy in FP64."""
import ctypes

import numpy as np
import pytest

from starpu_gb300 import DeviceBuffer
from starpu_gb300.native import check

pytestmark = pytest.mark.gpu

EPS = {np.float32: 2.0**-24, np.float64: 2.0**-53}
P = {np.float32: "s", np.float64: "d"}
BOTH = pytest.mark.parametrize("dtype", [np.float32, np.float64])


def up(a):
    return DeviceBuffer.from_array(np.asfortranarray(a))


def spd(n, seed, scale=None):
    rng = np.random.default_rng(seed)
    b = rng.standard_normal((n, n))
    a = b @ b.T / n + np.eye(n)
    return a if scale is None else a * scale[:, None] * scale[None, :]


def fn(gpu, dtype, name):
    return getattr(gpu, "starpu_gb300_" + P[dtype] + name)


@BOTH
@pytest.mark.parametrize("m,n", [(1, 1), (3, 64), (17, 127), (2047, 70), (2048, 64), (2049, 130), (5, 1025), (2100, 1100)])
def test_trsm_slabs(gpu, dtype, m, n):
    l = np.linalg.cholesky(spd(n, n)).astype(dtype)
    b = np.random.default_rng(m).uniform(-1, 1, (m, n)).astype(dtype)
    dl, db = up(l), up(np.vstack([b, np.full((2, n), 7, dtype)]))  # two rows of padding below
    check(fn(gpu, dtype, "trsm_rltn_tile")(None, m, n, 1.0, dl.ptr, n, db.ptr, m + 2))
    out = db.download((m + 2, n), dtype)
    assert np.all(out[m:] == 7)
    x = out[:m].astype(np.float64)
    # each row solves L x = b with backward error <= c n eps |L| |x|
    bound = 4 * n * EPS[dtype] * (np.abs(x) @ np.abs(l.astype(np.float64)).T + np.abs(b))
    assert np.all(np.abs(x @ l.astype(np.float64).T - b) <= bound)


@BOTH
@pytest.mark.parametrize("n,nrhs", [(1, 1), (31, 3), (33, 4), (256, 1), (257, 5), (511, 17), (700, 64), (1030, 2)])
def test_potrs_blocks(gpu, dtype, n, nrhs):
    l = np.linalg.cholesky(spd(n, n)).astype(dtype)
    l[np.triu_indices(n, 1)] = np.nan  # never read
    b = np.random.default_rng(n + nrhs).uniform(-1, 1, (n, nrhs)).astype(dtype)
    dl, db = up(l), up(b)
    check(fn(gpu, dtype, "potrs")(None, n, nrhs, dl.ptr, n, db.ptr, n))
    x = db.download((n, nrhs), dtype).astype(np.float64)
    l = np.tril(np.nan_to_num(l)).astype(np.float64)
    y = np.abs(l.T) @ np.abs(x)
    bound = 8 * n * EPS[dtype] * (np.abs(l) @ y + np.abs(b))
    assert np.all(np.abs(l @ (l.T @ x) - b) <= bound)


@BOTH
@pytest.mark.parametrize("m,n,k", [(33, 31, 64), (300, 290, 65), (640, 700, 33), (1200, 1100, 64), (1700, 1650, 17)])
@pytest.mark.parametrize("lower", [False, True])
def test_product_tiles(gpu, dtype, m, n, k, lower):
    n = m if lower else n
    rng = np.random.default_rng(m + k)
    a, b, c = (rng.standard_normal(s).astype(dtype) for s in ((m, k), (n, k), (m, n)))
    b = a if lower else b
    da, db, dc = up(a), up(b), up(c)
    if lower:
        check(fn(gpu, dtype, "syrk_ln_tile")(None, n, k, -1.0, da.ptr, n, 1.0, dc.ptr, n))
    else:
        check(fn(gpu, dtype, "gemm_nt_tile")(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
    out = dc.download((m, n), dtype).astype(np.float64)
    a, b, c = (v.astype(np.float64) for v in (a, b, c))
    ref, bound = c - a @ b.T, (k + 2) * EPS[dtype] * (np.abs(c) + np.abs(a) @ np.abs(b).T)
    keep = np.tril(np.ones((m, n), bool)) if lower else np.ones((m, n), bool)
    assert np.all(np.abs(out - ref)[keep] <= bound[keep])
    assert np.array_equal(out[~keep], c[~keep])


# k a multiple of 4 with a remainder of 16, ragged tiles; ld of B (k) and of A and C (m) off the 16-byte grid
@pytest.mark.parametrize("m,n,k", [(1024, 1024, 32), (1100, 1033, 36), (1156, 1000, 4), (1028, 1030, 33), (1027, 1024, 64), (1024, 1, 8)])
def test_product_nn_tiles(gpu, m, n, k):
    rng = np.random.default_rng(m + k)
    a, b, c = (rng.standard_normal(s).astype(np.float32) for s in ((m, k), (k, n), (m, n)))
    da, db, dc = up(a), up(b), up(c)
    check(gpu.starpu_gb300_sgemm_nn_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, k, 1.0, dc.ptr, m))
    out = dc.download((m, n), np.float32).astype(np.float64)
    a, b, c = (v.astype(np.float64) for v in (a, b, c))
    assert np.all(np.abs(out - (c - a @ b)) <= (k + 2) * EPS[np.float32] * (np.abs(c) + np.abs(a) @ np.abs(b)))


@BOTH
@pytest.mark.parametrize("n,nb", [(63, 64), (65, 16), (127, 64), (191, 64), (192, 512), (193, 512), (321, 100), (700, 512), (1281, 256), (3001, 512), (4097, 1024)])
def test_potrf_blocks(gpu, dtype, n, nb):
    # rows and columns scaled over 12 orders of magnitude (FP32: 6)
    d = np.power(10.0, np.random.default_rng(n).uniform(-6, 6, n) * (1.0 if dtype == np.float64 else 0.5))
    a = spd(n, n, d).astype(dtype)
    lda = n + 1
    pad = np.full((lda, n), 3, dtype, order="F")
    pad[:n] = a
    da, info = up(pad), up(np.full(1, 9, np.int32))
    check(fn(gpu, dtype, "potrf")(None, n, da.ptr, lda, nb, info.ptr))
    out = da.download((lda, n), dtype)
    assert info.download((1,), np.int32)[0] == 0
    iu = np.triu_indices(n, 1)
    assert np.array_equal(out[:n][iu], a[iu]) and np.all(out[n] == 3)
    l = np.tril(out[:n]).astype(np.float64)
    a = a.astype(np.float64)
    # |A - L L^T| <= c (n + 1) eps |L| |L|^T, and |L| |L|^T <= sqrt(a_ii a_jj)
    s = np.sqrt(np.diag(a))
    assert np.all(np.abs(np.tril(a - l @ l.T)) <= 2 * (n + 1) * EPS[dtype] * s[:, None] * s[None, :])


@BOTH
@pytest.mark.parametrize("n,k", [(1, 1), (40, 3), (64, 64), (100, 65), (500, 130), (500, 331), (1000, 1000)])
def test_first_bad_pivot_is_reported(gpu, dtype, n, k):
    a = spd(n, n).astype(dtype)
    a[k - 1, k - 1] = -1.0
    da, info = up(a), up(np.zeros(1, np.int32))
    check(fn(gpu, dtype, "potrf")(None, n, da.ptr, n, 256, info.ptr))
    assert info.download((1,), np.int32)[0] == k


def test_fp64_update_keeps_nan_in_its_row(gpu):
    n, i = 400, 250
    a = spd(n, n)
    a[i, 10] = a[10, i] = np.nan
    da, info = up(a), up(np.zeros(1, np.int32))
    check(gpu.starpu_gb300_dpotrf(None, n, da.ptr, n, 64, info.ptr))
    out = da.download((n, n), np.float64)
    assert info.download((1,), np.int32)[0] == i + 1
    ref = np.linalg.cholesky(spd(n, n)[:i, :i])
    assert np.allclose(np.tril(out[:i, :i]), ref, rtol=0, atol=1e-13)


@BOTH
@pytest.mark.parametrize("n", [1, 3, 4, 5, 31, 33, 36, 63, 64, 65, 130])
def test_getrf_blocks(gpu, dtype, n):
    a = (np.random.default_rng(n).uniform(-1, 1, (n, n)) + n * np.eye(n)).astype(dtype)
    da, info = up(a), up(np.full(1, 5, np.int32))
    check(fn(gpu, dtype, "getrf_tile")(None, n, da.ptr, n, info.ptr))
    out = da.download((n, n), dtype).astype(np.float64)
    assert info.download((1,), np.int32)[0] == 0
    l, u = np.tril(out), np.triu(out, 1) + np.eye(n)
    bound = 2 * (n + 1) * EPS[dtype] * (np.abs(l) @ np.abs(u))
    assert np.all(np.abs(l @ u - a) <= bound)


@BOTH
@pytest.mark.parametrize("m,n", [(1, 1100), (64, 65), (70, 700), (700, 70), (1030, 33)])
def test_lu_panel_solves(gpu, dtype, m, n):
    rng = np.random.default_rng(m + n)
    for name, k in (("trsm_llnn_tile", m), ("trsm_runu_tile", n)):
        t = rng.uniform(-1, 1, (k, k)) / k
        t = np.tril(t) + np.eye(k) if k == m and name == "trsm_llnn_tile" else np.triu(t, 1)
        b = rng.uniform(-1, 1, (m, n))
        t, b = t.astype(dtype), b.astype(dtype)
        dt, db = up(t), up(b)
        check(fn(gpu, dtype, name)(None, m, n, dt.ptr, k, db.ptr, m))
        x, t64 = db.download((m, n), dtype).astype(np.float64), t.astype(np.float64)
        if name == "trsm_llnn_tile":
            got, mag = t64 @ x, np.abs(t64) @ np.abs(x)
        else:
            u = t64 + np.eye(k)
            got, mag = x @ u, np.abs(x) @ np.abs(u)
        assert np.all(np.abs(got - b) <= 4 * k * EPS[dtype] * (mag + np.abs(b)))


@pytest.mark.parametrize("form", ["syrk", "nt", "nn"])
@pytest.mark.parametrize("m,n,k", [(512, 192, 16), (129, 800, 65), (641, 640, 200), (130, 2000, 17)])
@pytest.mark.parametrize("kind", ["random", "graded", "sparse", "special"])
def test_fp64_products_keep_the_componentwise_bound(gpu, form, m, n, k, kind):
    rng = np.random.default_rng(m + n + k)
    n = max(m, 500) if form == "syrk" else n
    m = n if form == "syrk" else m
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((n, k)), rng.standard_normal((m, n))
    if kind == "graded":  # large elements of A meet small ones of B
        s = np.power(10.0, np.linspace(-7, 7, k))
        a, b = a * s, b / s
    elif kind == "sparse":
        a[rng.uniform(size=a.shape) < 0.97] = 0
        b[::3] = 0
    elif kind == "special":
        a[3, 1], a[7, 0], b[5, 2 % k], a[11] = np.nan, np.inf, -np.inf, 1e-310
    if form == "syrk":
        b = a
    da, dc = up(a), up(c)
    db = up(b.T if form == "nn" else b)
    if form == "syrk":
        check(gpu.starpu_gb300_dsyrk_ln_tile(None, n, k, -1.0, da.ptr, n, 1.0, dc.ptr, n))
    elif form == "nt":
        check(gpu.starpu_gb300_dgemm_nt_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
    else:
        check(gpu.starpu_gb300_dgemm_nn_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, k, 1.0, dc.ptr, m))
    out = dc.download((m, n), np.float64)
    with np.errstate(all="ignore"):
        ref = c - a @ b.T
        bound = (k + 2) * EPS[np.float64] * (np.abs(c) + np.abs(a) @ np.abs(b).T)
    keep = np.tril(np.ones((m, n), bool)) if form == "syrk" else np.ones((m, n), bool)
    assert np.array_equal(out[~keep], c[~keep])
    fine = np.isfinite(ref) & keep
    assert np.all(np.abs(out - ref)[fine] <= bound[fine])
    assert np.array_equal(np.isfinite(out)[keep], np.isfinite(ref)[keep])


@pytest.mark.parametrize("n,nrhs", [(3000, 40), (1900, 64)])
def test_potrs_many_columns_graded(gpu, n, nrhs):
    d = np.power(10.0, np.random.default_rng(n).uniform(-5, 5, n))
    l = np.linalg.cholesky(spd(n, n, d))
    b = np.random.default_rng(nrhs).uniform(-1, 1, (n, nrhs))
    dl, db = up(l), up(b)
    check(gpu.starpu_gb300_dpotrs(None, n, nrhs, dl.ptr, n, db.ptr, n))
    x = db.download((n, nrhs), np.float64)
    y = np.abs(l.T) @ np.abs(x)
    assert np.all(np.abs(l @ (l.T @ x) - b) <= 8 * n * EPS[np.float64] * (np.abs(l) @ y + np.abs(b)))


@pytest.mark.parametrize("n,nrhs,extreme", [(1, 1, None), (33, 3, None), (1023, 2, None), (1025, 5, None),
                                            (1500, 2, np.nan), (1500, 2, np.inf)])
def test_backward_error_column_maxima(gpu, n, nrhs, extreme):
    rng = np.random.default_rng(n)
    a = rng.uniform(-1, 1, (n, n))
    a = np.tril(a) + np.tril(a, -1).T
    x, b = rng.uniform(-1, 1, (n, nrhs)), rng.uniform(-3, 3, (n, nrhs))
    x[n - 1, 0], b[n // 2, nrhs - 1] = -5.0, 9.0  # maxima in the last row and in the middle
    if extreme is not None:
        b[7, 1] = extreme
    with np.errstate(invalid="ignore"):
        r = np.abs(b - a @ x)
    anorm = np.abs(a).sum(1).max()
    ref = np.nanmax(r, 0) / (anorm * np.abs(x).max(0) + np.nanmax(np.abs(b), 0))  # NaN entries do not count
    da, dx, db = up(a), up(x), up(b)
    gpu.starpu_gb300_backward_error_workspace.restype = ctypes.c_size_t
    lwork = gpu.starpu_gb300_backward_error_workspace(n, nrhs)
    work, got = DeviceBuffer(lwork), (ctypes.c_double * nrhs)()
    vp = ctypes.c_void_p
    check(gpu.starpu_gb300_backward_error(vp(), n, nrhs, vp(da.ptr), n, vp(dx.ptr), n, vp(db.ptr), n, vp(work.ptr),
                                          ctypes.c_size_t(lwork), got))
    got = np.array(got)
    finite = np.isfinite(ref)
    # both residuals are within (n + 2) u of (|A| |x| + |b|), the denominator's bound
    assert np.all(np.abs(got - ref)[finite] <= 4 * (n + 2) * EPS[np.float64])
    assert np.all(np.isnan(got[~finite]))  # inf / inf


@pytest.mark.parametrize("n", [1, 31, 33, 64])
def test_dpotrf_leaf_diagonal_is_the_square_root(gpu, n):
    d = np.random.default_rng(n).uniform(1e-3, 1e3, n)
    d[0] = 5e-320  # below the normal range: the plain functions
    da, info = up(np.diag(d)), up(np.zeros(1, np.int32))
    check(gpu.starpu_gb300_dpotrf_tile(None, n, da.ptr, n, info.ptr))
    assert info.download((1,), np.int32)[0] == 0
    got, ref = np.diag(da.download((n, n), np.float64)), np.sqrt(d)
    # half an ulp, and the residual's and the step's rounding (2^-53 of the ulp-sized step)
    assert np.all(np.abs(got - ref) <= np.spacing(ref))


# an element of the result is Inf, NaN or finite as the FMA sum makes it: one and
# two infinities in a row, zeros against them, short and ragged last chunks
@pytest.mark.parametrize("form", ["syrk", "nt", "nn"])
@pytest.mark.parametrize("k", [16, 17, 32, 64, 80, 129])
def test_fp64_products_of_infinities(gpu, form, k):
    m, n = 512, 512 if form == "syrk" else 400
    rng = np.random.default_rng(k)
    a, b, c = rng.standard_normal((m, k)), rng.standard_normal((n, k)), rng.standard_normal((m, n))
    a[3, 1], a[200, k - 1], a[7, 0], a[7, 5] = np.inf, -np.inf, np.inf, -np.inf
    a[9, 2] = np.nan
    b[5, 1], b[6, 1], b[300, 3] = 0.0, -0.0, -np.inf
    c[3, 20], c[100, 40] = np.inf, -np.inf
    if form == "syrk":
        b = a
    with np.errstate(invalid="ignore"):
        ref = c.copy()
        for p in range(k):  # (a BLAS may treat infinities in blocks)
            ref -= a[:, p, None] * b[None, :, p]
    da, dc = up(a), up(c)
    db = up(b.T if form == "nn" else b)
    if form == "syrk":
        check(gpu.starpu_gb300_dsyrk_ln_tile(None, n, k, -1.0, da.ptr, n, 1.0, dc.ptr, n))
    elif form == "nt":
        check(gpu.starpu_gb300_dgemm_nt_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
    else:
        check(gpu.starpu_gb300_dgemm_nn_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, k, 1.0, dc.ptr, m))
    out = dc.download((m, n), np.float64)
    keep = np.tril(np.ones((m, n), bool)) if form == "syrk" else np.ones((m, n), bool)
    for f in (np.isnan, np.isposinf, np.isneginf):
        assert np.array_equal(f(out)[keep], f(ref)[keep])


def test_fp64_trailing_update_of_an_infinity(gpu):
    # the panel's row i is infinite: C_ij -= inf l_j, so -inf or +inf by the sign of l_j
    n, i = 400, 250
    a = spd(n, n)
    a[i, 10] = a[10, i] = np.inf
    da, info = up(a), up(np.zeros(1, np.int32))
    check(gpu.starpu_gb300_dpotrf(None, n, da.ptr, n, 64, info.ptr))
    assert info.download((1,), np.int32)[0] == i + 1
    out = da.download((n, n), np.float64)
    ref = np.linalg.cholesky(spd(n, n)[:i, :i])
    assert np.allclose(np.tril(out[:i, :i]), ref, rtol=0, atol=1e-13)
    assert np.isposinf(out[i, 10])


# rows in or near the subnormal range, elements spread over 52 powers of two, against large ones
@pytest.mark.parametrize("k", [16, 64, 100])
@pytest.mark.parametrize("top", [-1074, -1060, -1022, -1000, -970, -960])
def test_fp64_products_of_subnormal_rows(gpu, k, top):
    m, n = 512, 400
    rng = np.random.default_rng(k - top)
    a = np.ldexp(rng.uniform(0.5, 1, (m, k)), rng.integers(top - 50, top + 2, (m, k)))  # some round to subnormals or 0
    b = np.ldexp(rng.uniform(0.5, 1, (n, k)), 900)
    c = np.zeros((m, n))
    da, db, dc = up(a), up(b), up(c)
    check(gpu.starpu_gb300_dgemm_nt_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
    out = dc.download((m, n), np.float64)
    # scaled into the normal range (exact: powers of two), summed there
    ref, mag = -(np.ldexp(a, 600) @ np.ldexp(b, -900).T), np.abs(np.ldexp(a, 600)) @ np.abs(np.ldexp(b, -900)).T
    assert np.all(np.abs(np.ldexp(out, -300) - ref) <= 2 * (k + 2) * EPS[np.float64] * mag)


# single products in the last binade and beyond it, and around half the smallest number
@pytest.mark.parametrize("k", [16, 64])
@pytest.mark.parametrize("top", [True, False])
def test_fp64_products_at_the_ends_of_the_range(gpu, k, top):
    m, n = 512, 400
    rng = np.random.default_rng(k)
    a, b, c = np.zeros((m, k)), np.zeros((n, k)), np.zeros((m, n))
    a[:, 3] = np.ldexp(rng.uniform(1, 2, m), (511 + np.arange(m) % 3) if top else (-540 - np.arange(m) % 4))
    b[:, 3] = np.ldexp(rng.uniform(1, 2, n), 511 if top else -535)
    with np.errstate(over="ignore", under="ignore"):
        ref = -(a[:, 3, None] * b[None, :, 3])  # one rounding
    da, db, dc = up(a), up(b), up(c)
    check(gpu.starpu_gb300_dgemm_nt_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
    out = dc.download((m, n), np.float64)
    fine = np.isfinite(ref)
    assert np.array_equal(np.isneginf(out), ~fine) and fine.any() and (not top or not fine.all())
    assert np.all(np.abs(out - ref)[fine] <= np.spacing(np.abs(ref))[fine])


# one pair of larger elements, from a hundredth of the rows' maxima up to both, among elements whose digits
# below the first are all -128, so that the digit products left out add up; some of the elements zero
@pytest.mark.parametrize("k", [16, 17, 32, 64, 100])
@pytest.mark.parametrize("zeros", [0.0, 0.8])
def test_fp64_products_keep_the_bound_at_the_worst_digits(gpu, k, zeros):
    m, n = 512, 400
    rng = np.random.default_rng(k)
    low = sum(2.0 ** (8 * (7 - t)) for t in range(2, 8))
    cut = lambda first: np.ldexp(first * 2.0**48 - 128.0 * low, -55)  # first digit, then -128s: exact in FP64
    a, b = np.full((m, k), cut(1.0)), np.full((n, k), cut(1.0))
    a[:, 2:][rng.uniform(size=(m, k - 2)) < zeros] = 0
    b[:, 2:][rng.uniform(size=(n, k - 2)) < zeros] = 0
    a[:, 0], b[:, 0] = cut(128.0), 0.0  # the rows' maxima, against nothing
    a[:, 1], b[:, 1] = cut(1.0 + np.arange(m) % 128), cut(1.0 + np.arange(n) % 128)
    b[:, 0] = np.where(np.arange(n) % 2, 0.0, -cut(1.0))
    c = np.zeros((m, n))
    da, db, dc = up(a), up(b), up(c)
    check(gpu.starpu_gb300_dgemm_nt_tile(None, m, n, k, -1.0, da.ptr, m, db.ptr, n, 1.0, dc.ptr, m))
    out = dc.download((m, n), np.float64)
    ref, mag = np.zeros((m, n), np.longdouble), np.zeros((m, n))
    for p in range(k):
        ref -= a[:, p, None].astype(np.longdouble) * b[None, :, p]
        mag += np.abs(a[:, p, None] * b[None, :, p])
    assert np.all(np.abs((out - ref).astype(np.float64)) <= (k + 2) * EPS[np.float64] * mag)


# the leaf, one cooperative launch of several blocks, and panels
@pytest.mark.parametrize("n", [1, 31, 64, 65, 200, 4200])
def test_spotrf_diagonal_is_the_square_root(gpu, n):
    d = np.random.default_rng(n).uniform(1e-3, 1e3, n).astype(np.float32)
    d[0] = 1e-41  # below the normal range
    da, info = up(np.diag(d)), up(np.zeros(1, np.int32))
    check(gpu.starpu_gb300_spotrf(None, n, da.ptr, n, 512, info.ptr))
    assert info.download((1,), np.int32)[0] == 0
    assert np.array_equal(np.diag(da.download((n, n), np.float32)), np.sqrt(d))


# L of [[d, t], [t, 2.5 t^2 / d]] has t / sqrt(d) below the diagonal (t a power of two): 32 such blocks a
# matrix, d over the normal range and its powers of two, and beyond it
@BOTH
def test_leaf_reciprocal_root(gpu, dtype):
    lo, hi, t = (-126, 128, 2.0**-20) if dtype == np.float32 else (-1022, 1024, 2.0**-60)
    rng = np.random.default_rng(11)
    edges = np.concatenate([[1.0, 1.5, np.nextafter(dtype(2), dtype(0)), 2.0, 3.0, np.nextafter(dtype(4), dtype(0))]] * 8)
    e = rng.integers(lo, hi, 32 * 400)
    d = np.ldexp(rng.uniform(1, 2, e.size).astype(dtype), np.minimum(e, hi - 1))
    d[: edges.size] = np.ldexp(edges.astype(dtype), rng.integers(lo + 2, hi - 4, edges.size))
    d[-64:] = np.ldexp(dtype(1), np.linspace(lo - 10, lo, 64).astype(int)).astype(dtype)  # some subnormal
    d = d[np.isfinite(d)][: e.size // 32 * 32]
    info = up(np.zeros(1, np.int32))
    worst = 0.0
    for block in d.reshape(-1, 32):
        a = np.zeros((64, 64), dtype)
        i = 2 * np.arange(32)
        a[i, i], a[i + 1, i] = block, t
        a[i + 1, i + 1] = np.maximum(2.5 * t * (t / block.astype(np.float64)), 1e-30)
        da = up(a)
        check(fn(gpu, dtype, "potrf_tile")(None, 64, da.ptr, 64, info.ptr))
        r = da.download((64, 64), dtype)[i + 1, i].astype(np.longdouble) / t
        exact = 1 / np.sqrt(block.astype(np.longdouble))
        normal = block >= np.finfo(dtype).tiny
        err = np.abs(r / exact - 1).astype(np.float64) / EPS[dtype]
        # 1.5 u; outside the normal range 1 / sqrt(d) of two rounded operations, 2 u
        assert np.all(err <= np.where(normal, 1.5, 2.0) * (1 + 2.0**-9)), (block[np.argmax(err)], err.max())
        worst = max(worst, err.max())
    assert worst > 0.5


def test_dpotrf_leaf_sums_products_apart(gpu):
    """48 products of 2^-54 count 3 2^-50 together and nothing one by one beside 1:
    rounded into their element at every column they would be lost."""
    l = np.eye(64)
    l[48:, :48] = 2.0**-27
    a = l @ l.T  # exact
    da = up(a)
    check(gpu.starpu_gb300_dpotrf(None, 64, da.ptr, 64, 64, None))
    out = np.tril(da.download((64, 64), np.float64))
    assert np.all(np.diag(out) == 1.0)
    assert np.all(np.abs(out - l) <= 2.0**-52 * l)


@pytest.mark.parametrize("m", [1, 33, 800, 2100])
def test_dtrsm_slab_sums_products_apart(gpu, m):
    """The panel solve's counterpart of the leaf's: X = 1 in the last group of 16
    columns once the 48 products before it are summed apart."""
    l = np.eye(64)
    l[48:, :48] = 2.0**-27
    x = np.ones((m, 64))
    x[:, :48] = 2.0**-27
    b = x.copy()
    b[:, 48:] += 3 * 2.0**-50
    dl, db = up(l), up(b)
    check(gpu.starpu_gb300_dtrsm_rltn_tile(None, m, 64, 1.0, dl.ptr, 64, db.ptr, m))
    np.testing.assert_array_equal(db.download((m, 64), np.float64), x)


def test_dpotrs_sums_products_apart(gpu):
    """The same in the solve's blocks of 32 rows, whose groups are of eight: forward
    the last group has 24 products of 2^-54 before it, backward the others eight."""
    l = np.eye(32)
    l[24:, :24] = 2.0**-27
    b = np.full((32, 1), 2.0**-27)
    b[24:] = 1 + 3 * 2.0**-51
    x = np.full((32, 1), -7 * 2.0**-27)
    x[24:] = 1.0
    dl, db = up(l), up(b)
    check(gpu.starpu_gb300_dpotrs(None, 32, 1, dl.ptr, 32, db.ptr, 32))
    np.testing.assert_array_equal(db.download((32, 1), np.float64), x)

    sign = np.where(np.arange(24) % 2 == 0, 1.0, -1.0)  # so that forward every sum is exact
    l[24:, :24] = 2.0**-27 * sign
    b = np.full((32, 1), 2.0**-27 + 3 * 2.0**-75)
    b[:24, 0] = 1 + sign * 2.0**-51
    x = np.full((32, 1), 2.0**-27)
    x[:24] = 1.0
    dl, db = up(l), up(b)
    check(gpu.starpu_gb300_dpotrs(None, 32, 1, dl.ptr, 32, db.ptr, 32))
    np.testing.assert_array_equal(db.download((32, 1), np.float64), x)
