"""Performance cases of the GB300 Cholesky framework: the work its users have it do, through the public C ABI.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (matrices, right-hand sides, workspaces), `run` makes one pass, `work`
states the bytes and operations one pass cannot do without and `exact` gives
the same results from 64-bit torch arithmetic.

Matrices are column-major with the lower triangle significant.  The torch
tensors below hold them row-major, so a matrix in the library's layout is the
tensor's transpose: its lower triangle is the tensor's upper one.
"""
import ctypes as C
import math

import numpy as np
import torch

from starpu_gb300.native import IrInfo, check, load

REAL = {"f32": torch.float32, "f64": torch.float64}
LETTER = {"f32": "s", "f64": "d"}


def listed():
    return [
        # One step of the tiled Cholesky DAG on a 3 x 3 tile matrix, codelet by
        # codelet (POTRF, 2 TRSM, 2 SYRK, GEMM): what a StarPU program's tasks
        # run.  256 is the tile of the reference driver's default problem.
        {"name": "chol_step_f32_256", "op": "chol_step", "dtype": "f32", "nb": 256},
        # the same step in FP64 at the FP64 configuration's tile
        {"name": "chol_step_f64_512", "op": "chol_step", "dtype": "f64", "nb": 512},
        # the SYRK and GEMM codelets of large FP32 tiles, which run on the tensor cores
        {"name": "tile_tc_1024", "op": "tile_tc", "nb": 1024},
        # one step of the tiled LU DAG (GETRF, TRSM_LL, TRSM_RU, GEMM), a tile that is no power of two
        {"name": "lu_step_f32_480", "op": "lu_step", "dtype": "f32", "nb": 480},
        # plain FP32 factorisation and solve: the default problem of the reference driver ...
        {"name": "sposv_2048", "op": "posv", "dtype": "f32", "n": 2048, "nb": 256, "nrhs": 4},
        # ... and a large one of ragged order
        {"name": "sposv_10000", "op": "posv", "dtype": "f32", "n": 10000, "nb": 512, "nrhs": 16},
        # plain FP64 factorisation and solve: one small system, one right-hand side ...
        {"name": "dposv_1000", "op": "posv", "dtype": "f64", "n": 1000, "nb": 512, "nrhs": 1},
        # ... and a large one with the FP64 configuration's tile and 64 right-hand sides
        {"name": "dposv_8192", "op": "posv", "dtype": "f64", "n": 8192, "nb": 512, "nrhs": 64},
        # mixed-precision solve, as the serving loop's executors call it: a small
        # odd order, a middle one, and the headline configuration's size
        {"name": "dsposv_777", "op": "dsposv", "n": 777, "nb": 1024, "nrhs": 3, "kappa": 1000.0},
        {"name": "dsposv_4096", "op": "dsposv", "n": 4096, "nb": 1024, "nrhs": 16, "kappa": 1000.0},
        {"name": "dsposv_32768", "op": "dsposv", "n": 32768, "nb": 1024, "nrhs": 16, "kappa": 100.0},
        # many small systems of uneven orders in one launch
        {"name": "batched_1024", "op": "batched", "nsys": 1024, "nmin": 32, "nmax": 1024, "nrhs": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["chol_step", "tile_tc", "lu_step", "posv", "posv", "dsposv", "dsposv", "batched"])
    if op in ("chol_step", "lu_step"):
        return {"op": op, "dtype": rng.choice(["f32", "f64"]), "nb": _log(rng, 64, 1024)}
    if op == "tile_tc":
        return {"op": op, "nb": _log(rng, 512, 1536)}
    if op == "posv":
        dtype = rng.choice(["f32", "f64"])
        return {"op": op, "dtype": dtype, "n": _log(rng, 256, 12000 if dtype == "f32" else 8192),
                "nb": rng.choice([256, 512, 1024]), "nrhs": _log(rng, 1, 64)}
    if op == "dsposv":
        return {"op": op, "n": _log(rng, 64, 16384), "nb": rng.choice([512, 1024, 1024]), "nrhs": _log(rng, 1, 16),
                "kappa": 10.0 ** rng.uniform(1.0, 3.0)}
    nmax = _log(rng, 64, 1024)
    return {"op": op, "nsys": _log(rng, 64, 1024), "nmin": max(1, nmax // 32), "nmax": nmax, "nrhs": _log(rng, 1, 8)}


# ---------------------------------------------------------------- inputs

def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _spd(n, g, alpha):
    """G G^T / n + v v^T + alpha I in FP64 with G iid N(0, 1): spectrum about
    [alpha, 4 + alpha], every mantissa bit in use."""
    b = torch.randn(n, n, device="cuda", generator=g)
    if n > 4096:  # G to 11 bits, so that its product may run in TF32
        b = b.to(torch.float16).float()
    tf32 = torch.backends.cuda.matmul.allow_tf32
    torch.backends.cuda.matmul.allow_tf32 = n > 4096
    p = b @ b.T
    torch.backends.cuda.matmul.allow_tf32 = tf32
    del b
    a = p.double()
    del p
    a /= n
    v = (0.5 + 0.5 * torch.rand(n, device="cuda", generator=g, dtype=torch.float64)) / math.sqrt(n)
    a.addr_(v, v)
    a.diagonal().add_(alpha)
    return a


def _rhs(n, nrhs, g, dtype):
    return 2.0 * torch.rand(nrhs, n, device="cuda", generator=g, dtype=dtype) - 1.0


def _alpha(kappa):
    return 4.0 / (kappa - 1.0)


def _inputs(case, seed):
    g = _generator(seed)
    op = case["op"]
    if op == "chol_step":
        return {"a": _spd(3 * case["nb"], g, 1.0).to(REAL[case["dtype"]])}
    if op == "tile_tc":
        nb = case["nb"]
        l = torch.randn(2 * nb, nb, device="cuda", generator=g) / math.sqrt(nb)
        # two solved panel tiles and the two tiles they update, each column-major
        return {"l1": l[:nb].contiguous(), "l2": l[nb:2 * nb].contiguous(),
                "c1": torch.randn(nb, nb, device="cuda", generator=g),
                "c2": torch.randn(nb, nb, device="cuda", generator=g)}
    if op == "lu_step":
        n = 2 * case["nb"]
        a = torch.rand(n, n, device="cuda", generator=g, dtype=torch.float64)
        a.diagonal().add_(float(n))
        return {"a": a.to(REAL[case["dtype"]])}
    if op == "posv":
        d = REAL[case["dtype"]]
        return {"a": _spd(case["n"], g, 1.0).to(d), "b": _rhs(case["n"], case["nrhs"], g, d)}
    if op == "dsposv":
        return {"a": _spd(case["n"], g, _alpha(case["kappa"])), "b": _rhs(case["n"], case["nrhs"], g, torch.float64)}
    sizes = _batch_sizes(case, seed)
    total = int(sum(n * n for n in sizes))
    a = torch.empty(total, device="cuda", dtype=torch.float64)
    off = np.zeros(len(sizes), dtype=np.int64)
    o = 0
    for i, n in enumerate(sizes):
        off[i] = o
        r = torch.randn(n, n, device="cuda", generator=g)
        m = (r @ r.T).double() / n
        m = torch.triu(m) + torch.triu(m, 1).T
        m.diagonal().add_(1.0)
        a[o:o + n * n] = m.reshape(-1)
        o += n * n
    boff = np.concatenate([[0], np.cumsum([n * case["nrhs"] for n in sizes])]).astype(np.int64)
    b = 2.0 * torch.rand(int(boff[-1]), device="cuda", generator=g, dtype=torch.float64) - 1.0
    return {"a": a, "b": b, "sizes": np.asarray(sizes, dtype=np.int32), "a_off": off, "b_off": boff[:-1].copy()}


def _batch_sizes(case, seed):
    """Log-uniform orders in a random order; the middle of each of nsys equal
    parts of the range, so that the work hardly depends on the seed."""
    lo, hi, k = math.log(case["nmin"]), math.log(case["nmax"]), case["nsys"]
    s = np.exp(lo + (hi - lo) * (np.arange(k) + 0.5) / k).round().astype(np.int64)
    np.random.RandomState(int(seed) & 0x7FFFFFFF).shuffle(s)
    return [int(x) for x in s]


def _tol(n):
    """LAPACK dsposv's stopping rule for the backward error: sqrt(n) eps."""
    return math.sqrt(n) * np.finfo(np.float64).eps


def prepare(case, seed):
    lib = load()
    s = {"case": dict(case), "lib": lib, "in": _inputs(case, seed)}
    op = case["op"]
    info = torch.zeros(1, dtype=torch.int32, device="cuda")
    err = torch.zeros(1, dtype=torch.int32, device="cuda")
    s["info"], s["err"] = info, err
    if op in ("chol_step", "lu_step"):
        s["w"] = torch.empty_like(s["in"]["a"])
    elif op == "tile_tc":
        s["c1"], s["c2"] = torch.empty_like(s["in"]["c1"]), torch.empty_like(s["in"]["c2"])
        s["lwork"] = lib.starpu_gb300_tile_tc_workspace(case["nb"])
        s["work"] = torch.empty(s["lwork"], dtype=torch.uint8, device="cuda")
        check(lib.starpu_gb300_tile_tc_prepare(), "tile_tc_prepare")
    elif op == "posv":
        s["w"], s["x"] = torch.empty_like(s["in"]["a"]), torch.empty_like(s["in"]["b"])
    elif op == "dsposv":
        s["x"] = torch.empty_like(s["in"]["b"])
        s["lwork"] = lib.starpu_gb300_dsposv_workspace(case["n"], case["nrhs"], case["nb"])
        s["work"] = torch.empty(s["lwork"], dtype=torch.uint8, device="cuda")
    else:
        n = s["in"]["sizes"]
        s["x"] = torch.empty_like(s["in"]["b"])
        s["lwork"] = lib.starpu_gb300_dposv_batched_workspace(len(n), n.ctypes.data, case["nrhs"])
        s["work"] = torch.empty(s["lwork"], dtype=torch.uint8, device="cuda")
        s["status"] = np.zeros(len(n), dtype=np.int32)
        s["berr"] = np.zeros(len(n), dtype=np.float64)
    return s


# ---------------------------------------------------------------- one pass

def run(s):
    case, lib, inp = s["case"], s["lib"], s["in"]
    st = torch.cuda.current_stream().cuda_stream
    op = case["op"]
    if op == "chol_step":
        return _run_chol_step(s, case, lib, inp, st)
    if op == "tile_tc":
        nb = case["nb"]
        s["c1"].copy_(inp["c1"])
        s["c2"].copy_(inp["c2"])
        l1, l2, err = inp["l1"].data_ptr(), inp["l2"].data_ptr(), s["err"].data_ptr()
        work, lwork = s["work"].data_ptr(), s["lwork"]
        check(lib.starpu_gb300_sgemm_nt_tile_tc(st, nb, nb, nb, l1, nb, l1, nb, s["c1"].data_ptr(), nb, 1, work, lwork,
                                                err), "syrk")
        check(lib.starpu_gb300_sgemm_nt_tile_tc(st, nb, nb, nb, l2, nb, l1, nb, s["c2"].data_ptr(), nb, 0, work, lwork,
                                                err), "gemm")
        return {"syrk": s["c1"], "gemm": s["c2"], "err": s["err"]}
    if op == "lu_step":
        return _run_lu_step(s, case, lib, inp, st)
    if op == "posv":
        p, n, nrhs = LETTER[case["dtype"]], case["n"], case["nrhs"]
        s["w"].copy_(inp["a"])
        s["x"].copy_(inp["b"])
        check(getattr(lib, "starpu_gb300_%spotrf" % p)(st, n, s["w"].data_ptr(), n, case["nb"], s["info"].data_ptr()),
              "potrf")
        check(getattr(lib, "starpu_gb300_%spotrs" % p)(st, n, nrhs, s["w"].data_ptr(), n, s["x"].data_ptr(), n), "potrs")
        return {"l": s["w"], "x": s["x"], "info": s["info"]}
    if op == "dsposv":
        n, info = case["n"], IrInfo()
        check(lib.starpu_gb300_dsposv(st, n, case["nrhs"], inp["a"].data_ptr(), n, inp["b"].data_ptr(), n,
                                      s["x"].data_ptr(), n, case["nb"], 3, _tol(n), 30, s["work"].data_ptr(),
                                      s["lwork"], C.byref(info)), "dsposv")
        return {"x": s["x"], "status": info.status}
    n = inp["sizes"]
    check(lib.starpu_gb300_dposv_batched(st, len(n), n.ctypes.data, inp["a"].data_ptr(), inp["a_off"].ctypes.data,
                                         inp["b"].data_ptr(), inp["b_off"].ctypes.data, s["x"].data_ptr(), case["nrhs"],
                                         1e-13, 20, s["work"].data_ptr(), s["lwork"], s["status"].ctypes.data,
                                         s["berr"].ctypes.data), "dposv_batched")
    return {"x": s["x"], "converged": s["status"] >= 0}


def _run_chol_step(s, case, lib, inp, st):
    p, nb = LETTER[case["dtype"]], case["nb"]
    w = s["w"]
    w.copy_(inp["a"])
    ld, size, base = 3 * nb, w.element_size(), w.data_ptr()

    def tile(i, j):
        return base + (i * nb + j * nb * ld) * size

    f = {k: getattr(lib, "starpu_gb300_%s%s_tile" % (p, k)) for k in ("potrf", "trsm_rltn", "syrk_ln", "gemm_nt")}
    check(f["potrf"](st, nb, tile(0, 0), ld, s["info"].data_ptr()), "potrf")
    for i in (1, 2):
        check(f["trsm_rltn"](st, nb, nb, 1.0, tile(0, 0), ld, tile(i, 0), ld), "trsm")
    for i in (1, 2):
        check(f["syrk_ln"](st, nb, nb, -1.0, tile(i, 0), ld, 1.0, tile(i, i), ld), "syrk")
    check(f["gemm_nt"](st, nb, nb, nb, -1.0, tile(2, 0), ld, tile(1, 0), ld, 1.0, tile(2, 1), ld), "gemm")
    return {"a": w, "info": s["info"]}


def _run_lu_step(s, case, lib, inp, st):
    p, nb = LETTER[case["dtype"]], case["nb"]
    w = s["w"]
    w.copy_(inp["a"])
    ld, size, base = 2 * nb, w.element_size(), w.data_ptr()

    def tile(i, j):
        return base + (i * nb + j * nb * ld) * size

    f = {k: getattr(lib, "starpu_gb300_%s%s_tile" % (p, k)) for k in ("getrf", "trsm_llnn", "trsm_runu", "gemm_nn")}
    check(f["getrf"](st, nb, tile(0, 0), ld, s["info"].data_ptr()), "getrf")
    check(f["trsm_llnn"](st, nb, nb, tile(0, 0), ld, tile(0, 1), ld), "trsm_ll")
    check(f["trsm_runu"](st, nb, nb, tile(0, 0), ld, tile(1, 0), ld), "trsm_ru")
    check(f["gemm_nn"](st, nb, nb, nb, -1.0, tile(1, 0), ld, tile(0, 1), ld, 1.0, tile(1, 1), ld), "gemm")
    return {"a": w, "info": s["info"]}


# ---------------------------------------------------------------- the work of one pass

def work(case):
    op = case["op"]
    if op == "chol_step":
        nb, e = case["nb"], 4 if case["dtype"] == "f32" else 8
        # lower triangles of three diagonal tiles, three full tiles: read and written
        return {"bytes": 2.0 * e * (3 * nb * (nb + 1) / 2 + 3 * nb * nb),
                "flops": nb**3 / 3.0 + 2.0 * nb**3 + 2.0 * nb * nb * (nb + 1) + 2.0 * nb**3}
    if op == "tile_tc":
        nb = case["nb"]
        return {"bytes": 4.0 * (2 * nb * nb + nb * (nb + 1) + 2 * nb * nb), "flops": nb * nb * (nb + 1.0) + 2.0 * nb**3}
    if op == "lu_step":
        nb, e = case["nb"], 4 if case["dtype"] == "f32" else 8
        return {"bytes": 2.0 * e * 4 * nb * nb, "flops": 2.0 * nb**3 / 3.0 + 2.0 * nb**3 + 2.0 * nb**3}
    if op == "posv":
        n, k, e = case["n"], case["nrhs"], 4 if case["dtype"] == "f32" else 8
        return {"bytes": e * (n * (n + 1.0) + 2.0 * n * k), "flops": n**3 / 3.0 + 2.0 * n * n * k}
    if op == "dsposv":
        n, k = case["n"], case["nrhs"]
        return {"bytes": 8.0 * (n * (n + 1.0) / 2 + 2.0 * n * k), "flops": n**3 / 3.0 + 2.0 * n * n * k}
    k, sizes = case["nrhs"], _batch_sizes(case, 0)
    return {"bytes": float(sum(8.0 * (n * (n + 1.0) / 2 + 2.0 * n * k) for n in sizes)),
            "flops": float(sum(n**3 / 3.0 + 2.0 * n * n * k for n in sizes))}


# ---------------------------------------------------------------- the same results in 64 bits

def exact(case, seed):
    inp = _inputs(case, seed)
    op = case["op"]
    if op == "chol_step":
        nb = case["nb"]
        m = inp["a"].double().T.contiguous()  # the library's matrix
        t = [slice(i * nb, (i + 1) * nb) for i in range(3)]
        full = torch.tril(m[t[0], t[0]]) + torch.tril(m[t[0], t[0]], -1).T
        l = torch.linalg.cholesky(full)
        m[t[0], t[0]] = torch.tril(l) + torch.triu(m[t[0], t[0]], 1)
        for i in (1, 2):
            m[t[i], t[0]] = torch.linalg.solve_triangular(l, m[t[i], t[0]].T, upper=False).T
        for i in (1, 2):
            p = m[t[i], t[0]]
            m[t[i], t[i]] -= torch.tril(p @ p.T)
        m[t[2], t[1]] -= m[t[2], t[0]] @ m[t[1], t[0]].T
        return {"a": m.T.contiguous(), "info": None}
    if op == "tile_tc":
        l1, l2 = inp["l1"].double(), inp["l2"].double()
        # column-major operands: the library's A is l.T, so A B^T is l2.T @ l1, whose transpose is l1.T @ l2
        return {"syrk": inp["c1"].double() - torch.triu(l1.T @ l1), "gemm": inp["c2"].double() - l1.T @ l2, "err": None}
    if op == "lu_step":
        nb = case["nb"]
        m = inp["a"].double().T.contiguous()
        d = m[:nb, :nb].clone()
        for k in range(nb):  # no pivoting, the pivot in L
            d[k, k + 1:] /= d[k, k]
            d[k + 1:, k + 1:].addr_(d[k + 1:, k], d[k, k + 1:], alpha=-1.0)
        m[:nb, :nb] = d
        m[:nb, nb:] = torch.linalg.solve_triangular(torch.tril(d), m[:nb, nb:], upper=False)
        u = torch.triu(d, 1) + torch.eye(nb, device="cuda", dtype=torch.float64)
        m[nb:, :nb] = torch.linalg.solve_triangular(u, m[nb:, :nb], upper=True, left=False, unitriangular=True)
        m[nb:, nb:] -= m[nb:, :nb] @ m[:nb, nb:]
        return {"a": m.T.contiguous(), "info": None}
    if op == "posv":
        a, b = inp["a"].double(), inp["b"].double()
        u = torch.linalg.cholesky(torch.triu(a) + torch.triu(a, 1).T, upper=True)
        x = torch.cholesky_solve(b.T.contiguous(), u, upper=True)
        return {"l": u + torch.tril(a, -1), "x": x.T.contiguous(), "info": None}
    if op == "dsposv":
        a = torch.triu(inp["a"]) + torch.triu(inp["a"], 1).T
        b = inp["b"].T.contiguous()
        del inp
        if case["n"] <= 8192:
            l = torch.linalg.cholesky(a)
            x = torch.cholesky_solve(b, l)
            x += torch.cholesky_solve(b - a @ x, l)
        else:
            x = _cg(a, b, case["kappa"])
        return {"x": x.T.contiguous(), "status": None}
    k, x = case["nrhs"], torch.empty_like(inp["b"])
    for n, ao, bo in zip(inp["sizes"].tolist(), inp["a_off"].tolist(), inp["b_off"].tolist()):
        m = inp["a"][ao:ao + n * n].reshape(n, n)
        m = torch.triu(m) + torch.triu(m, 1).T
        b = inp["b"][bo:bo + n * k].reshape(k, n).T
        x[bo:bo + n * k] = torch.cholesky_solve(b, torch.linalg.cholesky(m)).T.reshape(-1)
    return {"x": x, "converged": None}


def _cg(a, b, kappa):
    """Conjugate gradients in FP64, restarted once from the true residual."""
    x = torch.zeros_like(b)
    rho = (math.sqrt(kappa) - 1.0) / (math.sqrt(kappa) + 1.0)
    for digits in (1e-14, 1e-6):
        r = b - a @ x
        p, rr = r.clone(), (r * r).sum(0)
        for _ in range(int(math.log(digits) / math.log(rho)) + 5):
            q = a @ p
            step = torch.where(rr > 0, rr / (p * q).sum(0), torch.zeros_like(rr))
            x += step * p
            r -= step * q
            new = (r * r).sum(0)
            p = r + torch.where(rr > 0, new / rr, torch.zeros_like(rr)) * p
            rr = new
    return x
