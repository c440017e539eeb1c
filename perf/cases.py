"""The workloads this library is measured on: one pass of each is one call of a
public entry point on device arrays, as a caller of NextLA.jl's
``unified_rectrxm!`` makes it (``run`` first restores the right-hand sides,
which every entry point overwrites).

A case names its entry point (``kind``), element type, flags and sizes:

  plain    unified_rectrxm_ in the caller's element type (real or complex);
           ``native`` runs the recursion inside the library, otherwise it is
           driven from the host as the Julia package does;
  mixed    unified_rectrxm_mixed_: Float64 answers from tensor-core updates;
  lu       getrf2_trsm_: the triangular solve inside a recursive LU, on views
           of one array;
  batch    BatchPlan.solve / solve_mixed over many uneven systems, the plan
           kept by the caller.

``pad`` is how far the leading dimensions exceed the row counts (views of
larger arrays).  Inputs have the repository's usual distributions:
off-diagonals N(0,1)/sqrt(n), diagonal 2 + |N(0,1)| (ones for an LU factor),
right-hand sides uniform on [-1, 1].
"""

import importlib.util
import math
import os
import sys

import numpy as np
import torch

_PKG = "nextla_gb300"
_DIR = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "nextla.jl_gb300")


def _package():
    """The package, whose folder name is not a Python identifier."""
    if _PKG not in sys.modules:
        spec = importlib.util.spec_from_file_location(_PKG, os.path.join(_DIR, "__init__.py"),
                                                      submodule_search_locations=[_DIR])
        mod = importlib.util.module_from_spec(spec)
        sys.modules[_PKG] = mod
        spec.loader.exec_module(mod)
    return sys.modules[_PKG]


def _batched():
    _package()
    return importlib.import_module(_PKG + ".batched")


_DTYPES = {"f16": torch.float16, "f32": torch.float32, "f64": torch.float64, "c32": torch.complex64,
           "c64": torch.complex128}


def _plain(name, dtype, func, side, uplo, trans, n, m, alpha=1.0, native=True, pad=0):
    return {"name": name, "kind": "plain", "dtype": dtype, "func": func, "side": side, "uplo": uplo, "trans": trans,
            "n": n, "m": m, "alpha": alpha, "native": native, "pad": pad}


def _mixed(name, func, side, uplo, trans, n, m, terms, sweeps, lowp="bf16", alpha=1.0, pad=0):
    return {"name": name, "kind": "mixed", "func": func, "side": side, "uplo": uplo, "trans": trans, "n": n, "m": m,
            "alpha": alpha, "terms": terms, "sweeps": sweeps, "lowp": lowp, "pad": pad}


def listed():
    return [
        # One small diagonal block, the call a blocked factorisation makes for
        # every panel: a single base case, so launch latency is all of it.
        _plain("f64 solve 96x24", "f64", "S", "L", "L", "N", 96, 24, native=False),
        # The reference tests' and the CPU comparison's problem: Float64,
        # 1024 unknowns, 256 right-hand sides, host-driven recursion.
        _plain("f64 solve 1024x256", "f64", "S", "L", "L", "N", 1024, 256, native=False),
        # A Float32 multiply of ragged size from the right with a transposed
        # upper triangle, through the default entry point.
        _plain("f32 multiply 1500x900", "f32", "M", "R", "U", "T", 1500, 900, alpha=0.5, native=False),
        # The dtype-preserving sweep's Float32 solve.
        _plain("f32 solve 8192x8192", "f32", "S", "L", "L", "N", 8192, 8192, alpha=0.5),
        # Float16 data on the FP16 tensor path.
        _plain("f16 solve 8192x4096", "f16", "S", "L", "L", "N", 8192, 4096),
        # Complex single precision (least squares and eigenvector back
        # substitution on complex data): adjoint triangle from the right.
        _plain("c32 solve 2048x1000", "c32", "S", "R", "U", "C", 2048, 1000),
        # The headline: Float64 answer with exact tensor-core updates.
        _mixed("mixed exact 16384x16384", "S", "L", "L", "N", 16384, 16384, 7, 0),
        # The triangular solve of an LU step of odd size, on views of the
        # array that is being factored.
        {"name": "lu solve 3001", "kind": "lu", "dtype": "f64", "n": 3001, "n1": 1500, "mixed": True},
        # The mixed form with its default options: three BF16 terms and two
        # refinement sweeps.
        _mixed("mixed refined 4096x2048", "S", "L", "U", "N", 4096, 2048, 3, 2),
        # The mixed multiply: three BF16 terms.
        _mixed("mixed multiply 6144x6144", "M", "R", "U", "T", 6144, 6144, 3, 0),
        # Thousands of uneven systems in one launch, in Float32.
        {"name": "batch f32 10000", "kind": "batch", "dtype": "f32", "count": 10000, "sizes": 7, "mixed": False,
         "sweeps": 0},
        # The Float64 batch in its mixed form with two refinement sweeps.
        {"name": "batch mixed 2000", "kind": "batch", "dtype": "f64", "count": 2000, "sizes": 7, "mixed": True,
         "sweeps": 2},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "mixed", "mixed", "lu", "batch"])
    if kind == "lu":
        n = _log_int(rng, 64, 8192)
        mixed = rng.random() < 0.7 or n > 4096
        return {"kind": "lu", "dtype": "f64", "n": n, "n1": max(1, n // 2 - rng.choice([0, 0, 1, n // 8])),
                "mixed": mixed}
    if kind == "batch":
        dtype = rng.choice(["f32", "f32", "f64"])
        mixed = dtype == "f64" and rng.random() < 0.7
        return {"kind": "batch", "dtype": dtype, "count": _log_int(rng, 50, 10000 if dtype == "f32" else 4000),
                "sizes": rng.randrange(1000), "mixed": mixed, "sweeps": rng.choice([1, 2]) if mixed else 0}
    side, uplo = rng.choice("LR"), rng.choice("LU")
    func = rng.choice("SSM")
    alpha, pad = rng.choice([1.0, 0.5, -1.25]), rng.choice([0, 0, 1, 64])
    if kind == "mixed":
        terms = rng.choice([7, 7, 3])
        top = 8192 if terms == 7 else 4096
        n, m = _log_int(rng, 200, top), _log_int(rng, 100, top)
        sweeps = 2 if terms == 3 and func == "S" else 0
        c = _mixed("", func, side, uplo, rng.choice("NT"), n, m, terms, sweeps, rng.choice(["bf16", "bf16", "f16"])
                   if terms == 3 else "bf16", alpha, pad)
    else:
        dtype = rng.choice(["f64", "f32", "f32", "f16", "c32"])
        top = {"f64": 3000, "f32": 8192, "f16": 8192, "c32": 2500}[dtype]
        n, m = _log_int(rng, 24, top), _log_int(rng, 8, top)
        c = _plain("", dtype, func, side, uplo, rng.choice("NTC" if dtype == "c32" else "NT"), n, m, alpha,
                   rng.random() < 0.6, pad)
    del c["name"]
    return c


def _col_major(rows, cols, dtype, pad=0):
    """An uninitialised column-major rows x cols array, a view of one with
    rows + pad rows."""
    return torch.empty((cols, rows + pad), dtype=dtype, device="cuda").T[:rows]


def _triangular(n, uplo, dtype, pad, g):
    work = torch.complex64 if dtype.is_complex else torch.float32 if dtype != torch.float64 else dtype
    A = _col_major(n, n, dtype, pad)
    Z = torch.randn((n, n), generator=g, device="cuda", dtype=work).mul_(1.0 / math.sqrt(n))
    Z.diagonal().copy_(torch.randn(n, generator=g, device="cuda", dtype=torch.float64).abs().add_(2.0))
    A.copy_(Z.tril_() if uplo == "L" else Z.triu_())
    return A


def _rhs(rows, cols, dtype, pad, g):
    work = torch.float64 if dtype == torch.float64 else torch.float32
    B = _col_major(rows, cols, dtype, pad)
    U = torch.rand((rows, cols, 2) if dtype.is_complex else (rows, cols), generator=g, device="cuda", dtype=work)
    U.mul_(2.0).sub_(1.0)
    B.copy_(torch.view_as_complex(U) if dtype.is_complex else U)
    return B


def _sizes(case):
    rng = np.random.default_rng(case["sizes"])
    n = np.rint(np.exp(rng.uniform(np.log(16), np.log(1024), case["count"]))).astype(np.int64).clip(16, 1024)
    return n, rng.integers(1, 129, case["count"])


def _offsets(sizes):
    return np.concatenate([[0], np.cumsum(sizes)[:-1]])


def _batch_inputs(case, g):
    """The pools of a batch and its systems (n, m, a_off, lda, b_off, ldb)."""
    dtype = _DTYPES[case["dtype"]]
    n, m = _sizes(case)
    a_off, b_off = _offsets(n * n), _offsets(n * m)
    nd = torch.from_numpy(n).to("cuda")
    A = torch.randn(int((n * n).sum()), generator=g, device="cuda", dtype=dtype)
    A.mul_(torch.repeat_interleave(nd.to(dtype).rsqrt(), nd * nd))
    first = torch.repeat_interleave(torch.from_numpy(a_off - _offsets(n) * (n + 1)).to("cuda"), nd)
    step = torch.repeat_interleave(nd + 1, nd)
    at = first + torch.arange(int(n.sum()), device="cuda") * step  # a_off + i (n + 1) for each row i of each system
    A[at] = torch.randn(at.numel(), generator=g, device="cuda", dtype=dtype).abs_().add_(2.0)
    B = torch.rand(int((n * m).sum()), generator=g, device="cuda", dtype=dtype).mul_(2.0).sub_(1.0)
    systems = [(int(n[i]), int(m[i]), int(a_off[i]), int(n[i]), int(b_off[i]), int(n[i])) for i in range(len(n))]
    return A, B, systems


def _single_inputs(case, g):
    n, m = case["n"], case["m"]
    dtype = _DTYPES[case.get("dtype", "f64")]
    A = _triangular(n, case["uplo"], dtype, case["pad"], g)
    rows, cols = (n, m) if case["side"] == "L" else (m, n)
    return A, _rhs(rows, cols, dtype, case["pad"], g)


def _lu_input(case, g):
    """An array in the middle of an LU: its first n1 columns are factored
    (unit lower L below the diagonal, U on and above it)."""
    n = case["n"]
    A = _col_major(n, n, torch.float64)
    A.copy_(torch.randn((n, n), generator=g, device="cuda", dtype=torch.float64).mul_(1.0 / math.sqrt(n)))
    return A


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def prepare(case, seed):
    g = _generator(seed)
    if case["kind"] == "batch":
        A, B0, systems = _batch_inputs(case, g)
        plan = _batched().BatchPlan(_DTYPES[case["dtype"]], "L", "N", systems)
        return {"case": case, "A": A, "B0": B0, "B": torch.empty_like(B0), "plan": plan}
    if case["kind"] == "lu":
        A0 = _lu_input(case, g)
        return {"case": case, "B0": A0, "B": torch.empty_strided(A0.shape, A0.stride(), dtype=A0.dtype, device="cuda")}
    A, B0 = _single_inputs(case, g)
    B = _col_major(B0.shape[0], B0.shape[1], B0.dtype, case["pad"])
    return {"case": case, "A": A, "B0": B0, "B": B}


def run(state):
    pkg, c, B = _package(), state["case"], state["B"]
    B.copy_(state["B0"])
    if c["kind"] == "plain":
        pkg.unified_rectrxm_(c["side"], c["uplo"], c["trans"], c["alpha"], c["func"], state["A"], B,
                             native=c["native"])
    elif c["kind"] == "mixed":
        pkg.unified_rectrxm_mixed_(c["side"], c["uplo"], c["trans"], c["alpha"], c["func"], state["A"], B,
                                   lowp=c["lowp"], split_terms=c["terms"], sweeps=c["sweeps"])
    elif c["kind"] == "lu":
        pkg.getrf2_trsm_(B, c["n1"], mixed=c["mixed"])
    elif c["mixed"]:
        state["plan"].solve_mixed(1.0, state["A"], B, sweeps=c["sweeps"])
    else:
        state["plan"].solve(1.0, state["A"], B)
    return B


def work(case):
    """Each referenced triangle and right-hand side read once, each result
    written once; n^2 m operations per solve or multiply (four times that on
    complex data)."""
    if case["kind"] == "batch":
        n, m = (v.astype(np.float64) for v in _sizes(case))
        es = 4 if case["dtype"] == "f32" else 8
        return {"bytes": float(es * (n * (n + 1) / 2 + 2 * n * m).sum()), "flops": float((n * n * m).sum())}
    if case["kind"] == "lu":
        n, m = case["n1"], case["n"] - case["n1"]
        return {"bytes": 8.0 * (n * (n - 1) / 2 + 2 * n * m), "flops": float(n) * n * m}
    n, m = case["n"], case["m"]
    dtype = _DTYPES[case.get("dtype", "f64")]
    return {"bytes": float(dtype.itemsize) * (n * (n + 1) / 2 + 2 * n * m),
            "flops": float(n) * n * m * (4 if dtype.is_complex else 1)}


def exact(case, seed):
    """The same result from torch in 64 bits."""
    g = _generator(seed)
    if case["kind"] == "batch":
        A, B, systems = _batch_inputs(case, g)
        X = torch.empty(B.shape, dtype=torch.float64, device="cuda")
        for n, m, a, _, b, _ in systems:
            T = A[a:a + n * n].view(n, n).T.double()
            R = B[b:b + n * m].view(m, n).T.double()
            X[b:b + n * m].view(m, n).T.copy_(torch.linalg.solve_triangular(T, R, upper=False))
        return X
    if case["kind"] == "lu":
        A, n1 = _lu_input(case, g), case["n1"]
        A[:n1, n1:] = torch.linalg.solve_triangular(A[:n1, :n1], A[:n1, n1:], upper=False, unitriangular=True)
        return A
    A, B = _single_inputs(case, g)
    wide = torch.complex128 if A.is_complex() else torch.float64
    A, B = A.to(wide), B.to(wide).mul_(case["alpha"])
    upper = case["uplo"] == "U"
    if case["trans"] != "N":
        A, upper = (A.T.conj() if case["trans"] == "C" else A.T).contiguous(), not upper
    left = case["side"] == "L"
    if case["func"] == "S":
        return torch.linalg.solve_triangular(A.resolve_conj(), B, upper=upper, left=left)
    return A @ B if left else B @ A
