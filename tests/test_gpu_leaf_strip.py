"""The strip kernel of the diagonal blocks, through the base cases, at the
edges of its panels (16 or 32 rows), its chunks of A (128 columns) and its
strips (2 to 64 right-hand sides), against BLAS in Float64.

Tolerances (relative Frobenius error): Float64 1e-14 and Float32 1e-5 (the
reference's own), Float16 2^-10: inputs exact in Float16, computed in Float32
and rounded once (at most 2^-11 per element)."""

import itertools

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = {np.float64: 1e-14, np.float32: 1e-5, np.float16: 2.0 ** -10}
SHAPES = [(1, 1), (15, 3), (16, 2), (17, 5), (31, 64), (32, 305), (33, 1), (97, 65), (128, 9), (129, 130), (160, 620),
          (257, 1300), (500, 7), (1000, 33), (1024, 2)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.float16])
@pytest.mark.parametrize("func", ["S", "M"])
def test_strip_edges(pkg, oracle, workloads, cuda, dtype, func):
    import torch

    rt = pkg.rectrxm
    for (n, m), (side, uplo, ta) in zip(SHAPES, itertools.cycle(itertools.product("LR", "LU", [False, True]))):
        A, B = workloads.problem(n, m, side, uplo, seed=n + m)
        A, B = A.astype(dtype), B.astype(dtype)
        An = A.copy()
        An[np.triu_indices(n, 1) if uplo == "L" else np.tril_indices(n, -1)] = np.nan  # never used
        stored = An.T if ta else An
        Ad = to_dev(stored, dtype, cuda, ld=n + 3)
        Bd = to_dev(B, dtype, cuda, ld=B.shape[0] + 1)
        rt._diag_block(func, side, uplo, Ad.T if ta else Ad, Bd)
        torch.cuda.synchronize()
        ref = oracle.blas_rectrxm(side, uplo, "N", 1.0, func, A.astype(np.float64), B.astype(np.float64))
        assert oracle.rel_err(to_host(Bd), ref) < TOL[dtype], (n, m, side, uplo, ta)


# Strips of 32 and 64 columns (16 warps in Float32 and Float16), whole and
# with a remainder, both orientations of B and of A; same tolerances.
@pytest.mark.parametrize("dtype", [np.float32, np.float16])
@pytest.mark.parametrize("n,m", [(33, 2500), (256, 2433), (130, 5001), (257, 9728)])
@pytest.mark.parametrize("func", ["S", "M"])
def test_strip_wide(pkg, oracle, workloads, cuda, dtype, func, n, m):
    import torch

    rt = pkg.rectrxm
    for side, uplo, ta in [("L", "L", False), ("L", "U", True), ("R", "L", True), ("R", "U", False)]:
        A, B = workloads.problem(n, m, side, uplo, seed=n + m)
        A, B = A.astype(dtype), B.astype(dtype)
        stored = A.T if ta else A
        Ad = to_dev(stored, dtype, cuda, ld=n + 3)
        Bd = to_dev(B, dtype, cuda, ld=B.shape[0] + 1)
        rt._diag_block(func, side, uplo, Ad.T if ta else Ad, Bd)
        torch.cuda.synchronize()
        ref = oracle.blas_rectrxm(side, uplo, "N", 1.0, func, A.astype(np.float64), B.astype(np.float64))
        assert oracle.rel_err(to_host(Bd), ref) < TOL[dtype], (side, uplo, ta)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("n,m", [(17, 3), (40, 24), (96, 300), (128, 2500)])
def test_strip_multiply_rows(pkg, workloads, cuda, dtype, n, m):
    """A row of a multiply takes nothing from the rows past it (Inf and NaN
    there do not reach it), and its largest term, the diagonal's, is rounded
    once.  Bound per element: at most n + 4 roundings of the off-diagonal sums
    plus one of the result, u (n + 4) S_off + 1.01 u |y| (u the unit roundoff,
    S_off = sum of |a x| left of the diagonal)."""
    import torch

    rng = np.random.default_rng(n)
    A = np.tril(rng.standard_normal((n, n)) / np.sqrt(n), -1) + np.diag(2 + np.abs(rng.standard_normal(n)))
    B = rng.uniform(-1, 1, (n, m))
    A, B = A.astype(dtype), B.astype(dtype)
    u = np.finfo(dtype).eps / 2
    for bad in (None, n // 2, n - 1):
        Bb = B.copy()
        if bad is not None:
            Bb[bad, 0], Bb[bad, m - 1] = np.inf, np.nan
        Ad, Bd = to_dev(A, dtype, cuda, ld=n + 1), to_dev(Bb, dtype, cuda, ld=n + 2)
        pkg.rectrxm._diag_block("M", "L", "L", Ad, Bd)
        torch.cuda.synchronize()
        got = to_host(Bd).astype(np.longdouble)
        with np.errstate(all="ignore"):
            A8, B8 = A.astype(np.longdouble), B.astype(np.longdouble)
            ref = A8 @ B8
            off = np.abs(np.tril(A8, -1)) @ np.abs(B8)
        rows = slice(0, n if bad is None else bad)
        err = np.abs(got - ref)[rows]
        assert (err <= (u * (n + 4) * off + u * 1.01 * np.abs(ref))[rows]).all(), (n, m, bad)
        if bad is not None:
            assert not np.isfinite(got[bad:, [0, m - 1]]).any()
            keep = slice(1, m - 1)
            assert np.isfinite(got[:, keep]).all()
