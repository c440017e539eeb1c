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
