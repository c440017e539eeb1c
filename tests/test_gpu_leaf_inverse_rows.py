"""Exact mixed solves through inverse leaves, with a singular or non-finite
triangle: a zero pivot or a NaN in A makes exactly those unknowns non-finite
that depend on it, and leaves the others as accurate as ever.

Unknown i of the order of substitution depends on pivot k for i >= k, and on the
element (k + 1, k) for i >= k + 1.  The others: 1e-13 of the solution, as for the
exact solves elsewhere."""

import itertools

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [64, 50, 128, 200])
@pytest.mark.parametrize("what", ["pivot", "nan"])
def test_only_dependent_unknowns_are_lost(pkg, workloads, cuda, n, what):
    import torch

    m = 700
    for (side, uplo, trans), k in itertools.product(itertools.product("LR", "LU", "NT"), (0, 3, 21, 40, n - 2)):
        A, B = workloads.problem(n, m, side, uplo, seed=n + k)
        A = A.copy()
        lower = (uplo == "L") != (trans == "T")  # of op(A)
        forward = lower == (side == "L")         # unknowns solved from the first on
        order = np.arange(n) if forward else np.arange(n)[::-1]
        clean = A.copy()
        if what == "pivot":
            A[order[k], order[k]] = 0.0
            lost = order[k:]
        else:
            r, c = order[k + 1], order[k]  # unknown r's equation meets unknown c
            r, c = (r, c) if (side == "L") != (trans == "T") else (c, r)
            A[r, c] = np.nan
            lost = order[k + 1:]
        X = to_dev(B, np.float64, cuda)
        pkg.unified_rectrxm_mixed_(side, uplo, trans, 1.0, "S", to_dev(A, np.float64, cuda), X, split_terms=7, sweeps=0,
                                   cutoff=64)
        torch.cuda.synchronize()
        pkg.device_status(X)
        got = to_host(X) if side == "L" else to_host(X).T
        bad = ~np.isfinite(got)
        want_bad = np.zeros((n, m), dtype=bool)
        want_bad[lost] = True
        assert np.array_equal(bad, want_bad), (side, uplo, trans, k)
        kept = np.setdiff1d(np.arange(n), lost)
        T = np.tril(clean) if uplo == "L" else np.triu(clean)
        T = T.T if trans == "T" else T
        T, R = (T, B) if side == "L" else (T.T, B.T)
        ref = np.linalg.solve(T[np.ix_(kept, kept)], R[kept]) if len(kept) else np.zeros((0, m))
        assert np.linalg.norm(got[kept] - ref) <= 1e-13 * max(np.linalg.norm(ref), 1e-300), (side, uplo, trans, k)
