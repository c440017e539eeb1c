"""unified_rec on the host, as the reference runs it (src/rectrxm.jl:101-198):
the recursion itself, and the calls of unified_rectrxm_ that only it can
express (a transposed or conjugated view of a complex A with transpose 'C', a
complex alpha with thresholds, thresholds outside 1..1024), against Float64
references.

Tolerances: 1e-13 in Float64 and ComplexF64, 1e-5 in Float32 and ComplexF32,
as for the native calls."""

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _problem(n, m, side, uplo, dtype, cuda, seed):
    import torch

    rng = np.random.default_rng(seed)
    cx = np.dtype(dtype).kind == "c"

    def make(*s):
        return rng.standard_normal(s) + (1j * rng.standard_normal(s) if cx else 0)

    A = make(n, n) / np.sqrt(n)
    A[np.diag_indices(n)] = 2 + np.abs(rng.standard_normal(n))
    A, B = A.astype(dtype), make(*((n, m) if side == "L" else (m, n))).astype(dtype)

    def dev(X):
        return torch.from_numpy(np.ascontiguousarray(X.T)).to(cuda).T

    return A, B, dev(A), dev(B)


def _want(A, B, side, uplo, op, alpha, func):
    T = np.tril(A) if uplo == "L" else np.triu(A)
    T = op(T.astype(np.complex128 if np.iscomplexobj(T) else np.float64))
    B = alpha * B
    if func == "M":
        return T @ B if side == "L" else B @ T
    return np.linalg.solve(T, B) if side == "L" else np.linalg.solve(T.T, B.T).T


def _close(X, want, dtype):
    got = X.cpu().numpy()
    return np.linalg.norm(got - want) <= (1e-13 if np.dtype(dtype).name in ("float64", "complex128") else 1e-5) * \
        np.linalg.norm(want)


@pytest.mark.parametrize("dtype", [np.float32, np.float64, np.complex64, np.complex128])
@pytest.mark.parametrize("threshold", [16, 256])
def test_unified_rec(pkg, cuda, dtype, threshold):
    from nextla_gb300 import rectrxm

    for (n, m), func, side, uplo in itertools.product([(70, 5), (300, 33)], "SM", "LR", "LU"):
        A, B, Ad, X = _problem(n, m, side, uplo, dtype, cuda, n)
        rectrxm.unified_rec(func, side, uplo, Ad, n, X, threshold)
        assert _close(X, _want(A, B, side, uplo, lambda T: T, 1.0, func), dtype), (n, func, side, uplo)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_conjugated_and_transposed_views(pkg, cuda, dtype):
    for n, func, side, uplo in itertools.product([40, 300], "SM", "LR", "LU"):
        # A passed as a view: the flags describe that view.
        forms = [(lambda X: X.T, "C", np.conj), (lambda X: X.T.conj(), "N", lambda T: T.conj().T),
                 (lambda X: X.conj(), "T", lambda T: T.conj().T), (lambda X: X.conj(), "C", lambda T: T.T)]
        for view, trans, op in forms:
            A, B, Ad, X = _problem(n, 9, side, uplo, dtype, cuda, n)
            transposed = view(Ad).stride() != Ad.stride()
            up = ("U" if uplo == "L" else "L") if transposed else uplo  # the triangle as the view shows it
            pkg.unified_rectrxm_(side, up, trans, 0.5, func, view(Ad), X)
            assert _close(X, _want(A, B, side, uplo, op, 0.5, func), dtype), (n, func, side, uplo, trans)


@pytest.mark.parametrize("dtype,alpha,thresholds", [(np.float64, -0.5, (2000, 1500)), (np.float32, 0.5, (5000, 1025)),
                                                     (np.complex128, 1 - 2j, (64, 16)), (np.complex64, 2j, (256, 16))])
def test_thresholds_only_the_host_takes(pkg, cuda, dtype, alpha, thresholds):
    """500 rows: below the first two thresholds, one base case; several levels
    of recursion for the others."""
    for func, side, uplo in itertools.product("SM", "LR", "LU"):
        A, B, Ad, X = _problem(500, 21, side, uplo, dtype, cuda, 7)
        pkg.unified_rectrxm_(side, uplo, "T", alpha, func, Ad, X, thresholds=thresholds)
        assert _close(X, _want(A, B, side, uplo, lambda T: T.T, alpha, func), dtype), (func, side, uplo)
