"""Complex diagonal blocks on the strip kernel at the edges of its panels and
strips, against numpy in ComplexF64.

Tolerances (relative Frobenius error): ComplexF64 1e-14 and ComplexF32 1e-5,
the real types' own."""

import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1), (15, 3), (17, 2), (32, 40), (33, 310), (100, 9), (128, 700), (128, 2500)]


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("func", ["S", "M"])
def test_complex_strip_edges(pkg, cuda, dtype, func):
    import torch

    rt = pkg.rectrxm
    rng = np.random.default_rng(12)
    forms = itertools.cycle(itertools.product("LR", "LU", "NTC"))
    for (n, m), (side, uplo, view) in zip(SHAPES * 2, forms):
        T = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))) / np.sqrt(n)
        T = np.tril(T, -1) if uplo == "L" else np.triu(T, 1)
        T += np.diag((2 + np.abs(rng.standard_normal(n))) * np.exp(1j * rng.uniform(0, 6, n)))
        T = T.astype(dtype)
        B = (rng.uniform(-1, 1, (n, m)) + 1j * rng.uniform(-1, 1, (n, m))).astype(dtype)
        B = B if side == "L" else np.ascontiguousarray(B.T)
        stored = {"N": T, "T": T.T, "C": T.conj().T}[view]
        Ad = torch.from_numpy(np.ascontiguousarray(stored.T)).to(cuda).T
        Ad = {"N": Ad, "T": Ad.T, "C": Ad.T.conj()}[view]
        Bd = torch.from_numpy(np.ascontiguousarray(B.T)).to(cuda).T
        rt._diag_block(func, side, uplo, Ad, Bd)
        torch.cuda.synchronize()
        T, B = T.astype(np.complex128), B.astype(np.complex128)
        if func == "M":
            ref = T @ B if side == "L" else B @ T
        else:
            ref = np.linalg.solve(T, B) if side == "L" else np.linalg.solve(T.T, B.T).T
        got = Bd.cpu().numpy()
        tol = 1e-5 if dtype == np.complex64 else 1e-14
        assert np.linalg.norm(got - ref) < tol * np.linalg.norm(ref), (n, m, side, uplo, view)
