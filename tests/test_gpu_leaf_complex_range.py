"""Complex diagonal blocks whose pivots have no finite reciprocal: the
quotients are finite all the same, and one that overflows is infinite.

Row i of the system is scaled by 2^s with s far below the type's smallest
normal exponent, so that 1 / a_ii overflows while a_ii x_i = b_i has the
solution of the unscaled row.  The scaled values are subnormal, with
p = (bits left) of precision: the solution is that of the stored values, and
each of a row's n + 2 operations rounds to the smallest subnormal at most,
2^-p of the row's scale, which the well-conditioned rows after it keep within
a factor of 4: (n + 2) 2^(2 - p)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (dtype, real parts, exponent of the scaled rows, bits of precision left there)
TYPES = [("complex64", np.float32, -130, 19), ("complex128", np.float64, -1026, 48)]


def _dev(X, dtype, cuda):
    import torch

    return torch.from_numpy(np.ascontiguousarray(X.T)).to(cuda, getattr(torch, dtype)).T


def _matrix(n, rng):
    A = np.tril(rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)), -1) / (4 * n)
    return A + np.diag(1.0 + 0.5 * rng.random(n) + 1j * rng.uniform(-0.5, 0.5, n))


@pytest.mark.parametrize("dtype,real,s,p", TYPES)
@pytest.mark.parametrize("side,m", [("L", 3), ("R", 70), ("L", 5000)])
def test_tiny_pivots(pkg, cuda, dtype, real, s, p, side, m):
    import torch

    n = 70
    rng = np.random.default_rng(n)
    wide = np.clongdouble
    A, B = _matrix(n, rng), rng.uniform(-1, 1, (n, m)) + 1j * rng.uniform(-1, 1, (n, m))
    rows = [0, 5, 17, 31, 32, 50, n - 1]
    A[rows, :] *= 2.0 ** s
    B[rows, :] *= 2.0 ** s
    A, B = A.astype(dtype), B.astype(dtype)
    X = _dev(B if side == "L" else B.T, dtype, cuda)
    pkg.unified_rectrxm_(side, "L", "N" if side == "L" else "T", 1.0, "S", _dev(A, dtype, cuda), X)
    torch.cuda.synchronize()
    got = X.cpu().numpy()
    got = got if side == "L" else got.T
    # The stored values' solution, with the scaled rows brought back to size.
    up = np.ones((n, 1), dtype=np.longdouble)
    up[rows] = np.ldexp(np.longdouble(1), -s)
    A, B = A.astype(wide) * up, B.astype(wide) * up
    want = np.zeros((n, m), dtype=wide)
    for i in range(n):
        want[i] = (B[i] - A[i, :i] @ want[:i]) / A[i, i]
    assert np.isfinite(got).all(), dtype
    assert np.abs(got - want).max() <= (n + 2) * 2.0 ** (2 - p) * np.abs(want).max()


@pytest.mark.parametrize("dtype,real,s,p", TYPES)
def test_quotient_overflows_to_infinity(pkg, cuda, dtype, real, s, p):
    import torch

    n, m = 40, 6
    rng = np.random.default_rng(n)
    A = _matrix(n, rng)
    A[n - 1, :] = 0
    A[n - 1, n - 1] = 2.0 ** (s + 10)
    B = rng.uniform(-1, 1, (n, m)) + 1j * rng.uniform(-1, 1, (n, m))
    B[n - 1, :] = [2.0 ** 20, -2.0 ** 20, 2.0 ** 30, 1e3, -1e3, 2.0 ** 25]
    X = _dev(B.astype(dtype), dtype, cuda)
    pkg.unified_rectrxm_("L", "L", "N", 1.0, "S", _dev(A.astype(dtype), dtype, cuda), X)
    torch.cuda.synchronize()
    got = X.cpu().numpy()
    assert np.isfinite(got[:n - 1]).all()
    big = np.isinf(np.float64(B[n - 1].real) / np.float64(2.0) ** (s + 10)) if real is np.float64 else np.abs(
        B[n - 1].real) * 2.0 ** -(s + 10) > np.finfo(np.float32).max
    assert np.array_equal(np.isinf(got[n - 1].real), big) and big.any()
    assert np.array_equal(np.sign(got[n - 1].real), np.sign(B[n - 1].real))
    assert np.array_equal(got[n - 1].imag, np.zeros(m, dtype=real))
