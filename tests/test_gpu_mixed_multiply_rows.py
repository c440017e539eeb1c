"""The diagonal blocks of a mixed multiply, row by row: every row takes
exactly the rows of B that its part of the triangle reads.

Up to 64 rows the multiply is one diagonal block in FP64, so each element is
within (n + 2) 2^-53 sum |t| |b| of the product (n products and additions and
the product with alpha, each rounded once), however far the rows of a column
of B are apart, and the reference here, a Float64 product, as far again.  Right-hand
sides enough that the library takes its wide blocks, and few of them with the
block size named by the caller."""

import itertools

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

FORMS = list(itertools.product("LR", "LU", "NT"))


def _multiply(pkg, cuda, side, uplo, trans, A, B, cutoff):
    import torch

    X = B if side == "L" else B.T
    Bd = to_dev(X, np.float64, cuda, ld=X.shape[0] + 1)
    pkg.unified_rectrxm_mixed_(side, uplo, trans, -0.5, "M", to_dev(A, np.float64, cuda), Bd, split_terms=7, sweeps=0,
                               cutoff=cutoff)
    torch.cuda.synchronize()
    pkg.device_status(Bd)
    got = to_host(Bd)
    return got if side == "L" else got.T


def _operand(side, uplo, trans, A):
    """T with result rows -0.5 T B: op(A) for side L, its transpose for side R."""
    T = np.tril(A) if uplo == "L" else np.triu(A)
    T = T.T if trans == "T" else T
    return T if side == "L" else T.T


@pytest.mark.parametrize("n,m,cutoff", [(64, 4000, 0), (37, 4000, 0), (64, 130, 64), (16, 200, 16)])
def test_graded_columns(pkg, cuda, n, m, cutoff):
    rng = np.random.default_rng(n + m)
    for side, uplo, trans in FORMS:
        A = rng.standard_normal((n, n))
        B = rng.uniform(-1, 1, (n, m)) * np.exp2(rng.integers(-60, 61, (n, m)))
        B[:, 0] = np.exp2(np.linspace(-60, 60, n))
        B[:, 1] = B[::-1, 0]
        got = _multiply(pkg, cuda, side, uplo, trans, A, B, cutoff)
        T = _operand(side, uplo, trans, A)
        bound = 2 * (n + 2) * 2.0 ** -53 * 0.5 * (np.abs(T) @ np.abs(B))
        assert (np.abs(got + 0.5 * (T @ B)) <= bound).all(), (side, uplo, trans)


@pytest.mark.parametrize("n,m,cutoff", [(64, 4000, 0), (200, 4000, 0), (200, 300, 64)])
def test_not_finite_rows(pkg, cuda, n, m, cutoff):
    """An Inf or NaN in row k of a column reaches the rows that read row k and
    no other."""
    rng = np.random.default_rng(n)
    for side, uplo, trans in FORMS:
        A, B = rng.standard_normal((n, n)), rng.uniform(-1, 1, (n, m))
        for j, k in enumerate((0, 1, 30, 63, n // 2, n - 1)):
            B[k, 20 * j], B[k, 20 * j + 1] = np.inf, np.nan
        got = _multiply(pkg, cuda, side, uplo, trans, A, B, cutoff)
        T = _operand(side, uplo, trans, A)
        reads = (T != 0).astype(float) @ (~np.isfinite(B)).astype(float) > 0
        assert np.array_equal(~np.isfinite(got), reads), (side, uplo, trans)
        clean = np.where(np.isfinite(B), B, 0.0)
        ref = -0.5 * (T @ clean)
        scale = np.abs(T) @ np.abs(clean)
        assert (np.abs(got - ref)[~reads] <= 2.0 ** -44 * scale.max()).all(), (side, uplo, trans)
