"""The exact update from residues (nla_crt.cu) through matmul_mixed_ with
split_terms=7, at the edges of its tiles (128 columns x 256 or 128 rows), its
64-wide K blocks and its 1024-wide exact chunks, and across the change of the
operands' bits at K = 14336.

Integer operands of few bits make every product and sum exact, so the update
must equal the integer result bit for bit.  Random operands: every element of
a row is rounded to 2^-56 of at most four times the row's largest value
(2^-55 past K = 14336) and the sum once to FP64, so the error is at most
K (2^-53 amax |bmax| 2) + 2^-53 |result|, written below with one factor two
to spare for the second-order term."""

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (64, 200, 64), (128, 129, 65), (129, 127, 128), (257, 300, 1024), (300, 513, 1025),
          (385, 100, 3000), (100, 70, 14400)]


def _update(pkg, cuda, A, B, C, ta, tb, alpha):
    import torch

    Ad = to_dev(A.T if ta else A, np.float64, cuda, ld=(A.shape[1] if ta else A.shape[0]) + 1)
    Bd = to_dev(B.T if tb else B, np.float64, cuda, ld=(B.shape[1] if tb else B.shape[0]) + 2)
    Cd = to_dev(C, np.float64, cuda, ld=C.shape[0] + 3)
    pkg.matmul_mixed_(Cd, Ad.T if ta else Ad, Bd.T if tb else Bd, alpha, split_terms=7)
    pkg.device_status(Cd)
    return to_host(Cd)


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 0), (0, 1), (1, 1)])
def test_integers_are_exact(pkg, cuda, ta, tb):
    rng = np.random.default_rng(1)
    for M, N, K in SHAPES:
        A = rng.integers(-1000, 1001, (M, K)).astype(np.float64)
        B = rng.integers(-1000, 1001, (K, N)).astype(np.float64)
        C = rng.integers(-1000, 1001, (M, N)).astype(np.float64)
        A[0, :] = 0.0
        assert np.array_equal(_update(pkg, cuda, A, B, C, ta, tb, -1.0), C - A @ B), (M, N, K)


@pytest.mark.parametrize("values", ["normal", "extremes"])
def test_random_within_the_rounding(pkg, cuda, values):
    """'extremes': every element +-(largest), the largest integers the
    residues have to carry, all of one sign in half of the rows."""
    rng = np.random.default_rng(2)
    for M, N, K in SHAPES:
        if values == "normal":
            A, B = rng.standard_normal((M, K)), rng.standard_normal((K, N))
        else:
            big = np.nextafter(1.0, 0.0)
            A, B = big * np.sign(rng.standard_normal((M, K))), np.full((K, N), big)
            A[::2] = big
        C = np.zeros((M, N))
        got = _update(pkg, cuda, A, B, C, 0, 0, 1.0)
        ref = (A.astype(np.longdouble) @ B.astype(np.longdouble)).astype(np.float64) if M * N * K < 3e7 else A @ B
        slack = 0.0 if M * N * K < 3e7 else K * 2.0 ** -53 * np.abs(A) @ np.abs(B)
        amax = np.abs(A).max(axis=1, keepdims=True)
        bmax = np.abs(B).max(axis=0, keepdims=True)
        bound = K * 2.0 ** -52 * amax * bmax + 2.0 ** -52 * np.abs(ref) + slack
        assert (np.abs(got - ref) <= bound).all(), (M, N, K)
        if values == "extremes":  # the products are exact sums of (1 - 2^-53)^2
            assert np.abs(got[0] - K * big * big).max() <= 2.0 ** -52 * K


def test_scales_and_special_values(pkg, cuda):
    """Rows and columns of very different scales keep their own precision;
    one that holds an Inf or NaN gives NaN, the others are untouched."""
    rng = np.random.default_rng(3)
    M, N, K = 140, 260, 96
    A, B = rng.integers(-9, 10, (M, K)).astype(np.float64), rng.integers(-9, 10, (K, N)).astype(np.float64)
    sa, sb = np.exp2(rng.integers(-300, 301, (M, 1))), np.exp2(rng.integers(-300, 301, (1, N)))
    C = np.zeros((M, N))
    assert np.array_equal(_update(pkg, cuda, A * sa, B * sb, C, 0, 0, 1.0), (A @ B) * (sa * sb))
    tiny = np.zeros((M, K))
    tiny[5] = 5e-324 * rng.integers(-4, 5, K)
    assert np.array_equal(_update(pkg, cuda, tiny, B, C, 0, 0, 1.0), tiny @ B)
    A[3, 7], A[130, 0], B[2, 259] = np.inf, np.nan, -np.inf
    got = _update(pkg, cuda, A, B, C, 0, 0, 1.0)
    assert np.isnan(got[[3, 130]]).all() and np.isnan(got[:, 259]).all()
    keep = np.ix_([i for i in range(M) if i not in (3, 130)], range(N - 1))
    A[3, 7], A[130, 0], B[2, 259] = 0.0, 0.0, 0.0
    assert np.array_equal(got[keep], (A @ B)[keep])
