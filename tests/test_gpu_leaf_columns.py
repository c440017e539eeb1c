"""Diagonal blocks of few rows with very many right-hand sides (one right-hand
side per thread), and the strips' panels at row counts that are no multiple of
a panel: solves and multiplies of every type at the edges of the four-row
groups and of the CTAs' 64 columns, against torch in 64 bits, element by
element.

Tolerance: an element of a product is n products and sums, rounded once each
at most, (n + 2) u sum |l| |x| (complex: four products to one, 4 u); a solve's
residual likewise, (n + 4) u (|L| |X| + |B|).  The reference of the 64-bit
types is as far off again: twice that.  Float16 results below its normal range
are rounded to multiples of 2^-24, an error of 2^-25 each."""

import itertools

import pytest

pytestmark = pytest.mark.gpu

U = {"float16": 2.0 ** -11, "float32": 2.0 ** -24, "float64": 2.0 ** -53, "complex64": 2.0 ** -22,
     "complex128": 2.0 ** -51}


def _check(pkg, cuda, dtype, side, uplo, func, n, m, special):
    import torch

    dt = getattr(torch, dtype)
    wide = torch.complex128 if dt.is_complex else torch.float64
    g = torch.Generator(device=cuda).manual_seed(n + m)

    def rand(r, c):
        X = torch.randn((c, r), generator=g, device=cuda, dtype=torch.float64)
        if dt.is_complex:
            X = torch.complex(X, torch.randn((c, r), generator=g, device=cuda, dtype=torch.float64))
        return X.T

    A = rand(n, n) / n ** 0.5
    A.diagonal().copy_(A.diagonal().abs() + 2)
    A = A.to(dt).T.contiguous().T
    B = rand(*((n, m) if side == "L" else (m, n))).to(dt)
    if special:
        k, j = n // 2, m - 3
        (B if side == "L" else B.T)[k, j] = float("nan")
    X = torch.empty((B.shape[1], B.shape[0] + 3), device=cuda, dtype=dt).T[:B.shape[0]]
    X.copy_(B)
    name = {"L": "Left", "R": "Right"}[side] + {"L": "Lower", "U": "Upper"}[uplo] + {"S": "TRSM_", "M": "TRMM_"}[func]
    from nextla_gb300 import rectrxm

    getattr(rectrxm, name)(A, X)
    torch.cuda.synchronize()
    T = A.to(wide).tril() if uplo == "L" else A.to(wide).triu()
    if side == "R":
        T, X, B = T.T, X.T, B.T
    X, B = X.to(wide), B.to(wide)
    if special:
        bad = ~torch.isfinite(X.abs())
        reads = (T.abs() > 0).double()  # rows that depend on row k: all of its side of the triangle
        want = (reads[:, k] > 0) if func == "M" else ((torch.arange(n, device=cuda) >= k) if T.triu(1).abs().sum() == 0
                                                      else (torch.arange(n, device=cuda) <= k))
        assert torch.equal(bad[:, j], want), (name, n, m)
        keep = torch.ones(m, dtype=torch.bool, device=cuda)
        keep[j] = False
        assert not bool(bad[:, keep].any())
        X, B = X[:, keep], B[:, keep]
    u, tiny = 2 * U[dtype], 2.0 ** -25 if dtype == "float16" else 0.0
    if func == "M":
        assert bool(((X - T @ B).abs() <= (n + 2) * u * (T.abs() @ B.abs()) + tiny).all()), (name, n, m)
    else:
        assert bool(((T @ X - B).abs() <= (n + 4) * u * (T.abs() @ X.abs() + B.abs()) + tiny * T.abs().sum(1, keepdim=True)).all()), (name, n, m)


@pytest.mark.parametrize("dtype", sorted(U))
@pytest.mark.parametrize("n", [1, 3, 4, 5, 16, 31, 32, 47, 48, 64])
def test_blocks_of_few_rows(pkg, cuda, dtype, n):
    """64 columns past the largest of the rule's lines, and one short of a CTA."""
    for side, uplo, func in ("LLS", "RUS", "LUS", "RLS", "LUM", "RLM"):
        _check(pkg, cuda, dtype, side, uplo, func, n, 21001, n > 1 and func == "M")
    _check(pkg, cuda, dtype, "L", "L", "S", n, 25000 + 63, n > 1)


@pytest.mark.parametrize("dtype", sorted(U))
@pytest.mark.parametrize("n", [15, 17, 33, 49, 65, 100, 127])
def test_strips_at_ragged_panels(pkg, cuda, dtype, n):
    for (side, uplo), func, m in itertools.product(("LL", "RU"), "SM", (1, 2500)):
        _check(pkg, cuda, dtype, side, uplo, func, n, m, False)


@pytest.mark.parametrize("n,m", [(49, 19000), (64, 15000), (113, 30000), (128, 36000), (100, 30000)])
def test_float64_wide_columns(pkg, cuda, n, m):
    for side, uplo in ("LL", "RU"):
        _check(pkg, cuda, "float64", side, uplo, "S", n, m, False)
