"""What exact solves keep on the device between calls: no more than the slices
of the operands' digits would take (14 bytes per operand element and 8 per
element of the updated block, in padded rows), or 1 GiB where that is less,
plus the narrowest panel of residues and the growth margin of an eighth.  And
the panels change no bit of the result."""

import pytest

pytestmark = pytest.mark.gpu

GIB = 1 << 30


def _problem(n, m, side, cuda, seed=0):
    import torch

    g = torch.Generator(device=cuda).manual_seed(seed)
    A = torch.randn((n, n), generator=g, device=cuda, dtype=torch.float64).div_(n ** 0.5)
    A.diagonal().abs_().add_(2.0)
    B = torch.rand((m, n) if side == "L" else (n, m), generator=g, device=cuda, dtype=torch.float64).T
    return A.T, B


def _held(fn, cuda):
    """Device memory that a call on a stream of its own leaves in use."""
    import torch

    torch.cuda.synchronize()
    s = torch.cuda.Stream()
    before = torch.cuda.mem_get_info(cuda)[0]
    with torch.cuda.stream(s):
        fn()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info(cuda)[0]


@pytest.mark.parametrize("side,n,m", [("L", 8192, 16384), ("R", 8192, 16384), ("L", 16384, 4096)])
def test_exact_solve_workspace(pkg, cuda, side, n, m):
    A, B = _problem(n, m, side, cuda)
    X = B.T.clone().T
    k = n // 2  # the largest update: k unknowns of K = k
    slices = 14 * (k * k + k * m) + 8 * k * m
    panel = 1024 * 32 * k + 1024 * 16 * max(k, m)
    held = _held(lambda: pkg.unified_rectrxm_mixed_(side, "L", "N", 1.0, "S", A, X, split_terms=7, sweeps=0), cuda)
    assert held <= 1.125 * max(slices, GIB, 32 * k * min(k, m) + panel) + GIB // 8, held / GIB


@pytest.mark.parametrize("side,n,m", [("L", 4096, 20000), ("R", 4096, 20000)])
def test_refined_solve_workspace(pkg, cuda, side, n, m):
    A, B = _problem(n, m, side, cuda)
    X = B.T.clone().T
    k = n // 2
    updates = 1.125 * max(6 * (k * k + k * m), GIB)  # three terms
    slices = 14 * (n * n + n * m)
    panel = 1024 * 32 * n + 1024 * 16 * n
    residual = 16 * n * m + max(slices, GIB, 32 * n * n + panel)
    held = _held(lambda: pkg.unified_rectrxm_mixed_(side, "L", "N", 1.0, "S", A, X, split_terms=3, sweeps=1), cuda)
    assert held <= updates + residual + GIB // 8, held / GIB


@pytest.mark.parametrize("side,n,m,sweeps", [("L", 4096, 9000, 0), ("R", 4096, 9000, 0), ("L", 6000, 2500, 0),
                                             ("R", 2048, 12000, 1), ("L", 2048, 12000, 1)])
def test_panels_change_no_bit(pkg, cuda, side, n, m, sweeps):
    """On a stream that already holds the memory for whole residues and on one
    that does not; refinement, whose panels do not depend on that, against a
    solve of its first and last columns alone."""
    import torch

    A, B = _problem(n, m, side, cuda, seed=n)

    def solve(X):
        pkg.unified_rectrxm_mixed_(side, "L", "T", 0.5, "S", A, X, split_terms=7, sweeps=sweeps, cutoff=64)
        return X

    X = solve(B.T.clone().T)
    if sweeps == 0:
        with torch.cuda.stream(torch.cuda.Stream()):
            big_A, big_B = _problem(8192, 12000, "L", cuda)
            pkg.unified_rectrxm_mixed_("L", "L", "N", 1.0, "S", big_A, big_B, split_terms=7, sweeps=0)
            Y = solve(B.T.clone().T)
        torch.cuda.synchronize()
        assert torch.equal(X, Y)
    for cols in (slice(0, 500), slice(m - 700, m)):
        part = B[:, cols] if side == "L" else B[cols, :]
        part = solve(part.T.clone().T)
        torch.cuda.synchronize()
        assert torch.equal(part, X[:, cols] if side == "L" else X[cols, :])
