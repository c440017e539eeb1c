"""Updates with more columns than the narrow tilings' grids reach: every
tiling puts the columns' tiles on a grid dimension of 65535, and one that does
not reach must not be chosen.  Just past 65535 times each tile width, against
torch's product.

Tolerance: K + 2 roundings of the element type's unit on sum |a||b| + |c|
(Float16 accumulates in Float32 and rounds once), doubled for the reference."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,N,M,u", [("float64", 16, 65535 * 16 + 3, 2.0 ** -53), ("float64", 32, 65535 * 32 + 5, 2.0 ** -53),
                                         ("float64", 16, 65535 * 32 + 5, 2.0 ** -53), ("float32", 32, 65535 * 32 + 1, 2.0 ** -24),
                                         ("float32", 64, 65535 * 64 + 7, 2.0 ** -24), ("float16", 64, 65535 * 64 + 7, 2.0 ** -11),
                                         ("complex64", 16, 65535 * 32 + 1, 2.0 ** -24)])
def test_update_of_many_columns(pkg, cuda, dtype, N, M, u):
    import torch

    dt = getattr(torch, dtype)
    g = torch.Generator(device=cuda).manual_seed(N + M)
    K = 3

    def make(r, c):
        work = dt if dt != torch.float16 else torch.float32
        return torch.randn((c, r), generator=g, device=cuda, dtype=work).to(dt).T

    A, B, C = make(N, K), make(K, M), make(N, M)
    X = C.T.clone().T
    pkg.matmul_(X, A, B, -1.0)
    torch.cuda.synchronize()
    work = torch.complex128 if dt.is_complex else torch.float64
    step = 1 << 20
    for c in range(0, M, step):
        s = slice(c, min(M, c + step))
        ref = C[:, s].to(work) - A.to(work) @ B[:, s].to(work)
        bound = 2 * (K + 2) * u * (C[:, s].abs().to(torch.float64) + A.abs().to(torch.float64) @ B[:, s].abs().to(torch.float64))
        assert bool(((X[:, s].to(work) - ref).abs() <= (2 if dt.is_complex else 1) * bound).all()), (dtype, N, M, c)


@pytest.mark.parametrize("n", [272])
def test_solve_of_many_right_hand_sides(pkg, cuda, n):
    """A left-side Float64 solve whose last split leaves a 16-row update."""
    import torch

    m = 65535 * 32 + 5
    g = torch.Generator(device=cuda).manual_seed(1)
    A = torch.randn((n, n), generator=g, device=cuda, dtype=torch.float64).div_(n ** 0.5).tril_()
    A.diagonal().abs_().add_(2.0)
    A = A.T.contiguous().T
    X = torch.rand((m, n), generator=g, device=cuda, dtype=torch.float64).T
    cols = torch.randint(0, m, (300,), generator=g, device=cuda)
    want = torch.linalg.solve_triangular(A, X[:, cols].contiguous(), upper=False)
    pkg.unified_rectrxm_("L", "L", "N", 1.0, "S", A, X)
    torch.cuda.synchronize()
    assert float((X[:, cols] - want).norm() / want.norm()) < 1e-14
