"""Updates on either side of the lines that choose between the CUDA cores and
the tensor cores (Float32, ComplexF32) and between digit slices and residues
(exact Float64): long and narrow, short K, in every layout, against torch in
64 bits, element by element.

Tolerances: (K + 12) 2^-24 (|C| + sum |a b|) in Float32, twice that with 2 K
products per real component for ComplexF32; exact updates are within
2^-50 of the product of a row's and a column's largest values, K times, plus
the rounding of C (2^-52 |C|), the bound of their 56-bit operands."""

import pytest

pytestmark = pytest.mark.gpu


def _make(r, c, dt, row_major, g, cuda):
    import torch

    shape = (r, c) if row_major else (c, r)
    X = torch.randn(shape, generator=g, device=cuda, dtype=torch.float64)
    if dt.is_complex:
        X = torch.complex(X, torch.randn(shape, generator=g, device=cuda, dtype=torch.float64))
    X = X.to(dt)
    return X if row_major else X.T


@pytest.mark.parametrize("dtype,N,K,M", [("float32", 64, 400, 13000), ("float32", 13000, 400, 64), ("float32", 13000, 513, 65),
                                         ("float32", 95, 130, 12300), ("complex64", 5000, 130, 70), ("complex64", 4000, 200, 90),
                                         ("complex64", 300, 65, 4100), ("complex64", 300, 64, 900), ("complex64", 1000, 127, 300)])
@pytest.mark.parametrize("layout", ["cc", "rr", "cr", "rc"])
def test_single_precision(pkg, cuda, dtype, N, K, M, layout):
    import torch

    dt = getattr(torch, dtype)
    wide = torch.complex128 if dt.is_complex else torch.float64
    g = torch.Generator(device=cuda).manual_seed(N + K)
    A, B, C = (_make(N, K, dt, layout[0] == "r", g, cuda), _make(K, M, dt, layout[1] == "r", g, cuda),
               _make(N, M, dt, False, g, cuda))
    X = C.T.clone().T
    pkg.matmul_(X, A, B, -1.0)
    torch.cuda.synchronize()
    pkg.device_status(X)
    ref = C.to(wide) - A.to(wide) @ B.to(wide)
    k = 2 * K if dt.is_complex else K
    bound = (2 if dt.is_complex else 1) * (k + 12) * 2.0 ** -24 * (C.abs().double() + A.abs().double() @ B.abs().double())
    assert bool(((X.to(wide) - ref).abs() <= bound).all())


@pytest.mark.parametrize("N,K,M", [(2000, 64, 2000), (1500, 64, 1500), (2200, 128, 2200), (128, 128, 40000), (128, 130, 30000),
                                   (3000, 192, 3000), (3000, 255, 3000), (3000, 256, 3000), (16, 16, 50000)])
def test_exact(pkg, cuda, N, K, M):
    import torch

    g = torch.Generator(device=cuda).manual_seed(N + K)
    A, B, C = (_make(r, c, torch.float64, False, g, cuda) for r, c in ((N, K), (K, M), (N, M)))
    X = C.T.clone().T
    pkg.matmul_mixed_(X, A, B, -1.0, split_terms=7)
    torch.cuda.synchronize()
    pkg.device_status(X)
    scale = K * A.abs().amax(1, keepdim=True) * B.abs().amax(0, keepdim=True)
    bound = 2.0 ** -50 * scale + 2.0 ** -52 * C.abs()
    assert bool(((X - (C - A @ B)).abs() <= bound).all())
