"""Float32 and ComplexF32 updates on the tensor cores where the operands
leave the range that three BF16 terms hold: element by element as accurate as
the plain product, and not much slower than it.

Tolerance per element: (12 + K) 2^-24 (|C| + sum |a b|), the bound of a chain
of K Float32 FMAs with the slack of the tensor-core form, plus 2^-140 for
products below Float32's normal range."""

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ta,tb", [(0, 0), (1, 1)])
def test_tiny_elements_in_rows_of_ordinary_ones(pkg, cuda, ta, tb):
    """Elements near 2^-123 whose partners are large while the row's large
    elements meet zeros: their products are all of the result."""
    import torch

    rng = np.random.default_rng(5)
    N, K, M = 300, 256, 1000
    A, B = rng.standard_normal((N, K)), rng.standard_normal((K, M))
    small = rng.random((N, K)) < 0.5
    A[small] *= 2.0 ** -123
    A[100:, :] = rng.standard_normal((N - 100, K))  # and rows without any
    B[:, :500] = rng.standard_normal((K, 500)) * 2.0 ** 30
    B[:, 7] *= 2.0 ** -148  # a column of tiny elements
    for i in range(100):  # column 500 + i meets row i's tiny elements only
        B[:, 500 + i] = np.where(small[i], B[:, 500 + i] * 2.0 ** 66, 0.0)
    A, B = A.astype(np.float32), B.astype(np.float32)
    C = np.zeros((N, M), dtype=np.float32)
    Ad = to_dev(A.T if ta else A, np.float32, cuda)
    Bd = to_dev(B.T if tb else B, np.float32, cuda)
    Cd = to_dev(C, np.float32, cuda)
    pkg.matmul_(Cd, Ad.T if ta else Ad, Bd.T if tb else Bd, 1.0)
    torch.cuda.synchronize()
    pkg.device_status(Cd)
    A8, B8 = A.astype(np.float64), B.astype(np.float64)
    bound = (12 + K) * 2.0 ** -24 * (np.abs(A8) @ np.abs(B8)) + 2.0 ** -140
    assert (np.abs(to_host(Cd) - A8 @ B8) <= bound).all()


def _ms(fn, reps=3):
    import torch

    fn()
    best = float("inf")
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        best = min(best, a.elapsed_time(b))
    return best


@pytest.mark.parametrize("dtype", ["float32", "complex64"])
@pytest.mark.parametrize("case", ["not finite", "tiny", "one row"])
def test_speed_does_not_collapse(pkg, cuda, dtype, case):
    """A whole update outside the range costs what the CUDA-core tiling does
    (about 6 times the tensor cores at this size), not a serial sum per
    element; 20 times leaves room for the clock and small launches."""
    import torch

    dt = getattr(torch, dtype)
    g = torch.Generator(device=cuda).manual_seed(2)
    n = 2048 if dtype == "float32" else 1024
    A, B = (torch.randn((n, n), generator=g, device=cuda, dtype=dt).T for _ in range(2))
    C = torch.zeros((n, n), device=cuda, dtype=dt).T
    usual = _ms(lambda: pkg.matmul_(C, A, B, 1e-6))
    if case == "not finite":
        B[5, :] = float("nan")
    elif case == "tiny":
        A, B = A * 2.0 ** -60, B * 2.0 ** -60
        A, B = A.T.contiguous().T, B.T.contiguous().T
    else:
        A[77, 9] = float("inf")
    C.zero_()
    special = _ms(lambda: pkg.matmul_(C, A, B, 1e-6))
    assert special < 20 * usual, (special, usual)


def test_c32_rows_outside_the_range(pkg, cuda):
    """ComplexF32: rows and columns of tiny, large and ordinary elements in
    every pairing, per real component, against Float64."""
    import torch

    rng = np.random.default_rng(12)
    N, K, M = 200, 150, 1500

    def make(r, c):
        return rng.standard_normal((r, c)) + 1j * rng.standard_normal((r, c))

    A, B = make(N, K), make(K, M)
    A[3] *= 2.0 ** -110
    A[4] *= 2.0 ** 60
    A[150, ::2] *= 2.0 ** -112
    B[:, 700] *= 2.0 ** 55
    B[:, 701] *= 2.0 ** -75
    A, B = A.astype(np.complex64), B.astype(np.complex64)
    for form in ("NN", "TC", "CT"):
        op = {"N": lambda X: X, "T": lambda X: X.T, "C": lambda X: X.conj().T}
        view = {"N": lambda X: X, "T": lambda X: X.T, "C": lambda X: X.T.conj()}
        Ad, Bd = (torch.from_numpy(np.ascontiguousarray(op[f](X).T)).to(cuda).T for f, X in zip(form, (A, B)))
        Cd = torch.zeros((M, N), device=cuda, dtype=torch.complex64).T
        pkg.matmul_(Cd, view[form[0]](Ad), view[form[1]](Bd), -1.0)
        torch.cuda.synchronize()
        got = Cd.cpu().numpy().astype(np.complex128)
        A8, B8 = A.astype(np.complex128), B.astype(np.complex128)
        ref = -(A8 @ B8)
        ar, ai, br, bi = np.abs(A8.real), np.abs(A8.imag), np.abs(B8.real), np.abs(B8.imag)
        u = (12 + 2 * K) * 2.0 ** -24
        assert (np.abs((got - ref).real) <= u * (ar @ br + ai @ bi) + 2.0 ** -140).all(), form
        assert (np.abs((got - ref).imag) <= u * (ar @ bi + ai @ br) + 2.0 ** -140).all(), form
