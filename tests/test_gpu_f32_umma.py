"""The Float32 update on the tensor cores (three BF16 terms per value) against
the product in Float64, element by element.

Tolerance per element: (12 + K / 64) 2^-24 (|C| + sum |a b|).  A chunk of 64
values of K is four tensor-core sums, truncated (at most 2^-23 each, so
8 x 2^-24), its two accumulators are added (2^-24), each of the K / 64 chunks
is one rounded addition (2^-24 each), the update of C one FMA (2^-24) and the
three products left out are below 2^-26 each."""

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

# (N, K, M, trans1, trans2): remainders of the 128 x 128 tiles and of the
# 64-wide blocks of K, and the smallest sizes that take this path.
SHAPES = [(64, 128, 16384, 0, 0), (129, 130, 8200, 1, 0), (8200, 191, 64, 0, 1), (300, 513, 1000, 1, 1),
          (1025, 200, 700, 0, 0), (700, 1500, 257, 1, 0)]


def _update(pkg, cuda, A, B, C, ta, tb, alpha):
    import torch

    Ad = to_dev(A.T if ta else A, np.float32, cuda, ld=(A.shape[1] if ta else A.shape[0]) + 1)
    Bd = to_dev(B.T if tb else B, np.float32, cuda, ld=(B.shape[1] if tb else B.shape[0]) + 3)
    Cd = to_dev(C, np.float32, cuda, ld=C.shape[0] + 5)
    pkg.matmul_(Cd, Ad.T if ta else Ad, Bd.T if tb else Bd, alpha)
    torch.cuda.synchronize()
    pkg.device_status(Cd)
    return to_host(Cd)


@pytest.mark.parametrize("values", ["normal", "positive", "graded"])
def test_f32_update(pkg, cuda, values):
    rng = np.random.default_rng(3)
    make = {"normal": lambda s: rng.standard_normal(s), "positive": lambda s: rng.random(s),
            "graded": lambda s: rng.standard_normal(s) * np.exp2(rng.integers(-20, 21, s))}[values]
    for N, K, M, ta, tb in SHAPES:
        A, B, C = (make(s).astype(np.float32) for s in ((N, K), (K, M), (N, M)))
        got = _update(pkg, cuda, A, B, C, ta, tb, -1.0)
        A, B, C = (X.astype(np.float64) for X in (A, B, C))
        bound = (12 + -(-K // 64)) * 2.0 ** -24 * (np.abs(C) + np.abs(A) @ np.abs(B))
        assert (np.abs(got - (C - A @ B)) <= bound).all(), (N, K, M, ta, tb)


def test_f32_update_special_values(pkg, cuda):
    """Inf, NaN, overflow and rows near the ends of Float32's range: the same
    infinities and NaNs as the plain product, and full precision elsewhere."""
    rng = np.random.default_rng(4)
    N, K, M = 300, 256, 2000
    A, B = (rng.integers(-8, 9, s).astype(np.float32) for s in ((N, K), (K, M)))
    C = rng.standard_normal((N, M)).astype(np.float32)
    A[7, 3], A[9, 0], A[130, 255] = np.inf, -np.inf, np.nan
    A[20, :] = rng.standard_normal(K) * 2.0 ** -120
    A[21, :] = rng.standard_normal(K) * 2.0 ** -140
    A[22, :] = 2.0 ** 125 * np.sign(A[22, :])
    A[23, :] = np.float32(3.4028234e38) * (np.arange(K) == 5)
    B[:, 1500] = rng.standard_normal(K) * 2.0 ** 100
    B[5, 1999] = np.inf
    B[:, 3] = 0.0
    with np.errstate(all="ignore"):
        got = _update(pkg, cuda, A, B, C, 0, 0, 1.0)
        P = A.astype(np.float64) @ B.astype(np.float64)
        ref = (P + C).astype(np.float32).astype(np.float64)
        S = np.abs(A.astype(np.float64)) @ np.abs(B.astype(np.float64)) + np.abs(C)
    big = np.abs(S) * 1.001 >= np.finfo(np.float32).max  # partial sums may overflow in any order
    assert np.array_equal(np.isnan(got)[~big], np.isnan(ref)[~big])
    rows = [7, 9, 130]
    assert np.array_equal(np.isnan(got[rows]), np.isnan(ref[rows]))
    assert np.array_equal(got[[7, 9]][np.isinf(ref[[7, 9]])], ref[[7, 9]][np.isinf(ref[[7, 9]])])
    ok = np.isfinite(ref) & ~big
    assert (np.abs(got - ref)[ok] <= ((K + 12) * 2.0 ** -24 * S + 2.0 ** -140)[ok]).all()


def test_f32_update_under_capture(pkg, cuda):
    """A captured solve takes no scratch: it replays on new data."""
    import torch

    rng = np.random.default_rng(6)
    n, m = 600, 1500
    A = np.tril(rng.standard_normal((n, n)) / np.sqrt(n), -1) + np.diag(2 + np.abs(rng.standard_normal(n)))
    B = rng.uniform(-1, 1, (n, m))
    Ad, B0 = to_dev(A, np.float32, cuda), to_dev(B, np.float32, cuda)
    X, Y = B0.T.clone().T, B0.T.clone().T
    pkg.unified_rectrxm_("L", "L", "N", 1.0, "S", Ad, X, native=True)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        pkg.unified_rectrxm_("L", "L", "N", 1.0, "S", Ad, Y, native=True)
    graph.replay()
    torch.cuda.synchronize()
    assert np.linalg.norm(to_host(X) - to_host(Y)) < 1e-5 * np.linalg.norm(to_host(X))


def _cdev(X, cuda, pad):
    import torch

    buf = torch.zeros((X.shape[1], X.shape[0] + pad), dtype=torch.complex64, device=cuda)
    buf[:, : X.shape[0]] = torch.from_numpy(np.ascontiguousarray(X.T))
    return buf.T[: X.shape[0]]


@pytest.mark.parametrize("form", ["NN", "TN", "CN", "NC", "TT", "CC"])
def test_c32_update(pkg, cuda, form):
    """ComplexF32 on the same kernel (2 M x 2 K real operands): every
    transposed and conjugated form, bound as above per real component with
    sums of 2 K products."""
    import torch

    rng = np.random.default_rng(8)
    for N, K, M in ((70, 130, 4000), (333, 129, 1000), (1001, 600, 130)):
        A, B, C = ((rng.standard_normal(s) + 1j * rng.standard_normal(s)).astype(np.complex64)
                   for s in ((N, K), (K, M), (N, M)))
        op = {"N": lambda X: X, "T": lambda X: X.T, "C": lambda X: X.conj().T}
        Ad, Bd, Cd = _cdev(op[form[0]](A), cuda, 1), _cdev(op[form[1]](B), cuda, 2), _cdev(C, cuda, 0)
        view = {"N": lambda X: X, "T": lambda X: X.T, "C": lambda X: X.T.conj()}
        pkg.matmul_(Cd, view[form[0]](Ad), view[form[1]](Bd), -1.0)
        torch.cuda.synchronize()
        got = Cd.cpu().numpy().astype(np.complex128)
        A, B, C = (X.astype(np.complex128) for X in (A, B, C))
        ref = C - A @ B
        ar, ai, br, bi = np.abs(A.real), np.abs(A.imag), np.abs(B.real), np.abs(B.imag)
        u = (12 + -(-2 * K // 64)) * 2.0 ** -24
        assert (np.abs((got - ref).real) <= u * (np.abs(C.real) + ar @ br + ai @ bi)).all(), (form, N, K, M)
        assert (np.abs((got - ref).imag) <= u * (np.abs(C.imag) + ar @ bi + ai @ br)).all(), (form, N, K, M)


def test_c32_update_not_finite(pkg, cuda):
    """An Inf or NaN component reaches exactly the outputs its products do."""
    import torch

    rng = np.random.default_rng(9)
    N, K, M = 200, 200, 2000
    A, B = ((rng.integers(-4, 5, s) + 1j * rng.integers(-4, 5, s)).astype(np.complex64) for s in ((N, K), (K, M)))
    A[3, 4] = complex(np.inf, 1.0)
    B[6, 77] = complex(2.0, np.nan)
    Cd = _cdev(np.zeros((N, M), dtype=np.complex64), cuda, 0)
    pkg.matmul_(Cd, _cdev(A, cuda, 0), _cdev(B, cuda, 0), 1.0)
    torch.cuda.synchronize()
    got = Cd.cpu().numpy()
    with np.errstate(all="ignore"):
        Ar, Ai, Br, Bi = (np.nan_to_num(X.astype(np.float64), nan=np.nan, posinf=np.inf) for X in
                          (A.real, A.imag, B.real, B.imag))
        re, im = Ar @ Br - Ai @ Bi, Ar @ Bi + Ai @ Br
    keep = np.ones((N, M), dtype=bool)
    keep[3, :] = False
    keep[:, 77] = False
    assert np.array_equal(got.real[keep], re[keep].astype(np.float32))
    assert np.array_equal(got.imag[keep], im[keep].astype(np.float32))
    rest = [j for j in range(M) if j != 77]
    assert np.array_equal(np.isnan(got.real[3, rest]), np.isnan(re[3, rest]))
    assert np.array_equal(np.isinf(got.real[3, rest]), np.isinf(re[3, rest]))
    assert np.isnan(got.imag[:, 77]).all() and np.isnan(got.real[:, 77]).all()


@pytest.mark.parametrize("shape", [(64, 300, 2000), (100, 200, 1601), (129, 140, 2400), (128, 256, 4900),
                                   (257, 130, 3100), (257, 128, 6500)])
@pytest.mark.parametrize("special", [False, True])
def test_f32_update_tile_widths(pkg, cuda, shape, special):
    """Tiles of 32, 64 and 128 columns (chosen by how many fill the GPU), from
    the smallest sizes that take this path, with remainders; the tolerance of
    this file, and with Inf and NaN the plain product's pattern of them."""
    N, K, M = shape
    rng = np.random.default_rng(N + M)
    A, B, C = (rng.standard_normal(s).astype(np.float32) for s in ((N, K), (K, M), (N, M)))
    if special:
        A[3, 5], A[N - 1, K - 1], B[1, M - 1], B[K - 1, 40] = np.inf, np.nan, -np.inf, np.nan
    for ta, tb in ((0, 0), (1, 1)):
        got = _update(pkg, cuda, A, B, C, ta, tb, -1.0)
        with np.errstate(all="ignore"):
            A8, B8, C8 = (X.astype(np.float64) for X in (A, B, C))
            ref = C8 - A8 @ B8
            bound = (12 + -(-K // 64)) * 2.0 ** -24 * (np.abs(C8) + np.abs(A8) @ np.abs(B8))
        ok = np.isfinite(ref)
        assert np.array_equal(np.isnan(got), np.isnan(ref)) and np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)])
        assert (np.abs(got - ref)[ok] <= bound[ok]).all(), (shape, ta, tb)
