"""The CUDA-core update at sizes that select each of its tilings and leave
remainders in every dimension, against the product in Float64.

Tolerances (relative Frobenius error of C + alpha A B): Float64 1e-14 and
Float32 1e-5 as in the reference's tests, Float16 2^-10 (Float32 sums, one
rounding of at most 2^-11)."""

import numpy as np
import pytest

from gpu_util import to_dev, to_host

pytestmark = pytest.mark.gpu

TOL = {np.float64: 1e-14, np.float32: 1e-5, np.float16: 2.0 ** -10}
# (N, K, M): one tile and less, 32 x 16, 32 x 32, 64 x 64 and 128 x 128 tiles
SHAPES = [(1, 1, 1), (7, 3, 17), (33, 17, 15), (250, 63, 31), (257, 129, 255), (700, 33, 1100), (1500, 40, 1300),
          (100, 50, 5000)]


@pytest.mark.parametrize("dtype", [np.float64, np.float32, np.float16])
def test_update_tilings(pkg, oracle, cuda, dtype):
    import torch

    rng = np.random.default_rng(5)
    for k, (N, K, M) in enumerate(SHAPES):
        ta, tb = k & 1, (k >> 1) & 1
        A, B, C = (rng.uniform(-1, 1, s).astype(dtype) for s in ((N, K), (K, M), (N, M)))
        Ad = to_dev(A.T if ta else A, dtype, cuda, ld=(K if ta else N) + 1)
        Bd = to_dev(B.T if tb else B, dtype, cuda, ld=(M if tb else K) + 2)
        Cd = to_dev(C, dtype, cuda, ld=N + 3)
        pkg.matmul_(Cd, Ad.T if ta else Ad, Bd.T if tb else Bd, -1.0)
        torch.cuda.synchronize()
        ref = C.astype(np.float64) - A.astype(np.float64) @ B.astype(np.float64)
        assert oracle.rel_err(to_host(Cd), ref) < TOL[dtype], (N, K, M)
