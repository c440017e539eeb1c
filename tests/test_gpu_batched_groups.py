"""Batches solved one group per CTA (enough systems that no group is longer
than a CTA's share): every orientation, orders at the edges of the 64-row
blocks, right-hand sides at the edges of the column templates, leaf orders 16
to 64, against the same batch solved one system at a time by torch in Float64.

Tolerances: Float64 1e-13 and Float32 1e-5 over the whole batch, as for the
batches elsewhere."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [("float32", 1e-5), ("float64", 1e-13)])
@pytest.mark.parametrize("uplo,trans", [("L", "N"), ("U", "N"), ("L", "T"), ("U", "T")])
def test_whole_groups(pkg, cuda, dtype, tol, uplo, trans):
    import torch

    from nextla_gb300 import batched

    dt = getattr(torch, dtype)
    rng = np.random.default_rng(31)
    count = 2600
    n, m = rng.integers(1, 140, count), rng.integers(1, 131, count)
    n[:10] = [1, 16, 63, 64, 65, 127, 128, 129, 200, 300]
    m[:10] = [1, 16, 17, 32, 33, 64, 65, 128, 129, 130]
    A, B, systems = batched.make_batch(n, m, dt, cuda, seed=4, uplo=uplo)
    for cutoff in (None, [16, 32, 64, 16, 32, 64]):
        plan = batched.BatchPlan(dt, uplo, trans, systems, cutoff=cutoff)
        groups = int(sum(-(-int(v) // 64) for v in m))
        assert plan.info()[0] == groups  # the queue holds groups, not recursion nodes
        X = B.clone()
        plan.solve(-0.5, A, X)
        torch.cuda.synchronize()
        plan.close()
        err = ref = 0.0
        for k in list(range(10)) + list(range(10, count, 97)):
            nk, mk, ao, _, bo, _ = systems[k]
            T = A[ao:ao + nk * nk].view(nk, nk).T.double()
            T = T.tril() if uplo == "L" else T.triu()
            T = T.T if trans == "T" else T
            R = -0.5 * B[bo:bo + nk * mk].view(mk, nk).T.double()
            want = torch.linalg.solve_triangular(T.contiguous(), R, upper=(uplo == "U") != (trans == "T"))
            got = X[bo:bo + nk * mk].view(mk, nk).T.double()
            err += float((got - want).square().sum())
            ref += float(want.square().sum())
        assert (err / ref) ** 0.5 < tol, (dtype, uplo, trans, cutoff)
