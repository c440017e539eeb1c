"""The error of a batch solved one group per CTA against extended precision,
beside that of the same systems solved by the node queue, whose updates are
separate sums: no larger (2 % for the chance of the draw), on long rows, in
both types."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("values", ["normal", "positive"])
def test_whole_groups_round_no_worse(pkg, cuda, dtype, values):
    import torch

    from nextla_gb300 import batched

    dt = getattr(torch, dtype)
    count, n, m = 640, 768, 8
    A, B, systems = batched.make_batch([n] * count, [m] * count, dt, cuda, seed=6)
    if values == "positive":  # off-diagonals and right-hand sides of one sign: sums of like terms
        T = A.view(count, n, n)
        T.copy_(torch.where(torch.eye(n, device=cuda, dtype=torch.bool), T, T.abs().neg() / n ** 0.5))
        B.abs_()
    whole = batched.BatchPlan(dt, "L", "N", systems)
    assert whole.info()[0] == count
    X = B.clone()
    whole.solve(1.0, A, X)
    Y = B.clone()
    for k in range(0, count, 16):
        plan = batched.BatchPlan(dt, "L", "N", systems[k:k + 16])
        assert plan.info()[0] > 16
        plan.solve(1.0, A, Y)
        plan.close()
    torch.cuda.synchronize()
    whole.close()
    err = {"whole": 0.0, "queue": 0.0}
    for k in range(0, count, 80):
        ao, bo = systems[k][2], systems[k][4]
        T = A[ao:ao + n * n].view(n, n).T.cpu().numpy().astype(np.longdouble)
        want = B[bo:bo + n * m].view(m, n).T.cpu().numpy().astype(np.longdouble)
        for j in range(n):
            want[j] /= T[j, j]
            want[j + 1:] -= np.outer(T[j + 1:, j], want[j])
        for name, Z in (("whole", X), ("queue", Y)):
            got = Z[bo:bo + n * m].view(m, n).T.cpu().numpy().astype(np.longdouble)
            err[name] += float(np.sum((got - want) ** 2) / np.sum(want ** 2))
    assert err["whole"] <= 1.02 ** 2 * err["queue"], err
