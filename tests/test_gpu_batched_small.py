"""Which batches are solved one group per CTA: those whose longest group is no
longer than a CTA's share of the work on the whole GPU, and fewer groups than
CTAs when they are short.  A few large systems, equal ones above all, are not:
their updates spread over the CTAs as nodes of the queue."""

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["float32", "float64"])
@pytest.mark.parametrize("count,n,m", [(1, 1024, 64), (8, 1024, 64), (20, 1024, 16), (1, 1024, 1)])
def test_few_equal_systems_keep_the_node_queue(pkg, cuda, dtype, count, n, m):
    import torch

    from nextla_gb300 import batched

    dt = getattr(torch, dtype)
    A, B, systems = batched.make_batch([n] * count, [m] * count, dt, cuda, seed=count)
    plan = batched.BatchPlan(dt, "L", "N", systems)
    leaves = -(-n // 64)
    assert plan.info()[0] >= count * (leaves + leaves // 2), plan.info()
    X = B.clone()
    plan.solve(0.5, A, X)
    torch.cuda.synchronize()
    plan.close()
    T = A.view(count, n, n).transpose(1, 2).double().tril()
    want = torch.linalg.solve_triangular(T, 0.5 * B.view(count, m, n).transpose(1, 2).double(), upper=False)
    got = X.view(count, m, n).transpose(1, 2).double()
    assert float((got - want).norm() / want.norm()) < (1e-5 if dtype == "float32" else 1e-13)


@pytest.mark.parametrize("count,n", [(2000, 96), (30, 200), (150, 380), (1, 64)])
def test_many_or_short_systems_go_whole(pkg, cuda, count, n):
    import torch

    from nextla_gb300 import batched

    _, _, systems = batched.make_batch([n] * count, [16] * count, torch.float32, cuda, seed=1)
    plan = batched.BatchPlan(torch.float32, "L", "N", systems)
    assert plan.info()[0] == count
    plan.close()
