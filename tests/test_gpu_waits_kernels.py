"""The wait limit (nla_set_wait_limit_ns) holds for the waits of the
tensor-core kernels of every translation unit: Float32 and ComplexF32 updates,
Float16 updates and the exact updates of a mixed solve.  With the limit at 1 ns
ordinary calls, whose waits would all complete, give up and report
NLA_ERR_TIMEOUT; with the default limit the next call gives the bits it gave
before.

The leaf products and pairs have the limit too, but a wait of theirs lasts a
few microseconds, less than one try of the hardware may wait by itself, so no
limit makes them give up on an ordinary call."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _make(rng, r, c, dev, dtype):
    import torch

    X = rng.uniform(-1, 1, (c, r))
    if dtype.is_complex:
        X = X + 1j * rng.uniform(-1, 1, (c, r))
    return torch.tensor(X, device=dev).to(dtype).T


def _update(dtype, N, K, M):
    def build(pkg, cuda, rng):
        import torch

        dt = getattr(torch, dtype)
        A, B, C = _make(rng, N, K, cuda, dt), _make(rng, K, M, cuda, dt), _make(rng, N, M, cuda, dt)

        def run():
            X = C.T.clone().T
            pkg.matmul_(X, A, B, -1.0)
            return X

        return run

    return build


def _solve(side, n, m):
    def build(pkg, cuda, rng):
        import torch

        A = _make(rng, n, n, cuda, torch.float64).div(n ** 0.5)
        A.diagonal().abs_().add_(2.0)
        B = _make(rng, *((n, m) if side == "L" else (m, n)), cuda, torch.float64)

        def run():
            X = B.T.clone().T
            pkg.unified_rectrxm_mixed_(side, "L", "N", 1.0, "S", A, X, split_terms=7, sweeps=0, cutoff=64)
            return X

        return run

    return build


CALLS = {"float32 update": _update("float32", 640, 700, 900), "complex64 update": _update("complex64", 300, 400, 900),
         "float32 wide update": _update("float32", 2000, 700, 3000), "float16 update": _update("float16", 640, 700, 900),
         "mixed solve": _solve("L", 700, 900), "mixed solve R": _solve("R", 700, 900)}


@pytest.mark.parametrize("call", sorted(CALLS))
def test_limit_reaches_every_kernel(pkg, lib, cuda, call):
    import torch

    from nextla_gb300 import _lib

    run = CALLS[call](pkg, cuda, np.random.default_rng(len(call)))
    ref = run()
    pkg.device_status(ref)
    try:
        _lib.check(lib.nla_set_wait_limit_ns(1))
        run()
        with pytest.raises(_lib.NLAError) as err:
            pkg.device_status()
        assert err.value.code == _lib.NLA_ERR_TIMEOUT
    finally:
        _lib.check(lib.nla_set_wait_limit_ns(0))
    pkg.device_status()
    for _ in range(2):
        again = run()
        pkg.device_status(again)
        assert torch.equal(torch.view_as_real(again) if again.is_complex() else again,
                           torch.view_as_real(ref) if ref.is_complex() else ref)
