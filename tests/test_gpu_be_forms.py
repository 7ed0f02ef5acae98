"""The forms of the backward-Euler solve beside the on-chip one: each grid here is
one that the dispatch sends to them.  Reference: the launch per phase
(PIRO_BE_PERSISTENT=0), both solved to a 1e-8 FP64 residual, so that 1e-6 of
max |u| bounds the difference (see the on-chip solve's test)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _solver(n, monkeypatch, env="1"):
    import torch
    from piro_b200 import ops
    N, dt = n[0] * n[1] * n[2], 5.0
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    alpha = torch.exp(torch.randn(N, generator=g, device="cuda").clamp(-2, 2))
    b = torch.rand(N, generator=g, device="cuda")
    L = ops.csr_laplacian(*n, 3, 1.0)
    ops.csr_rowscale(L[0], L[2], alpha)
    A = ops.csrgeam2(N, ops.csr_identity(N), -dt, L)
    monkeypatch.setenv("PIRO_BE_PERSISTENT", env)
    return ops.BESolver(*n, A, alpha, stencil=(dt, 1.0)), b


def _solve(s, b):
    import torch
    x = torch.full_like(b, float("nan"))
    for _ in range(2):
        info = s.solve(b, x, rtol=1e-8)
        assert info.status == 0 and info.rel_residual <= 1e-8
    s.close()
    return x.cpu().numpy().astype(np.float64), info


@pytest.mark.parametrize("n,env,form", [
    ((132, 132, 132), "1", "shared"),   # too large for the chip, not for p, d, q in shared memory
    ((141, 139, 137), "1", "global"),
    ((40, 32, 24), "1", "chip"),
    ((40, 32, 24), "g", "global"),
])
def test_plain_forms(cuda, n, env, form, monkeypatch):
    s, b = _solver(n, monkeypatch, env)
    assert s.forms[0] == form
    got, _ = _solve(s, b)
    s, _ = _solver(n, monkeypatch, "0")
    assert s.forms == ("launches", "launches")
    want, _ = _solve(s, b)
    assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()


@pytest.mark.parametrize("n,env,form", [
    ((128, 126, 127), "1", "shared"),   # seven groups per thread, float4 width
    ((141, 139, 137), "1", "global"),
    ((40, 32, 24), "g", "global"),
    ((40, 32, 24), "1", "chip"),
])
@pytest.mark.parametrize("with_net", [True, False])
def test_flexible_forms(cuda, n, env, form, with_net, monkeypatch):
    from piro_b200 import ops
    got = {}
    for e in (env, "0"):
        s, b = _solver(n, monkeypatch, e)
        assert s.forms[1] == (form if e == env else "launches")
        net = ops.PCNet(seed=3) if with_net else None
        s.set_preconditioner(net) if with_net else s.set_preconditioner(flexible_jacobi=True)
        got[e], info = _solve(s, b)
        assert info.fallbacks == 0
    assert np.abs(got[env] - got["0"]).max() <= 1e-6 * np.abs(got["0"]).max()


@pytest.mark.parametrize("n", [(40, 32, 24), (128, 126, 127)])  # alpha on chip, alpha streamed
def test_bytes_of_the_on_chip_solve(cuda, n, monkeypatch):
    s, b = _solver(n, monkeypatch)
    import torch
    x = torch.empty_like(b)
    s.solve(b, x)
    s.kernel_stats(reset=True)
    info = s.solve(b, x)
    N = b.numel()
    want = 24 + 32 * info.outer_iterations + (4 + 4 * info.inner_iterations if n[0] == 128 else 0)
    assert s.persistent_bytes() == want * N
    s.close()
