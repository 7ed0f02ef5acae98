"""A breakdown in the first sweep of a backward-Euler solve: the solution so far
is the start, b, not what the solver's FP64 vector held before.

A negative dt makes A = I - dt alpha L indefinite, -D^-1 A having mostly positive
eigenvalues, so that <p, S p> < 0 in the first iteration for a rough b."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["1", "g"])  # on chip, and the launch with grid barriers
@pytest.mark.parametrize("n", [(24, 20, 22), (29, 27, 31)])
def test_first_sweep_breakdown_returns_b(cuda, n, variant, monkeypatch):
    import torch
    from piro_b200 import ops
    monkeypatch.setenv("PIRO_BE_PERSISTENT", variant)
    N, dt = n[0] * n[1] * n[2], -5.0
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    alpha = torch.rand(N, generator=g, device="cuda") + 0.5
    L = ops.csr_laplacian(*n, 3, 1.0)
    ops.csr_rowscale(L[0], L[2], alpha)
    A = ops.csrgeam2(N, ops.csr_identity(N), -dt, L)
    s = ops.BESolver(*n, A, alpha, stencil=(dt, 1.0))
    assert s.persistent_variant == ("resident" if variant == "1" else "global")
    for _ in range(2):  # the second solve finds the first one's vectors
        b = torch.rand(N, generator=g, device="cuda") - 0.5
        x = torch.full((N,), float("nan"), device="cuda")
        info = s.solve(b, x, rtol=1e-8, strict=False)
        assert info.status != 0 and info.outer_iterations == 1 and np.isfinite(info.rel_residual)
        assert torch.equal(x, b)
    s.close()
