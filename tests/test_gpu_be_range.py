"""Fields far from 1 on widths whose dot products are taken term by term in FP64:
their FP32 products would vanish (8e-25 squared) or overflow (7e19 squared).

The solution is linear in b.  Scaling by a power of two is exact until single
entries of the vectors become denormal, which is below 1e-12 of their norms; so
the scaled solve has the unscaled one's status, and its field within the 1e-6 of
max |u| that a 1e-8 residual allows (see the on-chip solve's test)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(29, 27, 31), (87, 63, 75), (97, 95, 91), (117, 111, 113), (125, 127, 129)])
@pytest.mark.parametrize("flexible", [False, True])
@pytest.mark.parametrize("exponent", [-80, 66])
def test_scaled_field(cuda, n, flexible, exponent):
    import torch
    from piro_b200 import ops
    N, dt = n[0] * n[1] * n[2], 5.0
    assert N % 4
    g = torch.Generator(device="cuda")
    g.manual_seed(N)
    alpha = torch.rand(N, generator=g, device="cuda") + 0.5
    b = torch.rand(N, generator=g, device="cuda")
    L = ops.csr_laplacian(*n, 3, 1.0)
    ops.csr_rowscale(L[0], L[2], alpha)
    A = ops.csrgeam2(N, ops.csr_identity(N), -dt, L)
    s = ops.BESolver(*n, A, alpha, stencil=(dt, 1.0))
    assert s.persistent_variant == "resident"
    if flexible:
        s.set_preconditioner(flexible_jacobi=True)
    x, y = torch.empty_like(b), torch.empty_like(b)
    assert s.solve(b, x, rtol=1e-8).status == 0
    info = s.solve(b * 2.0 ** exponent, y, rtol=1e-8, strict=False)
    assert info.status == 0 and info.rel_residual <= 1e-8 and info.fallbacks == 0
    diff = (y.double() * 2.0 ** -exponent - x.double()).abs().max()
    assert float(diff) <= 1e-6 * float(x.abs().max())
    s.close()


@pytest.mark.parametrize("grouped", [False, True])
def test_batch_member_of_small_alpha(cuda, grouped):
    """alpha 2^-40 of another member's with dt 2^40 of its: the operator is the same, and
    so is the field, bit for bit, at any size of the field."""
    import numpy as np
    from piro_b200 import ops
    n = np.array([20, 20, 33, 33], np.int32)
    f = 2.0 ** np.array([0, -40, 0, -40])
    alpha, dt = (0.01 * f).astype(np.float32), (830.0 / f).astype(np.float32)
    B = ops.Batch(n, alpha, dt, np.ones(4, np.int32))
    B.set_schedule(grouped, 2)
    rng = np.random.default_rng(5)
    u = np.zeros(B.total, np.float32)
    for k in (0, 2):
        v = rng.random(int(n[k]) ** 3, dtype=np.float32) * np.float32(2.0 ** 36)
        for q in (k, k + 1):
            u[int(B.offsets[q]):int(B.offsets[q]) + v.size] = v
    B.set_fields(u)
    B.step(1)
    info, got = B.member_info(), B.get_fields()
    assert np.all(info["status"] == 0) and np.all(info["rel"] <= 1e-8), info
    for k in (0, 2):
        assert np.array_equal(B.member(got, k), B.member(got, k + 1))
    B.close()
