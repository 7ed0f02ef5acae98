"""The Jacobi iterations of a learned sweep on chip, which go on from the network
iteration's direction or (flexible Jacobi) start without one, on runs of one to
seven groups of cells per thread, odd widths, one CTA and many.  References: the
plain solve (the same tolerance: 1e-6 of max |u|, see the on-chip solve's test)
and the launch per phase (PIRO_BE_PERSISTENT=0), whose iterations they are up
to rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [(3, 3, 3), (6, 3, 50), (10, 17, 19), (33, 47, 29), (72, 65, 81), (92, 91, 93), (113, 112, 111),
                               (125, 127, 126)])
@pytest.mark.parametrize("with_net", [True, False])
def test_fcg_on_chip(cuda, n, with_net, monkeypatch):
    import torch
    from piro_b200 import learned, ops
    nx, ny, nz = n
    N = nx * ny * nz
    rng = np.random.default_rng(nx + 1000 * ny + nz)
    alpha = np.exp(np.clip(rng.standard_normal(N), -2, 2)).astype(np.float32)
    dt = np.float32(20.0 / (6.0 * alpha.max()))
    b_t = torch.from_numpy(rng.random(N, dtype=np.float32)).cuda()
    a_t = torch.from_numpy(alpha).cuda()
    L = ops.csr_laplacian(nx, ny, nz, 3, 1.0)
    ops.csr_rowscale(L[0], L[2], a_t)
    A = ops.csrgeam2(N, ops.csr_identity(N), -float(dt), L)
    net = ops.PCNet(seed=3)
    xs, its = [], []
    for kind in ("plain", "chip", "launches"):
        monkeypatch.setenv("PIRO_BE_PERSISTENT", "0" if kind == "launches" else "1")
        s = ops.BESolver(nx, ny, nz, A, a_t, stencil=(float(dt), 1.0))
        if kind != "plain":
            s.set_preconditioner(net) if with_net else s.set_preconditioner(flexible_jacobi=True)
        x = torch.empty_like(b_t)
        for _ in range(2):
            info = s.solve(b_t, x, rtol=1e-8)
            assert info.status == 0 and info.rel_residual <= 1e-8
        xs.append(x.cpu().numpy().astype(np.float64))
        its.append((info.inner_iterations, info.outer_iterations, info.fallbacks))
        s.close()
    net.close()
    # a sweep may end an iteration earlier or later by rounding
    assert its[1][1:] == its[2][1:] and abs(its[1][0] - its[2][0]) <= its[1][1], its
    for x in xs[1:]:
        assert np.abs(x - xs[0]).max() <= 1e-6 * np.abs(xs[0]).max()


def test_fcg_on_chip_wait_gives_up(cuda):
    import torch
    from piro_b200 import ops
    from piro_b200._lib import lib
    n = (40, 32, 25)
    N = n[0] * n[1] * n[2]
    a_t = torch.rand(N, device="cuda") + 0.5
    b_t = torch.rand(N, device="cuda")
    dt = 3.0
    L = ops.csr_laplacian(*n, 3, 1.0)
    ops.csr_rowscale(L[0], L[2], a_t)
    A = ops.csrgeam2(N, ops.csr_identity(N), -dt, L)
    s = ops.BESolver(*n, A, a_t, stencil=(dt, 1.0))
    s.set_preconditioner(flexible_jacobi=True)
    want, x = torch.empty_like(b_t), torch.empty_like(b_t)
    assert s.solve(b_t, want, rtol=1e-8).status == 0
    assert lib().piro_set_wait_limit(0) == 0
    try:
        info = s.solve(b_t, x, rtol=1e-8, strict=False)
        assert info.status == 6  # PIRO_ERR_CUDA
    finally:
        lib().piro_set_wait_limit(-1)
    for _ in range(2):
        assert s.solve(b_t, x, rtol=1e-8).status == 0
        assert torch.equal(x, want)
    s.close()
