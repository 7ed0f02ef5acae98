"""The on-chip backward-Euler solve (resident_cg.cuh) at the edges of its
splits: one CTA and many, one to seven groups of four cells per thread, lines
of one to four cells past a group, strips that cut the planes unevenly, grids
one cell thick, and nonzero boundary values (PIRO's 10.0 entries).

The reference is the oracle's FP64 CG to 1e-13.  Tolerance: the field is
rounded to FP32 (6e-8 of max |u|) and solved to ||b - A x|| <= 1e-8 ||b||; A's
smallest eigenvalue is at least 1 (A = I - dt alpha L), so the error's 2-norm
is at most 1e-8 ||b|| sqrt(max alpha / min alpha), and 1e-6 of max |u| covers
both with the diffusivities drawn here (ratio below 400)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.mark.parametrize("n,boundary", [
    ((3, 3, 3), True),        # one unknown
    ((3, 40, 5), False),      # one cell per line
    ((6, 3, 50), True),       # one line per plane, a full group
    ((5, 9, 3), True),        # one plane
    ((67, 4, 6), False),      # 65 cells: one past a group
    ((10, 17, 19), True),     # a few CTAs, uneven strips
    ((131, 12, 9), False),    # lines longer than a warp's groups
    ((33, 47, 29), True),     # one group per thread
    ((72, 65, 81), False),    # two
    ((92, 91, 93), False),    # three
    ((113, 112, 111), False),  # five
    ((127, 126, 129), True),  # seven
    ((190, 20, 130), False),  # few long lines
])
def test_resident_solve_matches_fp64(cuda, oracle, n, boundary):
    import torch
    from piro_b200 import ops
    nx, ny, nz = n
    N = nx * ny * nz
    rng = np.random.default_rng(nx * 10007 + ny * 101 + nz)
    alpha = np.exp(np.clip(rng.standard_normal(N), -3, 3)).astype(np.float32)
    dt = np.float32(20.0 / (6.0 * alpha.max()))
    b = rng.random(N, dtype=np.float32)
    inter = np.zeros((nz, ny, nx), bool)
    inter[1:-1, 1:-1, 1:-1] = True
    if not boundary:
        b[~inter.ravel()] = 0.0
    L = oracle.laplacian(nx, ny, nz, 3, np.float32(1.0))
    Ls = (L[0], L[1], oracle.csr_rowscale(N, L[0], L[2], alpha))
    I = (np.arange(N + 1, dtype=np.int32), np.arange(N, dtype=np.int32), np.ones(N, np.float32))
    A = oracle.csrgeam2(N, I, np.float32(-dt), Ls)
    u64, _, rel = oracle.be_cg_f64(nx, ny, nz, A, alpha, b, rtol=1e-13)
    assert rel <= 1e-12
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
    s = ops.BESolver(nx, ny, nz, tuple(dev(a) for a in A), dev(alpha), stencil=(dt, 1.0))
    assert s.persistent_variant == "resident"
    bd, x = dev(b), torch.full((N,), float("nan"), device="cuda")
    first = None
    for _ in range(2):  # the second solve goes on with the rounds of the first
        info = s.solve(bd, x, rtol=1e-8)
        assert info.status == 0 and info.rel_residual <= 1e-8
        got = x.cpu().numpy()
        assert np.array_equal(got[~inter.ravel()], b[~inter.ravel()])
        assert np.abs(got - u64).max() <= TOL * np.abs(u64).max()
        assert first is None or np.array_equal(first, got)  # the same bits on every run
        first = got
    s.close()
