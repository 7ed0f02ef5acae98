"""piro_csr_fe_run_bc against its steps one by one (piro_csr_fe_step_bc, itself
bit-exact with the oracle): the one-cluster form at the edges of its splits
(one CTA, one and two rows per thread, uneven last CTA, the largest grid it
takes and the first it does not), odd and even step counts, rows longer than
the registers hold, a bandwidth that reaches every CTA, and no face values.
Same arithmetic in the same order: bit for bit."""
import numpy as np
import pytest

from conftest import f32_bits_equal

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps", [((3, 3, 3), 1), ((4, 3, 5), 2), ((10, 10, 10), 7), ((11, 10, 10), 4),
                                     ((16, 16, 16), 3), ((26, 25, 25), 5), ((32, 32, 32), 6), ((33, 32, 31), 6),
                                     ((40, 33, 30), 3), ((32, 32, 33), 2), ((257, 5, 24), 5)])
@pytest.mark.parametrize("kind", ["heat", "upwind", "wide", "nobc"])
def test_run_equals_steps(cuda, n, steps, kind):
    import torch
    from piro_b200 import ops
    nx, ny, nz = n
    N = nx * ny * nz
    g = torch.Generator(device="cuda")
    g.manual_seed(N + steps)
    if kind == "upwind":
        v = torch.randn(3 * N, generator=g, device="cuda")
        A = ops.csrgeam3(N, *[ops.csr_gradient(nx, ny, nz, 1, a, 2.0) for a in range(3)], v)
    elif kind == "wide":  # rows of 3 to 12 entries at any column
        rng = np.random.default_rng(N)
        cnt = rng.integers(3, 13, N)
        rp = np.concatenate([[0], np.cumsum(cnt)]).astype(np.int32)
        A = tuple(torch.from_numpy(a).cuda() for a in (rp, rng.integers(0, N, rp[-1]).astype(np.int32),
                                                       rng.standard_normal(rp[-1]).astype(np.float32)))
    else:
        A = ops.csr_laplacian(nx, ny, nz, 3, 1.0)
        ops.csr_rowscale(A[0], A[2], torch.rand(N, generator=g, device="cuda"))
    u0 = torch.randn(N, generator=g, device="cuda")
    bc = None if kind == "nobc" else u0
    bufs = [torch.full_like(u0, float("nan")) for _ in range(2)]
    got = ops.csr_fe_run_bc(nx, ny, nz, A, 0.03, u0, bc, *bufs, steps)
    assert got.data_ptr() == bufs[steps & 1].data_ptr()
    u, out = u0.clone(), torch.empty_like(u0)
    for _ in range(steps):
        ops.csr_fe_step_bc(nx, ny, nz, A, 0.03, u, bc, out)
        u, out = out, u
    assert f32_bits_equal(got.cpu().numpy(), u.cpu().numpy())


@pytest.mark.parametrize("n", [(12, 10, 9), (40, 36, 33)])  # one cluster, a launch per step
def test_run_takes_what_the_step_loop_took(cuda, n):
    """Slices and step counts of zero and below; a permuted field and a fraction of a
    step refused; the face values kept for single steps."""
    import torch
    from piro_b200 import fe
    N = n[0] * n[1] * n[2]
    run = fe.FeRunner(*n, torch.full((N,), 0.01, device="cuda"), 3.0)
    wide = torch.rand(2 * N, device="cuda")
    u = wide[::2].clone()
    want = run.run(u, 3, graph=True)
    assert torch.equal(run.run(wide[::2], 3), want)
    for steps in (0, -2):
        got = run.run(u, steps)
        assert torch.equal(got, u) and got.data_ptr() != u.data_ptr()
    with pytest.raises(TypeError):
        run.run(u, 2.0)
    with pytest.raises(ValueError):
        run.run(u.reshape(n).permute(2, 1, 0), 3)
    v = torch.rand_like(u)
    out = run.run(v, 1)
    assert torch.equal(run.memD, v)
    one = torch.empty_like(v)
    run._step(v, one)
    assert torch.equal(one, out)
