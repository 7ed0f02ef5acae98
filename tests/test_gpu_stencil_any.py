"""The matrix-free step in groups of four cells for widths that are no multiple
of four: every remainder of nx and nx ny mod 4, groups over two lines and two
planes, array lengths with a rest, the narrowest width (8; 7 takes the
z-marching form), pointers off the 16-byte grid (the z-marching form): bit for
bit the update's operations in float32, in their order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


def _ref(n, c, dt, a, u):
    nx, ny, nz = n
    U, A, out = u.reshape(nz, ny, nx), a.reshape(nz, ny, nx), u.reshape(nz, ny, nx).copy()
    i = (slice(1, -1),) * 3
    C = U[i]
    c2 = f32(2) * C
    lx = ((U[1:-1, 1:-1, 2:] + U[1:-1, 1:-1, :-2]) - c2) * f32(c[0])
    ly = ((U[1:-1, 2:, 1:-1] + U[1:-1, :-2, 1:-1]) - c2) * f32(c[1])
    lz = ((U[2:, 1:-1, 1:-1] + U[:-2, 1:-1, 1:-1]) - c2) * f32(c[2])
    out[i] = C + f32(dt) * (A[i] * ((lx + ly) + lz))
    return out.reshape(-1)


@pytest.mark.parametrize("n", [(8, 3, 3), (7, 9, 5), (9, 3, 3), (9, 4, 5), (10, 3, 7), (10, 5, 4), (11, 3, 3), (11, 7, 6),
                               (13, 4, 3), (14, 11, 9), (15, 15, 15), (251, 17, 5), (33, 129, 7), (8, 5, 5)])
@pytest.mark.parametrize("with_alpha", [True, False])
@pytest.mark.parametrize("off", [0, 1])
def test_stencil_any_width(cuda, n, with_alpha, off):
    import torch
    from piro_b200 import ops
    N = n[0] * n[1] * n[2]
    rng = np.random.default_rng(N)
    u = rng.standard_normal(N).astype(f32)
    u[rng.integers(0, N, 3)] = [np.inf, -0.0, 1e-42]
    a = rng.random(N).astype(f32) if with_alpha else np.ones(N, f32)
    T = lambda v: torch.from_numpy(np.concatenate([np.zeros(off, f32), v])).cuda()[off:]  # noqa: E731
    out = torch.full((N + 8,), 7.0, device="cuda")
    c, dt = (3.0, 2.0, 0.7), 0.11
    ops.stencil_fe_step(*n, dt, T(u), out[off:off + N], T(a) if with_alpha else None, *c)
    got = out.cpu().numpy()
    with np.errstate(invalid="ignore"):
        want = _ref(n, c, dt, a, u)
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got[off:off + N]), nan)
    assert np.array_equal(got[off:off + N][~nan].view(np.uint32), want[~nan].view(np.uint32))
    assert (got[:off] == 7).all() and (got[off + N:] == 7).all()
