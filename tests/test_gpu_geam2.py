"""csrgeam2 (A + beta B) and the row scale on rows that the fast forms hand to
the general ones and back: empty rows, repeated and unsorted columns, 8 and 9
entries (the register limit), chunks longer than the stages, a last chunk of
fewer than 32 rows.  The reference adds a row's entries in the order the
kernels state (A's, then B's, per column), in float32: bit for bit."""
import numpy as np
import pytest

from conftest import f32_bits_equal

pytestmark = pytest.mark.gpu


def _csr(rng, N, lens, ncol):
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    return rp, rng.integers(0, ncol, rp[-1]).astype(np.int32), rng.standard_normal(rp[-1]).astype(np.float32)


def _ref(N, A, beta, B):
    rp, cols, vals = [0], [], []
    for r in range(N):
        acc = {}
        for k in range(A[0][r], A[0][r + 1]):
            c = int(A[1][k])
            acc[c] = np.float32(acc[c] + A[2][k]) if c in acc else A[2][k]
        for k in range(B[0][r], B[0][r + 1]):
            c, v = int(B[1][k]), np.float32(np.float32(beta) * B[2][k])
            acc[c] = np.float32(acc[c] + v) if c in acc else v
        for c in sorted(acc):
            cols.append(c)
            vals.append(acc[c])
        rp.append(len(cols))
    return np.array(rp, np.int32), np.array(cols, np.int32), np.array(vals, np.float32)


@pytest.mark.parametrize("N,la,lb,ncol", [(1, (1, 2), (7, 8), 20), (31, (0, 2), (0, 8), 5), (33, (1, 2), (7, 8), 40),
                                          (500, (0, 5), (0, 5), 6), (1000, (0, 10), (0, 12), 30),
                                          (700, (8, 9), (0, 2), 50), (200, (20, 33), (20, 33), 1000)])
def test_geam2_and_rowscale(cuda, N, la, lb, ncol):
    import torch
    from piro_b200 import ops
    rng = np.random.default_rng(N + la[1] * 7 + lb[1])
    A = _csr(rng, N, rng.integers(*la, N), ncol)
    B = _csr(rng, N, rng.integers(*lb, N), ncol)
    dev = lambda m: tuple(torch.from_numpy(a).cuda() for a in m)  # noqa: E731
    want = _ref(N, A, -0.37, B)
    got = ops.csrgeam2(N, dev(A), -0.37, dev(B))
    assert np.array_equal(got[0].cpu().numpy(), want[0]) and np.array_equal(got[1].cpu().numpy(), want[1])
    assert f32_bits_equal(got[2].cpu().numpy(), want[2])
    s = rng.standard_normal(N).astype(np.float32)
    Bd = dev(B)
    ops.csr_rowscale(Bd[0], Bd[2], torch.from_numpy(s).cuda())
    assert f32_bits_equal(Bd[2].cpu().numpy(), B[2] * np.repeat(s, np.diff(B[0])))


def test_geam2_too_long_row_is_reported(cuda):
    import torch
    from piro_b200 import ops
    from piro_b200._lib import PiroError
    rng = np.random.default_rng(1)
    A = _csr(rng, 40, np.where(np.arange(40) == 17, 40, 1), 100)
    with pytest.raises(PiroError) as e:
        ops.csrgeam2(40, *[tuple(torch.from_numpy(a).cuda() for a in A)], 1.0, tuple(torch.from_numpy(a).cuda() for a in A))
    assert e.value.status == 1
