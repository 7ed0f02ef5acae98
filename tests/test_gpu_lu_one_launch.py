"""The band LU in one cooperative launch and its one-block solve at the edges of
their rules: bandwidths 15 | 16 (the launches per panel below), 632 | 633 (the
solve's registers), 720 | 721 (a thread's two rows per panel), sizes that are
no multiple of the 16-column panel, exchanges in nearly every column.  The
factor's order of operations is that of the column launches: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _table(ops, N, bw, seed, zero_col=None):
    """About 7 entries a row at random places in the band."""
    import torch
    rng = np.random.default_rng(seed)
    rows = []
    for r in range(N):
        c = np.unique(np.concatenate([[r], np.clip(rng.integers(r - bw, r + bw + 1, 6), 0, N - 1)]))
        c = c[np.abs(c - r) <= bw]
        rows.append(c[c != zero_col])
    rp = np.concatenate([[0], np.cumsum([len(c) for c in rows])]).astype(np.int32)
    col = np.concatenate(rows).astype(np.int32)
    val = rng.standard_normal(len(col)).astype(np.float32)
    A = [torch.from_numpy(t).cuda() for t in (rp, col, val)]
    ts = ops.ht_table_size(len(col), N, 1)
    return ops.ht_build(N, *A, ts), ts, (rp, col, val)


def _parts(lu, N, bw):
    nb = 8 * N * (3 * bw + 1)
    off = (nb + 255) // 256 * 256
    band = lu.band[:nb].cpu().numpy().view(np.uint64)
    lc = lu.band[off:off + 8 * N * bw].cpu().numpy().view(np.uint64).reshape(N, bw)
    span = np.minimum(bw, N - 1 - np.arange(N))
    return band, lc[np.arange(bw)[None, :] < span[:, None]], lu.pivots()


@pytest.mark.parametrize("N,bw", [(17, 15), (16, 16), (17, 17), (33, 16), (100, 17), (255, 40), (700, 300), (1301, 632),
                                  (1290, 633), (1500, 720), (1480, 721)])
def test_lu_one_launch_equals_column_launches(cuda, N, bw, monkeypatch):
    import torch
    from piro_b200 import ops
    (keys, vals), ts, (rp, col, val) = _table(ops, N, bw, 7 * N + bw)
    lu = ops.HtLu(N, bw, keys, vals, ts, 0.0, 1.0)
    b = torch.from_numpy(np.random.default_rng(3).random(N).astype(np.float32)).cuda()
    x = lu.solve(b).cpu().numpy()
    monkeypatch.setenv("PIRO_LU_NO_RING", "1")
    assert np.array_equal(x.view(np.uint32), lu.solve(b).cpu().numpy().view(np.uint32))
    monkeypatch.setenv("PIRO_LU_UNBLOCKED", "1")
    col_lu = ops.HtLu(N, bw, keys, vals, ts, 0.0, 1.0)
    assert (np.arange(N) != lu.pivots()).sum() > N // 3
    for got, want in zip(_parts(lu, N, bw), _parts(col_lu, N, bw)):
        assert np.array_equal(got, want)
    Ad = np.zeros((N, N))
    Ad[np.repeat(np.arange(N), np.diff(rp)), col] = val
    ref = np.linalg.solve(Ad, b.cpu().numpy().astype(np.float64))
    # float32 rounding of x, and the backward error of a pivoted elimination
    # (growth up to 2^7 allowed for)
    assert np.abs(x - ref).max() <= (1.2e-7 + 128 * N * 1.2e-16 * np.linalg.cond(Ad)) * np.abs(ref).max()


@pytest.mark.parametrize("zero_col", [0, 16, 37, 99])
def test_lu_one_launch_singular(cuda, zero_col):
    from piro_b200 import ops
    from piro_b200._lib import PiroError
    (keys, vals), ts, _ = _table(ops, 100, 20, 5, zero_col)
    with pytest.raises(PiroError, match=f"column {zero_col} ") as e:
        ops.HtLu(100, 20, keys, vals, ts, 0.0, 1.0)
    assert e.value.status == 12  # PIRO_ERR_ZERO_PIVOT


def test_lu_one_launch_wait_gives_up(cuda):
    from piro_b200 import ops
    from piro_b200._lib import PiroError, lib
    (keys, vals), ts, _ = _table(ops, 300, 60, 6)
    want = _parts(ops.HtLu(300, 60, keys, vals, ts, 0.0, 1.0), 300, 60)
    assert lib().piro_set_wait_limit(0) == 0
    try:
        with pytest.raises(PiroError, match="timed out"):
            ops.HtLu(300, 60, keys, vals, ts, 0.0, 1.0)
    finally:
        lib().piro_set_wait_limit(-1)
    for got, ref in zip(_parts(ops.HtLu(300, 60, keys, vals, ts, 0.0, 1.0), 300, 60), want):
        assert np.array_equal(got, ref)


def test_lu_one_launch_singular_beside_a_wait_that_gave_up(cuda):
    """A zero first column, found without a wait, while the other blocks' first wait gives up."""
    from piro_b200 import ops
    from piro_b200._lib import PiroError, lib
    (keys, vals), ts, _ = _table(ops, 100, 20, 5, 0)
    assert lib().piro_set_wait_limit(0) == 0
    try:
        with pytest.raises(PiroError, match="column 0 ") as e:
            ops.HtLu(100, 20, keys, vals, ts, 0.0, 1.0)
        assert e.value.status == 12  # PIRO_ERR_ZERO_PIVOT
    finally:
        lib().piro_set_wait_limit(-1)
