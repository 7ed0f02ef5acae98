"""The grouped batched step on chip (k_batch_resident): teams of one and of
many CTAs, members from 3^3 up to the largest that fits, a member that does
not fit (the batch then takes k_batch_groups), and waits that run out.

Reference: the lockstep schedule, itself checked against FP64 direct solves.
Forward-Euler members agree bit for bit; both schedules solve backward-Euler
members to a 1e-8 FP64 residual, and with A's eigenvalues >= 1 each is within
1e-8 ||b|| of the solution, so 1e-6 of max |u| bounds their difference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(n, scheme):
    from piro_b200 import ops
    n = np.array(n, np.int32)
    rng = np.random.default_rng(int(n.sum()))
    alpha = (10.0 ** rng.uniform(-3.0, -1.0, size=n.size)).astype(np.float32)
    scheme = np.array(scheme, np.int32)
    dt = np.where(scheme == 0, 0.2 / (6.0 * alpha), 50.0 / (6.0 * alpha)).astype(np.float32)
    B = ops.Batch(n, alpha, dt, scheme)
    u0 = np.zeros(B.total, np.float32)
    for o, m in zip(B.offsets, n):  # nonzero boundary values too
        u0[int(o):int(o) + int(m) ** 3] = rng.random(int(m) ** 3, dtype=np.float32)
    return B, u0, n, scheme


@pytest.mark.parametrize("n,scheme", [
    ((3, 4, 5, 6, 7, 3), (1, 1, 1, 1, 1, 0)),
    ((16, 34, 33, 20), (1, 1, 1, 0)),
    ((96, 17, 64, 81, 50), (1, 1, 0, 1, 1)),
    ((127,), (1,)),
    ((134, 20, 19), (1, 1, 0)),  # the first does not fit on chip
])
def test_grouped_matches_lockstep(cuda, n, scheme):
    out = {}
    for grouped in (False, True):
        B, u0, nn, sc = _batch(n, scheme)
        B.set_schedule(grouped, 2)
        B.set_fields(u0)
        B.step(2)
        info = B.member_info()
        assert np.all(info["status"] == 0) and np.all(info["rel"][sc == 1] <= 1e-8)
        out[grouped] = B.get_fields()
        if grouped:  # the same bits again
            B.set_fields(u0)
            B.step(2)
            assert np.array_equal(B.get_fields(), out[True])
        off = B.offsets
        B.close()
    for k in range(len(nn)):
        s = slice(int(off[k]), int(off[k]) + int(nn[k]) ** 3)
        a, b = out[False][s], out[True][s]
        if sc[k]:
            assert np.abs(a - b).max() <= 1e-6 * np.abs(a).max(), k
        else:
            assert np.array_equal(a, b), k


def test_grouped_waits_give_up(cuda):
    from piro_b200._lib import PiroError, lib
    B, u0, n, sc = _batch((40, 33, 20, 9), (1, 1, 0, 1))
    B.set_schedule(True, 2)
    B.set_fields(u0)
    B.step(1)
    want = B.get_fields()
    B.set_fields(u0)
    try:
        assert lib().piro_set_wait_limit(0) == 0
        with pytest.raises(PiroError) as e:
            B.step(1)
        assert e.value.status == 6 and "timed out" in str(e.value)
    finally:
        lib().piro_set_wait_limit(-1)
    B.set_fields(u0)
    B.step(1)
    assert np.array_equal(B.get_fields(), want)
    B.close()


@pytest.mark.parametrize("steps", [2, 3, "autotune"])
def test_grouped_waits_give_up_in_any_launch(cuda, steps):
    """Several launches whose waits give up, in one call: the call says so, and nothing
    of their rounds is taken for a later launch's (other fields, so that it would show)."""
    from piro_b200._lib import PiroError, lib
    B, u0, n, sc = _batch((40, 33, 20, 9), (1, 1, 0, 1))
    B.set_schedule(True, 2)
    u1 = np.ascontiguousarray(u0[::-1])
    B.set_fields(u1)
    B.step(3)
    want = B.get_fields()
    B.set_fields(u0)
    try:
        assert lib().piro_set_wait_limit(0) == 0
        with pytest.raises(PiroError) as e:
            B.autotune(1e-8) if steps == "autotune" else B.step(steps)
        assert e.value.status == 6 and "timed out" in str(e.value)
    finally:
        lib().piro_set_wait_limit(-1)
    B.set_schedule(True, 2) if steps == "autotune" else None
    B.set_fields(u1)
    B.step(3)
    got = B.get_fields()
    for k in range(len(n)):  # the cells between the members belong to none
        assert np.array_equal(B.member(got, k), B.member(want, k)), k
    B.close()
