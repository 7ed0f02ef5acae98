"""With device memory for the older forms but not for the on-chip form's exchange
buffers, solvers and batches are created all the same and solve in an older form.
The rest of the device memory is held by one allocation meanwhile."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MIB = 1 << 20


class _Full:
    """All free device memory but `leave` bytes."""

    def __init__(self, torch, leave):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.torch = torch
        size = torch.cuda.mem_get_info()[0] - leave
        while True:  # the last MiB may not be had in one piece
            try:
                self.t = torch.empty(size // (2 * MIB) * 2 * MIB, dtype=torch.uint8, device="cuda")
                break
            except torch.cuda.OutOfMemoryError:
                size -= 2 * MIB

    def __enter__(self):
        return self

    def __exit__(self, *a):
        del self.t
        self.torch.cuda.empty_cache()


def test_be_solver_without_the_exchange_buffer(cuda, monkeypatch):
    import torch
    from piro_b200 import ops
    n, dt = (128, 128, 128), 5.0
    N = n[0] ** 3
    alpha = torch.rand(N, device="cuda") + 0.5
    b = torch.rand(N, device="cuda")
    L = ops.csr_laplacian(*n, 3, 1.0)
    ops.csr_rowscale(L[0], L[2], alpha)
    A = ops.csrgeam2(N, ops.csr_identity(N), -dt, L)
    x, want = torch.empty_like(b), torch.empty_like(b)

    def run(out):
        s = ops.BESolver(*n, A, alpha, stencil=(dt, 1.0))
        used, form = torch.cuda.mem_get_info()[0], s.forms[0]
        assert s.solve(b, out, rtol=1e-8).status == 0
        s.close()
        return used, form

    assert run(want)[1] == "chip"
    monkeypatch.setenv("PIRO_BE_PERSISTENT", "g")
    run(x)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    used, form = run(x)
    assert form == "global"
    monkeypatch.setenv("PIRO_BE_PERSISTENT", "1")
    with _Full(torch, free - used + 10 * MIB):  # the exchange buffer and alpha take 24 MB
        assert run(x)[1] == "shared"
    assert float((x - want).abs().max()) <= 1e-6 * float(want.abs().max())


def test_batch_without_the_exchange_buffer(cuda):
    import torch
    from piro_b200 import ops
    n = np.array([127], np.int32)  # 16 MB
    alpha, dt = np.array([0.01], np.float32), np.array([830.0], np.float32)
    u = np.random.default_rng(0).random(int(n[0]) ** 3, dtype=np.float32)
    got = []
    for low in (False, True):
        B = ops.Batch(n, alpha, dt, np.ones(1, np.int32))
        u0 = np.zeros(B.total, np.float32)
        u0[:u.size] = u
        if low:
            B.set_schedule(False, 4)
            B.set_fields(u0)
            B.step(1)
            with _Full(torch, 8 * MIB):
                B.set_schedule(True, 2)
                B.set_fields(u0)
                B.step(1)
        else:
            B.set_schedule(True, 2)
            B.set_fields(u0)
            B.step(1)
        assert np.all(B.member_info()["rel"] <= 1e-8)
        got.append(B.member(B.get_fields(), 0))
        B.close()
    assert np.abs(got[0] - got[1]).max() <= 1e-6 * np.abs(got[0]).max()
