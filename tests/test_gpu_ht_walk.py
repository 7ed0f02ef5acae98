"""The hash-table step's lookups along chains of every length: walks of 1 to 12
slots, over the table's end, past deleted entries (-2), to an empty slot, in a
full table (no empty slot) and with absent keys: bit for bit the plain linear
probing, in all three forms of the step."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
f32 = np.float32


@pytest.mark.parametrize("ts", [331, 401, 360, 300, 293])
@pytest.mark.parametrize("dead,drop", [(0.0, 0.0), (0.15, 0.1), (0.0, 0.3)])
def test_ht_walks(cuda, ts, dead, drop):
    import torch
    from piro_b200 import ops
    n = (5, 4, 3)
    nx, ny, nz = n
    N = nx * ny * nz
    rng = np.random.default_rng(int(ts + 100 * dead + 10 * drop))
    A = ops.csr_laplacian(nx, ny, nz, 3, 1.0)
    rp, col = A[0].cpu().numpy(), A[1].cpu().numpy()
    ent = [(r, int(c)) for r in range(N) for c in col[rp[r]:rp[r + 1]]]
    ent = [e for e in ent if rng.random() >= drop]
    ent = [ent[i] for i in rng.permutation(len(ent))]
    keys, vals, walks = np.full(ts, -1, np.int64), np.zeros(ts, f32), []
    for r, c in ent:
        h, w = (r * N + c) % ts, 0
        while keys[h] != -1:
            h, w = (h + 1) % ts, w + 1
            if w == ts:
                break
        if w < ts:
            keys[h], vals[h] = r * N + c, f32(rng.standard_normal())
            walks.append(w)
    gone = (rng.random(ts) < dead) & (keys >= 0)
    keys[gone] = -2
    if dead == 0 and drop == 0:
        assert max(walks) > 4
    if ts == 293:  # no empty slot: absent keys end after the whole table
        keys[keys == -1] = -2
    u, dt = rng.standard_normal(N).astype(f32), f32(0.3)

    def get(key):
        h = key % ts
        for _ in range(ts + 1):
            if keys[h] == key:
                return vals[h]
            if keys[h] == -1:
                break
            h = (h + 1) % ts
        return f32(0)

    want = np.zeros(N, f32)
    for i in range(N):
        x, y, z = i % nx, i // nx % ny, i // (nx * ny)
        s = f32(0)
        for o, ok in ((-nx * ny, z > 0), (-nx, y > 0), (-1, x > 0), (0, True), (1, x < nx - 1), (nx, y < ny - 1),
                      (nx * ny, z < nz - 1)):
            if ok:
                s = f32(s + f32(get(i * N + i + o) * u[i + o]))
        want[i] = f32(dt * s)
    K, V, U = (torch.from_numpy(a).cuda() for a in (keys, vals, u))
    order = ops.ht_row_order(N, ts)
    outs = [torch.empty(N, device="cuda") for _ in range(3)]
    ops.ht_spmv(nx, ny, nz, K, V, dt, U, outs[0])
    ops.ht_spmv_ordered(nx, ny, nz, K, V, dt, order, U, outs[1])
    ops.ht_spmv_staged(nx, ny, nz, K, V, dt, order, ops.ht_stage(N), U, outs[2])
    for o in outs:
        assert np.array_equal(o.cpu().numpy().view(np.uint32), want.view(np.uint32))
