"""The two-plane activation arrays of the tensor-core layers at their ends:
array lengths of every remainder mod 8, grids with as few boundary cells after
the last interior one as there can be, windows that start before the array and
end after it, and buffers that a larger grid has used before (the rows after
the last cell then held another grid's values)."""
import numpy as np
import pytest

from oracle import pcnet_oracle as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,B", [((3, 3, 3), 1), ((3, 3, 6), 1), ((3, 3, 4), 1), ((3, 3, 5), 3), ((3, 4, 7), 1),
                                 ((5, 3, 3), 1), ((3, 5, 7), 5), ((11, 3, 4), 1), ((43, 3, 3), 2)])
def test_planes_do_not_depend_on_what_was_there(cuda, n, B):
    import torch
    from piro_b200 import ops
    p = P.init_params(7).astype(np.float32)
    rng = np.random.default_rng(9)
    N = n[0] * n[1] * n[2]
    r, f, t = (rng.standard_normal((B, N)).astype(np.float32) for _ in range(3))
    m = np.ones((B, N), np.float32)
    T = lambda a: torch.from_numpy(a.reshape(-1)).cuda()  # noqa: E731
    got = []
    for used in (False, True):
        net = ops.PCNet(seed=0)
        net.set_params(p)
        if used:  # large values everywhere, then the small grid in the same buffers
            big = (16, 15, 14)
            h = torch.full((3360,), 3.0e4, device="cuda")
            net.loss_grad(*big, h, h, h, torch.ones_like(h), batch=1, want_grad=True)
            net.forward(*big, h, h)
        loss, g = net.loss_grad(*n, T(r), T(f), T(t), T(m), batch=B, want_grad=True)
        got.append((loss, g, net.forward(*n, T(r), T(f), batch=B).cpu().numpy()))
        net.close()
    assert got[0][0] == got[1][0] and np.array_equal(got[0][1], got[1][1]) and np.array_equal(got[0][2], got[1][2])
    rl, rg = P.loss_grad(p.astype(np.float64), n, r, f, t, m, emulate=True)
    assert abs(got[0][0] - rl) <= 1e-3 * abs(rl)
    wo, total = P.layout()
    ends = wo[1:] + [total]
    for l in range(4):  # BF16 activations and gradients: 2^-8 per rounding, a few roundings deep
        a, b = got[0][1][wo[l]:ends[l]].astype(np.float64), rg[wo[l]:ends[l]]
        assert np.sqrt(((a - b) ** 2).sum()) <= 2e-2 * np.sqrt((b ** 2).sum()), l


@pytest.mark.parametrize("n,B", [((33, 31, 6), 40), ((34, 34, 9), 12), ((6, 5, 3), 700), ((12, 12, 400), 3)])
def test_shares_of_the_tiles_do_not_matter(cuda, n, B):
    """A batch and its members alone, whose tiles fall to other blocks (one tile
    a block, shares that end inside a column, at its end and in the next
    member): the same bits."""
    import torch
    from piro_b200 import ops
    rng = np.random.default_rng(4)
    N = n[0] * n[1] * n[2]
    r, f = (torch.from_numpy(rng.standard_normal(B * N).astype(np.float32)).cuda() for _ in range(2))
    net = ops.PCNet(seed=0)
    out = net.forward(*n, r, f, batch=B)
    for b in sorted({0, 1, B // 2, B - 2, B - 1}):
        s = slice(b * N, (b + 1) * N)
        one = net.forward(*n, r[s].contiguous(), f[s].contiguous())
        assert torch.equal(out[s].view(torch.int32), one.view(torch.int32)), b
    net.close()
