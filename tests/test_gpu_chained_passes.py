"""Alternating solves on the tensor cores stage each half-step's potential as the column bias of the next in its epilogue;
the CUDA-core engine, which reads potentials, gives the same potentials, iteration counts included."""
import pytest
import torch

pytestmark = pytest.mark.gpu


# exact products on both sides: potentials of size |x|^2 differ by its fp32 rounding per half-step (1e-5 allows 100 ulp)
@pytest.mark.parametrize("ott", [False, True])
@pytest.mark.parametrize("threshold,check_every", [(None, 5), (1e-2, 1), (1e-2, 3)])
@pytest.mark.parametrize("n,m,d,tiles", [(1, 1, 3, False), (257, 300, 3, False), (700, 900, 64, False), (300, 400, 80, False),
                                         (300, 260, 200, False), (700, 900, 3, True)])
def test_chained_half_steps(monkeypatch, n, m, d, tiles, threshold, check_every, ott):
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_alternating
    g = torch.Generator().manual_seed(n + d)
    x, y = torch.randn(n, d, generator=g).cuda(), (0.3 + torch.randn(m, d, generator=g)).cuda()
    a, b = (torch.softmax(torch.randn(k, generator=g), 0).cuda() for k in (n, m))
    mask = None
    if tiles:  # some row and column blocks keep a single tile
        mask = torch.rand((n + 127) // 128, (m + 127) // 128, generator=g) < 0.5
        mask[:, 0] = True
        mask[0, :] = True
    kw = dict(eps_list=[0.2 * d, 0.1 * d, 0.05 * d], iters_per_eps=4, rho_x=3.0 * d, threshold=threshold, check_every=check_every,
              return_n_iters=True, ott_convention=ott, tile_mask=mask, allow_tf32=False)
    got = sinkhorn_flashstyle_alternating(x, y, a, b, **kw)
    monkeypatch.setenv("FLASH_SINKHORN_B200_PREC", "simt")
    want = sinkhorn_flashstyle_alternating(x, y, a, b, **kw)
    size = float((x * x).sum(1).max() + (y * y).sum(1).max())
    assert got[2] == want[2]
    for u, v in zip(got[:2], want[:2]):
        assert float((u - v).abs().max()) < 1e-5 * size


# TF32 coordinates move each squared distance by up to 2^-11 of |x||y| (2e-3 of the largest potential). A point far from its
# cloud, without weight, gives every point a scale of its own, the staged biases too. One cloud has it: its shifted potential
# is 1e10 with an ulp of 1e3, and what it adds to the other cloud's sums lies 1e5 eps > 1e4 lower. (Two such points of
# either cloud meet at 1e17, where rounding alone, 1e10, decides what they add.)
@pytest.mark.parametrize("tf32,far", [(True, None), (True, "x"), (False, "x"), (True, "y"), (False, "y")])
@pytest.mark.parametrize("n,m,d,tiles", [(700, 900, 64, False), (300, 260, 100, False), (700, 900, 3, True), (513, 385, 20, True)])
def test_chained_half_steps_tf32_and_far_points(monkeypatch, n, m, d, tiles, tf32, far):
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_alternating
    g = torch.Generator().manual_seed(n + d)
    x, y = torch.randn(n, d, generator=g), 0.3 + torch.randn(m, d, generator=g)
    a, b = (torch.softmax(torch.randn(k, generator=g), 0) for k in (n, m))
    size = float((x * x).sum(1).max() + (y * y).sum(1).max())
    keep_x, keep_y = torch.ones(n, dtype=torch.bool), torch.ones(m, dtype=torch.bool)
    for name, pts, w, keep, k in (("x", x, a, keep_x, 1), ("y", y, b, keep_y, 130)):
        if far == name:
            pts[k] *= 1e8
            w[k] = 0.0
            keep[k] = False
    mask = None
    if tiles:
        mask = torch.rand((n + 127) // 128, (m + 127) // 128, generator=g) < 0.5
        mask[:, 0] = True
        mask[0, :] = True
    args = [t.cuda() for t in (x, y, a, b)]
    kw = dict(eps_list=[0.2 * d, 0.1 * d, 0.05 * d], iters_per_eps=4, tile_mask=mask)
    got = sinkhorn_flashstyle_alternating(*args, allow_tf32=tf32, **kw)
    monkeypatch.setenv("FLASH_SINKHORN_B200_PREC", "simt")
    want = sinkhorn_flashstyle_alternating(*args, allow_tf32=False, **kw)
    for u, v, keep in zip(got, want, (keep_x.cuda(), keep_y.cuda())):
        assert float((u - v)[keep].abs().max()) < (2e-3 if tf32 else 1e-5) * size
