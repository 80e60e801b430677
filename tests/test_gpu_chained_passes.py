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
