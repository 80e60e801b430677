"""Early stop of symmetric solves: a test after every step, on each kernel that serves them, and a stop behind the first table of
step records (256 of them), so that later tables and launches find the solve converged."""
import pytest
import torch

from test_gpu_two_sided import _clouds, cta_limit  # noqa: F401

pytestmark = pytest.mark.gpu


def _dense(x, y, a, b, sched, every, stop):
    """The textbook iteration in fp64 up to `stop` steps behind the first one, and the move of the potentials at every check
    so far: {step: largest change since the check before}."""
    cost = (x * x).sum(1)[:, None] + (y * y).sum(1)[None] - 2.0 * x @ y.T
    f, g, moves, last = torch.zeros_like(a), torch.zeros_like(b), {}, None

    def step(eps, w):
        nf = -eps * torch.logsumexp((g[None] - cost) / eps + b.log()[None], dim=1)
        ng = -eps * torch.logsumexp((f[:, None] - cost) / eps + a.log()[:, None], dim=0)
        return (1 - w) * f + w * nf, (1 - w) * g + w * ng

    f, g = step(sched[0], 1.0)
    for t, eps in enumerate(sched[:stop], 1):
        f, g = step(eps, 0.5)
        if t % every == 0:
            if last:
                moves[t] = max(float((f - last[0]).abs().max()), float((g - last[1]).abs().max()))
            last = f, g
    pre = f, g
    f, g = step(sched[-1], 1.0)
    return (f, g) + pre, moves


def _check(n, m, d, sched, every, stop):
    """The threshold lies halfway (in octaves) between the moves at the stop and at the check before, at least 1 % from any
    move up to there: several times what rounding does to one."""
    from flash_sinkhorn_b200 import _lib
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    x, y, a, b = (torch.as_tensor(v).cuda() for v in _clouds(n, m, d, seed=40))
    want, moves = _dense(x, y, a, b, sched, every, stop)
    threshold = (moves[stop - every] * moves[stop]) ** 0.5
    assert moves[stop] < threshold / 1.01 and min(v for t, v in moves.items() if t < stop) > 1.01 * threshold
    got = sinkhorn_flashstyle_symmetric(*(v.float() for v in (x, y, a, b)), eps_list=sched, threshold=threshold, check_every=every,
                                        allow_tf32=False, return_prelast=True, return_n_iters=True)
    assert int(got[-1]) == stop + 2
    size = float((x * x).sum(1).max())
    for u, v in zip(got[:4], want):  # potentials of size |x|^2 carry 2^-24 of it per step (100 ulp)
        assert float((u.double() - v).abs().max()) < 1e-5 * size
    assert _lib.load().fs_device_error() == 0


# points as in the test of every kernel of the two-sided steps: operands resident, streamed, 256 x 256 and 128 x 128 tiles
@pytest.mark.parametrize("limit", [40, 0])
@pytest.mark.parametrize("every,stop", [(1, 15), (3, 15)])
@pytest.mark.parametrize("n,m,d,kernel", [(1900, 1430, 64, 1), (2100, 1950, 200, 2), (2200, 2050, 512, 3), (300, 515, 200, 4)])
def test_stop_on_every_kernel(cta_limit, n, m, d, kernel, every, stop, limit):  # noqa: F811
    from flash_sinkhorn_b200 import _lib
    cta_limit(limit)
    assert _lib.load().fs_two_sided_kernel(n, m, d, _lib.PREC_FP32) == kernel
    _check(n, m, d, [0.05 * d] * 40, every, stop)


@pytest.mark.parametrize("every,stop", [(1, 264), (4, 268), (1, 600)])
def test_stop_behind_the_first_table(cta_limit, every, stop):  # noqa: F811
    """Slow steps at a small eps, then quick ones at a larger one; further tables follow the one with the stop."""
    cta_limit(5)
    _check(300, 260, 3, [0.05] * (stop - 28) + [2.0] * 300, every, stop)
