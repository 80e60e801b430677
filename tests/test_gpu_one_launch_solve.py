"""Symmetric solves whose steps share one cooperative launch: more runs of tiles per CTA than its list holds, more steps
than a problem's table holds, problems of a lockstep call that end at different steps, capture, and solves side by side."""
import threading

import pytest
import torch

from test_gpu_two_sided import _clouds, _dense, cta_limit  # noqa: F401

pytestmark = pytest.mark.gpu


def _problem(n, m, d, seed):
    x, y, a, b = _clouds(n, m, d, seed=seed)
    return (x, y, a, b), tuple(torch.as_tensor(v, dtype=torch.float32).cuda() for v in (x, y, a, b))


def _size(*refs):
    """Largest |x|^2 of either cloud: potentials carry 2^-24 of it per step, which averaged steps do not amplify."""
    return max((v ** 2).sum(1).max() for r in refs for v in r[:2])


def _close(got, want, size):
    assert max(float((g.double() - w).abs().max()) for g, w in zip(got, want)) < 1e-5 * size


@pytest.mark.parametrize("n,m,d", [(130, 20000, 5), (20000, 130, 5), (130, 14000, 200), (1, 9000, 3)])
def test_more_runs_than_a_list_holds(cta_limit, n, m, d):  # noqa: F811
    """Two CTAs share 36 to 79 column tiles of one or two row tiles each; the list has 24 entries."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    cta_limit(2)
    ref, args = _problem(n, m, d, seed=7)
    eps = 0.05 * d
    got = sinkhorn_flashstyle_symmetric(*args, use_epsilon_scaling=False, eps=eps, n_iters=9, allow_tf32=False,
                                        return_prelast=True)
    _close(got, _dense(*ref, eps, 9), _size(ref))


@pytest.mark.parametrize("iters", [253, 254, 255, 256, 300, 520])
def test_more_steps_than_a_table_holds(cta_limit, iters):  # noqa: F811
    """A table has 256 steps, a solve iters + 2; alone and with problems that end before it in the same call."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric, sinkhorn_flashstyle_symmetric_batched
    cta_limit(5)
    eps = 3.0
    probs = [_problem(300, 520, 8, seed=s) for s in (1, 2, 3)]
    wants = [_dense(*p[0], eps, k) for p, k in zip(probs, (iters, 254, 7))]
    size = _size(*(p[0] for p in probs))
    kw = dict(use_epsilon_scaling=False, eps=eps, allow_tf32=False)
    _close(sinkhorn_flashstyle_symmetric(*probs[0][1], n_iters=iters, return_prelast=True, **kw), wants[0], size)
    got = sinkhorn_flashstyle_symmetric_batched([p[1] for p in probs], schedules=[[eps] * k for k in (iters, 254, 7)], **kw)
    for g, w in zip(got, wants):
        _close(g[:4], w, size)


def test_capture_and_side_by_side():
    """A captured solve replays to the same bits, and solves on streams of their own threads do not disturb one another."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    kw = dict(use_epsilon_scaling=False, eps=2.0, n_iters=12, allow_tf32=False)
    sets = [_problem(1500 + 100 * k, 1400, 16, seed=k)[1] for k in range(3)]
    wants = [sinkhorn_flashstyle_symmetric(*s, **kw) for s in sets]
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = sinkhorn_flashstyle_symmetric(*sets[0], **kw)
    for _ in range(2):
        out[0].zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(out, wants[0]))
    bad = []

    def work(args, want):
        stream = torch.cuda.Stream()
        with torch.cuda.stream(stream):
            for _ in range(10):
                got = sinkhorn_flashstyle_symmetric(*args, **kw)
                if not all(torch.equal(p, q) for p, q in zip(got, want)):
                    bad.append(args)
        stream.synchronize()

    threads = [threading.Thread(target=work, args=p) for p in zip(sets, wants)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


@pytest.mark.parametrize("limit", [5, 0])
def test_launch_that_ends_while_steps_are_one_sided(cta_limit, limit):  # noqa: F811
    """At a small eps the first steps are one-sided; problems of the same call end among them, and the launch with them."""
    from flash_sinkhorn_b200 import _lib
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric_batched
    cta_limit(limit)
    lib, eps, d = _lib.load(), 0.02, 8
    sizes = [(300, 520), (1500, 1400), (2100, 1700)]
    probs = [_problem(n, m, d, seed=k) for k, (n, m) in enumerate(sizes)]
    kw = dict(use_epsilon_scaling=False, eps=eps, allow_tf32=False)
    before = lib.fs_two_sided_steps()
    sinkhorn_flashstyle_symmetric_batched([p[1] for p in probs], schedules=[[eps]] * 3, **kw)
    assert lib.fs_two_sided_steps() == before  # three steps, all one-sided
    lengths = (1, 30, 2)
    got = sinkhorn_flashstyle_symmetric_batched([p[1] for p in probs], schedules=[[eps] * k for k in lengths], **kw)
    assert lib.fs_two_sided_steps() > before
    for g, p, k in zip(got, probs, lengths):
        _close(g[:4], _dense(*p[0], eps, k), _size(p[0]))


# column tiles of y = pairs per point of x that the end of a one-sided step adds: eight warps with eight offsets, four with four pairs
# in flight each (64 and 16 pairs a round), at the edges of a round; x has two pairs per point of y
@pytest.mark.parametrize("zeros", [False, True])
@pytest.mark.parametrize("tiles", [1, 8, 9, 16, 17, 31, 33, 64, 65, 97])
def test_pairs_of_one_sided_steps(tiles, zeros):
    from flash_sinkhorn_b200 import _lib
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    x, y, a, b = _clouds(130, 128 * (tiles - 1) + 5, 8, seed=tiles)
    if zeros and tiles > 1:  # a tile of columns that add nothing
        b[:128] = 0.0
    args = [torch.as_tensor(v, dtype=torch.float32).cuda() for v in (x, y, a, b)]
    before = _lib.load().fs_two_sided_steps()
    got = sinkhorn_flashstyle_symmetric(*args, use_epsilon_scaling=False, eps=0.02, n_iters=1, allow_tf32=False, return_prelast=True)
    assert _lib.load().fs_two_sided_steps() == before  # three steps, all one-sided
    _close(got, _dense(x, y, a, b, 0.02, 1), _size((x, y, a, b)))
