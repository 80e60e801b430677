"""Symmetric solves that take one exponential per score entry for both potentials: edges of the tiles, every kernel that
serves them, self-transport triangles, and inputs that force the one-sided steps."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host, rel
from oracle import dense_sinkhorn as O

pytestmark = pytest.mark.gpu


@pytest.fixture
def cta_limit():
    """Few CTAs: small problems then share tiles and column runs the way large ones do on all SMs."""
    from flash_sinkhorn_b200 import _lib
    lib = _lib.load()
    previous = lib.fs_set_cta_limit(0)
    yield lib.fs_set_cta_limit
    lib.fs_set_cta_limit(previous)


def _clouds(n, m, d, seed=0, zeros=False):
    r = np.random.default_rng(seed)
    x, y = r.normal(size=(n, d)), 0.3 + r.normal(size=(m, d))
    a, b = r.uniform(0.1, 1.1, n), r.uniform(0.1, 1.1, m)
    if zeros:
        a[::3] = 0.0
    x, y, a, b = (np.float32(v).astype(np.float64) for v in (x, y, a / a.sum(), b / b.sum()))
    return x, y, a, b


def _solve(x, y, a, b, prec, **kw):
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    xd, ad = dev(x), dev(a)
    yd, bd = (xd, ad) if y is x else (dev(y), dev(b))
    return sinkhorn_flashstyle_symmetric(xd, yd, ad, bd, allow_tf32=prec == "tf32", return_prelast=True,
                                         use_epsilon_scaling=False, **kw)


# (n, m, d): single points, one less and one more than a tile, runs that end inside a column tile; contractions that
# stay in shared memory (3 to 64) and streamed ones on tiles of 128 x 128 (the other streamed kernels serve larger clouds:
# test_every_kernel_of_the_two_sided_steps)
SHAPES = [(1, 1, 3), (1, 300, 7), (257, 1, 40), (128, 256, 64), (129, 257, 64), (511, 769, 3), (900, 640, 64),
          (300, 515, 200), (513, 300, 330), (260, 520, 1100)]


@pytest.mark.parametrize("limit", [1, 3, 0])
@pytest.mark.parametrize("prec", ["fp32", "tf32"])
@pytest.mark.parametrize("n,m,d", SHAPES)
def test_potentials_against_the_oracle(cta_limit, n, m, d, prec, limit):
    """eps small enough for one-sided first steps, then two-sided ones. Tolerances: fp32 potentials of size |x|^2
    carry 2^-24 of it per step, which 14 averaged steps do not amplify (1e-5 allows 100 ulp); TF32 coordinates
    move each squared distance by up to 2^-11 of |x||y|, 2e-3 of the largest potential."""
    cta_limit(limit)
    x, y, a, b = _clouds(n, m, d)
    eps = 0.02 * d
    want = O.solve_symmetric(x, y, a, b, [eps] * 14)
    got = _solve(x, y, a, b, prec, eps=eps, n_iters=14)
    tol = 1e-5 if prec == "fp32" else 2e-3
    size = max(np.abs(want["f"]).max(), (x * x).sum(1).max())
    for g, k in zip(got, ("f", "g", "f_pre", "g_pre")):
        assert np.abs(host(g) - want[k]).max() < tol * size


def _dense(x, y, a, b, eps, iters):
    """The textbook iteration in fp64 on the device (the numpy oracle takes minutes at these sizes)."""
    x, y, a, b = (torch.as_tensor(v).cuda() for v in (x, y, a, b))
    cost = (x * x).sum(1)[:, None] + (y * y).sum(1)[None] - 2.0 * x @ y.T
    f, g = torch.zeros_like(a), torch.zeros_like(b)
    for w in [1.0] + [0.5] * iters + [1.0]:
        pre = (f, g)
        nf = -eps * torch.logsumexp((g[None] - cost) / eps + b.log()[None], dim=1)
        ng = -eps * torch.logsumexp((f[:, None] - cost) / eps + a.log()[:, None], dim=0)
        f, g = (1 - w) * f + w * nf, (1 - w) * g + w * ng
    return f, g, pre[0], pre[1]


@pytest.mark.parametrize("limit", [40, 0])
@pytest.mark.parametrize("prec", ["fp32", "tf32"])
@pytest.mark.parametrize("n,m,d,kernel", [(1900, 1430, 64, 1), (2100, 1950, 200, 2), (2200, 2050, 512, 3), (300, 515, 200, 4)])
def test_every_kernel_of_the_two_sided_steps(cta_limit, n, m, d, kernel, prec, limit):
    """Ragged clouds on each of the four kernels: against each other, against themselves, and the three problems of a
    divergence in one call, with two-sided steps among theirs (all but the first ones; on all SMs the smallest have a CTA
    for every one-sided tile and nothing to share). Tolerances as in test_potentials_against_the_oracle."""
    from flash_sinkhorn_b200 import _lib
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric_batched
    lib = _lib.load()
    cta_limit(limit)
    prec_id = _lib.PREC_TF32 if prec == "tf32" else _lib.PREC_FP32
    sizes = ((n, m), (n, n), (m, m))
    assert lib.fs_two_sided_kernel(n, m, d, prec_id) == kernel
    x, y, a, b = _clouds(n, m, d, seed=40)
    eps, iters = 0.02 * d, 10
    wants = [_dense(*p, eps, iters) for p in ((x, y, a, b), (x, x, a, a), (y, y, b, b))]
    tol = (1e-5 if prec == "fp32" else 2e-3) * max((x * x).sum(1).max(), (y * y).sum(1).max())

    def check(out, want):
        for t, w in zip(out, want):
            assert float((t.double() - w).abs().max()) < tol

    def tiles(k, t):
        return (k + t - 1) // t

    bm, bn = {1: (128, 256), 2: (128, 256), 3: (256, 256), 4: (128, 128)}[kernel]
    shared = [tiles(p, bm) * tiles(q, bn) + (tiles(q, bm) * tiles(p, bn) if p != q else 0) > (limit or 148) for p, q in sizes]
    before = lib.fs_two_sided_steps()
    check(_solve(x, y, a, b, prec, eps=eps, n_iters=iters), wants[0])
    crossed = lib.fs_two_sided_steps()
    assert (crossed - before >= 4) == shared[0]
    check(_solve(x, x, a, a, prec, eps=eps, n_iters=iters), wants[1])
    assert (lib.fs_two_sided_steps() - crossed >= 4) == shared[1]
    xd, yd, ad, bd = (dev(v) for v in (x, y, a, b))
    before = lib.fs_two_sided_steps()
    got = sinkhorn_flashstyle_symmetric_batched([(xd, yd, ad, bd), (xd, xd, ad, ad), (yd, yd, bd, bd)], eps=eps, n_iters=iters,
                                                use_epsilon_scaling=False, allow_tf32=prec == "tf32")
    assert lib.fs_two_sided_steps() - before >= 4 * sum(shared)
    for out, want in zip(got, wants):
        check(out, want)
    assert lib.fs_device_error() == 0


@pytest.mark.parametrize("limit", [2, 0])
@pytest.mark.parametrize("n,d", [(1, 5), (130, 64), (385, 16), (640, 64), (300, 200), (515, 1100)])
def test_self_transport_triangle(cta_limit, n, d, limit):
    """One cloud against itself: only one side of the diagonal is evaluated."""
    cta_limit(limit)
    x, _, a, _ = _clouds(n, n, d, seed=1)
    eps = 0.02 * d
    want = O.solve_symmetric(x, x, a, a, [eps] * 10, rho_x=4.0, rho_y=4.0)
    got = _solve(x, x, a, a, "fp32", eps=eps, n_iters=10, reach=2.0)
    size = max(np.abs(want["f"]).max(), (x * x).sum(1).max())
    assert torch.equal(got[0], got[1])
    assert np.abs(host(got[0]) - want["f"]).max() < 1e-5 * size


@pytest.mark.parametrize("limit", [2, 0])
def test_zero_weights_schedules_and_early_stop(cta_limit, limit):
    """Zero weights and a rising eps have no bound on the next step's range: one-sided throughout, same results."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    cta_limit(limit)
    x, y, a, b = _clouds(400, 300, 32, seed=2, zeros=True)
    sched = [4.0, 1.0, 0.5, 2.0, 0.25, 0.25]
    want = O.solve_symmetric(x, y, a, b, sched)
    got = sinkhorn_flashstyle_symmetric(dev(x), dev(y), dev(a), dev(b), eps_list=sched, allow_tf32=False)
    size = (x * x).sum(1).max()
    assert np.abs(host(got[0]) - want["f"]).max() < 1e-5 * size
    assert np.abs(host(got[1]) - want["g"]).max() < 1e-5 * size
    x, y, a, b = _clouds(400, 300, 32, seed=3)
    want = O.solve_symmetric(x, y, a, b, [8.0] * 60, threshold=1e-3, check_every=4)
    got = sinkhorn_flashstyle_symmetric(dev(x), dev(y), dev(a), dev(b), eps=8.0, n_iters=60, use_epsilon_scaling=False,
                                        threshold=1e-3, check_every=4, allow_tf32=False, return_n_iters=True)
    assert got[2] == want["n_iters"] and np.abs(host(got[0]) - want["f"]).max() < 1e-5 * size


@pytest.mark.parametrize("limit", [2, 0])
@pytest.mark.parametrize("extrapolate", [True, False])
@pytest.mark.parametrize("zeros", [True, False])
def test_early_stop_inside_a_varying_schedule(cta_limit, limit, extrapolate, zeros):
    """The steps that are skipped have other eps than the last one, which runs all the same, at its own eps."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric
    cta_limit(limit)
    x, y, a, b = _clouds(400, 300, 32, seed=9, zeros=zeros)
    sched = [16.0] * 30 + [8.0, 4.0, 2.0, 1.0]
    want = O.solve_symmetric(x, y, a, b, sched, threshold=1e-2, check_every=4, last_extrapolation=extrapolate)
    assert want["n_iters"] < 25
    got = sinkhorn_flashstyle_symmetric(dev(x), dev(y), dev(a), dev(b), eps_list=sched, threshold=1e-2, check_every=4,
                                        last_extrapolation=extrapolate, allow_tf32=False, return_n_iters=True)
    size = (x * x).sum(1).max()
    assert got[2] == want["n_iters"]
    assert np.abs(host(got[0]) - want["f"]).max() < 1e-5 * size and np.abs(host(got[1]) - want["g"]).max() < 1e-5 * size


def test_not_a_number_stays_with_its_point(cta_limit):
    """No bound on the range can be given: one-sided steps to the end, and no wait runs out."""
    from flash_sinkhorn_b200 import _lib
    cta_limit(2)
    x, y, a, b = _clouds(300, 300, 64, seed=4)
    x[17, 3] = np.nan
    f = _solve(x, y, a, b, "tf32", eps=1.0, n_iters=5)[0]
    torch.cuda.synchronize()
    assert torch.isnan(f[17]) and _lib.load().fs_device_error() == 0


@pytest.mark.parametrize("zeros", [True, False])
@pytest.mark.parametrize("n,m,d", [(300, 20, 3), (20, 300, 3), (295, 260, 8), (130, 70, 2)])
def test_eps_at_which_the_mask_of_padded_points_leaves_fp32(n, m, d, zeros):
    """Clouds in units of 1e-3 and eps = 1e-9: the exponent of a padded point is -inf, also where a stretch of columns holds
    nothing else, in one-sided steps (weights of zero keep all of them so), soft-mins and alternating solves. Scores are 2e3
    to 2e4 times eps: the tolerance of the other tests, 1e-5 of |x|^2."""
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_alternating
    x, y, a, b = _clouds(n, m, d, seed=11, zeros=zeros)
    x, y = (np.float32(1e-3 * v).astype(np.float64) for v in (x, y))
    eps, size = 1e-9, max((x * x).sum(1).max(), (y * y).sum(1).max())
    bias = np.float32(np.random.default_rng(12).normal(size=m)).astype(np.float64)
    got = flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=eps, allow_tf32=False)
    assert np.abs(host(got) - O.lse_update(x, y, bias, eps)).max() < 1e-5 * size
    want = O.solve_symmetric(x, y, a, b, [eps] * 6)
    got = _solve(x, y, a, b, "fp32", eps=eps, n_iters=6)
    assert np.abs(host(got[0]) - want["f"]).max() < 1e-5 * size and np.abs(host(got[1]) - want["g"]).max() < 1e-5 * size
    want = O.solve_alternating(x, y, a, b, [eps], 3)
    got = sinkhorn_flashstyle_alternating(*(dev(v) for v in (x, y, a, b)), eps_list=[eps], iters_per_eps=3, allow_tf32=False)
    assert np.abs(host(got[0]) - want["f"]).max() < 1e-5 * size and np.abs(host(got[1]) - want["g"]).max() < 1e-5 * size


@pytest.mark.parametrize("scale", [1e-9, 1e-4, 1.0, 3e4, 1e9])
def test_operand_scale_follows_the_clouds(scale):
    """Coordinates ride as fp16 scaled by a power of two per cloud: any size of the clouds, also very different ones
    and with one far larger coordinate, gives the soft-min the precision of the 3-product mode (22 bits of every
    product against a largest potential of the size of the logits: 2e-6)."""
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    r = np.random.default_rng(5)
    x, y = np.float32(scale * r.normal(size=(300, 48))), np.float32(0.1 / scale * r.normal(size=(260, 48)))
    x[0, 0] *= 1000.0
    bias = np.float32(r.normal(size=260))
    got = flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=0.05, allow_tf32=False)
    want = O.lse_update(x.astype(np.float64), y.astype(np.float64), bias.astype(np.float64), 0.05)
    assert rel(host(got), want) < 2e-6


@pytest.mark.parametrize("d", [1, 8, 13, 14, 16, 17, 63, 80, 81])
@pytest.mark.parametrize("prec", ["fp32", "tf32"])
def test_every_operand_layout(prec, d):
    """Feature dimensions around the change from TF32 to fp16 columns and the ends of 16-coordinate steps: soft-min,
    nearest target, gradient and plan application against fp64 (the operand rounding is the only TF32 error: 2^-11 of
    |x||y| in the exponent of a weight)."""
    from flash_sinkhorn_b200.c_transform import c_transform_fwd
    from flash_sinkhorn_b200.kernels.apply_flash import apply_plan_mat_flashstyle
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    x, y, a, b = _clouds(200, 333, d, seed=7)
    tf32, eps = prec == "tf32", 0.5 * d
    r = np.random.default_rng(8)
    bias, mat = np.float32(r.normal(size=333)), np.float32(r.normal(size=(333, d)))
    got = flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=eps, allow_tf32=tf32)
    assert rel(host(got), O.lse_update(x, y, bias.astype(np.float64), eps)) < (3e-3 if tf32 else 2e-6)
    val, _ = c_transform_fwd(dev(x), dev(y), dev(bias), allow_tf32=tf32)
    assert rel(host(val), O.c_transform(x, y, bias.astype(np.float64))[0]) < (3e-3 if tf32 else 2e-6)
    fh, gh = -(x * x).sum(1), -(y * y).sum(1)
    args = [dev(v) for v in (x, y, fh, gh, np.log(a), np.log(b), mat)]
    got = apply_plan_mat_flashstyle(*args, eps=eps, axis=1, allow_tf32=tf32)
    want = O.apply_mat(x, y, fh, gh, np.log(a), np.log(b), mat.astype(np.float64), eps, 1)
    assert rel(host(got), want) < (5e-3 if tf32 else 3e-5)


def test_divergence_solves_share_their_launches(cta_limit):
    """The three solves of a debiased loss go out as one lockstep call; values and gradients equal the dense ones."""
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = _clouds(700, 450, 24, seed=6)
    want = O.samples_loss(x, y, a, b, [0.5] * 20, debias=True, want_grad_x=True)
    for limit in (5, 0):
        cta_limit(limit)
        xs = dev(x).requires_grad_(True)
        val = SamplesLoss("sinkhorn", use_epsilon_scaling=False, eps=0.5, n_iters=20, blur=0.5**0.5, debias=True,
                          allow_tf32=False)(dev(a), xs, dev(b), dev(y))
        (gx,) = torch.autograd.grad(val, xs)
        assert abs(float(val) - want["loss"]) < 2e-5 * abs(want["loss"])
        assert rel(host(gx), want["grad_x"]) < 3e-4


def _problems(sizes, d=20):
    out, wants = [], []
    for k, (n, m) in enumerate(sizes):
        x, y, a, b = _clouds(n, m, d, seed=20 + k)
        if k % 3 == 2:
            y, b = x, a
        wants.append(O.solve_symmetric(x, y, a, b, [6.0] * 5))
        xd, ad = dev(x), dev(a)
        out.append((xd, xd, ad, ad) if y is x else (xd, dev(y), ad, dev(b)))
    return out, wants


def _check(got, wants):
    for out, want in zip(got, wants):
        size = np.abs(want["f"]).max() + 40.0
        for t, k in zip(out, ("f", "g", "f_pre", "g_pre")):
            assert np.abs(host(t) - want[k]).max() < 1e-5 * size


@pytest.mark.parametrize("count", [1, 3, 24, 25, 60])
def test_lockstep_calls_of_many_problems(count):
    """More problems than one launch takes (24), of different sizes and kinds."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_symmetric_batched
    r = np.random.default_rng(count)
    probs, wants = _problems([(int(r.integers(1, 400)), int(r.integers(1, 400))) for _ in range(count)])
    _check(sinkhorn_flashstyle_symmetric_batched(probs, use_epsilon_scaling=False, eps=6.0, n_iters=5, allow_tf32=False), wants)


def test_lockstep_calls_split_where_their_sums_take_too_much(monkeypatch):
    from flash_sinkhorn_b200 import _lib, sinkhorn_solvers as S
    r = torch.Generator().manual_seed(3)
    probs = []
    for n in (6000, 6500, 7000, 8000):
        x, y = torch.randn(n, 20, generator=r).cuda(), torch.randn(n - 100, 20, generator=r).cuda()
        probs.append((x, y, torch.full((n,), 1.0 / n).cuda(), torch.full((n - 100,), 1.0 / (n - 100)).cuda()))
    probs[2] = (probs[2][0], probs[2][0], probs[2][2], probs[2][2])
    kw = dict(use_epsilon_scaling=False, eps=6.0, n_iters=5, allow_tf32=False)
    want = [S.sinkhorn_flashstyle_symmetric(*p, return_prelast=True, **kw) for p in probs]
    launches = []
    for limit in (1 << 30, 3 << 20, 0):
        monkeypatch.setattr(S, "LOCKSTEP_SCRATCH_BYTES", limit)
        before = _lib.load().fs_launch_count()
        got = S.sinkhorn_flashstyle_symmetric_batched(probs, **kw)
        launches.append(_lib.load().fs_launch_count() - before)
        for g, w in zip(got, want):  # another order of the partial sums: rounding of potentials below 100
            assert max(float((p - q).abs().max()) for p, q in zip(g[:4], w[:4])) < 1e-4
    assert launches[0] < launches[1] < launches[2]


def test_scratch_too_small_for_two_sided_steps():
    """Callers that bring the smaller scratch, and a device that has no room for the larger one, get the solve that evaluates
    the scores once per side: same results, alone and in a lockstep call."""
    from flash_sinkhorn_b200 import _lib, sinkhorn_solvers as S
    x, y, a, b = _clouds(40000, 36000, 16, seed=30)
    args = [dev(v) for v in (x, y, a, b)]
    kw = dict(use_epsilon_scaling=False, eps=4.0, n_iters=3, allow_tf32=False)
    full = S.sinkhorn_flashstyle_symmetric(*args, **kw)
    own = S.sinkhorn_flashstyle_symmetric(args[0], args[0], args[2], args[2], **kw)
    need = [_lib.symmetric_bytes(40000, 36000, 16, _lib.PREC_FP32, two_sided=t) for t in (True, False)]
    assert need[0] - need[1] > 5e7
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    total = torch.cuda.get_device_properties(0).total_memory
    room = torch.cuda.memory_reserved(0) + need[1] + 4.5e7
    torch.cuda.set_per_process_memory_fraction(room / total)
    try:
        small = S.sinkhorn_flashstyle_symmetric(*args, **kw)
        torch.cuda.empty_cache()
        both = S.sinkhorn_flashstyle_symmetric_batched([tuple(args), (args[0], args[0], args[2], args[2])], **kw)
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    size = (x * x).sum(1).max()
    for got, want in ((small, full), (both[0], full), (both[1], own)):
        assert max(float((g - w).abs().max()) for g, w in zip(got[:2], want)) < 1e-5 * size


@pytest.mark.parametrize("far", [1.0, 1e8])
def test_lockstep_calls_that_step_side_by_side(monkeypatch, far):
    """A lockstep call whose items bring the smaller scratch: several soft-min passes per launch, one per potential, also with a
    point far from its cloud (and without weight) in one of them."""
    from flash_sinkhorn_b200 import _lib, sinkhorn_solvers as S
    r = torch.Generator().manual_seed(4)
    probs = []
    for n, m in ((6000, 5800), (7000, 6100), (6400, 6300)):
        x, y = torch.randn(n, 20, generator=r), 0.2 + torch.randn(m, 20, generator=r)
        a, b = torch.softmax(torch.randn(n, generator=r), 0), torch.softmax(torch.randn(m, generator=r), 0)
        if n == 7000:
            x[0] *= far
            a[0] = 0.0
        probs.append(tuple(t.cuda() for t in (x, y, a, b)))
    kw = dict(use_epsilon_scaling=False, eps=6.0, n_iters=5, allow_tf32=False)
    want = S.sinkhorn_flashstyle_symmetric_batched(probs, **kw)
    full = _lib.symmetric_bytes
    monkeypatch.setattr(_lib, "symmetric_bytes", lambda n, m, d, prec, *a, **k: full(n, m, d, prec, two_sided=False))
    before = _lib.load().fs_two_sided_steps()
    got = S.sinkhorn_flashstyle_symmetric_batched(probs, **kw)
    assert _lib.load().fs_two_sided_steps() == before
    for g, w in zip(got, want):
        assert max(float((p - q)[1:].abs().max()) for p, q in zip(g[:4], w[:4])) < 1e-4
