"""A point far from its cloud (an outlier, a padding sentinel) takes no significant bits from the others.

The score contractions take fp16 coordinates scaled by a power of two, one for a whole cloud where that carries every
point. Here it cannot: one point is 1e6 to 1e13 times as far out as the rest, all rows but its own are compared with
fp64, each against its own size. What remains is the rounding that every input shows. Exact mode: three products drop
2^-22 of |x||y|, the fp32 contraction rounds at 2^-23 of its largest partial sum a few times; 2^-18 of
|x_i| max|y_j| + max|bias| covers both, times 2 for the logit's factor. TF32 mode: 2^-11 of either factor, 2^-9 in all.
"""
import numpy as np
import pytest
import torch

from gpu_util import dev, host
from oracle import dense_sinkhorn as O

pytestmark = pytest.mark.gpu

N, M = 400, 300


def _points(d, far, where, seed=0, n=N, m=M):
    """Clouds of unit-variance coordinates in fp32, as fp64 arrays; row 5 of x and/or row 7 of y is far away."""
    r = np.random.default_rng(seed)
    x, y = r.normal(size=(n, d)), 0.3 + r.normal(size=(m, d))
    for cloud, at, name in ((x, 5, "x"), (y, 7, "y")):
        if name in where:
            cloud[at] = far * (r.integers(0, 2, size=d) * 2 - 1)
    return np.float32(x).astype(np.float64), np.float32(y).astype(np.float64)


def _near(count, where, name):
    keep = np.ones(count, bool)
    if name in where:
        keep[5 if name == "x" else 7] = False
    return keep


def _norm(v):
    return np.sqrt((v * v).sum(1))


FAR = [(1e6, "x"), (1e8, "y"), (1e10, "x"), (1e10, "xy"), (1e13, "y")]
DIMS = [16, 64, 200, 520]  # fp16 operands resident in shared memory and K-streamed


@pytest.mark.parametrize("prec", ["fp32", "tf32"])
@pytest.mark.parametrize("d", DIMS)
@pytest.mark.parametrize("far,where", FAR)
def test_soft_min_and_nearest_target(prec, d, far, where):
    from flash_sinkhorn_b200.c_transform import c_transform_fwd
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    tf32 = prec == "tf32"
    x, y = _points(d, far, where)
    ny = _near(M, where, "y")
    eps = 0.5 * d
    bias = np.float32(np.where(ny, np.random.default_rng(1).normal(size=M), -2.0 * (y * y).sum(1) / eps)).astype(np.float64)
    keep = _near(N, where, "x")
    tol = 2.0 * (2.0**-9 if tf32 else 2.0**-18) * (_norm(x) * _norm(y[ny]).max() + eps * np.abs(bias[ny]).max())
    got = flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=eps, allow_tf32=tf32)
    assert (np.abs(host(got) - O.lse_update(x, y, bias, eps)) < tol)[keep].all()
    psi = np.float32(np.random.default_rng(2).normal(size=M))
    val, idx = c_transform_fwd(dev(x), dev(y), dev(psi), allow_tf32=tf32)
    cost = (x * x).sum(1)[:, None] - 2.0 * x @ y.T + (y * y).sum(1)[None] - psi.astype(np.float64)[None]
    size = 2.0 * _norm(x) * _norm(y[ny]).max() + (_norm(y[ny])**2).max() + _norm(x)**2
    tol = (2.0**-9 if tf32 else 2.0**-18) * size
    assert (np.abs(host(val) - cost.min(1)) < tol)[keep].all()
    picked = cost[np.arange(N), idx.cpu().numpy()]  # the target it names is within the error of the nearest one
    assert (picked - cost.min(1) < 2.0 * tol)[keep].all()


@pytest.mark.parametrize("prec", ["fp32", "tf32"])
@pytest.mark.parametrize("d", DIMS)
@pytest.mark.parametrize("far,where", FAR)
def test_plan_applications_and_gradient(prec, d, far, where):
    """Weights are exponentials of scores divided by eps = d / 2 (errors: a few times 2^-18 or 2^-9 of |x||y| / eps, about 4
    here); in TF32 mode weights and matrix are rounded for the second GEMM too."""
    from flash_sinkhorn_b200.kernels.apply_flash import apply_plan_mat_flashstyle, apply_plan_vec_flashstyle
    from flash_sinkhorn_b200.kernels.apply_ott import mat5_sqeuclid
    from flash_sinkhorn_b200.kernels.grad_sqeuclid import sinkhorn_geomloss_online_grad_sqeuclid
    tf32 = prec == "tf32"
    tol = 4e-2 if tf32 else 1e-4
    x, y = _points(d, far, where, seed=3)
    kx, ky = _near(N, where, "x"), _near(M, where, "y")
    eps = 0.5 * d
    r = np.random.default_rng(4)
    la, lb = np.full(N, -np.log(N)), np.full(M, -np.log(M))
    g = np.where(ky, r.normal(size=M), 0.0)
    # row potentials from the near columns; a far point has no mass in any other point's row or column
    gh = np.float32(g - (y * y).sum(1)).astype(np.float64)
    fh = np.float32(np.where(kx, O.lse_update(x, y[ky], gh[ky] / eps + lb[ky], eps), -2.0 * (x * x).sum(1))).astype(np.float64)
    plan = np.exp((2.0 * x[kx] @ y[ky].T + fh[kx][:, None] + gh[ky][None]) / eps + la[kx][:, None] + lb[ky][None])
    args = [dev(v) for v in (x, y, fh, gh, la, lb)]
    kw = dict(eps=eps, allow_tf32=tf32)

    def close(got, want, keep):
        got = host(got)[keep]
        size = np.abs(want).max(axis=-1, keepdims=True) if want.ndim == 2 else np.abs(want).max()
        assert (np.abs(got - want) < tol * size).all()

    v, u = r.uniform(0.5, 1.5, M), r.uniform(0.5, 1.5, N)
    close(apply_plan_vec_flashstyle(*args, dev(v), axis=1, **kw), plan @ v[ky], kx)
    close(apply_plan_vec_flashstyle(*args, dev(u), axis=0, **kw), plan.T @ u[kx], ky)
    mv, mu = r.normal(size=(M, d)), r.normal(size=(N, d))
    rows, cols = plan.sum(1)[:, None], plan.sum(0)[None]
    mv, mu = mv + 3.0, mu + 3.0  # means well above the noise: a relative error per row is meaningful
    close(apply_plan_mat_flashstyle(*args, dev(mv), axis=1, **kw), plan @ mv[ky], kx)
    close(apply_plan_mat_flashstyle(*args, dev(mu), axis=0, **kw), plan.T @ mu[kx], ky)
    f = np.where(kx, fh + (x * x).sum(1), 0.0)
    gx, gy = sinkhorn_geomloss_online_grad_sqeuclid(dev(x), dev(y), dev(np.exp(la)), dev(np.exp(lb)), dev(f), dev(g), **kw)
    want = 2.0 * np.exp(la)[kx][:, None] * (x[kx] - (plan / rows) @ y[ky])
    close(gx, want, kx)
    want = 2.0 * np.exp(lb)[ky][:, None] * (y[ky] - (plan / cols).T @ x[kx])
    close(gy, want, ky)
    # the second row operand has a range of its own
    fo, go = eps * la + np.where(kx, f, 0.0), eps * lb + g
    amat = 3.0 + r.normal(size=(N, d))
    amat[[5, 50]] *= far
    got = mat5_sqeuclid(dev(x), dev(y), dev(fo), dev(go), dev(amat), **kw)
    want = (-4.0 / eps) * ((plan * (np.float32(amat[kx]).astype(np.float64) @ y[ky].T)) @ y[ky])
    got, scale = host(got)[kx], (4.0 / eps) * (plan.sum(1) * _norm(amat[kx]) * (_norm(y[ky])**2).mean())[:, None]
    assert (np.abs(got - want) < tol * scale).all()


@pytest.mark.parametrize("prec", ["fp32", "tf32"])
@pytest.mark.parametrize("n,m,d", [(400, 300, 16), (400, 300, 64), (400, 300, 200), (2100, 1950, 200), (4100, 3900, 512)])
@pytest.mark.parametrize("weight", [0.0, 1.0])
def test_symmetric_and_alternating_solves(prec, n, m, d, weight):
    """Every kernel of the solvers: a far point without weight in a balanced problem, two with weight in a relaxed one (two
    without would meet in a product of 1e16 that their potentials, in fp32, cannot cancel). The far point's potential starts
    at 1e16 d and must not enter its own sums either. Tolerances as for ordinary clouds: 1e-5 and 2e-3 of the largest near
    potential."""
    from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_alternating, sinkhorn_flashstyle_symmetric
    tf32, eps, iters = prec == "tf32", 0.5 * d, 3
    where = "xy" if weight else "x"
    x, y = _points(d, 1e8, where, seed=5, n=n, m=m)
    kx, ky = _near(n, where, "x"), _near(m, where, "y")
    r = np.random.default_rng(6)
    a, b = r.uniform(0.5, 1.5, n), r.uniform(0.5, 1.5, m)
    a[5] *= weight
    a, b = (np.float32(w / w.sum()).astype(np.float64) for w in (a, b))
    rho = None if weight == 0.0 else 4.0
    want = O.solve_symmetric(x, y, a, b, [eps] * iters, rho_x=rho, rho_y=rho)
    reach = None if rho is None else 2.0
    size = max(np.abs(want["f"][kx]).max(), (_norm(x[kx])**2).max(), (_norm(y[ky])**2).max())
    tol = (2e-3 if tf32 else 1e-5) * size
    args = [dev(v) for v in (x, y, a, b)]
    got = sinkhorn_flashstyle_symmetric(*args, eps=eps, n_iters=iters, use_epsilon_scaling=False, reach=reach, allow_tf32=tf32)
    assert np.abs(host(got[0]) - want["f"])[kx].max() < tol
    assert np.abs(host(got[1]) - want["g"])[ky].max() < tol
    if n * m < 1e6 and rho is None:
        want = O.solve_alternating(x, y, a, b, [eps], iters)
        got = sinkhorn_flashstyle_alternating(*args, eps_list=[eps], iters_per_eps=iters, allow_tf32=tf32)
        assert np.abs(host(got[0]) - want["f"])[kx].max() < tol
        assert np.abs(host(got[1]) - want["g"])[ky].max() < tol


def test_lockstep_labels_and_tile_lists_with_a_far_point():
    """One far problem among ordinary ones of a lockstep launch, the label table, and a list of kept tiles."""
    from flash_sinkhorn_b200.sinkhorn_solvers import (sinkhorn_flashstyle_alternating, sinkhorn_flashstyle_symmetric,
                                                      sinkhorn_flashstyle_symmetric_batched)
    d, eps = 24, 12.0
    r = np.random.default_rng(7)
    probs, wants = [], []
    for far in (1.0, 1e9, 1.0):
        x, y = _points(d, far, "x", seed=8)
        a, b = r.uniform(0.5, 1.5, N), r.uniform(0.5, 1.5, M)
        a[5] = 0.0
        a, b = (np.float32(w / w.sum()).astype(np.float64) for w in (a, b))
        wants.append(O.solve_symmetric(x, y, a, b, [eps] * 4))
        probs.append(tuple(dev(v) for v in (x, y, a, b)))
    got = sinkhorn_flashstyle_symmetric_batched(probs, use_epsilon_scaling=False, eps=eps, n_iters=4, allow_tf32=False)
    kx = _near(N, "x", "x")
    tol = 1e-5 * max((_norm(x[kx])**2).max(), (_norm(y)**2).max())
    for out, want in zip(got, wants):
        assert np.abs(host(out[0]) - want["f"])[kx].max() < tol and np.abs(host(out[1]) - want["g"]).max() < tol

    x, y = _points(d, 1e9, "x", seed=8)
    lx, ly = r.integers(0, 4, N), r.integers(0, 4, M)
    table = r.uniform(0.0, 5.0, (4, 4))
    table = np.float32(table + table.T).astype(np.float64)
    want = O.label_solve_symmetric(x, y, a, b, [eps] * 4, lx, ly, table)
    out = sinkhorn_flashstyle_symmetric(
        *(dev(v) for v in (x, y, a, b)), eps=eps, n_iters=4, use_epsilon_scaling=False, allow_tf32=False,
        label_x=torch.as_tensor(lx).cuda(), label_y=torch.as_tensor(ly).cuda(), label_cost_matrix=dev(table), lambda_y=1.0)
    assert np.abs(host(out[0]) - want["f"])[kx].max() < tol and np.abs(host(out[1]) - want["g"]).max() < tol

    mask = np.ones((4, 3), bool)
    mask[1, 2] = mask[3, 0] = False
    want = O.solve_alternating(x, y, a, b, [eps], 4, tile_mask=mask)
    out = sinkhorn_flashstyle_alternating(*(dev(v) for v in (x, y, a, b)), eps_list=[eps], iters_per_eps=4,
                                          tile_mask=torch.as_tensor(mask), allow_tf32=False)
    assert np.abs(host(out[0]) - want["f"])[kx].max() < tol and np.abs(host(out[1]) - want["g"]).max() < tol


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("d", [64, 520])
def test_a_non_finite_point_leaves_the_rows_of_its_own_cloud_alone(bad, d):
    """Rows of a soft-min do not meet: one that is not a number costs the others nothing, whatever their size."""
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    x, y = _points(d, 1.0, "x", seed=9)
    x, y = np.float32(1e6 * x).astype(np.float64), np.float32(1e-6 * y).astype(np.float64)
    x[5, 2] = bad
    bias = np.float32(np.random.default_rng(10).normal(size=M)).astype(np.float64)
    got = host(flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=0.5 * d, allow_tf32=False))
    x[5] = 0.0
    want = O.lse_update(x, y, bias, 0.5 * d)
    keep = _near(N, "x", "x")
    tol = 2.0 * 2.0**-18 * (_norm(x) * _norm(y).max() + 0.5 * d * np.abs(bias).max())
    assert (np.abs(got - want) < tol)[keep].all()


@pytest.mark.parametrize("column", range(40, 48))
@pytest.mark.parametrize("d,tf32", [(64, True), (64, False), (520, True)])
def test_a_target_that_is_not_a_number_counts_wherever_it_stands(column, d, tf32):
    """The soft-min of every source then has its sum at the floor of the logarithm (1e-40 of the largest other term) and the
    weighted sum is not a number, for every place of the target in a chunk of columns."""
    from flash_sinkhorn_b200.kernels.apply_flash import apply_plan_vec_flashstyle
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    x, y = _points(d, 1.0, "", seed=13)
    bias = np.float32(np.random.default_rng(14).normal(size=M)).astype(np.float64)
    eps = 0.5 * d
    top = np.delete(2.0 / eps * x @ y.T + bias, column, axis=1).max(1)
    y[column, 3] = np.nan
    got = host(flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=eps, allow_tf32=tf32))
    assert np.allclose(got / -eps, top + np.log(1e-40), rtol=0, atol=0.05)
    r = [dev(v) for v in (-(x * x).sum(1), np.zeros(M), np.full(N, -np.log(N)), np.full(M, -np.log(M)))]
    out = apply_plan_vec_flashstyle(dev(x), dev(y), *r, dev(np.ones(M)), eps=eps, axis=1, allow_tf32=tf32)
    assert torch.isnan(out).all()


@pytest.mark.parametrize("size", [1e-14, 1e-12, 1e-9])
def test_clouds_near_the_origin_keep_their_bits(size):
    """Tiny coordinates against a large cloud: the products are of order one and carry 22 bits."""
    from flash_sinkhorn_b200.kernels.sinkhorn_flashstyle_sqeuclid import flashsinkhorn_lse
    x, y = _points(48, 1.0, "", seed=11)
    x, y = np.float32(size * x).astype(np.float64), np.float32(y / size).astype(np.float64)
    bias = np.float32(np.random.default_rng(12).normal(size=M)).astype(np.float64)
    got = host(flashsinkhorn_lse(dev(x), dev(y), dev(bias), eps=24.0, allow_tf32=False))
    want = O.lse_update(x, y, bias, 24.0)
    tol = 2.0 * 2.0**-18 * (_norm(x) * _norm(y).max() + 24.0 * np.abs(bias).max())
    assert (np.abs(got - want) < tol).all()
