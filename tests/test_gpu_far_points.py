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
