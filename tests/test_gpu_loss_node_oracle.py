"""Losses whose terms are one autograd node, and gradients that share launches, against the fp64 oracle."""
import numpy as np
import pytest
import torch

from gpu_util import dev, host, rel
from oracle import dense_sinkhorn as O

pytestmark = pytest.mark.gpu


def _clouds(B, n, m, d, seed=0):
    r = np.random.default_rng(seed)
    x, y = r.normal(size=(B, n, d)), 0.4 + r.normal(size=(B, m, d))
    x *= np.linspace(0.7, 1.3, B)[:, None, None]
    a, b = r.uniform(0.1, 1.1, (B, n)), r.uniform(0.1, 1.1, (B, m))
    return [np.float32(v).astype(np.float64) for v in (x, y, a / a.sum(1, keepdims=True), b / b.sum(1, keepdims=True))]


def _oracle(x, y, a, b, sched, debias, cs, rho_x, rho_y, labels):
    """Loss and its gradients to both clouds and both weights; sched(u, v): eps list of a term."""
    def term(u, v, wu, wv, lu, lv):
        eps = sched(u, v)
        if labels:
            kw = dict(lambda_x=0.7, lambda_y=1.3, cost_scale=cs)
            s = O.label_solve_symmetric(u, v, wu, wv, eps, lu, lv, labels[2], **kw)
            gu, gv = O.label_grad_xy(u, v, wu, wv, s["f_pre"], s["g_pre"], eps[-1], lu, lv, labels[2], **kw)
        else:
            s = O.solve_symmetric(u, v, wu, wv, eps, cost_scale=cs, rho_x=rho_x, rho_y=rho_y)
            gu, gv = O.grad_xy(u, v, wu, wv, s["f_pre"], s["g_pre"], eps[-1], cs)
        return [np.array(O.ot_cost(wu, wv, s["f"], s["g"], eps[-1], rho_x, rho_y)), gu, gv, s["f"], s["g"]]

    lx, ly = labels[:2] if labels else (None, None)
    out = term(x, y, a, b, lx, ly)
    if debias:
        for k, (w, own, lab) in enumerate(((a, x, lx), (b, y, ly))):
            val, gu, gv, f, g = term(own, own, w, w, lab, lab)
            out[0] = out[0] - 0.5 * val
            out[1 + k] = out[1 + k] - 0.5 * (gu + gv)
            out[3 + k] = out[3 + k] - 0.5 * (f + g)
    return out


FIXED = dict(eps=0.5, n_iters=10, use_epsilon_scaling=False)
CASES = [(FIXED, None, None), (dict(FIXED, half_cost=True), 2.0, None), (dict(FIXED), 2.0, 3.0),
         (dict(blur=0.4, scaling=0.6), None, None),
         (dict(blur=0.2, scaling=0.8, n_iters=6), None, None),     # schedules cut: every term ends at an eps of its own
         (dict(blur=0.2, scaling=0.8, n_iters=6), 2.0, 3.0)]


# exact products. Values: 1e-5 of the potentials' size (100 ulp of |x|^2); gradients to clouds: rounding of potentials over
# eps, 3e-4 as in the other tests of gradients against the oracle; those to weights are potentials
@pytest.mark.parametrize("kw,rho_x,rho_y", CASES)
@pytest.mark.parametrize("B,n,m,d,debias", [(1, 257, 300, 40, True), (3, 130, 97, 5, True), (3, 130, 97, 5, False)])
def test_values_and_gradients(B, n, m, d, debias, kw, rho_x, rho_y):
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = _clouds(B, n, m, d)
    cs = 0.5 if kw.get("half_cost") else 1.0

    def sched(u, v):
        if not kw.get("use_epsilon_scaling", True):
            return [kw["eps"]] * kw["n_iters"]
        return O.epsilon_schedule(O.max_diameter(u, v), kw["blur"], kw["scaling"])[: kw.get("n_iters")]

    loss = SamplesLoss("sinkhorn", debias=debias, allow_tf32=False, normalize=False, **kw,
                       reach_x=rho_x and rho_x ** 0.5, reach_y=rho_y and rho_y ** 0.5)
    args = [dev(v if B > 1 else v[0]).requires_grad_(True) for v in (a, x, b, y)]
    val = loss(*args)
    assert type(val.grad_fn).__name__ == "_SinkhornLossFnBackward"
    ga, gx, gb, gy = (host(t).reshape((B,) + t.shape[-1 - (k % 2):]) for k, t in
                      enumerate(torch.autograd.grad(val.sum(), args)))
    vals = np.atleast_1d(host(val))
    for i in range(B):
        want = _oracle(x[i], y[i], a[i], b[i], sched, debias, cs, rho_x, rho_y, None)
        size = (x[i] ** 2).sum(1).max() + (y[i] ** 2).sum(1).max()
        assert abs(vals[i] - want[0]) < 1e-5 * size
        assert rel(gx[i], want[1]) < 3e-4 and rel(gy[i], want[2]) < 3e-4
        assert np.abs(ga[i] - want[3]).max() < 1e-5 * size and np.abs(gb[i] - want[4]).max() < 1e-5 * size


@pytest.mark.parametrize("symmetric", [False, True])
def test_labelled_divergence(symmetric):
    from flash_sinkhorn_b200 import SamplesLoss
    n, m, V = 300, 260, 4
    x, y, a, b = (v[0] for v in _clouds(1, n, m, 16, seed=7))
    r = np.random.default_rng(3)
    table = np.float32(3.0 * r.random((V, V))).astype(np.float64)
    if symmetric:
        table = table + table.T
    lx, ly = r.integers(0, V, n), r.integers(0, V, m)
    want = _oracle(x, y, a, b, lambda u, v: [0.5] * 10, True, 1.0, None, None, (lx, ly, table))
    loss = SamplesLoss("sinkhorn", debias=True, allow_tf32=False, normalize=False, label_cost_matrix=dev(table), lambda_x=0.7,
                       lambda_y=1.3, **FIXED)
    args = [dev(v).requires_grad_(True) for v in (a, x, b, y)]
    val = loss(*args, label_x=torch.as_tensor(lx).cuda(), label_y=torch.as_tensor(ly).cuda())
    ga, gx, gb, gy = (host(t) for t in torch.autograd.grad(val, args))
    size = (x ** 2).sum(1).max() + (y ** 2).sum(1).max()
    assert abs(float(val.detach()) - want[0]) < 1e-5 * size
    assert rel(gx, want[1]) < 3e-4 and rel(gy, want[2]) < 3e-4
    assert np.abs(ga - want[3]).max() < 1e-5 * size and np.abs(gb - want[4]).max() < 1e-5 * size


@pytest.mark.parametrize("mode", ["fp32", "tf32"])
@pytest.mark.parametrize("B,n,m,d", [(1, 300, 1200, 30), (1, 700, 300, 64), (1, 500, 600, 128), (17, 40, 50, 64), (5, 257, 129, 100)])
def test_shared_gradients(monkeypatch, mode, B, n, m, d):
    """One problem (either form of the plan-times-matrix kernel) and several. The exponents are |x||y| cs 2 / eps < 10 in size:
    split products give them to 2^-22 of that (1e-5 of a weight, 2e-5 with the sums), TF32 ones to 2^-11 (5e-3)."""
    from flash_sinkhorn_b200 import _autograd, _lib
    monkeypatch.setenv("FLASH_SINKHORN_B200_PREC", mode)
    prec = _lib.precision_id(True)
    if not _lib.load().fs_grad_many_bytes(n, m, d, prec):
        pytest.skip("streamed operands")
    x, y, a, b = _clouds(B, n, m, d, seed=11)
    pot = np.float32(np.random.default_rng(1).normal(size=(B, m))).astype(np.float64)
    scales, eps = np.linspace(0.5, 2.0, B), [0.3 * d if i % 2 else 0.35 * d for i in range(B)]
    xd, yd, ad, bd, sd = (dev(v) for v in (x, y, a, b, scales))
    out = torch.empty_like(xd)
    _autograd._gradients_together([((xd, ad, ad.log(), n), (yd, bd, bd.log(), m), dev(pot), sd, out)], B, d, [eps], 0.5, prec,
                                  xd.device)
    for i in range(B):
        want, _ = O.grad_xy(x[i], y[i], a[i], b[i], np.zeros(n), pot[i], eps[i], 0.5, scales[i])
        assert rel(host(out[i]), want) < (2e-5 if mode == "fp32" else 5e-3)
