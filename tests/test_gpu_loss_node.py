"""Losses whose terms are one autograd node (debiased losses and batches) against the nodes of single terms, which
``threshold=0`` (an early stop that never comes) keeps: values, gradients to clouds and weights, second order, refusals."""
import pytest
import torch

from gpu_util import dev  # noqa: F401

pytestmark = pytest.mark.gpu


def _inputs(B, n, m, d, seed=0):
    g = torch.Generator().manual_seed(seed)
    x = torch.randn(B, n, d, generator=g)
    y = 0.4 + torch.randn(B, m, d, generator=g)
    a, b = (torch.softmax(torch.randn(B, k, generator=g), 1) for k in (n, m))
    return [t.cuda() for t in (x, y, a, b)]


def _err(u, v):
    return float((u.double() - v.double()).norm() / v.double().norm().clamp(min=1e-30))


CASES = [dict(eps=0.5, n_iters=12, use_epsilon_scaling=False),
         dict(eps=0.5, n_iters=9, use_epsilon_scaling=False, last_extrapolation=False, reach=2.0, half_cost=True),
         dict(eps=0.5, n_iters=9, use_epsilon_scaling=False, reach_x=1.5),
         dict(eps=0.5, n_iters=9, use_epsilon_scaling=False, reach_x=1.5, reach_y=2.5),
         dict(blur=0.4, scaling=0.6)]


# fp32-exact products: values agree to 1e-5, gradients to 3e-4 (rounding of potentials over eps, as in the other tests of
# this suite); the terms of one node are summed in another order
@pytest.mark.parametrize("kw", CASES)
@pytest.mark.parametrize("debias", [True, False])
@pytest.mark.parametrize("B,n,m,d", [(3, 130, 97, 5), (1, 257, 300, 40), (2, 60, 1, 3)])
def test_against_single_terms(B, n, m, d, debias, kw):
    from flash_sinkhorn_b200 import SamplesLoss
    if kw.get("blur") and m == 1:
        kw = dict(kw, n_iters=3, eps=0.5, use_epsilon_scaling=False)  # one point has no diameter
    x, y, a, b = _inputs(B, n, m, d)
    one = SamplesLoss("sinkhorn", debias=debias, allow_tf32=False, normalize=False, **kw)
    ref = SamplesLoss("sinkhorn", debias=debias, allow_tf32=False, normalize=False, threshold=0.0, **kw)
    w = torch.linspace(0.5, 1.5, B, device="cuda")
    outs = []
    for loss in (one, ref):
        args = [t.clone().requires_grad_(True) for t in (a, x, b, y)]
        val = loss(*args)
        outs.append((val, torch.autograd.grad((val * w).sum(), args)))
    assert outs[0][0].shape == (B,)
    scale = float(outs[1][0].abs().max()) + float((a * (x * x).sum(-1)).sum(-1).max())
    assert float((outs[0][0] - outs[1][0]).abs().max()) < 1e-5 * scale
    for u, v in zip(*(o[1] for o in outs)):
        assert u.shape == v.shape and _err(u, v) < 3e-4
    # the same loss, item by item
    for i in range(B):
        xi = x[i].clone().requires_grad_(True)
        vi = one(a[i], xi, b[i], y[i])
        assert vi.dim() == 0 and abs(float(vi) - float(outs[1][0][i])) < 1e-5 * scale
        assert _err(w[i] * torch.autograd.grad(vi, xi)[0], outs[1][1][1][i]) < 3e-4


def test_strided_half_and_shared_inputs():
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = _inputs(2, 150, 140, 6, seed=3)
    kw = dict(eps=0.5, n_iters=8, use_epsilon_scaling=False, debias=True, allow_tf32=False)
    one, ref = SamplesLoss("sinkhorn", **kw), SamplesLoss("sinkhorn", threshold=0.0, **kw)
    wide = torch.randn(150, 2, 12, device="cuda").requires_grad_(True)
    xs = wide.transpose(0, 1)[..., ::2]  # strides of its own in every axis
    half = y.half().requires_grad_(True)
    got, want = (torch.autograd.grad(f(xs, half).sum(), (wide, half)) for f in (one, ref))
    assert got[1].dtype == torch.float16
    assert _err(got[0], want[0]) < 3e-4 and _err(got[1], want[1]) < 2e-3
    same = x.clone().requires_grad_(True)  # both clouds are one tensor
    got, want = (torch.autograd.grad(f(same, same).sum(), same)[0] for f in (one, ref))
    assert float((got - want).abs().max()) < 1e-6
    big = x.double().requires_grad_(True)  # the value is computed in fp32, the gradient refused
    val = one(big, y.double())
    with pytest.raises(ValueError, match="Unsupported dtype"):
        val.sum().backward()


def test_second_order():
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = _inputs(2, 120, 110, 4, seed=5)
    v = torch.randn_like(x)
    kw = dict(eps=1.0, n_iters=30, use_epsilon_scaling=False, allow_tf32=False)
    outs = []
    for loss in (SamplesLoss("sinkhorn", **kw), SamplesLoss("sinkhorn", threshold=0.0, **kw)):
        xs = x.clone().requires_grad_(True)
        (gx,) = torch.autograd.grad((loss(xs, y) * torch.tensor([1.0, 2.0], device="cuda")).sum(), xs, create_graph=True)
        outs.append(torch.autograd.grad((gx * v).sum(), xs)[0])
    assert _err(*outs) < 1e-3  # each ends where its conjugate gradients meet rtol = 1e-6
    xs = x.clone().requires_grad_(True)
    (gx,) = torch.autograd.grad(SamplesLoss("sinkhorn", debias=True, **kw)(xs, y).sum(), xs, create_graph=True)
    with pytest.raises(NotImplementedError):
        torch.autograd.grad((gx * v).sum(), xs)


@pytest.mark.parametrize("symmetric", [False, True])
@pytest.mark.parametrize("n,m,V", [(300, 260, 4), (2900, 2701, 7)])
def test_labels_in_lockstep(n, m, V, symmetric):
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = (t[0] for t in _inputs(1, n, m, 16, seed=7))
    g = torch.Generator().manual_seed(1)
    table = 3.0 * torch.rand(V, V, generator=g).cuda()
    if symmetric:
        table = table + table.t()
    lx, ly = torch.randint(0, V, (n,), generator=g).cuda(), torch.randint(0, V, (m,), generator=g).cuda()
    kw = dict(eps=0.5, n_iters=10, use_epsilon_scaling=False, debias=True, allow_tf32=False, label_cost_matrix=table, lambda_x=0.7,
              lambda_y=1.3)
    outs = []
    for extra in ({}, dict(threshold=0.0)):
        args = [t.clone().requires_grad_(True) for t in (a, x, b, y)]
        val = SamplesLoss("sinkhorn", **kw, **extra)(*args, label_x=lx, label_y=ly)
        outs.append((val, torch.autograd.grad(val, args)))
    assert abs(float(outs[0][0]) - float(outs[1][0])) < 1e-5 * (abs(float(outs[1][0])) + float((x * x).sum(1).max()))
    for u, v in zip(outs[0][1], outs[1][1]):
        assert _err(u, v) < 3e-4
    with pytest.raises(ValueError, match="label_y values"):
        SamplesLoss("sinkhorn", **kw)(a, x, b, y, label_x=lx, label_y=ly + V)
    labels = lx.to(torch.int32)  # used as they were at the call
    xs = x.clone().requires_grad_(True)
    val = SamplesLoss("sinkhorn", **kw)(a, xs, b, y, label_x=labels, label_y=ly)
    labels.fill_(1 << 20)
    assert _err(torch.autograd.grad(val, xs)[0], outs[1][1][1]) < 3e-4


@pytest.mark.parametrize("mode", ["fp32", "tf32"])
@pytest.mark.parametrize("B,n,m,d", [(9, 300, 200, 12), (17, 40, 50, 64), (1, 2300, 4100, 64), (2, 1, 1, 2), (3, 129, 257, 100),
                                     (1, 700, 300, 128)])
def test_gradients_that_share_launches(monkeypatch, mode, B, n, m, d):
    """Against the same gradients one by one (more items than a call takes, column shares, one point, plans of one and two
    128-row halves, one item with a far point). Same products and normalisers; sums in another order: 2e-5 of the
    gradient's size in the exact mode, of TF32 weights up to 2^-11."""
    from flash_sinkhorn_b200 import _autograd, _lib
    monkeypatch.setenv("FLASH_SINKHORN_B200_PREC", mode)
    lib = _lib.load()
    prec = _lib.precision_id(True)
    if not lib.fs_grad_many_bytes(n, m, d, prec):
        pytest.skip("streamed operands")
    x, y, a, b = _inputs(B, n, m, d, seed=11)
    if B == 3:
        x[1, 0] *= 1e9
    la, lb, pot = a.log(), b.log(), torch.randn(B, m, device="cuda")
    scales = torch.linspace(0.5, 2.0, B, device="cuda")
    out, want = torch.empty_like(x), torch.empty_like(x)
    _autograd._gradients_together([((x, a, la, n), (y, b, lb, m), pot, scales, out)], B, d, 0.3 * d, 0.5, prec, x.device)
    ws = _lib.workspace(_lib.OP_GRAD, n, m, d, prec, x.device)
    f = torch.zeros(n, device="cuda")
    for i in range(B):
        _lib.call("fs_grad", x.device, _lib.ptr(x[i]), _lib.ptr(y[i]), n, m, d, _lib.ptr(a[i]), _lib.ptr(b[i]), _lib.ptr(la[i]),
                  _lib.ptr(lb[i]), _lib.ptr(f), _lib.ptr(pot[i]), _lib.ptr(scales[i]), _lib.ptr(want[i]), None, 0.3 * d, 0.5, prec,
                  _lib.ptr(ws), ws.numel(), _lib.stream_ptr(x.device), None)
    keep = x.abs().amax(dim=-1) < 1e6
    assert _err(out[keep], want[keep]) < (2e-5 if mode == "fp32" else 5e-4)
    assert _err(out[~keep], want[~keep]) < 1e-3 or bool(keep.all())
    assert lib.fs_device_error() == 0


@pytest.mark.parametrize("B,debias", [(90, True), (257, False)])
def test_batches_beyond_one_library_call(B, debias):
    """More problems (270, 257) than the library solves in one call (256): every item as on its own."""
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = _inputs(B, 20, 17, 3, seed=9)
    loss = SamplesLoss("sinkhorn", eps=0.5, n_iters=6, use_epsilon_scaling=False, debias=debias, allow_tf32=False)
    xs = x.clone().requires_grad_(True)
    vals = loss(a, xs, b, y)
    (gx,) = torch.autograd.grad(vals.sum(), xs)
    for i in (0, 79, 80, B - 1):
        xi = x[i].clone().requires_grad_(True)
        vi = loss(a[i], xi, b[i], y[i])
        assert abs(float(vi.detach()) - float(vals[i].detach())) < 1e-5 * float((x[i] * x[i]).sum(-1).max())
        assert _err(gx[i], torch.autograd.grad(vi, xi)[0]) < 3e-4


@pytest.mark.parametrize("kw", [dict(), dict(reach=2.0), dict(label_cost_matrix=True, lambda_y=1.0)])
@pytest.mark.parametrize("single,debias", [(True, True), (False, True), (False, False)])
def test_terms_that_end_at_different_eps(single, debias, kw):
    """``n_iters`` cuts annealed schedules that start at the diameters of their clouds: every term (and item) has an eps of its
    own, and the loss stays one node. Tolerances as in test_against_single_terms."""
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = _inputs(3, 140, 150, 5, seed=13)
    x = x * torch.tensor([1.0, 1.4, 0.6], device="cuda")[:, None, None]
    if single:
        x, y, a, b = (t[0] for t in (x, y, a, b))
    labels = {}
    if kw.get("label_cost_matrix"):
        if not single:
            pytest.skip("labels go item by item")
        g = torch.Generator().manual_seed(2)
        table = torch.rand(3, 3, generator=g).cuda()
        kw = dict(kw, label_cost_matrix=table + table.t())
        labels = {k: torch.randint(0, 3, (n,), generator=g).cuda() for k, n in (("label_x", 140), ("label_y", 150))}
    kw = dict(blur=0.2, scaling=0.8, n_iters=5, debias=debias, allow_tf32=False, normalize=False, **kw)
    outs = []
    for extra in ({}, dict(threshold=0.0)):
        args = [t.clone().requires_grad_(True) for t in (a, x, b, y)]
        val = SamplesLoss("sinkhorn", **kw, **extra)(*args, **labels)
        outs.append((val.detach(), torch.autograd.grad(val.sum(), args)))
        assert (type(val.grad_fn).__name__ == "_SinkhornLossFnBackward") == (not extra)
    assert float((outs[0][0] - outs[1][0]).abs().max()) < 1e-5 * float((x * x).sum(-1).max())
    for u, v in zip(outs[0][1], outs[1][1]):
        assert _err(u, v) < 3e-4


def test_label_table_of_the_call():
    """A table that is overwritten between the loss and its gradient, also by one that is not symmetric any more."""
    from flash_sinkhorn_b200 import SamplesLoss
    x, y, a, b = (t[0] for t in _inputs(1, 300, 260, 16, seed=7))
    g = torch.Generator().manual_seed(1)
    first = 3.0 * torch.rand(4, 4, generator=g).cuda()
    first = first + first.t()
    lx, ly = torch.randint(0, 4, (300,), generator=g).cuda(), torch.randint(0, 4, (260,), generator=g).cuda()
    grads = []
    for overwrite in (False, True):
        table = first.clone()
        loss = SamplesLoss("sinkhorn", eps=0.5, n_iters=10, use_epsilon_scaling=False, debias=True, label_cost_matrix=table,
                           lambda_x=0.7, lambda_y=1.3)
        xs = x.clone().requires_grad_(True)
        val = loss(a, xs, b, y, label_x=lx, label_y=ly)
        if overwrite:
            table.copy_(torch.arange(16.0).reshape(4, 4))
        grads.append(torch.autograd.grad(val, xs)[0])
    assert _err(grads[1], grads[0]) < 1e-6  # the same numbers go in


@pytest.mark.parametrize("kw", [dict(), dict(reach=2.0), dict(reach_x=2.0)])
@pytest.mark.parametrize("single,debias", [(True, True), (False, True), (False, False)])
def test_cloud_against_itself(monkeypatch, single, debias, kw):
    """The same cloud and weights on both sides: OT(x,y) is a self-transport problem too (of equal relaxations), with the values and
    gradients of a copy of the cloud."""
    from flash_sinkhorn_b200 import SamplesLoss, samples_loss
    x, _, a, _ = _inputs(2, 300, 1, 20, seed=5)
    if single:
        x, a = x[0], a[0]
    outs, solves, solve = [], [], samples_loss.solve_loss_terms
    monkeypatch.setattr(samples_loss, "solve_loss_terms", lambda *args, **kws: solves.append(solve(*args, **kws)) or solves[-1])
    loss = SamplesLoss("sinkhorn", eps=3.0, n_iters=12, use_epsilon_scaling=False, debias=debias, normalize=False, allow_tf32=False, **kw)
    for copy in (False, True):
        u, w = x.clone().requires_grad_(True), a.clone().requires_grad_(True)
        val = loss(w, u, w.clone() if copy else w, u.clone() if copy else u)
        outs.append((val.detach(), torch.autograd.grad(val.sum(), (u, w))))
        f, g = solves[-1][0][:2]
        assert (f is g) == (not copy and "reach_x" not in kw)
    size = float((x * x).sum(-1).max())
    assert float((outs[0][0] - outs[1][0]).abs().max()) < 1e-5 * size
    (gx, ga), (want_gx, want_ga) = outs[0][1], outs[1][1]
    # a debiased loss is at its minimum: what the terms' gradients leave is rounding of 4 w |x|, in weights that of a potential
    assert float((gx - want_gx).abs().max()) < 3e-4 * 4 * float(a.max()) * size ** 0.5
    assert float((ga - want_ga).abs().max()) < 2e-5 * size
