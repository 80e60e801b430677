"""The work that users have this package do, as a list of cases with the range that each one stands for.

``listed()`` names the cases, ``draw()`` gives further ones from the same ranges, ``prepare()`` makes what a program
has in hand before the call, ``run()`` is one pass through the public entry points and returns its whole result,
``work()`` counts what a pass cannot do without and ``tolerance()`` says how far two correct implementations of the
same precision may be apart. Everything is synthetic: Gaussian clouds, points of a mixture, rows on the unit sphere.
"""
from __future__ import annotations

import math

import torch

from flash_sinkhorn_b200 import SamplesLoss
from flash_sinkhorn_b200.c_transform import c_transform_fwd
from flash_sinkhorn_b200.kernels.apply_flash import apply_plan_mat_flashstyle, apply_plan_vec_flashstyle
from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_alternating

# ---------------------------------------------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------------------------------------------


def listed():
    return [
        # Shape matching of two small 3-D scans with the constructor's defaults (annealed eps, debiased): a loss in
        # a registration loop. The GPU work is tiny; launches and host time are what a user waits for.
        dict(name="scan3d_annealed", kind="loss", data="cube", n=500, m=450, d=3, anneal=True, blur=0.05, debias=True,
             tf32=True),
        # A mini-batch of small clouds, (B, N, D) form: feature-distribution loss inside a network's training step.
        dict(name="minibatch", kind="batch", batch=8, n=600, m=500, d=32, eps=1.0, iters=30, debias=True, tf32=True),
        # The debiased divergence between two feature clouds at the size that tests and benchmark use for parity.
        dict(name="divergence_4k", kind="loss", data="gauss", n=4096, m=4096, d=64, eps=0.01, iters=100, debias=True,
             tf32=True),
        # The headline benchmark: the same divergence at 50,000 points a side.
        dict(name="divergence_50k", kind="loss", data="gauss", n=50000, m=50000, d=64, eps=0.01, iters=100,
             debias=True, tf32=True),
        # Exact-fp32 products, Gauss-Seidel backend, both marginals relaxed, gradients to both clouds: domain
        # adaptation with outliers, 10 iterations as in the published table of the alternating solver.
        dict(name="exact_unbalanced", kind="loss", data="gauss", n=10007, m=8001, d=64, eps=1.0, iters=10,
             backend="alternating", reach=4.0, debias=False, tf32=False, grad_y=True),
        # Wide rows with early stopping (1,000 images of 784 pixels is the documented example): the solver runs far
        # fewer steps than it was given.
        dict(name="early_stop_d784", kind="loss", data="sphere", n=1000, m=1000, d=784, eps=0.1, iters=100,
             threshold=1e-4, debias=False, tf32=True),
        # Embedding clouds, semi-unbalanced, half cost: the large contraction, bound by the tensor cores.
        dict(name="embedding_d2048", kind="loss", data="sphere", n=16384, m=16384, d=2048, eps=0.0025, iters=50,
             reach_x=1.0, half_cost=True, debias=False, tf32=True),
        # Large 3-D clouds of a mixture, annealed alternating solve that skips 128 x 128 tiles of far-apart parts.
        dict(name="tiles3d_annealed", kind="tiles", n=200000, m=190017, blur=0.02, per_stage=4, tf32=True),
        # Dataset distance with labels: the ground cost has a class-to-class table.
        dict(name="labelled_otdd", kind="loss", data="gauss", n=6000, m=5003, d=64, eps=0.5, iters=50, debias=True,
             tf32=True, classes=10, lambda_y=1.0),
        # Second order: loss, gradient and Hessian-vector product of a Newton-type point-cloud flow (the products of
        # the second order are always fp32-exact).
        dict(name="newton_hvp", kind="hvp", n=8192, m=6000, d=64, eps=4.0, iters=60, cg=30, tf32=True),
        # Transporting features and one weight vector with a plan that is at hand (exact products, the default).
        dict(name="plan_apply", kind="plan", n=20000, m=15001, d=64, eps=2.0, tf32=False),
        # The hard c-transform of the semi-dual: nearest target under a price vector, values and indices.
        dict(name="c_transform", kind="ctrans", n=30000, m=20001, d=64, tf32=True),
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _fit(rng, n, m, weight, limit=1.0e12):
    """Shrinks (n, m) until weight * n * m stays below `limit` (score entries, or flops, of the largest listed)."""
    while weight * float(n) * m > limit:
        n, m = max(64, int(n * rng.uniform(0.6, 0.9))), max(64, int(m * rng.uniform(0.6, 0.9)))
    return n, m


def draw(rng):
    kind = rng.choice(["scan", "loss", "loss", "exact", "batch", "early", "wide", "tiles", "labels", "hvp", "plan",
                       "ctrans"])
    if kind == "scan":
        return dict(kind="loss", data="cube", n=_log_uniform(rng, 150, 6000), m=_log_uniform(rng, 150, 6000),
                    d=rng.choice([2, 3, 3, 6]), anneal=True, blur=rng.choice([0.02, 0.05, 0.1]),
                    debias=rng.random() < 0.7, tf32=True)
    if kind == "loss":
        n, d = _log_uniform(rng, 300, 50000), _log_uniform(rng, 8, 256)
        m = max(64, min(50000, int(n * rng.uniform(0.5, 1.6))))
        iters = rng.randint(20, 100)
        n, m = _fit(rng, n, m, 4.0 * iters * max(1.0, d / 64.0))
        return dict(kind="loss", data="gauss", n=n, m=m, d=d, eps=d * rng.choice([0.0002, 0.002, 0.01]), iters=iters,
                    debias=rng.random() < 0.6, tf32=True)
    if kind == "exact":
        n, d = _log_uniform(rng, 300, 20000), _log_uniform(rng, 8, 160)
        m = max(64, int(n * rng.uniform(0.5, 1.6)))
        iters = rng.randint(5, 40)
        n, m = _fit(rng, n, m, 6.0 * iters * max(1.0, d / 64.0))
        return dict(kind="loss", data="gauss", n=n, m=m, d=d, eps=d * rng.choice([0.01, 0.02]), iters=iters,
                    backend=rng.choice(["alternating", "symmetric"]), reach=4.0, debias=False, tf32=False,
                    grad_y=rng.random() < 0.5)
    if kind == "batch":
        return dict(kind="batch", batch=rng.randint(2, 16), n=_log_uniform(rng, 100, 2000),
                    m=_log_uniform(rng, 100, 2000), d=(d := rng.randint(3, 96)), eps=d / 32.0,
                    iters=rng.randint(10, 50), debias=rng.random() < 0.7, tf32=True)
    if kind == "early":
        return dict(kind="loss", data="sphere", n=_log_uniform(rng, 400, 5000), m=_log_uniform(rng, 400, 5000),
                    d=rng.choice([96, 128, 300, 512, 784, 1000]), eps=0.1, iters=100, threshold=1e-4, debias=False,
                    tf32=True)
    if kind == "wide":
        n, d = _log_uniform(rng, 2000, 16384), _log_uniform(rng, 300, 2048)
        m = max(256, min(16384, int(n * rng.uniform(0.6, 1.4))))
        iters = rng.randint(10, 50)
        return dict(kind="loss", data="sphere", n=n, m=m, d=d, eps=rng.choice([0.0025, 0.01]), iters=iters,
                    reach_x=1.0, half_cost=True, debias=False, tf32=True)
    if kind == "tiles":
        n = _log_uniform(rng, 20000, 200000)
        return dict(kind="tiles", n=n, m=max(10000, min(200000, int(n * rng.uniform(0.7, 1.3)))),
                    blur=rng.choice([0.02, 0.05]), per_stage=rng.randint(2, 4), tf32=True)
    if kind == "labels":
        d = _log_uniform(rng, 8, 96)
        return dict(kind="loss", data="gauss", n=_log_uniform(rng, 500, 10000), m=_log_uniform(rng, 500, 10000), d=d,
                    eps=d / 128.0, iters=rng.randint(20, 50), debias=rng.random() < 0.5, tf32=True,
                    classes=rng.randint(2, 10), lambda_y=rng.choice([0.5, 1.0]))
    if kind == "hvp":
        d = _log_uniform(rng, 8, 128)
        return dict(kind="hvp", n=_log_uniform(rng, 500, 12000), m=_log_uniform(rng, 500, 12000), d=d, eps=d / 16.0,
                    iters=rng.randint(40, 60), cg=rng.randint(10, 30), tf32=rng.random() < 0.5)
    if kind == "plan":
        d = _log_uniform(rng, 8, 200)
        return dict(kind="plan", n=_log_uniform(rng, 500, 30000), m=_log_uniform(rng, 500, 30000), d=d, eps=d / 32.0,
                    tf32=rng.random() < 0.3)
    return dict(kind="ctrans", n=_log_uniform(rng, 500, 50000), m=_log_uniform(rng, 500, 50000),
                d=_log_uniform(rng, 16, 128), tf32=rng.random() < 0.8)


# ---------------------------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------------------------


def _clouds(case, gen):
    n, m, d = case["n"], case["m"], case["d"]
    kw = dict(device="cuda", generator=gen)
    if case["data"] == "cube":     # scans scaled into the unit cube, the target slightly deformed
        return torch.rand(n, d, **kw), 0.1 + 0.8 * torch.rand(m, d, **kw)
    x, y = torch.randn(n, d, **kw), torch.randn(m, d, **kw)
    if case["data"] == "sphere":   # normalised embeddings
        return torch.nn.functional.normalize(x, dim=1), torch.nn.functional.normalize(y, dim=1)
    return x, 0.5 + y


def _weights(n, gen):
    w = torch.rand(n, device="cuda", generator=gen) + 0.1
    return w / w.sum()


def _loss_module(case, table=None):
    kw = dict(blur=case.get("blur", math.sqrt(case.get("eps", 0.0025))), debias=case["debias"],
              allow_tf32=case["tf32"], backend=case.get("backend", "symmetric"), half_cost=case.get("half_cost", False),
              reach=case.get("reach"), reach_x=case.get("reach_x"), threshold=case.get("threshold"),
              label_cost_matrix=table, lambda_y=case.get("lambda_y", 0.0), hvp_max_cg_iter=case.get("cg", 300))
    if not case.get("anneal", False):
        kw.update(use_epsilon_scaling=False, eps=case["eps"], n_iters=case["iters"])
    return SamplesLoss("sinkhorn", **kw)


def _mixture(n, centres, gen):
    """n points of a 64-part mixture in 3-D, sorted by part, and the part of each."""
    part = torch.sort(torch.randint(0, centres.shape[0], (n,), device="cuda", generator=gen)).values
    return centres[part] + 0.05 * torch.randn(n, 3, device="cuda", generator=gen), part


def _near_tiles(centres, part_x, part_y, radius=0.5):
    """Tile pairs some of whose parts have centres closer than `radius` (parts are sorted: a tile is a range)."""
    near = (torch.cdist(centres, centres) < radius).long()
    k = centres.shape[0]
    pre = torch.zeros(k + 1, k + 1, dtype=torch.long, device=centres.device)
    pre[1:, 1:] = near.cumsum(0).cumsum(1)

    def bounds(part):
        last = torch.clamp(torch.arange(127, part.shape[0] + 127, 128, device=part.device), max=part.shape[0] - 1)
        return part[::128], part[last] + 1

    (x0, x1), (y0, y1) = bounds(part_x), bounds(part_y)
    return (pre[x1][:, y1] - pre[x0][:, y1] - pre[x1][:, y0] + pre[x0][:, y0]) > 0


def _soft_min(rows, cols, pot, log_w, eps):
    """-eps * log sum_j exp((2 rows.cols + pot_j)/eps + log_w_j), by blocks of rows (plain torch)."""
    bias = pot / eps + log_w
    return torch.cat([-eps * torch.logsumexp((2.0 / eps) * (r @ cols.T) + bias, dim=1) for r in rows.split(2048)])


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    s = dict(case=case)
    if kind == "loss":
        x, y = _clouds(case, gen)
        s.update(x=x.requires_grad_(True), y=y.requires_grad_(bool(case.get("grad_y"))),
                 a=_weights(case["n"], gen), b=_weights(case["m"], gen))
        table = None
        if case.get("classes"):
            k = case["classes"]
            table = 4.0 * torch.rand(k, k, device="cuda", generator=gen)
            table = 0.5 * (table + table.T)
            table.fill_diagonal_(0.0)
            s.update(label_x=torch.randint(0, k, (case["n"],), device="cuda", generator=gen),
                     label_y=torch.randint(0, k, (case["m"],), device="cuda", generator=gen))
        s["loss"] = _loss_module(case, table)
    elif kind == "batch":
        shape = (case["batch"], case["n"], case["d"])
        x = torch.randn(*shape, device="cuda", generator=gen)
        y = 0.5 + torch.randn(case["batch"], case["m"], case["d"], device="cuda", generator=gen)
        s.update(x=x.requires_grad_(True), y=y, loss=_loss_module(case))
    elif kind == "tiles":
        centres = 2.0 * torch.rand(64, 3, device="cuda", generator=gen) - 1.0
        (x, px), (y, py) = _mixture(case["n"], centres, gen), _mixture(case["m"], centres, gen)
        s.update(x=x, y=y, a=torch.full((case["n"],), 1.0 / case["n"], device="cuda"),
                 b=torch.full((case["m"],), 1.0 / case["m"], device="cuda"), mask=_near_tiles(centres, px, py),
                 eps_list=_stages(case))
    elif kind == "hvp":
        x, y = _clouds(dict(case, data="gauss"), gen)
        s.update(x=x.requires_grad_(True), y=y, loss=_loss_module(dict(case, debias=False)),
                 v=torch.randn(case["n"], case["d"], device="cuda", generator=gen))
    elif kind == "plan":
        x, y = _clouds(dict(case, data="gauss"), gen)
        la, lb = _weights(case["n"], gen).log(), _weights(case["m"], gen).log()
        g = _soft_min(y, x, -(x * x).sum(1), la, case["eps"])
        f = _soft_min(x, y, g, lb, case["eps"])
        s.update(x=x, y=y, f=f, g=g, la=la, lb=lb,
                 mat=torch.randn(case["m"], case["d"], device="cuda", generator=gen),
                 vec=torch.rand(case["n"], device="cuda", generator=gen))
    else:
        x, y = _clouds(dict(case, data="gauss"), gen)
        s.update(x=x, y=y, psi=torch.randn(case["m"], device="cuda", generator=gen))
    return s


def _stages(case):
    """eps of the annealed alternating solve: from the squared extent of the mixture down to blur**2, by quarters."""
    out, e = [], 12.0
    while e > case["blur"] ** 2:
        out.append(e)
        e *= 0.25
    return out + [case["blur"] ** 2]


# ---------------------------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------------------------


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "loss":
        labels = dict(label_x=s["label_x"], label_y=s["label_y"]) if case.get("classes") else {}
        val = s["loss"](s["a"], s["x"], s["b"], s["y"], **labels)
        wrt = [s["x"]] + ([s["y"]] if case.get("grad_y") else [])
        return dict(loss=val, grads=torch.autograd.grad(val, wrt))
    if kind == "batch":
        val = s["loss"](s["x"], s["y"])
        return dict(loss=val, grads=torch.autograd.grad(val.sum(), [s["x"]]))
    if kind == "tiles":
        return sinkhorn_flashstyle_alternating(
            s["x"], s["y"], s["a"], s["b"], eps_list=s["eps_list"], iters_per_eps=case["per_stage"],
            tile_mask=s["mask"], allow_tf32=case["tf32"])
    if kind == "hvp":
        val = s["loss"](s["x"], s["y"])
        (grad,) = torch.autograd.grad(val, s["x"], create_graph=True)
        (hv,) = torch.autograd.grad((grad * s["v"]).sum(), s["x"])
        return dict(loss=val, grad=grad, hvp=hv)
    if kind == "plan":
        args = (s["x"], s["y"], s["f"], s["g"], s["la"], s["lb"])
        return dict(
            moved=apply_plan_mat_flashstyle(*args, s["mat"], eps=case["eps"], axis=1, allow_tf32=case["tf32"]),
            mass=apply_plan_vec_flashstyle(*args, s["vec"], eps=case["eps"], axis=0, allow_tf32=case["tf32"]))
    values, index = c_transform_fwd(s["x"], s["y"], s["psi"], allow_tf32=case["tf32"])
    return dict(values=values, index=index)


# ---------------------------------------------------------------------------------------------------------------
# What a pass needs, and how exact it is
# ---------------------------------------------------------------------------------------------------------------


def _steps(case):
    """Potential updates per side of one solve (the early-stop cases meet their threshold after about 20)."""
    if case.get("anneal"):
        stages = max(0.0, math.log(0.97 * math.sqrt(case["d"]) / case["blur"]) / math.log(2.0))
        return int(math.ceil(stages)) + 4
    if case.get("threshold") is not None:
        return min(case["iters"], 20) + 2
    return case["iters"] + (2 if case.get("backend", "symmetric") == "symmetric" else 0)


def work(case):
    """Bytes: each input read once, each result written once. Flops: two per coordinate and score entry, once per
    soft-min (one per step in a self-transport term, whose two potentials are equal) and plan application, twice
    where a plan meets a matrix."""
    kind, n, m = case["kind"], float(case["n"]), float(case["m"])
    d = 3 if kind == "tiles" else case["d"]
    clouds = 4.0 * (n + m) * d
    if kind in ("loss", "batch"):
        steps, grads = _steps(case), 2.0 if case.get("grad_y") else 1.0
        entries = (2.0 * steps + 2.0 * grads) * n * m
        if case["debias"]:
            entries += (steps + 4.0) * n * n + steps * m * m
        k = case.get("batch", 1)
        return dict(bytes=k * (clouds + 4.0 * (n + m) + 4.0 * n * d * grads), flops=k * 2.0 * d * entries)
    if kind == "tiles":
        kept = 0.06  # share of the tiles that the mixture keeps
        return dict(bytes=clouds + 12.0 * (n + m) + n * m / 128.0**2,
                    flops=2.0 * d * 2.0 * case["per_stage"] * len(_stages(case)) * kept * n * m)
    if kind == "hvp":
        passes = 2.0 * (_steps(case) + 1) + 2.0 + 6.0 + 2.0 * 4.0 + 2.0 * 8  # solve, gradient, vectors, matrices, CG
        return dict(bytes=clouds + 12.0 * n * d, flops=2.0 * d * passes * n * m)
    if kind == "plan":
        return dict(bytes=clouds + 4.0 * (n + m) * d + 16.0 * (n + m), flops=2.0 * d * 3.0 * n * m)
    return dict(bytes=clouds + 4.0 * m + 12.0 * n, flops=2.0 * d * n * m)


def tolerance(case):
    """About four times what the same pass shows when points and coordinates come in another order, which changes
    every fp32 sum and nothing else: 2e-4 (largest entry 6e-3) on a gradient at eps = 0.01, 4e-4 (8e-3) with annealed
    eps in the unit cube, 2e-5 (3e-4) with exact products, 6e-5 (2e-3) on a Hessian-vector product, 5e-6 (7e-5) on a
    plan application, 2e-7 (9e-7) on a c-transform, 5e-8 (5e-7) on potentials. Weights that are rounded to TF32 before
    they meet a matrix move by 2**-12 when a normaliser moves, so TF32 plan applications get 1e-3."""
    kind = case["kind"]
    if kind == "hvp":
        return {"rel": 5e-4, "max": 1e-2}
    if kind == "plan":
        return {"rel": 1e-3, "max": 2e-2} if case["tf32"] else {"rel": 3e-5, "max": 5e-4}
    if kind == "ctrans":
        return {"rel": 2e-6, "max": 2e-5, "differ": 5e-4}
    if kind == "tiles":
        return {"rel": 1e-6, "max": 1e-5}
    return {"rel": 2e-3, "max": 4e-2} if case["tf32"] else {"rel": 6e-5, "max": 1.5e-3}


# ---------------------------------------------------------------------------------------------------------------
# The same results in 64 bits
# ---------------------------------------------------------------------------------------------------------------


def _lse(dots, scale, bias, axis):
    """log sum exp(scale * dots + bias) along an axis, the bias running along that axis, by blocks of rows."""
    if axis == 1:
        return torch.cat([torch.logsumexp(scale * r + bias, dim=1) for r in dots.split(2048)])
    return torch.cat([torch.logsumexp(scale * c + bias[:, None], dim=0) for c in dots.split(2048, dim=1)])


def _solve(case, x, y, a, b, eps_list, extra=0.0):
    """Potentials (f, g) and those before the last extrapolation, by the textbook iteration. `extra` is added to the
    products x.y (the label table)."""
    cs = 0.5 if case.get("half_cost") else 1.0
    rx = case.get("reach_x", case.get("reach"))
    rx, ry = (None if r is None else r * r for r in (rx, case.get("reach")))
    al, be, la, lb = cs * (x * x).sum(1), cs * (y * y).sum(1), a.log(), b.log()
    dots = x @ y.T + extra
    f, g = -al, -be

    def half(axis, pot, logw, eps, rho):
        damp = 1.0 if rho is None else 1.0 / (1.0 + eps / rho)
        return -eps * damp * _lse(dots, 2.0 * cs / eps, pot / eps + logw, axis), damp

    if case.get("backend") == "alternating":
        for eps in eps_list:
            f, _ = half(1, g, lb, eps, rx)
            g, _ = half(0, f, la, eps, ry)
        return f + al, g + be, f + al, g + be

    def step(f, g, eps, w):
        (nf, df), (ng, dg) = half(1, g, lb, eps, rx), half(0, f, la, eps, ry)
        return ((1 - w) * f + w * (nf - al * (1 - df)), (1 - w) * g + w * (ng - be * (1 - dg)))

    f, g = step(f, g, eps_list[0], 1.0)
    seen = None
    for i, eps in enumerate(eps_list):
        f, g = step(f, g, eps, 0.5)
        if case.get("threshold") is not None and (i + 1) % 10 == 0:
            if seen is not None and max((f - seen[0]).abs().max(), (g - seen[1]).abs().max()) < case["threshold"]:
                break
            seen = (f, g)
    last = step(f, g, eps_list[-1], 1.0)
    return last[0] + al, last[1] + be, f + al, g + be


def _barycentres(x, y, pot, logw, eps, cs, extra=0.0):
    """Rows of the plan's normalised weights times y."""
    scores = (2.0 * cs / eps) * (x @ y.T + extra) + ((pot - cs * (y * y).sum(1)) / eps + logw)
    return torch.softmax(scores, dim=1) @ y


def _schedule(case, x, y):
    if not case.get("anneal"):
        return [case["eps"]] * case["iters"]
    both = torch.cat([x, y])
    diam = float((both.max(0).values - both.min(0).values).norm())
    out, lg = [diam**2], 2.0 * math.log(diam)
    while lg > 2.0 * math.log(case["blur"]):
        out.append(math.exp(lg))
        lg += 2.0 * math.log(0.5)
    return out + [case["blur"] ** 2]


def _term(case, x, y, a, b, same, extra=0.0):
    """OT value and its gradients to x and y (of a self term: the whole one, and nothing)."""
    cs = 0.5 if case.get("half_cost") else 1.0
    eps_list = _schedule(case, x, y)
    f, g, fg, gg = _solve(case, x, y, a, b, eps_list, extra)
    eps, turned = eps_list[-1], extra.T if torch.is_tensor(extra) else extra
    if case.get("reach") is not None and case.get("backend", "symmetric") == "symmetric":
        rho = case["reach"] ** 2
        val = (rho + eps / 2) * ((a * (1 - (-f / rho).exp())).sum() + (b * (1 - (-g / rho).exp())).sum())
    else:
        val = (a * f).sum() + (b * g).sum()
    gx = 2.0 * cs * a[:, None] * (x - _barycentres(x, y, gg, b.log(), eps, cs, extra))
    gy = 2.0 * cs * b[:, None] * (y - _barycentres(y, x, fg, a.log(), eps, cs, turned))
    return (val, gx + gy, None) if same else (val, gx, gy)


def _divergence(case, x, y, a, b, table=None, lx=None, ly=None):
    def extra(p, q):
        return 0.0 if table is None else -0.5 * case["lambda_y"] * table[p][:, q]

    val, gx, gy = _term(case, x, y, a, b, False, extra(lx, ly))
    if case["debias"]:
        vx, gxx, _ = _term(case, x, x, a, a, True, extra(lx, lx))
        vy, _, _ = _term(case, y, y, b, b, True, extra(ly, ly))
        val, gx = val - 0.5 * (vx + vy), gx - 0.5 * gxx
    return val, gx, gy


def _hessian_product(case, x, y, v):
    """Loss, gradient and Hessian-vector product with uniform weights and the plan as a matrix; the Schur system is
    solved by conjugate gradients under the module's defaults."""
    n, m, eps = x.shape[0], y.shape[0], case["eps"]
    a, b = x.new_full((n,), 1.0 / n), y.new_full((m,), 1.0 / m)
    f, g, fg, gg = _solve(case, x, y, a, b, [eps] * case["iters"])
    grad = 2.0 * a[:, None] * (x - _barycentres(x, y, gg, b.log(), eps, 1.0))
    plan = (2.0 / eps) * (x @ y.T) + ((fg - (x * x).sum(1)) / eps + a.log())[:, None]
    plan = (plan + (gg - (y * y).sum(1)) / eps + b.log()).exp_()
    pa, pb = plan.sum(1), plan.sum(0)
    xv, py = (x * v).sum(1), plan @ y
    rx, ry = 2.0 * (pa * xv - (v * py).sum(1)), 2.0 * (plan.T @ xv - (y * (plan.T @ v)).sum(1))
    z, r = torch.zeros_like(pb), ry - plan.T @ (rx / pa)
    p, tol = r.clone(), max(1e-6, 1e-6 * float(r.norm()))
    for _ in range(case["cg"]):
        ap = (pb + eps * 1e-5) * p - plan.T @ ((plan @ p) / pa)
        rr = r @ r
        step = rr / (p @ ap)
        z, r = z + step * p, r - step * ap
        if float(r.norm()) <= tol:
            break
        p = r + (r @ r) / rr * p
    pz = plan @ z
    z1 = (rx - pz) / pa
    hv = (2.0 / eps) * (x * (pa * z1 + pz)[:, None] - py * z1[:, None] - plan @ (y * z[:, None]))
    k = 4.0 / eps
    hv += 2.0 * pa[:, None] * v + k * (x * ((py * v).sum(1) - xv * pa)[:, None] + py * xv[:, None])
    hv -= k * ((plan * (v @ y.T)) @ y)
    return dict(loss=(a * f).sum() + (b * g).sum(), grad=grad, hvp=hv)


def exact(case, seed):
    """What run() returns for these inputs in 64 bits, by dense formulas; None where that would take too long."""
    n, m, kind = case["n"], case["m"], case["kind"]
    passes = {"plan": 2, "ctrans": 1, "tiles": 100, "batch": case.get("batch", 1) * 6 * case.get("iters", 1)}.get(
        kind, 6 * case.get("iters", 12))
    if float(max(n, m)) ** 2 * passes > 2.0e11 or max(n, m) > 50000 or kind == "tiles":
        return None
    s = prepare(case, seed)
    x, y = s["x"].detach().double(), s["y"].detach().double()
    if kind == "loss":
        table = s["loss"].label_cost_matrix
        val, gx, gy = _divergence(case, x, y, s["a"].double(), s["b"].double(),
                                  None if table is None else table.double(), s.get("label_x"), s.get("label_y"))
        return dict(loss=val, grads=(gx, gy) if case.get("grad_y") else (gx,))
    if kind == "batch":
        a, b = x.new_full((n,), 1.0 / n), x.new_full((m,), 1.0 / m)
        out = [_divergence(case, p, q, a, b) for p, q in zip(x, y)]
        return dict(loss=torch.stack([o[0] for o in out]), grads=(torch.stack([o[1] for o in out]),))
    if kind == "hvp":
        return _hessian_product(case, x, y, s["v"].double())
    if kind == "plan":
        # f and g are the shifted potentials
        f, g, eps = s["f"].double(), s["g"].double(), case["eps"]
        left, right = f / eps + s["la"].double(), g / eps + s["lb"].double()
        mat, vec = s["mat"].double(), s["vec"].double()
        moved, mass = [], 0.0
        for r, l, v in zip(x.split(2048), left.split(2048), vec.split(2048)):
            p = ((2.0 / eps) * (r @ y.T) + l[:, None] + right).exp_()
            moved.append(p @ mat)
            mass = mass + p.T @ v
        return dict(moved=torch.cat(moved), mass=mass)
    price = (y * y).sum(1) - s["psi"].double()
    best = [torch.min((r * r).sum(1)[:, None] - 2.0 * (r @ y.T) + price, dim=1) for r in x.split(2048)]
    return dict(values=torch.cat([v for v, _ in best]), index=torch.cat([i for _, i in best]))
