"""Autograd glue: OT cost with an analytic backward, and a gradient node whose backward is the HVP.

Behaviour follows the reference's ``_autograd.py`` (``_SinkhornConfig`` :33-76,
``_SinkhornGradFn`` :84-283, ``_SinkhornCostFn`` :291-519):

* forward = Sinkhorn solve + dual cost; the cost uses the final potentials, the
  gradient the potentials *before* the last extrapolation step (GeomLoss convention);
* ``d cost / d a = f``, ``d cost / d b = g`` (times the incoming gradient);
* ``d cost / d x`` comes from the barycentric gradient kernel and is itself
  differentiable w.r.t. x: its backward is the streaming-CG Hessian-vector product,
  always evaluated with fp32-exact products;
* double backward w.r.t. y raises ``NotImplementedError``.
"""
from __future__ import annotations

import ctypes
from dataclasses import dataclass
from typing import Optional, Tuple

import torch

from flash_sinkhorn_b200 import _lib
from flash_sinkhorn_b200.hvp import geomloss_to_ott_potentials, hvp_x_sqeuclid_from_potentials
from flash_sinkhorn_b200.kernels.grad_sqeuclid import sinkhorn_geomloss_online_grad_sqeuclid
from flash_sinkhorn_b200.sinkhorn_solvers import sinkhorn_flashstyle_alternating, sinkhorn_flashstyle_symmetric


@dataclass(frozen=True)
class _SinkhornConfig:
    """Immutable snapshot of a ``SamplesLoss`` configuration, carried on the autograd context."""

    backend: str
    blur: float
    scaling: float
    use_epsilon_scaling: bool
    eps: Optional[float]
    n_iters: Optional[int]
    cost_scale: float
    rho_x: Optional[float]
    rho_y: Optional[float]
    last_extrapolation: bool
    allow_tf32: bool
    use_exp2: bool
    autotune: bool
    block_m: Optional[int]
    block_n: Optional[int]
    block_k: Optional[int]
    num_warps: Optional[int]
    num_stages: int
    hvp_tau2: float
    hvp_max_cg_iter: int
    hvp_cg_rtol: float
    hvp_cg_atol: float
    hvp_cg_stabilise_every: int
    hvp_preconditioner: str
    hvp_precond_terms: int
    hvp_use_preconditioner: bool
    lambda_x: float
    lambda_y: float
    threshold: Optional[float]
    inner_iterations: int
    # Extension: torch.distributed group for row-sharded multi-GPU solves (None = single GPU).
    process_group: object = None


class _SinkhornGradFn(torch.autograd.Function):
    """``(grad_x, grad_y)`` of the OT cost; differentiable once more w.r.t. x (HVP)."""

    @staticmethod
    def forward(ctx, x, y, a, b, f_grad, g_grad, grad_scale, eps: float, config: _SinkhornConfig,
                want_x: bool, want_y: bool, label_x=None, label_y=None, label_cost_matrix=None):
        gx, gy = sinkhorn_geomloss_online_grad_sqeuclid(
            x, y, a, b, f_grad, g_grad,
            eps=float(eps), allow_tf32=config.allow_tf32, grad_scale=grad_scale,
            compute_grad_x=bool(want_x), compute_grad_y=bool(want_y), cost_scale=config.cost_scale,
            label_x=label_x, label_y=label_y, label_cost_matrix=label_cost_matrix,
            lambda_x=config.lambda_x, lambda_y=config.lambda_y,
            process_group=config.process_group,
        )
        ctx.save_for_backward(x, y, a, b, f_grad, g_grad, grad_scale)
        ctx.eps = float(eps)
        ctx.config = config
        ctx.use_label_cost = (label_x is not None and label_y is not None and label_cost_matrix is not None
                              and config.lambda_y != 0.0)
        return gx, gy

    @staticmethod
    def backward(ctx, v_x, v_y):
        x, y, a, b, f_grad, g_grad, grad_scale = ctx.saved_tensors
        cfg = ctx.config
        if v_y is not None:
            raise NotImplementedError("Double backward w.r.t y is not implemented yet.")
        if ctx.use_label_cost:
            raise NotImplementedError("Double backward (HVP) is not supported with OTDD label-augmented cost. "
                                      "Use gradient flow without HVP.")
        out_x = None
        if v_x is not None:
            if v_x.shape != x.shape:
                raise ValueError("grad_grad_x must have the same shape as x.")
            if not v_x.is_cuda:
                raise ValueError("grad_grad_x must be a CUDA tensor.")
            with torch.no_grad():
                f_ott, g_ott = geomloss_to_ott_potentials(f_grad, g_grad, a, b, eps=ctx.eps)
                hv, _ = hvp_x_sqeuclid_from_potentials(
                    x, y, f_ott, g_ott, v_x,
                    eps=ctx.eps, rho_x=cfg.rho_x, rho_y=cfg.rho_y, cost_scale=cfg.cost_scale,
                    tau2=cfg.hvp_tau2, max_cg_iter=cfg.hvp_max_cg_iter,
                    cg_rtol=cfg.hvp_cg_rtol, cg_atol=cfg.hvp_cg_atol,
                    cg_stabilise_every=cfg.hvp_cg_stabilise_every,
                    preconditioner=cfg.hvp_preconditioner, precond_terms=cfg.hvp_precond_terms,
                    use_preconditioner=cfg.hvp_use_preconditioner,
                    allow_tf32=False,  # second-order products need fp32-exact scores
                )
                out_x = hv * grad_scale
        return (out_x,) + (None,) * 13


@dataclass(frozen=True)
class _LossTerms:
    """What the node of a batch of losses knows beside its tensors."""

    eps: Tuple[Tuple[float, ...], ...]  # where the schedules end: [term][item]
    config: _SinkhornConfig
    debias: bool
    labels: Optional[list]  # label costs of the terms


def _loss_gradients(x, y, a, b, log_a, log_b, scale, meta, pots, want_x, want_y):
    """Gradients of ``sum_i scale_i loss_i`` to the clouds ``[B, n, d]``, ``[B, m, d]`` (or one item without the leading
    axis); pots: ``f, g, f_pre, g_pre`` of every term."""
    if x.dtype not in (torch.float16, torch.bfloat16, torch.float32):
        raise ValueError(f"Unsupported dtype for x/y: {x.dtype}")
    cfg, dev = meta.config, x.device
    n, m, d = x.shape[-2], y.shape[-2], x.shape[-1]
    x32, y32, a32, b32, la, lb = map(_lib.f32c, (x, y, a, b, log_a, log_b))
    pots = [_lib.f32c(p) for p in pots]
    gs = _lib.f32c(scale.detach().reshape(-1))
    prec = _lib.precision_id(cfg.allow_tf32)
    X, Y = (x32, a32, la, n), (y32, b32, lb, m)

    # gradients of row clouds that share launches: (rows, columns, potential of the columns, scales, out), and their eps
    waiting, waiting_eps = [], []

    def term(k, u, v, scales, out_u, out_v):
        (pu, wu, lu, r), (pv, wv, lv, c) = u, v
        if not meta.labels and all(_lib.load().fs_grad_many_bytes(p, q, d, prec) for p, q in ((r, c), (c, r))):
            if out_u is not None:
                waiting.append((u, v, pots[4 * k + 3], scales, out_u))
                waiting_eps.append(meta.eps[k])
            if out_v is not None:
                waiting.append((v, u, pots[4 * k + 2], scales, out_v))
                waiting_eps.append(meta.eps[k])
            return
        f_pre, g_pre = pots[4 * k + 2], pots[4 * k + 3]
        label = meta.labels[k] if meta.labels else None
        ws = _lib.workspace(_lib.OP_GRAD, r, c, d, prec, dev, label.V if label else 0)
        tensors = (pu, pv, wu, wv, lu, lv, f_pre, g_pre, scales, out_u, out_v)
        pitch = [4 * q for q in (r * d, c * d, r, c, r, c, r, c, 1, r * d, c * d)]
        addr = [_lib.ptr(t) for t in tensors]
        for i in range(gs.numel()):
            at = [None if p is None else p + i * q for p, q in zip(addr, pitch)]
            _lib.call("fs_grad", dev, at[0], at[1], r, c, d, *at[2:], meta.eps[k][i], float(cfg.cost_scale), prec, _lib.ptr(ws),
                      ws.numel(), _lib.stream_ptr(dev), label.ref if label else None)

    gx = torch.empty(x.shape, device=dev, dtype=torch.float32) if want_x else None
    gy = torch.empty(y.shape, device=dev, dtype=torch.float32) if want_y else None
    term(0, X, Y, gs, gx, gy)
    added = []
    for k, side, out in ((1, X, gx), (2, Y, gy)):
        if not meta.debias or out is None:
            continue
        if pots[4 * k + 2].data_ptr() == pots[4 * k + 3].data_ptr():  # equal potentials: the two sides' gradients are equal
            own = torch.empty_like(out)
            term(k, side, side, -gs, own, None)
            added.append((out, own))
        else:
            own, other = torch.empty_like(out), torch.empty_like(out)
            term(k, side, side, -0.5 * gs, own, other)
            added += [(out, own), (out, other)]
    _gradients_together(waiting, gs.numel(), d, waiting_eps, float(cfg.cost_scale), prec, dev)
    for out, own in added:
        out += own
    return gx, gy


# Scratch of one call of shared gradients: a single gradient of 50,000 points in 64 dimensions takes 71 MB (exact mode 108). It
# bounds memory, not time: sixteen gradients of 4,096 points share launches in 0.42 ms and take 1.18 in turn (108 MB), four of 16,384 0.94 and
# 1.27 (172 MB), four of 32,000 2.99 and 3.33 (235 MB; in the exact mode 6.48 and 6.52).
SHARED_GRADIENT_BYTES = 1 << 27


def _gradients_together(terms, B, d, eps, cost_scale, prec, dev):
    """Runs the gradients of row clouds ``(rows, columns, column potential, scales, out)`` of B items each, 16 of one eps per
    call. ``eps``: a number, or one per term and item."""
    lib = _lib.load()
    by_eps = {}  # eps -> (items, sizes)
    for t, ((pu, wu, _, r), (pv, _, lv, c), pot, scales, out) in enumerate(terms):
        base = [_lib.ptr(t) for t in (pu, pv, wu, lv, pot, scales, out)]
        pitch = [4 * q for q in (r * d, c * d, r, c, c, 1, r * d)]
        nbytes = int(lib.fs_grad_many_bytes(r, c, d, prec))
        for i in range(B):
            x, y, weight, log_w, at_pot, scale, at_out = (p + i * q for p, q in zip(base, pitch))
            items, sizes = by_eps.setdefault(float(eps[t][i] if isinstance(eps, list) else eps), ([], []))
            items.append((x, y, r, c, weight, log_w, at_pot, scale, at_out))
            sizes.append(nbytes)
    for at_eps, (items, sizes) in by_eps.items():
        while items:
            k = 1
            while k < min(len(items), 16) and sum(sizes[: k + 1]) <= SHARED_GRADIENT_BYTES:
                k += 1
            ws = torch.empty(sum(sizes[:k]), dtype=torch.uint8, device=dev)
            arr = (_lib.GradItem * k)(*items[:k])
            _lib.call("fs_grad_many", dev, ctypes.cast(arr, ctypes.c_void_p), k, d, at_eps, cost_scale, prec, _lib.ptr(ws),
                      ws.numel(), _lib.stream_ptr(dev))
            items, sizes = items[k:], sizes[k:]


class _SinkhornLossGradFn(torch.autograd.Function):
    """Gradients of a batch of losses; differentiable once more w.r.t. x where they are not debiased."""

    @staticmethod
    def forward(ctx, x, y, a, b, log_a, log_b, scale, meta, want_x, want_y, *pots):
        ctx.save_for_backward(x, y, a, b, scale, *pots[2:4])
        ctx.meta = meta
        return _loss_gradients(x, y, a, b, log_a, log_b, scale, meta, pots, want_x, want_y)

    @staticmethod
    def backward(ctx, v_x, v_y):
        x, y, a, b, scale, f_pre, g_pre = ctx.saved_tensors
        if v_y is not None or ctx.meta.debias:  # a self term has its cloud on both sides
            raise NotImplementedError("Double backward w.r.t y is not implemented yet.")
        out = None
        if v_x is not None:
            items = []
            for i in range(x.shape[0]):
                sub = _HvpContext((x[i], y[i], a[i], b[i], f_pre[i], g_pre[i], scale[i]), ctx.meta.eps[0][i],
                                  ctx.meta.config)
                items.append(_SinkhornGradFn.backward(sub, v_x[i], None)[0])
            out = torch.stack(items, dim=0)
        return (out,) + (None,) * (len(ctx.needs_input_grad) - 1)


@dataclass
class _HvpContext:
    """The part of an autograd context that the Hessian-vector product of one item reads."""

    saved_tensors: tuple
    eps: float
    config: _SinkhornConfig
    use_label_cost: bool = False


class _SinkhornLossFn(torch.autograd.Function):
    """A batch of losses ``OT(x,y) - OT(x,x)/2 - OT(y,y)/2`` (or ``OT(x,y)`` alone) from finished potentials as ONE node:
    the values of :class:`_SinkhornCostFn` for every term, combined, and their gradients in one pass over the terms. ``x``,
    ``y``, ``a``, ``b`` have a leading batch axis or describe one item; ``pots`` are ``f, g, f_pre, g_pre`` of every term
    (the last two those that gradients are taken at), shaped like the weights."""

    @staticmethod
    def forward(ctx, x, y, a, b, log_a, log_b, meta, *pots):
        ctx.save_for_backward(x, y, a, b, log_a, log_b, *pots)
        ctx.meta = meta
        cfg = meta.config

        def value(term, w, pot, rho):
            if cfg.rho_x is None or cfg.rho_y is None:  # balanced or semi-unbalanced
                return w * pot
            eps = meta.eps[term]
            mass = rho + eps[0] / 2
            if len(set(eps)) > 1:
                mass = torch.tensor([[rho + e / 2] for e in eps], device=pot.device, dtype=torch.float32)
            return mass * (w * (1 - (-pot / rho).exp()))

        def side(k, w, rho, own, other):
            # the potential of this side in OT(x,y), minus half of both potentials of the self term (number own // 4)
            if not meta.debias:
                return value(0, w, pots[k], rho).sum(dim=-1)
            if cfg.rho_x is None or cfg.rho_y is None:
                return (w * (pots[k] - _half_sum(pots[own], pots[other]))).sum(dim=-1)
            both = value(own // 4, w, pots[own], cfg.rho_x) + value(own // 4, w, pots[other], cfg.rho_y)
            return (value(0, w, pots[k], rho) - 0.5 * both).sum(dim=-1)

        return side(0, a, cfg.rho_x, 4, 5) + side(1, b, cfg.rho_y, 8, 9)

    @staticmethod
    def backward(ctx, grad_out):
        x, y, a, b, log_a, log_b, *pots = ctx.saved_tensors
        gx = gy = ga = gb = None
        if x.requires_grad or y.requires_grad:
            gx, gy = _SinkhornLossGradFn.apply(x, y, a, b, log_a, log_b, grad_out, ctx.meta, x.requires_grad, y.requires_grad,
                                               *(pots if ctx.meta.debias else pots[:4]))
        debias = ctx.meta.debias
        if a.requires_grad:
            ga = grad_out.unsqueeze(-1) * (pots[0] - _half_sum(pots[4], pots[5]) if debias else pots[0])
        if b.requires_grad:
            gb = grad_out.unsqueeze(-1) * (pots[1] - _half_sum(pots[8], pots[9]) if debias else pots[1])
        return (gx, gy, ga, gb) + (None,) * (3 + len(pots))


def _half_sum(u, v):
    return u if u.data_ptr() == v.data_ptr() else 0.5 * (u + v)


class _SinkhornCostFn(torch.autograd.Function):
    """Entropic OT cost ``OT_eps(a, x; b, y)`` with an analytic (envelope-theorem) backward."""

    @staticmethod
    def forward(ctx, x, y, a, b, eps_list: Tuple[float, ...], config: _SinkhornConfig,
                label_x, label_y, label_cost_matrix, presolved=None):
        # `presolved` (extension): (f_cost, g_cost, f_grad, g_grad) from a solve done elsewhere - the multi-GPU
        # divergence solves its three problems interleaved before building the three cost nodes.
        label_kw = dict(label_x=label_x, label_y=label_y, label_cost_matrix=label_cost_matrix,
                        lambda_x=config.lambda_x, lambda_y=config.lambda_y)
        if presolved is not None:
            eps = float(eps_list[-1])
            f_cost, g_cost, f_grad, g_grad = presolved
            plain_dual = config.backend == "alternating" or config.rho_x is None or config.rho_y is None
        elif config.backend == "alternating":
            eps = float(eps_list[-1])
            f_cost, g_cost = sinkhorn_flashstyle_alternating(
                x, y, a, b, eps=eps, n_iters=len(eps_list), cost_scale=config.cost_scale,
                rho_x=config.rho_x, rho_y=config.rho_y, allow_tf32=config.allow_tf32,
                process_group=config.process_group,
            )
            f_grad, g_grad = f_cost, g_cost
            plain_dual = True  # the reference's alternating branch always returns <a,f>+<b,g>
        else:
            eps = float(eps_list[-1])
            common = dict(
                blur=config.blur, scaling=config.scaling, use_epsilon_scaling=config.use_epsilon_scaling,
                eps=config.eps, n_iters=config.n_iters, allow_tf32=config.allow_tf32,
                cost_scale=config.cost_scale, rho_x=config.rho_x, rho_y=config.rho_y,
                threshold=config.threshold, check_every=config.inner_iterations,
                process_group=config.process_group,
            )
            if config.last_extrapolation:
                f_cost, g_cost, f_grad, g_grad = sinkhorn_flashstyle_symmetric(
                    x, y, a, b, last_extrapolation=True, return_prelast=True, **common, **label_kw)
            else:
                f_cost, g_cost = sinkhorn_flashstyle_symmetric(x, y, a, b, last_extrapolation=False, **common,
                                                               **label_kw)
                f_grad, g_grad = f_cost, g_cost
            plain_dual = config.rho_x is None or config.rho_y is None  # balanced or semi-unbalanced

        ctx.save_for_backward(x, y, a, b, f_cost, g_cost, f_grad, g_grad)
        ctx.eps = eps
        ctx.config = config
        ctx.labels = (label_x, label_y, label_cost_matrix)

        if plain_dual:
            return (a * f_cost).sum() + (b * g_cost).sum()
        # Both marginals relaxed: (rho + eps/2) * <w, 1 - exp(-potential/rho)> per side.
        total = torch.tensor(0.0, device=x.device, dtype=torch.float32)
        total = total + (config.rho_x + eps / 2) * (a * (1 - (-f_cost / config.rho_x).exp())).sum()
        total = total + (config.rho_y + eps / 2) * (b * (1 - (-g_cost / config.rho_y).exp())).sum()
        return total

    @staticmethod
    def backward(ctx, grad_out):
        x, y, a, b, f_cost, g_cost, f_grad, g_grad = ctx.saved_tensors
        gx = gy = ga = gb = None
        if x.requires_grad or y.requires_grad:
            gx, gy = _SinkhornGradFn.apply(
                x, y, a, b, f_grad, g_grad, grad_out, ctx.eps, ctx.config, x.requires_grad, y.requires_grad,
                *ctx.labels)
            if not x.requires_grad:
                gx = None
            if not y.requires_grad:
                gy = None
        if a.requires_grad:
            ga = grad_out * f_cost
        if b.requires_grad:
            gb = grad_out * g_cost
        return gx, gy, ga, gb, None, None, None, None, None, None
