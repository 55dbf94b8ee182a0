"""Differentiable P_l(k): gradients with respect to particle positions and weights.

The reference exists to differentiate its estimator (tests/lognormal.py:60-103
optimises particle positions through cic_mas_vec -> powspec_vec with JAX
autodiff).  `power_multipoles_diff` is the same capability for the production
estimator (B-spline deposit, optional interlacing, mass normalisation, shot
noise), as a torch.autograd.Function whose backward pass runs on the GPU:

    pk = power_multipoles_diff(x, y, z, w, box_size=1000.0, n_mesh=64)   # [nb, 3]
    loss = ((pk[:, 0] - target) ** 2).sum()
    loss.backward()                                                      # x.grad, y.grad, z.grad, w.grad

Forward: deposit (gbp_deposit) -> packed transform + binning (gbp_fft_power, the
packed spectrum kept) -> normalisation.  Backward: gbp_power_backward_packed
forms the adjoint spectrum from dLoss/dP and transforms it back to gradient
meshes; gbp_deposit_backward_total gathers them at the particles with the
B-spline derivatives and adds the explicit dependence of L^3/M^2 and of the
shot noise on the weights (M = sum w, Q = sum w^2):
    dP_l/dM = -2 P_l / M,   dP_0/dQ = -L^3 / M^2.
Meshes that need cuFFT go through gbp_fft_r2c, gbp_power and
gbp_power_backward.  Empty bins (NaN) carry no gradient.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from . import _lib, _native
from ._lib import check
from .pipeline import PkConfig

__all__ = ["power_multipoles_diff"]


def _p(t):
    return None if t is None else C.c_void_p(t.data_ptr())


class _PowerFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, y, z, w, cfg: PkConfig):
        dev = x.device
        N, G = cfg.n_mesh, cfg.grids
        xs, ys, zs = (t.detach().contiguous().to(torch.float32) for t in (x, y, z))
        ws = None if w is None else w.detach().contiguous().to(torch.float32)
        inv = np.float32(N / cfg.box_size)
        mesh, stats = _native.deposit(xs, ys, zs, ws, n_mesh=N, inv_cell=inv, origin=cfg.origin,
                                      mas=cfg.mas_order, interlace=cfg.interlace)
        plan = _native.fft_plan(N, G, dev)
        spec = torch.empty(plan.spectrum_floats, dtype=torch.float32, device=dev)
        bins = _native.bins_for(cfg.kedges_grid(), N, dev)
        mask = _lib.ELL0 | _lib.ELL2 | _lib.ELL4
        ctx.packed = _native.fft_power_workspace_size(plan, bins, mask) is not None
        if ctx.packed:
            sums = _native.fft_power(plan, mesh, spec, bins, mas_order=cfg.mas_order, ells=mask, mass=stats)
        else:
            plan.execute(mesh, spec)
            sums = _native.power(spec, G, bins, mas_order=cfg.mas_order, ells=mask, z_pitch=plan.pitch, mass=stats)
        pk, _ = _native.normalize(sums, n_mesh=N, box_size=cfg.box_size, mass=stats, stats=stats,
                                  subtract_shot=cfg.shot_noise)
        ctx.cfg, ctx.plan, ctx.bins = cfg, plan, bins
        ctx.has_w = w is not None
        ctx.save_for_backward(xs, ys, zs, ws if ws is not None else torch.empty(0, device=dev), spec, stats,
                              sums.nmodes, pk)
        return pk

    @staticmethod
    def backward(ctx, grad_pk):
        xs, ys, zs, ws, spec, stats, nmodes, pk = ctx.saved_tensors
        cfg, plan, bins = ctx.cfg, ctx.plan, ctx.bins
        dev = xs.device
        N, G = cfg.n_mesh, cfg.grids
        ws = ws if ctx.has_w else None
        lib = _lib.load()
        gmesh = torch.empty((G, N, N, N), dtype=torch.float32, device=dev)
        stream = _native._stream_of(dev)
        need = C.c_size_t(0)
        n = xs.numel()
        gx, gy, gz = (torch.empty(n, dtype=torch.float32, device=dev) for _ in range(3))
        want_w = ctx.has_w and ctx.needs_input_grad[3]
        gw = torch.empty(n, dtype=torch.float32, device=dev) if want_w else None
        inv = float(np.float32(N / cfg.box_size))
        o = [float(np.float32(v)) for v in cfg.origin]
        if ctx.packed:
            g = grad_pk.detach().to(torch.float64).contiguous()
            check(lib.gbp_power_backward_packed_workspace_size(plan.handle, bins.handle, C.byref(need)),
                  "gbp_power_backward_packed_workspace_size")
            wsb = _native.workspace(need.value, dev)
            scal = torch.empty(2, dtype=torch.float64, device=dev)
            check(lib.gbp_power_backward_packed(_p(spec), plan.handle, bins.handle, cfg.mas_order, _p(g), _p(pk),
                                                _p(nmodes), _p(stats), float(cfg.box_size), int(cfg.shot_noise),
                                                _p(gmesh), _p(scal), _p(wsb), wsb.numel(), stream),
                  "gbp_power_backward_packed")
        else:
            g = torch.nan_to_num(grad_pk.detach().to(torch.float64), nan=0.0).contiguous()
            g = torch.where(torch.isfinite(pk), g, torch.zeros_like(g))
            check(lib.gbp_power_backward_workspace_size(plan.handle, C.byref(need)),
                  "gbp_power_backward_workspace_size")
            wsb = _native.workspace(need.value, dev)
            check(lib.gbp_power_backward(_p(spec), plan.handle, bins.handle, cfg.mas_order, _p(g), _p(nmodes),
                                         _p(stats), float(cfg.box_size), _p(gmesh), _p(wsb), wsb.numel(), stream),
                  "gbp_power_backward")
            scal = None
            if want_w:
                M = stats[:8].view(torch.float64)                          # gbp_deposit_stats starts with mass[2]
                pk0 = torch.nan_to_num(pk, nan=0.0)
                shot = -2.0 * cfg.box_size ** 3 * int(cfg.shot_noise)
                scal = torch.cat([(g * (-2.0 * pk0 / M)).sum().reshape(1),  # dP_l/dM = -2 P_l / M
                                  shot / M ** 2 * g[:, 0].sum()])
        check(lib.gbp_deposit_backward_total(_p(xs), _p(ys), _p(zs), _p(ws), n, o[0], o[1], o[2], inv, N,
                                             cfg.mas_order, int(cfg.interlace), _p(gmesh), _p(scal), _p(gx), _p(gy),
                                             _p(gz), _p(gw), stream), "gbp_deposit_backward_total")
        return gx, gy, gz, gw, None


def power_multipoles_diff(x, y, z, w=None, *, box_size: float, n_mesh: int, mas: str = "tsc", interlace: bool = True,
                          shot_noise: bool = True, k_edges=None, origin=(0.0, 0.0, 0.0)) -> torch.Tensor:
    """P_0,2,4(k) [nb, 3] (float64) of float32 CUDA particle tensors, differentiable in x, y, z and w."""
    cfg = PkConfig(n_mesh=int(n_mesh), box_size=float(box_size), mas=mas, interlace=bool(interlace),
                   shot_noise=bool(shot_noise),
                   k_edges=None if k_edges is None else tuple(np.asarray(k_edges, np.float32).tolist()),
                   origin=tuple(float(v) for v in origin))
    return _PowerFn.apply(x, y, z, w, cfg)
