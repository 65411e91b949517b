"""Volume-rendering composite ops (weights scan and weighted colour/depth sums).

CPU tensors run the PyTorch statement of the math (the oracle); CUDA tensors run the warp-scan
kernels in ``csrc/composite.cu``.  Reference behaviour:
landmark/nerf_components/model_components/renderers/volume_renderer.py:20-67.
"""
from __future__ import annotations

from ctypes import c_float, c_int
from typing import Optional, Tuple

import torch

from . import native

P = native.P
native.register_signature("lmb_weights_select", [P, P, c_float, c_float, c_int, c_int, P, P, P])
native.register_signature("lmb_render_rows", [P, P, P, P, c_int, c_int, c_float, P, P, P])


def weights_reference(sigma: torch.Tensor, dists: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    alpha = 1.0 - torch.exp(-sigma * dists)
    trans = torch.cumprod(torch.cat([torch.ones_like(alpha[:, :1]), 1.0 - alpha + 1e-10], -1), -1)
    return alpha * trans[:, :-1], trans[:, -1]


def render_reference(weights, rgbs, z_vals, bg: float):
    acc = weights.sum(-1)
    rgb = (weights[..., None] * rgbs).sum(-2) + bg * (1.0 - acc[..., None])
    depth = (weights * z_vals).sum(-1)
    return rgb, depth, acc


class _Weights(torch.autograd.Function):
    @staticmethod
    def forward(ctx, sigma, dists):
        R, S = sigma.shape
        weights = torch.empty_like(sigma)
        bg = torch.empty(R, device=sigma.device, dtype=torch.float32)
        native.check(native.lib().lmb_weights_fwd(sigma.data_ptr(), dists.data_ptr(), R, S, weights.data_ptr(),
                                                  bg.data_ptr(), native.stream_ptr()), "weights_fwd")
        ctx.save_for_backward(sigma, dists)
        return weights, bg

    @staticmethod
    def backward(ctx, dweights, dbg):
        sigma, dists = ctx.saved_tensors
        R, S = sigma.shape
        dsigma = torch.empty_like(sigma)
        dweights = dweights.contiguous()
        dbg = None if dbg is None else dbg.contiguous()
        native.check(native.lib().lmb_weights_bwd(sigma.data_ptr(), dists.data_ptr(), dweights.data_ptr(),
                                                  native.ptr(dbg), R, S, dsigma.data_ptr(), native.stream_ptr()),
                     "weights_bwd")
        return dsigma, None


class _Render(torch.autograd.Function):
    @staticmethod
    def forward(ctx, weights, rgbs, z_vals, bg):
        R, S = weights.shape
        rgb = torch.empty((R, 3), device=weights.device, dtype=torch.float32)
        depth = torch.empty(R, device=weights.device, dtype=torch.float32)
        acc = torch.empty(R, device=weights.device, dtype=torch.float32)
        native.check(native.lib().lmb_render_fwd(weights.data_ptr(), rgbs.data_ptr(), z_vals.data_ptr(), R, S,
                                                 float(bg), rgb.data_ptr(), depth.data_ptr(), acc.data_ptr(),
                                                 native.stream_ptr()), "render_fwd")
        ctx.save_for_backward(weights, rgbs)
        ctx.bg = float(bg)
        ctx.mark_non_differentiable(depth, acc)
        return rgb, depth, acc

    @staticmethod
    def backward(ctx, drgb, _ddepth, _dacc):
        weights, rgbs = ctx.saved_tensors
        R, S = weights.shape
        dweights = torch.empty_like(weights)
        drgbs = torch.empty_like(rgbs)
        drgb = drgb.contiguous()
        native.check(native.lib().lmb_render_bwd(weights.data_ptr(), rgbs.data_ptr(), drgb.data_ptr(), R, S, ctx.bg,
                                                 dweights.data_ptr(), drgbs.data_ptr(), native.stream_ptr()),
                     "render_bwd")
        return dweights, drgbs, None, None


def composite_weights(sigma: torch.Tensor, dists: torch.Tensor) -> Tuple[torch.Tensor, torch.Tensor]:
    """``(weights [R,S], bg_transmittance [R])`` from densities and inter-sample distances."""
    if not sigma.is_cuda:
        return weights_reference(sigma, dists)
    return _Weights.apply(sigma.contiguous().float(), dists.contiguous().float())


def composite_render(weights: torch.Tensor, rgbs: torch.Tensor, z_vals: torch.Tensor, bg: float = 0.0):
    """``(rgb [R,3] unclamped, depth [R], acc [R])``; depth/acc carry no gradient (as in the reference)."""
    if not weights.is_cuda:
        rgb, depth, acc = render_reference(weights, rgbs, z_vals, bg)
        return rgb, depth.detach(), acc.detach()
    return _Render.apply(weights.contiguous().float(), rgbs.contiguous().float(), z_vals.contiguous().float(), bg)


@torch.no_grad()
def weights_select(sigma: torch.Tensor, dists: torch.Tensor, scale: float, threshold: float) -> Tuple[torch.Tensor, torch.Tensor]:
    """``(weights [R,S], weights > threshold)`` of densities and ``dists * scale`` (CUDA, no gradients)."""
    sigma, dists = sigma.contiguous().float(), dists.contiguous().float()
    R, S = sigma.shape
    weights, mask = torch.empty_like(sigma), torch.empty(R, S, dtype=torch.bool, device=sigma.device)
    native.check(native.lib().lmb_weights_select(sigma.data_ptr(), dists.data_ptr(), float(scale), float(threshold), R, S,
                                                 weights.data_ptr(), mask.data_ptr(), native.stream_ptr()), "weights_select")
    return weights, mask


@torch.no_grad()
def composite_rows(weights: torch.Tensor, vals: torch.Tensor, slot: torch.Tensor, z_vals: torch.Tensor, bg: float = 0.0):
    """:func:`composite_render` with the colours of the selected samples in ``vals [*, 3]``: ``slot int32 [R*S]`` holds a
    sample's row, -1 for black.  ``(rgb [R,3] unclamped, depth [R])``, CUDA, no gradients."""
    weights, vals, z_vals = weights.contiguous().float(), vals.contiguous().float(), z_vals.contiguous().float()
    R, S = weights.shape
    rgb, depth = torch.empty(R, 3, device=weights.device), torch.empty(R, device=weights.device)
    native.check(native.lib().lmb_render_rows(weights.data_ptr(), vals.data_ptr(), slot.data_ptr(), z_vals.data_ptr(), R, S, float(bg),
                                              rgb.data_ptr(), depth.data_ptr(), native.stream_ptr()), "render_rows")
    return rgb, depth
