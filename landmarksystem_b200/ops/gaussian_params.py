"""Per-Gaussian parameter passes (``csrc/gs_params.cu``): the three activations in one launch each way, and the
densification statistics of a step in one launch.  Callers check :func:`fusable` / :func:`stats_fusable` and otherwise
keep the tensor operations."""
from __future__ import annotations

from ctypes import c_longlong

import torch
from torch.autograd.function import once_differentiable

from . import native

P = native.P
native.register_signature("lmb_gs_activate", [c_longlong, P, P, P, P, P, P, P])
native.register_signature("lmb_gs_activate_bwd", [c_longlong, P, P, P, P, P, P, P, P, P, P])
native.register_signature("lmb_gs_view_stats", [c_longlong, P, P, P, P, P, P, P])


def _plain(t: torch.Tensor, shape) -> bool:
    return type(t) in (torch.Tensor, torch.nn.Parameter) and t.is_cuda and t.dtype == torch.float32 and t.is_contiguous() \
        and tuple(t.shape) == tuple(shape)


def fusable(scaling, rotation, opacity) -> bool:
    """Contiguous fp32 CUDA tensors ``[N, 3]``, ``[N, 4]`` (on 16 bytes) and ``[N, 1]`` of one device."""
    n = scaling.shape[0]
    return _plain(scaling, (n, 3)) and _plain(rotation, (n, 4)) and _plain(opacity, (n, 1)) and rotation.data_ptr() % 16 == 0 \
        and scaling.device == rotation.device == opacity.device


class _Activate(torch.autograd.Function):
    @staticmethod
    def forward(ctx, scaling, rotation, opacity):
        scales, quats, alphas = torch.empty_like(scaling), torch.empty_like(rotation), torch.empty_like(opacity)
        native.check(native.lib().lmb_gs_activate(scaling.shape[0], scaling.data_ptr(), rotation.data_ptr(), opacity.data_ptr(),
                                                  scales.data_ptr(), quats.data_ptr(), alphas.data_ptr(), native.stream_ptr()),
                     "gs_activate")
        ctx.save_for_backward(scales, rotation, alphas)
        return scales, quats, alphas

    @staticmethod
    @once_differentiable
    def backward(ctx, d_scales, d_quats, d_alphas):
        scales, rotation, alphas = ctx.saved_tensors
        d_scales, d_quats, d_alphas = d_scales.contiguous(), d_quats.contiguous(), d_alphas.contiguous()
        if d_quats.data_ptr() % 16:
            d_quats = d_quats.clone()
        grads = torch.empty_like(scales), torch.empty_like(rotation), torch.empty_like(alphas)
        native.check(native.lib().lmb_gs_activate_bwd(scales.shape[0], scales.data_ptr(), rotation.data_ptr(), alphas.data_ptr(),
                                                      d_scales.data_ptr(), d_quats.data_ptr(), d_alphas.data_ptr(),
                                                      *(g.data_ptr() for g in grads), native.stream_ptr()), "gs_activate_bwd")
        return grads


def activate(scaling, rotation, opacity):
    """``exp(scaling)``, unit ``rotation`` and ``sigmoid(opacity)``."""
    return _Activate.apply(scaling, rotation, opacity)


def stats_fusable(visible, radii, grad, max_radii, accum, denom) -> bool:
    n = radii.shape[0]
    return radii.is_cuda and radii.dtype == torch.int32 and radii.is_contiguous() \
        and visible.dtype == torch.bool and visible.is_contiguous() and tuple(visible.shape) == (n,) \
        and _plain(grad, (n, 3)) and _plain(max_radii, (n,)) and _plain(accum, (n, 1)) and _plain(denom, (n, 1)) \
        and len({t.device for t in (visible, radii, grad, max_radii, accum, denom)}) == 1


def view_stats(visible, radii, grad, max_radii, accum, denom) -> None:
    """Where ``visible``: ``max_radii = max(max_radii, radii)``, ``accum += |grad[:2]|``, ``denom += 1`` (in place)."""
    native.check(native.lib().lmb_gs_view_stats(radii.shape[0], visible.data_ptr(), radii.data_ptr(), grad.data_ptr(),
                                                max_radii.data_ptr(), accum.data_ptr(), denom.data_ptr(), native.stream_ptr()),
                 "gs_view_stats")
