"""Proposal-network density in one kernel each way (``csrc/prop_density.cu``) and the contraction to the unit cube that it
shares with the field.  Callers check :func:`prop_density_supported` / :func:`unit_positions_supported` and otherwise keep the
tensor operations."""
from __future__ import annotations

from ctypes import POINTER, byref, c_float, c_int, c_longlong
from typing import Optional

import torch
from torch.autograd.function import once_differentiable

from . import native
from .hashgrid import _LevelMeta, _meta_struct

HIDDEN, MAX_LEVELS = 16, 8


P = native.P
native.register_signature("lmb_unit_position", [c_longlong, P, P, c_int, P, P, P])
native.register_signature("lmb_spacing_to_euclid", [c_longlong, P, c_float, c_float, P, P])
native.register_signature("lmb_midpoints", [c_longlong, c_int, P, P, P, P, c_longlong, P, P])
native.register_signature("lmb_prop_density", [c_longlong, P, P, c_int, POINTER(_LevelMeta), P, P, P, P, P])
native.register_signature("lmb_prop_density_bwd", [c_longlong, P, P, c_int, POINTER(_LevelMeta), P, P, P, P, P, P, P, P, P])


def unit_positions_supported(pos: torch.Tensor, box: Optional[torch.Tensor]) -> bool:
    """fp32 CUDA positions that need no gradient, and a box ``[2, 3]`` beside them (None: positions are contracted as they are)."""
    if not (native.available() and type(pos) is torch.Tensor and pos.is_cuda and pos.dtype == torch.float32):
        return False
    if pos.requires_grad and torch.is_grad_enabled():
        return False
    return box is None or (box.device == pos.device and box.dtype == torch.float32 and box.is_contiguous() and box.numel() == 6
                           and not box.requires_grad)


def unit_positions(pos: torch.Tensor, box: Optional[torch.Tensor], contract: bool):
    """``pos [N, 3]`` -> (coordinates ``[N, 3]`` in the unit cube, zero outside of it; inside mask ``[N]``)."""
    pos = pos.contiguous()
    out, inside = torch.empty_like(pos), torch.empty(pos.shape[0], dtype=torch.bool, device=pos.device)
    native.check(native.lib().lmb_unit_position(pos.shape[0], pos.data_ptr(), native.ptr(box), int(contract), out.data_ptr(), inside.data_ptr(),
                                                native.stream_ptr()), "unit_position")
    return out, inside


def _value(t: torch.Tensor) -> bool:
    """A plain fp32 CUDA tensor through which no gradient is wanted."""
    return type(t) is torch.Tensor and t.is_cuda and t.dtype == torch.float32 and not (t.requires_grad and torch.is_grad_enabled())


def spacing_supported(s: torch.Tensor) -> bool:
    return native.available() and _value(s) and s.is_contiguous()


def spacing_to_euclid(s: torch.Tensor, near: float, far: float) -> torch.Tensor:
    """Distances of the spacing coordinates ``s``; ``near`` and ``far`` are the spacing coordinates of the range's ends."""
    out = torch.empty_like(s)
    native.check(native.lib().lmb_spacing_to_euclid(s.numel(), s.data_ptr(), near, far, out.data_ptr(), native.stream_ptr()), "spacing")
    return out


def midpoints_supported(o: torch.Tensor, d: torch.Tensor, starts: torch.Tensor, ends: torch.Tensor) -> bool:
    """Rays ``[R, 3]`` and intervals ``[R, S, 1]`` whose rows are equally far apart in both."""
    if not (native.available() and all(_value(t) for t in (o, d, starts, ends)) and starts.dim() == 3 and o.dim() == 2):
        return False
    return (o.is_contiguous() and d.is_contiguous() and o.shape == d.shape == (starts.shape[0], 3) and starts.shape == ends.shape
            and starts.shape[2] == 1 and starts.stride()[:2] == ends.stride()[:2] and starts.stride(1) == 1
            and len({t.device for t in (o, d, starts, ends)}) == 1)


def midpoints(o: torch.Tensor, d: torch.Tensor, starts: torch.Tensor, ends: torch.Tensor) -> torch.Tensor:
    """``[R, S, 3]``: the middle of every interval on its ray."""
    R, S = starts.shape[:2]
    out = torch.empty(R, S, 3, device=o.device)
    native.check(native.lib().lmb_midpoints(R, S, o.data_ptr(), d.data_ptr(), starts.data_ptr(), ends.data_ptr(), starts.stride(0),
                                            out.data_ptr(), native.stream_ptr()), "midpoints")
    return out


def prop_density_supported(pos: torch.Tensor, encoding, mlp, box: Optional[torch.Tensor]) -> bool:
    """fp32 CUDA positions; one fp32 hash table of at most 8 levels with two features, 16 hidden units, no biases, no output
    activation: the shipped proposal networks."""
    from ..components.fields.encodings.hash_encoding import HashEncoding
    from ..components.fields.mlp_decoder import MLPDecoder
    from ..components.utils.general_utils import has_hooks

    if not unit_positions_supported(pos, box) or torch.is_autocast_enabled("cuda"):
        return False
    if type(encoding) is not HashEncoding or type(mlp) is not MLPDecoder or mlp.use_fused or mlp.out_activation is not None:
        return False
    meta, lin = encoding.meta, mlp.linears()
    if encoding.num_hash_table != 1 or meta.n_features != 2 or meta.n_levels > MAX_LEVELS or len(lin) != 2:
        return False
    table = encoding.tables()[0].params
    weights = [l.weight for l in lin]
    return (getattr(table, "_lmb_shadow", None) is None and table.numel() >= meta.n_params and table.data_ptr() % 8 == 0
            and tuple(weights[0].shape) == (HIDDEN, 2 * meta.n_levels) and tuple(weights[1].shape) == (1, HIDDEN)
            and all(l.bias is None for l in lin)
            and all(t.is_cuda and t.device == pos.device and t.dtype == torch.float32 and t.is_contiguous() for t in [table] + weights)
            and not has_hooks(encoding, mlp, mlp.mlp, *mlp.mlp, encoding.tables()[0]))


class _PropDensity(torch.autograd.Function):
    @staticmethod
    def forward(ctx, pos, table, w1, w2, meta, box, sink):
        out = torch.empty(pos.shape[0], device=pos.device)
        ms = _meta_struct(meta)
        native.check(native.lib().lmb_prop_density(pos.shape[0], pos.data_ptr(), native.ptr(box), int(box is None), byref(ms), table.data_ptr(),
                                                   w1.data_ptr(), w2.data_ptr(), out.data_ptr(), native.stream_ptr()), "prop_density")
        ctx.save_for_backward(pos, table, w1, w2, box)
        ctx.meta, ctx.sink = meta, sink
        return out

    @staticmethod
    @once_differentiable
    def backward(ctx, d_out):
        pos, table, w1, w2, box = ctx.saved_tensors
        n, lib = pos.shape[0], native.lib()
        ms = _meta_struct(ctx.meta)
        unit, d_feat = torch.empty_like(pos), torch.empty(n, ctx.meta.out_dim, device=pos.device)
        d_w1, d_w2 = torch.zeros_like(w1), torch.zeros_like(w2)
        d_out = d_out.contiguous()
        native.check(lib.lmb_prop_density_bwd(n, pos.data_ptr(), native.ptr(box), int(box is None), byref(ms), table.data_ptr(), w1.data_ptr(),
                                              w2.data_ptr(), d_out.data_ptr(), unit.data_ptr(), d_feat.data_ptr(), d_w1.data_ptr(),
                                              d_w2.data_ptr(), native.stream_ptr()), "prop_density_bwd")
        grad = ctx.sink if ctx.sink is not None else torch.zeros_like(table)
        native.check(lib.lmb_hashgrid_bwd(unit.data_ptr(), n, byref(ms), d_feat.data_ptr(), native.DTYPE_CODE[d_feat.dtype],
                                          grad.data_ptr(), native.stream_ptr()), "hashgrid_bwd")
        return None, (None if ctx.sink is not None else grad), d_w1, d_w2, None, None, None


def prop_density(pos: torch.Tensor, encoding, mlp, box: Optional[torch.Tensor]) -> torch.Tensor:
    """Density ``[N]`` at ``pos [N, 3]``, normalised by ``box`` or (None) contracted, zero outside of the unit cube; gradients go
    to the table and the weights."""
    table = encoding.tables()[0].params
    w1, w2 = (l.weight for l in mlp.linears())
    return _PropDensity.apply(pos.contiguous(), table, w1, w2, encoding.meta, box, getattr(table, "_lmb_grad_sink", None))
