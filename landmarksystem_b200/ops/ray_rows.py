"""Marched samples as rows (``csrc/ray_rows.cu``): the samples of ray ``r`` are rows ``offsets[r] .. offsets[r + 1]`` of compact
arrays, in order."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong
from typing import List, Optional, Tuple

import torch
from torch.autograd.function import once_differentiable

from . import native

P = native.P
native.register_signature("lmb_row_index", [c_int, c_int, P, P, P])
native.register_signature("lmb_rows_composite", [c_int, c_int, P, P, P, P, P, c_float, P, P, P])
native.register_signature("lmb_rows_composite_bwd", [c_int, c_int, P, P, P, P, P, c_float, P, P, P, P])
native.register_signature("lmb_exclusive_scan_u32", [P, P, c_longlong, P, P])


class RowCounts:
    """Numbers of rows up to the end of every ``chunk`` rays on their way to the host: :meth:`wait` waits for the scan alone, not for
    work queued after it."""

    def __init__(self, offsets: torch.Tensor, chunk: int):
        ends = offsets[-1:] if offsets.shape[0] - 1 <= chunk else torch.cat((offsets[chunk:-1:chunk], offsets[-1:]))
        self.value = torch.empty(ends.shape[0], dtype=offsets.dtype, pin_memory=True)
        self.value.copy_(ends, non_blocking=True)
        self.event = torch.cuda.Event()
        self.event.record()

    def wait(self) -> List[int]:
        self.event.synchronize()
        return self.value.tolist()


def row_offsets(counts: torch.Tensor) -> Tuple[torch.Tensor, int]:
    """``counts int32 [R]`` -> ``(offsets int32 [R + 1], number of rows)``; the one host read of a marched batch."""
    offsets = scan_counts(counts)
    return offsets, int(offsets[-1].item())


@torch.no_grad()
def scan_counts(counts: torch.Tensor) -> torch.Tensor:
    """``counts int32 [R]`` -> offsets ``int32 [R + 1]``, the last of which is the number of rows."""
    lib, R = native.lib(), counts.shape[0]
    padded = torch.nn.functional.pad(counts, (0, 1))
    offsets = torch.empty_like(padded)
    scratch = torch.empty(lib.lmb_scan_scratch_bytes(R + 1), dtype=torch.uint8, device=counts.device)
    native.check(lib.lmb_exclusive_scan_u32(padded.data_ptr(), offsets.data_ptr(), R + 1, scratch.data_ptr(), native.stream_ptr()), "scan")
    return offsets


@torch.no_grad()
def row_index(offsets: torch.Tensor, rows: int, samples_per_ray: int) -> Optional[torch.Tensor]:
    """Flat slot ``ray * samples_per_ray + s`` of every row (int64), None when every slot is a row."""
    R = offsets.shape[0] - 1
    if rows == R * samples_per_ray:
        return None
    idx = torch.empty(rows, dtype=torch.int64, device=offsets.device)
    native.check(native.lib().lmb_row_index(R, samples_per_ray, offsets.data_ptr(), idx.data_ptr(), native.stream_ptr()), "row_index")
    return idx


class _Composite(torch.autograd.Function):
    @staticmethod
    def forward(ctx, sigma, rgb, offsets, ts, te, bg):
        R, S = ts.shape
        out, depth = torch.empty(R, 3, device=ts.device), torch.empty(R, device=ts.device)
        native.check(native.lib().lmb_rows_composite(R, S, offsets.data_ptr(), sigma.data_ptr(), rgb.data_ptr(), ts.data_ptr(),
                                                     te.data_ptr(), bg, out.data_ptr(), depth.data_ptr(), native.stream_ptr()),
                     "rows_composite")
        ctx.save_for_backward(sigma, rgb, offsets, ts, te)
        ctx.bg = bg
        ctx.mark_non_differentiable(depth)
        return out, depth

    @staticmethod
    @once_differentiable
    def backward(ctx, d_out, _d_depth):
        sigma, rgb, offsets, ts, te = ctx.saved_tensors
        R, S = ts.shape
        d_sigma, d_rgb, d_out = torch.empty_like(sigma), torch.empty_like(rgb), d_out.contiguous()
        native.check(native.lib().lmb_rows_composite_bwd(R, S, offsets.data_ptr(), sigma.data_ptr(), rgb.data_ptr(), ts.data_ptr(),
                                                         te.data_ptr(), ctx.bg, d_out.data_ptr(), d_sigma.data_ptr(), d_rgb.data_ptr(),
                                                         native.stream_ptr()), "rows_composite_bwd")
        return d_sigma, d_rgb, None, None, None, None


def composite_rows_of_rays(sigma: torch.Tensor, rgb: torch.Tensor, offsets: torch.Tensor, ts: torch.Tensor, te: torch.Tensor,
                           bg: float = 0.0) -> Tuple[torch.Tensor, torch.Tensor]:
    """Densities ``[M]`` and colours ``[M, 3]`` of the rows, intervals ``ts / te [R, S]`` -> ``(rgb [R, 3] unclamped, depth [R])``:
    the volume renderer's weights and composite; gradients go to densities and colours."""
    return _Composite.apply(sigma.contiguous().float(), rgb.contiguous().float(), offsets, ts.contiguous().float(),
                            te.contiguous().float(), float(bg))
