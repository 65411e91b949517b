"""Anchor -> neural-Gaussian decoder of Scaffold-GS / Octree-GS (reference:
landmark/nerf_components/model_components/fields/anchor_decoder.py:10-242 and its fused variant
fused_anchor_decoder.py:16-244).

For each visible anchor: view direction and distance to the camera, an optional view-conditioned
blend of the feature at three strides ("feature bank"), then three 2-layer MLP heads -> per-offset
opacity (tanh), covariance (7 values: 3 scale gates + quaternion) and colour (sigmoid).  Offsets with
positive opacity become Gaussians: ``xyz = anchor + offset * scale[:3]``,
``scale = scale[3:] * sigmoid(cov[:3])``, ``rot = normalize(cov[3:7])``.

Two documented deviations from the reference: with ``add_level`` the reference overwrites the
distance-carrying input by the distance-free one (anchor_decoder.py:181-182) - here each head gets
the input its ``add_*_dist`` flag asks for; and an appearance code is an embedding vector, not a
raw camera index.
"""
from __future__ import annotations

from ctypes import c_int, c_longlong
from typing import Optional

import torch
from torch import nn

from ...ops import native
from ..model.base_module import BaseModule

P = native.P
native.register_signature("lmb_anchor_rows", [c_longlong, P, P, c_int, P, P, c_int, P, P, P])
native.register_signature("lmb_anchor_epilogue", [P, P, P, P, P, P, P, c_longlong, c_int, P, P, P, P, P, P, P, P, P, P])


class AnchorDecoder(BaseModule):
    def __init__(self, use_feat_bank: bool, add_opacity_dist: bool, add_color_dist: bool, add_cov_dist: bool,
                 view_dim: int, feat_dim: int, n_offsets: int, appearance_dim: int = 0, add_level: bool = False,
                 dist2level: Optional[str] = None):
        super().__init__()
        self.use_feat_bank, self.add_opacity_dist = use_feat_bank, add_opacity_dist
        self.add_color_dist, self.add_cov_dist = add_color_dist, add_cov_dist
        self.add_level, self.dist2level = add_level, dist2level
        self.view_dim, self.feat_dim, self.n_offsets, self.appearance_dim = view_dim, feat_dim, n_offsets, appearance_dim
        lvl = 1 if add_level else 0
        base = feat_dim + view_dim + lvl
        if use_feat_bank:
            self.mlp_feature_bank = nn.Sequential(nn.Linear(view_dim + lvl, feat_dim), nn.ReLU(True),
                                                  nn.Linear(feat_dim, 3), nn.Softmax(dim=1))
        self.mlp_opacity = nn.Sequential(nn.Linear(base + int(add_opacity_dist), feat_dim), nn.ReLU(True),
                                         nn.Linear(feat_dim, n_offsets), nn.Tanh())
        self.mlp_cov = nn.Sequential(nn.Linear(base + int(add_cov_dist), feat_dim), nn.ReLU(True),
                                     nn.Linear(feat_dim, 7 * n_offsets))
        self.mlp_color = nn.Sequential(nn.Linear(base + int(add_color_dist) + appearance_dim, feat_dim), nn.ReLU(True),
                                       nn.Linear(feat_dim, 3 * n_offsets), nn.Sigmoid())
        self.use_fused = False
        self.save_init_kwargs(locals())

    def _heads(self, feat, ob_view, ob_dist, level, appearance):
        parts = [feat, ob_view]
        tail = [level] if (self.add_level and level is not None) else []
        with_dist = torch.cat(parts + [ob_dist] + tail, dim=1)
        without = torch.cat(parts + tail, dim=1)
        op_in = with_dist if self.add_opacity_dist else without
        cov_in = with_dist if self.add_cov_dist else without
        col_in = with_dist if self.add_color_dist else without
        if self.appearance_dim > 0:
            if appearance is None:
                appearance = torch.zeros(feat.shape[0], self.appearance_dim, device=feat.device, dtype=feat.dtype)
            elif appearance.dim() == 1:
                appearance = appearance[None].expand(feat.shape[0], -1)
            col_in = torch.cat((col_in, appearance), dim=1)
        if self.use_fused and feat.is_cuda and not torch.is_grad_enabled():
            from ...ops.fused_mlp import anchor_heads_forward, anchor_heads_supported

            if anchor_heads_supported(self, op_in, cov_in, col_in):
                return anchor_heads_forward(self, op_in, cov_in, col_in)
        return self.mlp_opacity(op_in), self.mlp_cov(cov_in), self.mlp_color(col_in)

    def _rows_ok(self, camera_center, anchor, anchor_feat, offset, scaling, visible_mask, level, prog_ratio, transition_mask) -> bool:
        """Whether a view is decoded without selecting anchors by tensor operations: rendering with the fused heads, whose inputs
        are features, direction and distance alone, on plain fp32 tensors."""
        if self.training or torch.is_grad_enabled() or not self.use_fused or not anchor.is_cuda:
            return False
        if self.use_feat_bank or self.appearance_dim > 0 or (self.add_level and level is not None):
            return False
        if self.dist2level == "progressive" and prog_ratio is not None and transition_mask is not None:
            return False
        if type(self)._heads is not AnchorDecoder._heads:
            return False
        n, k = anchor.shape[0], self.n_offsets
        tensors = ((anchor, (n, 3)), (anchor_feat, (n, self.feat_dim)), (offset, (n, k, 3)), (scaling, (n, 6)))
        if any(tuple(t.shape) != shape or t.dtype != torch.float32 or not t.is_contiguous() or t.device != anchor.device
               for t, shape in tensors):
            return False
        if visible_mask.dtype != torch.bool or tuple(visible_mask.shape) != (n,) or visible_mask.device != anchor.device:
            return False
        if not (torch.is_tensor(camera_center) and tuple(camera_center.shape) in ((3,), (1, 3)) and camera_center.dtype == torch.float32
                and camera_center.is_contiguous() and camera_center.device == anchor.device):
            return False
        from ...ops.fused_mlp import anchor_heads_supported

        base = self.feat_dim + 3
        widths = [seq[0].weight.shape[1] == base + int(dist) for seq, dist in
                  ((self.mlp_opacity, self.add_opacity_dist), (self.mlp_cov, self.add_cov_dist), (self.mlp_color, self.add_color_dist))]
        return all(widths) and anchor_heads_supported(self)

    def _forward_rows(self, camera_center, anchor, anchor_feat, offset, scaling, visible_mask):
        """The visible anchors by index: one kernel writes the heads' bf16 input rows, the last one reads anchors, offsets and
        scales in place (``ops/csrc/gs_aux.cu``)."""
        from ...ops.fused_mlp import anchor_heads_on_rows, anchor_rows_width

        idx = visible_mask.nonzero(as_tuple=True)[0]
        n, dists = idx.shape[0], (self.add_opacity_dist, self.add_cov_dist, self.add_color_dist)
        widths = {d: anchor_rows_width(self.feat_dim + 3 + int(d)) for d in set(dists)}
        rows = {d: torch.empty(n, w, dtype=torch.bfloat16, device=idx.device) for d, w in widths.items()}
        for w in set(widths.values()):
            part = {d: rows[d] for d in rows if widths[d] == w}
            native.check(native.lib().lmb_anchor_rows(n, idx.data_ptr(), anchor_feat.data_ptr(), self.feat_dim, anchor.data_ptr(),
                                                      camera_center.data_ptr(), w, native.ptr(part.get(True)),
                                                      native.ptr(part.get(False)), native.stream_ptr()), "anchor_rows")
        opacity, scale_rot, color = anchor_heads_on_rows(self, *(rows[d] for d in dists))
        return (*_decode_epilogue(anchor, offset, scaling, opacity, color, scale_rot, self.n_offsets, idx), None, None)

    def forward(self, camera_center, anchor, anchor_feat, offset, scaling, visible_mask=None, level=None,
                prog_ratio=None, transition_mask=None, appearance_code=None):
        if visible_mask is None:
            visible_mask = torch.ones(anchor.shape[0], dtype=torch.bool, device=anchor.device)
        if self._rows_ok(camera_center, anchor, anchor_feat, offset, scaling, visible_mask, level, prog_ratio, transition_mask):
            return self._forward_rows(camera_center, anchor, anchor_feat, offset, scaling, visible_mask)
        anchor, feat = anchor[visible_mask], anchor_feat[visible_mask]
        grid_offsets, grid_scaling = offset[visible_mask], scaling[visible_mask]
        if self.add_level and level is not None:
            level = level[visible_mask].reshape(-1, 1).to(feat.dtype)
        ob_view = anchor - camera_center
        ob_dist = ob_view.norm(dim=1, keepdim=True)
        ob_view = ob_view / ob_dist
        if self.use_feat_bank:
            bank_in = torch.cat((ob_view, level), dim=1) if (self.add_level and level is not None) else ob_view
            w = self.mlp_feature_bank(bank_in)                                  # [n, 3]
            feat = (feat[:, ::4].repeat(1, 4) * w[:, 0:1] + feat[:, ::2].repeat(1, 2) * w[:, 1:2]
                    + feat * w[:, 2:3])
        neural_opacity, scale_rot, color = self._heads(feat, ob_view, ob_dist, level, appearance_code)
        if self.dist2level == "progressive" and prog_ratio is not None and transition_mask is not None:
            prog = prog_ratio[visible_mask].clone().reshape(-1, 1)
            prog[~transition_mask[visible_mask]] = 1.0
            neural_opacity = neural_opacity * prog
        k = self.n_offsets
        if not self.training and not torch.is_grad_enabled() and anchor.is_cuda and neural_opacity.dtype == torch.float32:
            from ...ops import native

            if native.available():
                return (*_decode_epilogue(anchor, grid_offsets, grid_scaling, neural_opacity, color, scale_rot, k), None, None)
        neural_opacity = neural_opacity.reshape(-1, 1)
        mask = (neural_opacity > 0.0).view(-1)
        opacity = neural_opacity[mask]
        color = color.reshape(-1, 3)[mask]
        scale_rot = scale_rot.reshape(-1, 7)[mask]
        offsets = grid_offsets.reshape(-1, 3)[mask]
        idx = torch.arange(anchor.shape[0], device=anchor.device).repeat_interleave(k)[mask]
        scaling_rep, anchor_rep = grid_scaling[idx], anchor[idx]
        out_scaling = scaling_rep[:, 3:] * torch.sigmoid(scale_rot[:, :3])
        rot = torch.nn.functional.normalize(scale_rot[:, 3:7])
        xyz = anchor_rep + offsets * scaling_rep[:, :3]
        if self.training:
            return xyz, color, opacity, out_scaling, rot, neural_opacity, mask
        return xyz, color, opacity, out_scaling, rot, None, None


def _decode_epilogue(anchor, offsets, scaling, opacity, color, scale_rot, k: int, idx=None):
    """Render-time tail of the decoder as one flag / scan / scatter kernel sequence (``ops/csrc/gs_aux.cu``): opacity mask,
    order-preserving compaction and the Gaussian attributes of the kept candidates.  ``idx``: the rows of ``anchor``, ``offsets`` and
    ``scaling`` that were decoded (all of them without it).  One host read (the count)."""
    lib, dev = native.lib(), anchor.device
    n = (anchor if idx is None else idx).shape[0] * k
    f = lambda t: t.detach().contiguous().float()  # noqa: E731
    anchor, offsets, scaling, opacity, color, scale_rot = map(f, (anchor, offsets, scaling, opacity, color, scale_rot))
    work = torch.empty(2, max(n, 1), dtype=torch.int32, device=dev)
    scratch = torch.empty(max(lib.lmb_scan_scratch_bytes(max(n, 1)), 4), dtype=torch.uint8, device=dev)
    xyz, col, scl, rot, opa = (torch.empty(max(n, 1), w, dtype=torch.float32, device=dev) for w in (3, 3, 3, 4, 1))
    count = torch.zeros(1, dtype=torch.int32, device=dev)
    native.check(lib.lmb_anchor_epilogue(anchor.data_ptr(), offsets.data_ptr(), scaling.data_ptr(), opacity.data_ptr(),
                                         color.data_ptr(), scale_rot.data_ptr(), native.ptr(idx), n, k, work[0].data_ptr(),
                                         work[1].data_ptr(), scratch.data_ptr(), xyz.data_ptr(), col.data_ptr(), opa.data_ptr(), scl.data_ptr(),
                                         rot.data_ptr(), count.data_ptr(), native.stream_ptr()), "anchor_epilogue")
    m = int(count.item())
    return xyz[:m], col[:m], opa[:m], scl[:m], rot[:m]


class FusedAnchorDecoder(AnchorDecoder):
    """Same decoder with the three heads evaluated by the fused MLP kernel at render time."""

    def __init__(self, *args, **kwargs):
        super().__init__(*args, **kwargs)
        self.use_fused = True
