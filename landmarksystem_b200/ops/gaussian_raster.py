"""3D Gaussian splatting rasteriser: public module API, CUDA path and PyTorch oracle.

API mirrors what the reference imports from its rasteriser extension
(``GaussianRasterizationSettings`` / ``GaussianRasterizer(...)(means3D, means2D, shs, colors_precomp,
opacities, scales, rotations, cov3D_precomp) -> (image [3,H,W], radii [N], extra)`` and
``.visible_filter(...) -> radii``; call sites benchmarks/nerf/origin_gs/gs_model.py:82-97,148-162,
211-220).  CUDA tensors run ``csrc/gs_raster.cu`` + ``csrc/sort_scan.cu``; CPU tensors run
:func:`rasterize_reference`, a dense differentiable PyTorch statement of the same math that serves as
the numerics oracle (small scenes only).
"""
from __future__ import annotations

from ctypes import POINTER, Structure, byref, c_float, c_int, c_longlong
from typing import NamedTuple, Optional

import torch
from torch import nn

from . import native

TILE = 16
MAX_COEFFS = 16


class GaussianRasterizationSettings(NamedTuple):
    image_height: int
    image_width: int
    tanfovx: float
    tanfovy: float
    bg: torch.Tensor
    scale_modifier: float
    viewmatrix: torch.Tensor      # [4,4] transposed world-to-view (row-vector convention)
    projmatrix: torch.Tensor      # [4,4] viewmatrix @ projection
    sh_degree: int
    campos: torch.Tensor
    prefiltered: bool = False
    debug: bool = False


class GSCameraInfo(Structure):
    _fields_ = [("tanfovx", c_float), ("tanfovy", c_float), ("W", c_int), ("H", c_int), ("scale_modifier", c_float),
                ("sh_degree", c_int), ("sh_coeffs", c_int)]


P = native.P
native.register_signature("lmb_gs_project", [c_int, P, P, P, P, P, P, P, P, P, POINTER(GSCameraInfo), P, P, P, P, P, P, P, c_int, P])
native.register_signature("lmb_gs_draw", [c_int, P, P, P, P, c_int, c_int, c_longlong, c_longlong, P, P, P, P, P, P, P, P, P, P])
native.register_signature("lmb_gs_tile_words", [c_int, c_int, c_int])
native.register_signature("lmb_gs_sort_scratch_bytes", [c_int, c_longlong, c_longlong], c_longlong)
native.register_signature("lmb_gs_render_bwd", [P, P, c_int, c_int, P, P, P, P, P, P, P])
native.register_signature("lmb_gs_preprocess_bwd", [c_int, P, P, P, P, P, P, P, POINTER(GSCameraInfo), P, P, P, P, P, P, P, P,
                                                     P, P, P])
native.register_signature("lmb_exclusive_scan_u32", [P, P, c_longlong, P, P])
native.register_signature("lmb_radix_sort_pairs", [P, P, P, c_longlong, c_int, c_int, P, P])


def _lib_ll(name):
    return getattr(native.lib(), name)


def _camera_info(s: GaussianRasterizationSettings, sh_coeffs: int) -> GSCameraInfo:
    return GSCameraInfo(s.tanfovx, s.tanfovy, s.image_width, s.image_height, s.scale_modifier, s.sh_degree, sh_coeffs)


def _camera_pose(s: GaussianRasterizationSettings, device) -> torch.Tensor:
    """View and projection matrix and camera position as 35 floats on ``device``; nothing waits for them on the host."""
    pose = torch.cat([t.detach().reshape(-1)[:n].to(device=device, dtype=torch.float32)      # a position may be homogeneous
                      for t, n in ((s.viewmatrix, 16), (s.projmatrix, 16), (s.campos, 3))])
    if pose.numel() != 35:
        raise ValueError("viewmatrix and projmatrix are [4, 4], campos is [3]")
    return pose


# ---------------------------------------------------------------------------------------------------
# PyTorch oracle
# ---------------------------------------------------------------------------------------------------
def _quat_to_rot(q):
    r, x, y, z = q.unbind(-1)
    return torch.stack((1 - 2 * (y * y + z * z), 2 * (x * y - r * z), 2 * (x * z + r * y),
                        2 * (x * y + r * z), 1 - 2 * (x * x + z * z), 2 * (y * z - r * x),
                        2 * (x * z - r * y), 2 * (y * z + r * x), 1 - 2 * (x * x + y * y)), -1).reshape(-1, 3, 3)


def project_reference(means3D, scales, rotations, cov3D_precomp, s: GaussianRasterizationSettings):
    """Per-Gaussian screen quantities: ``(xy [N,2], depth [N], conic [N,3], radii [N], valid [N])``."""
    N = means3D.shape[0]
    V, Pm = s.viewmatrix.to(means3D), s.projmatrix.to(means3D)
    hom = torch.cat((means3D, torch.ones(N, 1, dtype=means3D.dtype, device=means3D.device)), -1)
    t = (hom @ V)[:, :3]
    ph = hom @ Pm
    ndc = ph[:, :2] / (ph[:, 3:4] + 1e-7)
    if cov3D_precomp is not None:
        c = cov3D_precomp
        Sigma = torch.stack((c[:, 0], c[:, 1], c[:, 2], c[:, 1], c[:, 3], c[:, 4], c[:, 2], c[:, 4], c[:, 5]), -1).reshape(-1, 3, 3)
    else:
        R = _quat_to_rot(rotations)
        M = R * (scales * s.scale_modifier)[:, None, :]
        Sigma = M @ M.transpose(1, 2)
    W, H = s.image_width, s.image_height
    fx, fy = W / (2 * s.tanfovx), H / (2 * s.tanfovy)
    tz = t[:, 2]
    limx, limy = 1.3 * s.tanfovx, 1.3 * s.tanfovy
    txz = torch.clamp(t[:, 0] / tz, -limx, limx) * tz
    tyz = torch.clamp(t[:, 1] / tz, -limy, limy) * tz
    zeros = torch.zeros_like(tz)
    J = torch.stack((fx / tz, zeros, -fx * txz / (tz * tz), zeros, fy / tz, -fy * tyz / (tz * tz)), -1).reshape(-1, 2, 3)
    Wr = V[:3, :3].t()
    T = J @ Wr
    cov = T @ Sigma @ T.transpose(1, 2)
    a, b, c = cov[:, 0, 0] + 0.3, cov[:, 0, 1], cov[:, 1, 1] + 0.3
    det = a * c - b * b
    conic = torch.stack((c / det, -b / det, a / det), -1)
    mid = 0.5 * (a + c)
    lam = mid + torch.sqrt(torch.clamp(mid * mid - det, min=0.1))
    radii = torch.ceil(3.0 * torch.sqrt(lam)).int()
    xy = torch.stack((((ndc[:, 0] + 1) * W - 1) * 0.5, ((ndc[:, 1] + 1) * H - 1) * 0.5), -1)
    valid = (tz > 0.2) & (det != 0)
    return xy, tz, conic, radii, valid


def _tile_rect(xy, radii, W, H):
    tx, ty = (W + TILE - 1) // TILE, (H + TILE - 1) // TILE
    r = radii.to(xy.dtype)
    x0 = torch.clamp(((xy[:, 0] - r) / TILE).int(), 0, tx)
    y0 = torch.clamp(((xy[:, 1] - r) / TILE).int(), 0, ty)
    x1 = torch.clamp(((xy[:, 0] + r + TILE - 1) / TILE).int(), 0, tx)
    y1 = torch.clamp(((xy[:, 1] + r + TILE - 1) / TILE).int(), 0, ty)
    return x0, y0, x1, y1


def rasterize_reference(means3D, opacities, s: GaussianRasterizationSettings, shs=None, colors_precomp=None, scales=None,
                        rotations=None, cov3D_precomp=None, visible=None):
    """Dense differentiable oracle: every pixel blends all Gaussians whose tile rectangle covers it."""
    from ..components.utils.sh_utils import eval_sh

    W, H = s.image_width, s.image_height
    xy, depth, conic, radii, valid = project_reference(means3D, scales, rotations, cov3D_precomp, s)
    x0, y0, x1, y1 = _tile_rect(xy.detach(), radii, W, H)
    valid = valid & ((x1 - x0) * (y1 - y0) > 0)
    if visible is not None:
        valid = valid & visible.bool()
    if colors_precomp is None:
        dirs = means3D - s.campos.to(means3D)
        dirs = dirs / dirs.norm(dim=-1, keepdim=True)
        colors = torch.clamp_min(eval_sh(s.sh_degree, shs.transpose(1, 2), dirs) + 0.5, 0.0)
    else:
        colors = colors_precomp
    order = torch.argsort(depth.detach() + (~valid) * 1e10, stable=True)
    order = order[valid[order]]
    ys, xs = torch.meshgrid(torch.arange(H, device=means3D.device), torch.arange(W, device=means3D.device), indexing="ij")
    pix = torch.stack((xs, ys), -1).reshape(-1, 2).to(means3D.dtype)          # [P, 2]
    tile_x, tile_y = (xs // TILE).reshape(-1), (ys // TILE).reshape(-1)
    T = torch.ones(H * W, dtype=means3D.dtype, device=means3D.device)
    C = torch.zeros(H * W, 3, dtype=means3D.dtype, device=means3D.device)
    done = torch.zeros(H * W, dtype=torch.bool, device=means3D.device)
    for g in order.tolist():
        cover = (tile_x >= x0[g]) & (tile_x < x1[g]) & (tile_y >= y0[g]) & (tile_y < y1[g]) & ~done
        d = xy[g][None] - pix
        power = -0.5 * (conic[g, 0] * d[:, 0] ** 2 + conic[g, 2] * d[:, 1] ** 2) - conic[g, 1] * d[:, 0] * d[:, 1]
        alpha = torch.clamp(opacities[g].reshape(()) * torch.exp(power), max=0.99)
        use = cover & (power <= 0) & (alpha >= 1.0 / 255.0)
        test_T = T * (1 - alpha)
        stop = use & (test_T < 1e-4)
        done = done | stop
        use = use & ~stop
        w = torch.where(use, alpha * T, torch.zeros_like(T))
        C = C + w[:, None] * colors[g][None]
        T = torch.where(use, test_T, T)
    img = C + T[:, None] * s.bg.to(means3D)[None]
    out_radii = torch.where(valid, radii, torch.zeros_like(radii))
    return img.t().reshape(3, H, W), out_radii, (1.0 - T).reshape(H, W).detach()


# ---------------------------------------------------------------------------------------------------
# CUDA path
# ---------------------------------------------------------------------------------------------------
def _f32(t: Optional[torch.Tensor]) -> Optional[torch.Tensor]:
    """Contiguous fp32 on a 16-byte boundary: the kernels read rows of several floats as float4."""
    if t is None:
        return None
    t = t.contiguous().float()
    return t if t.data_ptr() % 16 == 0 else t.clone()


def _sort_scratch(N: int, total: int, most: int, device) -> torch.Tensor:
    """Temporary storage of the draw on the current stream (from the caching allocator: safe with several streams)."""
    return torch.empty(native.lib().lmb_gs_sort_scratch_bytes(N, total, most), dtype=torch.uint8, device=device)


def _project(means3D, scales, rotations, opacities, shs, sh_rest, colors_precomp, cov3D_precomp, visible, info, pose, radius_only):
    """``radii`` alone, or ``(radii, records [N, 12], tiles touched [N], tiles)``; tiles: where every
    tile's pairs go (the first word is their start; one draw uses it up), their ranges ``[tiles, 2]`` and the totals ``[2]``, all pairs
    and those of the fullest tile."""
    N, dev = means3D.shape[0], means3D.device
    radii = torch.empty(N, dtype=torch.int32, device=dev)
    rec = touched = cursors = ranges = totals = None
    if not radius_only:
        n_tiles = ((info.W + TILE - 1) // TILE) * ((info.H + TILE - 1) // TILE)
        rec = torch.empty(N, 12, device=dev)
        touched = torch.empty(N, dtype=torch.int32, device=dev)
        words = native.lib().lmb_gs_tile_words(N, info.W, info.H)
        cursors, ranges = (torch.empty(n_tiles, w, dtype=torch.int32, device=dev) for w in (words, 2))
        totals = torch.empty(2, dtype=torch.int32, device=dev)
    native.check(native.lib().lmb_gs_project(N, means3D.data_ptr(), native.ptr(scales), native.ptr(rotations), native.ptr(opacities),
                                             native.ptr(shs), native.ptr(sh_rest), native.ptr(colors_precomp),
                                             native.ptr(cov3D_precomp), native.ptr(visible), byref(info), pose.data_ptr(),
                                             radii.data_ptr(), native.ptr(rec), native.ptr(touched), native.ptr(cursors),
                                             native.ptr(ranges), native.ptr(totals), int(radius_only), native.stream_ptr()), "gs_project")
    return radii if radius_only else (radii, rec, touched, (cursors, ranges, totals))


class _Rasterize(torch.autograd.Function):
    """``shs``: all coefficients ``[N, K, 3]``, or the constant ones ``[N, 1, 3]`` with the others in ``sh_rest``."""

    @staticmethod
    def forward(ctx, means3D, means2D, shs, sh_rest, colors_precomp, opacities, scales, rotations, cov3D_precomp, visible, settings):
        s = settings
        N, dev = means3D.shape[0], means3D.device
        W, H = s.image_width, s.image_height
        info = _camera_info(s, 0 if shs is None else shs.shape[1] + (0 if sh_rest is None else sh_rest.shape[1]))
        pose = _camera_pose(s, dev)
        means3D, shs, sh_rest, colors_precomp = _f32(means3D), _f32(shs), _f32(sh_rest), _f32(colors_precomp)
        opacities, scales, rotations, cov3D_precomp = _f32(opacities), _f32(scales), _f32(rotations), _f32(cov3D_precomp)
        vis = None if visible is None else visible.to(torch.uint8).contiguous()
        radii, rec, touched, (cursors, ranges, totals) = _project(means3D, scales, rotations, opacities, shs, sh_rest, colors_precomp, cov3D_precomp,
                                                                  vis, info, pose, False)
        total, most = totals.tolist()                                      # one host sync per frame
        keys = torch.empty(total, dtype=torch.int64, device=dev)
        vals = torch.empty(total, dtype=torch.int32, device=dev)
        scratch = _sort_scratch(N, total, most, dev)
        color, alpha, final_T = torch.empty(3, H, W, device=dev), torch.empty(H, W, device=dev), torch.empty(H, W, device=dev)
        n_contrib = torch.empty(H, W, dtype=torch.int32, device=dev)
        bg = s.bg.to(dev).float().contiguous()
        native.check(native.lib().lmb_gs_draw(N, rec.data_ptr(), radii.data_ptr(), touched.data_ptr(), cursors.data_ptr(), W, H, total,
                                              most, keys.data_ptr(), vals.data_ptr(), scratch.data_ptr(), ranges.data_ptr(), bg.data_ptr(),
                                              color.data_ptr(), alpha.data_ptr(), final_T.data_ptr(), n_contrib.data_ptr(),
                                              native.stream_ptr()), "gs_draw")
        ctx.settings, ctx.info = s, info
        ctx.save_for_backward(means3D, scales, rotations, shs, sh_rest, cov3D_precomp, radii, rec, final_T, n_contrib, ranges, vals,
                              bg, pose)
        ctx.mark_non_differentiable(radii, alpha)
        return color, radii, alpha

    @staticmethod
    def backward(ctx, dcolor, _dradii, _dalpha):
        (means3D, scales, rotations, shs, sh_rest, cov3D, radii, rec, final_T, n_contrib, ranges, vals, bg,
         pose) = ctx.saved_tensors
        s = ctx.settings
        N, dev = means3D.shape[0], means3D.device
        W, H = s.image_width, s.image_height
        lib = native.lib()
        dcolor = dcolor.contiguous().float()
        grad = torch.zeros(N, 12, device=dev)
        native.check(lib.lmb_gs_render_bwd(ranges.data_ptr(), vals.data_ptr(), W, H, bg.data_ptr(), rec.data_ptr(),
                                           final_T.data_ptr(), n_contrib.data_ptr(), dcolor.data_ptr(), grad.data_ptr(),
                                           native.stream_ptr()), "gs_render_bwd")
        d_means, d_means2D, d_opacity = torch.empty(N, 3, device=dev), torch.empty(N, 3, device=dev), torch.empty(N, 1, device=dev)
        d_scales = None if scales is None else torch.empty(N, 3, device=dev)
        d_rots = None if scales is None else torch.empty(N, 4, device=dev)
        d_shs = None if shs is None else torch.empty_like(shs)
        d_rest = None if sh_rest is None else torch.empty_like(sh_rest)
        d_cols = torch.empty(N, 3, device=dev) if shs is None else None
        native.check(lib.lmb_gs_preprocess_bwd(N, means3D.data_ptr(), native.ptr(scales), native.ptr(rotations), native.ptr(shs),
                                               native.ptr(sh_rest), native.ptr(cov3D), radii.data_ptr(), byref(ctx.info),
                                               pose.data_ptr(), grad.data_ptr(), d_means.data_ptr(), d_means2D.data_ptr(),
                                               d_opacity.data_ptr(), native.ptr(d_scales), native.ptr(d_rots), native.ptr(d_shs),
                                               native.ptr(d_rest), native.ptr(d_cols), native.stream_ptr()), "gs_preprocess_bwd")
        # means2D receives the NDC-space screen gradient (what densification statistics accumulate)
        return d_means, d_means2D, d_shs, d_rest, d_cols, d_opacity, d_scales, d_rots, None, None, None


class GaussianRasterizer(nn.Module):
    def __init__(self, raster_settings: GaussianRasterizationSettings):
        super().__init__()
        self.raster_settings = raster_settings

    def visible_filter(self, means3D, scales=None, rotations=None, cov3D_precomp=None):
        """Radii of the Gaussians for this view without rendering (0 = culled)."""
        s = self.raster_settings
        with torch.no_grad():
            if not means3D.is_cuda:
                xy, _, _, radii, valid = project_reference(means3D, scales, rotations, cov3D_precomp, s)
                x0, y0, x1, y1 = _tile_rect(xy, radii, s.image_width, s.image_height)
                return torch.where(valid & ((x1 - x0) * (y1 - y0) > 0), radii, torch.zeros_like(radii))
            return _project(_f32(means3D), _f32(scales), _f32(rotations), None, None, None, None, _f32(cov3D_precomp), None,
                            _camera_info(s, 0), _camera_pose(s, means3D.device), True)

    def forward(self, means3D, means2D, opacities, shs=None, colors_precomp=None, scales=None, rotations=None,
                cov3D_precomp=None, visible_mask=None):
        """``shs``: ``[N, K, 3]``, or the pair ``([N, 1, 3], [N, K - 1, 3])`` in which a Gaussian model stores them."""
        s = self.raster_settings
        assert (shs is None) != (colors_precomp is None), "provide exactly one of shs / colors_precomp"
        assert ((scales is None or rotations is None) != (cov3D_precomp is None)), \
            "provide exactly one of (scales, rotations) / cov3D_precomp"
        sh_rest = None
        if isinstance(shs, (tuple, list)):
            shs, sh_rest = shs if means3D.is_cuda and shs[0].shape[1] == 1 else (torch.cat(tuple(shs), dim=1), None)
        if not means3D.is_cuda:
            img, radii, alpha = rasterize_reference(means3D, opacities, s, shs, colors_precomp, scales, rotations,
                                                    cov3D_precomp, visible_mask)
            return img, radii, alpha
        # the kernels evaluate 16 coefficients and stage a Gaussian's whole row: any others stay out of it (their gradient is zero)
        if shs is not None and shs.shape[1] > MAX_COEFFS:
            shs = shs[:, :MAX_COEFFS]
        if sh_rest is not None and sh_rest.shape[1] > MAX_COEFFS - 1:
            sh_rest = sh_rest[:, :MAX_COEFFS - 1]
        if means2D is None:
            means2D = torch.zeros_like(means3D, requires_grad=means3D.requires_grad)
        return _Rasterize.apply(means3D, means2D, shs, sh_rest, colors_precomp, opacities, scales, rotations, cov3D_precomp,
                                visible_mask, s)
