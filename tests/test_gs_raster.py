"""Gaussian rasteriser: CPU oracle self-checks and CUDA kernels vs the oracle (forward and backward)."""
import math

import pytest
import torch

from landmarksystem_b200.components.data.cameras import Camera
from landmarksystem_b200.ops.gaussian_raster import GaussianRasterizationSettings, GaussianRasterizer
from landmarksystem_b200.synthetic import look_at


def _scene(n=60, W=48, H=32, seed=0, sh=True):
    g = torch.Generator().manual_seed(seed)
    means = (torch.rand(n, 3, generator=g) - 0.5) * torch.tensor([2.0, 1.4, 1.0])
    scales = torch.exp(torch.randn(n, 3, generator=g) * 0.3 - 2.2)
    rots = torch.nn.functional.normalize(torch.randn(n, 4, generator=g), dim=-1)
    opac = torch.sigmoid(torch.randn(n, 1, generator=g))
    shs = torch.randn(n, 16, 3, generator=g) * 0.2 if sh else None
    cols = None if sh else torch.rand(n, 3, generator=g)
    c2w = look_at(torch.tensor([0.3, -0.2, 3.0]), torch.zeros(3), up=(0.0, 1.0, 0.0)).numpy()
    cam = Camera.from_c2w(c2w, W, H, focal_x=40.0)
    s = GaussianRasterizationSettings(H, W, cam.tanfovx, cam.tanfovy, torch.tensor([0.1, 0.2, 0.3]), 1.0,
                                      cam.world_view_transform, cam.full_proj_transform, 3 if sh else 0, cam.camera_center)
    return means, scales, rots, opac, shs, cols, s


def test_reference_renders_something_and_is_differentiable():
    means, scales, rots, opac, shs, cols, s = _scene(n=20)
    means.requires_grad_()
    img, radii, alpha = GaussianRasterizer(s)(means, None, opac, shs=shs, scales=scales, rotations=rots)
    assert img.shape == (3, 32, 48) and (radii > 0).sum() > 5 and alpha.max() > 0.1
    img.sum().backward()
    assert torch.isfinite(means.grad).all() and means.grad.abs().sum() > 0


@pytest.mark.gpu
@pytest.mark.parametrize("sh", [True, False])
def test_cuda_matches_reference_forward_backward(sh):
    means, scales, rots, opac, shs, cols, s = _scene(sh=sh)
    leaves_c = [t.clone().requires_grad_() for t in (means, scales, rots, opac, shs if sh else cols)]
    mc, sc, rc, oc, cc = leaves_c
    img_ref, radii_ref, _ = GaussianRasterizer(s)(mc, None, oc, shs=cc if sh else None, colors_precomp=None if sh else cc,
                                                   scales=sc, rotations=rc)
    w = torch.rand(3, s.image_height, s.image_width, generator=torch.Generator().manual_seed(1))
    (img_ref * w).sum().backward()
    leaves_g = [t.clone().cuda().requires_grad_() for t in (means, scales, rots, opac, shs if sh else cols)]
    mg, sg, rg, og, cg = leaves_g
    img, radii, _ = GaussianRasterizer(s)(mg, None, og, shs=cg if sh else None, colors_precomp=None if sh else cg,
                                           scales=sg, rotations=rg)
    assert torch.equal(radii.cpu(), radii_ref)
    assert torch.allclose(img.cpu(), img_ref, atol=2e-4), (img.cpu() - img_ref).abs().max()
    (img * w.cuda()).sum().backward()
    for name, a, b in zip(("means", "scales", "rots", "opacity", "colour"), leaves_g, leaves_c):
        scale = b.grad.abs().max().item() + 1e-8
        assert torch.allclose(a.grad.cpu(), b.grad, atol=2e-3 * scale + 1e-6, rtol=1e-2), (name, (a.grad.cpu() - b.grad).abs().max(), scale)


@pytest.mark.gpu
@pytest.mark.parametrize("n,W,H,degree", [(1, 17, 5, 0), (33, 16, 16, 1), (97, 53, 37, 2), (300, 31, 66, 3)])
def test_cuda_matches_reference_at_partial_tiles(n, W, H, degree):
    """Partial tiles and warps, fewer SH coefficients than the maximum, opacities on both sides of the 1/255 cut, splats
    from sub-pixel to larger than a tile (same tolerances as the test above: fp32 sums in another order)."""
    means, scales, rots, opac, shs, _, s = _scene(n=n, W=W, H=H, seed=n)
    g = torch.Generator().manual_seed(n + 1)
    scales = scales * torch.exp(torch.rand(n, 1, generator=g) * 4.0 - 2.5)
    opac = torch.exp(-7.0 * torch.rand(n, 1, generator=g))
    shs = shs[:, :(degree + 1) ** 2].contiguous()
    s = s._replace(sh_degree=degree)
    w = torch.rand(3, H, W, generator=g)
    out = []
    for dev in ("cpu", "cuda"):
        leaves = [t.clone().to(dev).requires_grad_() for t in (means, scales, rots, opac, shs)]
        img, radii, alpha = GaussianRasterizer(s)(leaves[0], None, leaves[3], shs=leaves[4], scales=leaves[1], rotations=leaves[2])
        (img * w.to(dev)).sum().backward()
        out.append((img.detach().cpu(), radii.cpu(), alpha.cpu(), [t.grad.cpu() for t in leaves]))
    (img_ref, radii_ref, alpha_ref, grads_ref), (img, radii, alpha, grads) = out
    assert torch.equal(radii, radii_ref)
    assert torch.allclose(img, img_ref, atol=2e-4) and torch.allclose(alpha, alpha_ref, atol=2e-4)
    for a, b in zip(grads, grads_ref):
        assert torch.allclose(a, b, atol=2e-3 * float(b.abs().max()) + 1e-6, rtol=1e-2), float((a - b).abs().max())


@pytest.mark.gpu
def test_visible_filter_matches_radii():
    means, scales, rots, opac, shs, cols, s = _scene(n=500)
    r_cpu = GaussianRasterizer(s).visible_filter(means, scales, rots)
    r_gpu = GaussianRasterizer(s).visible_filter(means.cuda(), scales.cuda(), rots.cuda())
    assert torch.equal(r_cpu, r_gpu.cpu())


@pytest.mark.gpu
def test_radix_sort_and_scan():
    from landmarksystem_b200.ops import native
    from landmarksystem_b200.ops.gaussian_raster import _lib_ll

    torch.manual_seed(0)
    n = 300_000
    keys = torch.randint(0, 2 ** 44, (n,), dtype=torch.int64, device="cuda")
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    ref_keys, order = torch.sort(keys, stable=True)
    ws = torch.empty(_lib_ll("lmb_radix_sort_scratch_bytes")(n), dtype=torch.uint8, device="cuda")
    native.check(native.lib().lmb_radix_sort_pairs(keys.data_ptr(), vals.data_ptr(), None, n, 0, 48, ws.data_ptr(),
                                                   native.stream_ptr()), "sort")
    assert torch.equal(keys, ref_keys) and torch.equal(vals.long(), order)
    x = torch.randint(0, 50, (n,), dtype=torch.int32, device="cuda")
    out = torch.empty_like(x)
    ws2 = torch.empty(_lib_ll("lmb_scan_scratch_bytes")(n), dtype=torch.uint8, device="cuda")
    native.check(native.lib().lmb_exclusive_scan_u32(x.data_ptr(), out.data_ptr(), n, ws2.data_ptr(), native.stream_ptr()), "scan")
    assert torch.equal(out.long(), torch.cumsum(x.long(), 0) - x.long())


def test_baseline_restatement_agrees_with_the_oracle():
    """The PyTorch restatement timed as the 3DGS baseline (``baseline/gs_restatement.py``, written independently of the
    oracle in ``ops/gaussian_raster.py``) renders the same image from the same parameters."""
    import os
    import sys

    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    from baseline.gs_restatement import render

    means, scales, rots, opac, shs, _, s = _scene(n=80)
    want, _, _ = GaussianRasterizer(s)(means, None, opac, shs=shs, scales=scales, rotations=rots)
    got = render(means, scales.log(), rots, torch.logit(opac), shs, s.viewmatrix, s.projmatrix, s.campos, s.image_width,
                 s.image_height, s.tanfovx, s.tanfovy, s.bg)
    assert got.shape == want.shape
    assert float((got - want).abs().max()) < 2e-3, float((got - want).abs().max())


def test_baseline_orbit_camera_equals_the_framework_camera():
    import os
    import sys

    sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))
    import bench
    from baseline.gs_restatement import orbit_camera

    for k in (0, 7, 123):
        cam = bench.gs_orbit_camera(k, "cpu")
        view, proj, campos, tanx, tany = orbit_camera(k, "cpu")
        torch.testing.assert_close(view, cam.world_view_transform, rtol=1e-4, atol=1e-3)
        torch.testing.assert_close(proj, cam.full_proj_transform, rtol=1e-4, atol=1e-3)
        torch.testing.assert_close(campos, cam.camera_center, rtol=1e-5, atol=1e-3)
        assert abs(tanx - cam.tanfovx) < 1e-6 and abs(tany - cam.tanfovy) < 1e-6


def test_camera_pose_takes_batched_matrices_and_a_homogeneous_position():
    from landmarksystem_b200.ops.gaussian_raster import _camera_pose

    _, _, _, _, _, _, s = _scene(n=1)
    pose = _camera_pose(s._replace(viewmatrix=s.viewmatrix[None], campos=torch.cat((s.campos, torch.ones(1)))), "cpu")
    assert torch.equal(pose, _camera_pose(s, "cpu")) and torch.equal(pose[32:], s.campos.float())
    with pytest.raises(ValueError):
        _camera_pose(s._replace(campos=s.campos[:2]), "cpu")


@pytest.mark.gpu
@pytest.mark.parametrize("n,degree,stored", [(1, 0, 0), (33, 1, 1), (127, 2, 3), (129, 3, 3)])
def test_split_sh_equals_joined(n, degree, stored):
    """Constant and higher coefficients read in place give the bits of the joined tensor, image and gradients alike (the
    projection backward has no atomics over SH rows); partial warps and blocks, no higher coefficients, inactive degrees."""
    means, scales, rots, opac, shs, _, s = _scene(n=n, seed=n)
    shs = shs[:, :(stored + 1) ** 2].contiguous().cuda()
    s = s._replace(sh_degree=degree)
    means, scales, rots, opac = (t.cuda() for t in (means, scales, rots, opac))
    joined = shs.clone().requires_grad_()
    dc, rest = shs[:, :1].contiguous().requires_grad_(), shs[:, 1:].contiguous().requires_grad_()
    g = torch.rand(3, s.image_height, s.image_width, generator=torch.Generator().manual_seed(2)).cuda()
    out = []
    for coeffs in (joined, (dc, rest)):
        img, radii, _ = GaussianRasterizer(s)(means, None, opac, shs=coeffs, scales=scales, rotations=rots)
        (img * g).sum().backward()
        out.append((img, radii))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    split = torch.cat((dc.grad, rest.grad), 1)
    # atomics add a Gaussian's colour gradient in any order: at most 48 warp sums of one sign, 48 x 2^-24 = 3e-6 of their sum
    assert torch.allclose(split, joined.grad, rtol=1e-5, atol=1e-6 * float(joined.grad.abs().max()) + 1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("stored", [17, 31, 32, 200])
@pytest.mark.parametrize("split", [False, True])
def test_more_coefficients_than_are_evaluated(stored, split):
    """Rows longer than the 16 coefficients of degree 3: the image of the first 16, bit for bit, and no gradient for the others."""
    means, scales, rots, opac, shs, _, s = _scene(n=70, seed=3)
    means, scales, rots, opac, shs = (t.cuda() for t in (means, scales, rots, opac, shs))
    wide = torch.cat((shs, torch.randn(70, stored - 16, 3).cuda()), 1)
    short, wide = shs.requires_grad_(), wide.requires_grad_()
    out = []
    for c in (short, wide):
        coeffs = (c[:, :1], c[:, 1:]) if split else c
        img, _, _ = GaussianRasterizer(s)(means, None, opac, shs=coeffs, scales=scales, rotations=rots)
        img.sum().backward()
        out.append(img)
    assert torch.equal(out[0], out[1]) and float(wide.grad[:, 16:].abs().sum()) == 0.0
    # sums by atomics in any order, as in the test above
    assert torch.allclose(wide.grad[:, :16], short.grad, rtol=1e-5, atol=1e-6 * float(short.grad.abs().max()) + 1e-12)


@pytest.mark.gpu
@pytest.mark.parametrize("n,distinct,spin_limit", [(1, 1, None), (31, 3, None), (1023, 2 ** 44, None), (1025, 5, 0), (70_000, 700, 0), (2 ** 18 - 777, 11, 0),
                                                   (2 ** 20 + 4097, 2 ** 44, 0), (5 * 2 ** 18 - 777, 9, None), (2 ** 21 + 1, 2 ** 44, None)])
def test_radix_sort_edges(n, distinct, spin_limit):
    """Tiles of either size with remainders, digits that all keys share, and the path of a block whose bounded wait for the
    blocks before it runs out (limit 0).  Stable order, so the result is exact."""
    from ctypes import c_int, c_longlong, c_void_p

    from landmarksystem_b200.ops import native
    from landmarksystem_b200.ops.gaussian_raster import _lib_ll

    g = torch.Generator().manual_seed(n)
    keys = (torch.randint(0, distinct, (n,), dtype=torch.int64, generator=g) * (2 ** 44 // distinct)).cuda()
    vals = torch.arange(n, dtype=torch.int32, device="cuda")
    ref_keys, order = torch.sort(keys, stable=True)
    cap = n + 777                                                  # capacity beyond the device-side count
    k, v = torch.full((cap,), 2 ** 45, dtype=torch.int64, device="cuda"), torch.full((cap,), -1, dtype=torch.int32, device="cuda")
    k[:n], v[:n] = keys, vals
    count = torch.tensor([n], dtype=torch.int32, device="cuda")
    ws = torch.empty(_lib_ll("lmb_radix_sort_scratch_bytes")(cap), dtype=torch.uint8, device="cuda")
    if spin_limit is None:
        rc = native.lib().lmb_radix_sort_pairs(k.data_ptr(), v.data_ptr(), count.data_ptr(), cap, 0, 48, ws.data_ptr(),
                                               native.stream_ptr())
    else:
        fn = native.lib().lmb_radix_sort_pairs_bounded
        fn.argtypes = [c_void_p, c_void_p, c_void_p, c_longlong, c_int, c_int, c_void_p, c_int, c_void_p]
        rc = fn(k.data_ptr(), v.data_ptr(), count.data_ptr(), cap, 0, 48, ws.data_ptr(), spin_limit, native.stream_ptr())
    assert rc == 0
    assert torch.equal(k[:n], ref_keys) and torch.equal(v[:n].long(), order)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 255, 257])
def test_activations_and_view_statistics(n):
    """One-launch activations against the tensor operations in 64 bits (fp32 results: a few roundings, 1e-6), with a zero
    quaternion (floored norm), large logits and infinities; statistics against the masked statements."""
    from landmarksystem_b200.components.fields.encodings.gaussian_encoding import GaussianEncoding

    g = torch.Generator().manual_seed(n)
    raw = [torch.randn(n, 3, generator=g) * 3.0, torch.randn(n, 4, generator=g), torch.randn(n, 1, generator=g) * 20.0]
    raw[1][0] = 0.0
    raw[2][-1] = float("-inf") if n > 1 else 0.0
    enc = GaussianEncoding(device="cuda")
    for name, t in zip(("_scaling", "_rotation", "_opacity"), raw):
        setattr(enc, name, torch.nn.Parameter(t.cuda()))
    wide = [t.double().requires_grad_() for t in raw]
    want = torch.exp(wide[0]), torch.nn.functional.normalize(wide[1]), torch.sigmoid(wide[2])
    got = enc.activated()
    ups = [torch.randn(t.shape, generator=g, dtype=torch.float64) for t in raw]
    ups[1][0] *= 1e-12                                             # keeps the gradient through the floored norm representable
    sum((w * u).sum() for w, u in zip(want, ups)).backward()
    sum((w * u.float().cuda()).sum() for w, u in zip(got, ups)).backward()
    for p, w, a, b in zip((enc._scaling, enc._rotation, enc._opacity), wide, got, want):
        assert torch.allclose(a.detach().cpu().double(), b.detach(), rtol=1e-6, atol=1e-7)
        assert torch.allclose(p.grad.cpu().double(), w.grad, rtol=1e-5, atol=1e-6)
    radii = torch.randint(0, 9, (n,), generator=g, dtype=torch.int32).cuda()
    points = torch.zeros(n, 3, device="cuda", requires_grad=True)
    points.grad = torch.randn(n, 3, generator=g).cuda()
    visible = radii > 2
    enc.max_radii2D = torch.rand(n, generator=g).cuda() * 9
    enc.xyz_gradient_accum, enc.denom = torch.rand(n, 1, generator=g).cuda(), torch.ones(n, 1, device="cuda")
    top = torch.where(visible, torch.maximum(enc.max_radii2D, radii.float()), enc.max_radii2D)
    accum = enc.xyz_gradient_accum + torch.where(visible, points.grad[:, :2].norm(dim=-1), 0.0)[:, None]
    enc.track_view(points, visible, radii)
    assert torch.equal(enc.max_radii2D, top) and torch.equal(enc.denom[:, 0], 1.0 + visible.float())
    assert torch.allclose(enc.xyz_gradient_accum, accum, rtol=1e-6, atol=0)


@pytest.mark.gpu
@pytest.mark.parametrize("sigma_px", [18.0, 100.0, 300.0, 1000.0])
def test_reach_of_long_splats_holds_the_walk(sigma_px):
    """Oblique splats 0.55 pixels wide, whose determinant has lost bits: every pixel that the walk's conic takes above 1/255 inside
    the square of the radius lies within the record's reach, by which tiles and warps are cut (1e-4 for the walk's exponential)."""
    from landmarksystem_b200.ops import gaussian_raster as gr

    n, W, H, focal, depth = 200, 1024, 1024, 2000.0, 4.0
    g = torch.Generator().manual_seed(int(sigma_px))
    proj = torch.zeros(4, 4)
    proj[0, 0], proj[1, 1], proj[2, 3] = 2 * focal / W, 2 * focal / H, 1.0
    s = GaussianRasterizationSettings(H, W, W / (2 * focal), H / (2 * focal), torch.zeros(3).cuda(), 1.0, torch.eye(4).cuda(), proj.cuda(), 0,
                                      torch.zeros(3).cuda())
    means = torch.cat((0.1 * torch.randn(n, 2, generator=g), torch.full((n, 1), depth)), 1).cuda()
    theta = (0.1 + 1.3 * torch.rand(n, generator=g)).double()
    long2, short2 = (sigma_px * depth / focal) ** 2, (0.05 * depth / focal) ** 2
    cov = torch.zeros(n, 6, dtype=torch.float64)
    cov[:, 0] = long2 * theta.cos() ** 2 + short2 * theta.sin() ** 2
    cov[:, 3] = long2 * theta.sin() ** 2 + short2 * theta.cos() ** 2
    cov[:, 1] = (long2 - short2) * theta.sin() * theta.cos()
    cov, opac, cols = cov.float().cuda(), torch.rand(n, 1, generator=g).clamp_min(0.05).cuda(), torch.ones(n, 3).cuda()
    radii, rec, _, _ = gr._project(means, None, None, opac, None, None, cols, cov, None, gr._camera_info(s, 0), gr._camera_pose(s, "cuda"), False)
    assert int((radii > 0).sum()) > n // 2
    for i in radii.nonzero()[:, 0].tolist():
        x, y, reach_x, reach_y, ca, cb, cc, op = rec[i, :8]
        r = int(radii[i])
        # pixels along the long axis and 3 to either side, also beyond the image
        t, off = torch.arange(-1.1 * r, 1.1 * r, 0.5, device="cuda")[:, None], torch.arange(-3, 3.1, 0.5, device="cuda")[None]
        co, si = math.cos(theta[i]), math.sin(theta[i])
        dx, dy = x - (x + t * co - off * si).round(), y - (y + t * si + off * co).round()
        power = -0.5 * (ca * dx * dx + cc * dy * dy) - cb * dx * dy
        hit = (power <= 0) & (op * power.exp() >= (1 + 1e-4) / 255) & (dx.abs() <= r) & (dy.abs() <= r)
        assert bool((dx.abs() <= reach_x)[hit].all()) and bool((dy.abs() <= reach_y)[hit].all())


@pytest.mark.gpu
@pytest.mark.parametrize("n,spread", [(1, 0.0), (7, 0.0), (8, 0.0), (9, 0.0), (256, 0.0), (257, 0.0), (2048, 0.0), (2049, 0.0), (8192, 0.0),
                                      (8193, 0.0), (20_000, 0.0), (6000, 0.6)])
def test_pairs_are_in_tile_depth_and_index_order(n, spread):
    """Whole numbers: the pairs of every tile, by depth and, at one depth, by index - for tiles of every sorting class, beyond
    the largest and for a view that mixes them."""
    from landmarksystem_b200.ops import gaussian_raster as gr
    from landmarksystem_b200.ops import native

    s = _scene(n=4)[-1]._replace(image_width=150, image_height=90)
    g = torch.Generator().manual_seed(n)
    depth = 4.0 + 2.0 * torch.rand(n, generator=g).double()              # points in front of the camera
    depth[::5] = 5.0                                                     # equal depths
    side = (torch.rand(n, 3, generator=g).double() - 0.5) * spread * depth[:, None]
    means = (s.campos.double() + s.viewmatrix.double()[:3, 2] * depth[:, None] + side).float().cuda()
    scales, rots = torch.full((n, 3), 1e-3).cuda(), torch.tensor([1.0, 0.0, 0.0, 0.0]).repeat(n, 1).cuda()
    opac, cols = torch.full((n, 1), 0.5).cuda(), torch.rand(n, 3, generator=g).cuda()
    info, pose = gr._camera_info(s, 0), gr._camera_pose(s, means.device)
    radii, rec, touched, (cursors, ranges, totals) = gr._project(means, scales, rots, opac, None, None, cols, None, None, info, pose, False)
    total, most = totals.tolist()
    assert total == int(touched.sum()) and (spread or most == n) and total >= n * 0.5
    keys, vals = torch.empty(total, dtype=torch.int64, device="cuda"), torch.empty(total, dtype=torch.int32, device="cuda")
    H, W, start = s.image_height, s.image_width, cursors[:, 0].clone()
    out = [torch.empty(3, H, W, device="cuda"), torch.empty(H, W, device="cuda"), torch.empty(H, W, device="cuda"),
           torch.empty(H, W, dtype=torch.int32, device="cuda")]
    bg, ws = s.bg.cuda().float(), gr._sort_scratch(n, total, most, means.device)
    native.check(native.lib().lmb_gs_draw(n, rec.data_ptr(), radii.data_ptr(), touched.data_ptr(), cursors.data_ptr(), W, H, total, most,
                                          keys.data_ptr(), vals.data_ptr(), ws.data_ptr(), ranges.data_ptr(), bg.data_ptr(),
                                          *(o.data_ptr() for o in out), native.stream_ptr()), "gs_draw")
    assert torch.equal(ranges[:, 0], start) and torch.equal(ranges[1:, 0], ranges[:-1, 1]) and int(ranges[-1, 1]) == total
    counts = (ranges[:, 1] - ranges[:, 0]).long()
    tile = torch.repeat_interleave(torch.arange(counts.numel(), device="cuda"), counts)
    z = rec[:, 11].contiguous().view(torch.int32).long()[vals.long()]
    order = z << 32 | vals.long()
    assert bool(((tile[1:] > tile[:-1]) | (order[1:] > order[:-1])).all())
    assert torch.equal(torch.bincount(vals.long(), minlength=n), touched.long())


@pytest.mark.gpu
@pytest.mark.parametrize("n,size,spread", [(2_000, (150, 90), 0.6), (5_000, (150, 90), 0.6), (40_000, (40, 25), 0.5), (9_000, (17, 16), 0.05),
                                           (300_000, (2000, 1100), 1.5)])
def test_pairs_of_crowded_views_are_in_order(n, size, spread):
    """Whole numbers, as above, where a tile has 1, 4, 32 and 2 counters, of which the last view scans three chunks: ranges by the tiles of
    the pairs that a splat touches, and the order of pairs that are sorted in their tiles and all together."""
    from landmarksystem_b200.ops import gaussian_raster as gr
    from landmarksystem_b200.ops import native

    W, H = size
    n_tiles = ((W + 15) // 16) * ((H + 15) // 16)
    words = native.lib().lmb_gs_tile_words(n, W, H)
    assert words % 8 == 0 and (words == 8 or words // 8 * n_tiles <= n // 16) and (words > 8) == (n_tiles * 2 <= n // 16)
    s = _scene(n=4)[-1]._replace(image_width=W, image_height=H)
    g = torch.Generator().manual_seed(n)
    depth = 4.0 + 2.0 * torch.rand(n, generator=g).double()
    depth[::5] = 5.0
    side = (torch.rand(n, 3, generator=g).double() - 0.5) * spread * depth[:, None]
    means = (s.campos.double() + s.viewmatrix.double()[:3, 2] * depth[:, None] + side).float().cuda()
    scales, rots = torch.full((n, 3), 1e-3).cuda(), torch.tensor([1.0, 0.0, 0.0, 0.0]).repeat(n, 1).cuda()
    opac, cols = torch.full((n, 1), 0.5).cuda(), torch.rand(n, 3, generator=g).cuda()
    info, pose = gr._camera_info(s, 0), gr._camera_pose(s, means.device)
    radii, rec, touched, (cursors, ranges, totals) = gr._project(means, scales, rots, opac, None, None, cols, None, None, info, pose, False)
    total, most = totals.tolist()
    counts = (ranges[:, 1] - ranges[:, 0]).long()
    assert total == int(touched.sum()) == int(counts.sum()) and most == int(counts.max()) and total >= n * 0.3
    assert torch.equal(ranges[:, 0], cursors[:, 0]) and torch.equal(ranges[1:, 0], ranges[:-1, 1])
    keys, vals = torch.empty(total, dtype=torch.int64, device="cuda"), torch.empty(total, dtype=torch.int32, device="cuda")
    out = [torch.empty(3, H, W, device="cuda"), torch.empty(H, W, device="cuda"), torch.empty(H, W, device="cuda"),
           torch.empty(H, W, dtype=torch.int32, device="cuda")]
    bg, ws = s.bg.cuda().float(), gr._sort_scratch(n, total, most, means.device)
    native.check(native.lib().lmb_gs_draw(n, rec.data_ptr(), radii.data_ptr(), touched.data_ptr(), cursors.data_ptr(), W, H, total, most,
                                          keys.data_ptr(), vals.data_ptr(), ws.data_ptr(), ranges.data_ptr(), bg.data_ptr(),
                                          *(o.data_ptr() for o in out), native.stream_ptr()), "gs_draw")
    tile = torch.repeat_interleave(torch.arange(n_tiles, device="cuda"), counts)
    v = vals.long()
    order = rec[:, 11].contiguous().view(torch.int32).long()[v] << 32 | v
    assert bool(((tile[1:] > tile[:-1]) | (order[1:] > order[:-1])).all())
    assert torch.equal(torch.bincount(v, minlength=n), touched.long())
    # a pair's tile is one that its splat's square of 3 sigma reaches
    tx, ty, r = tile % ((W + 15) // 16), tile // ((W + 15) // 16), radii[v].float()
    x, y = rec[v, 0], rec[v, 1]
    assert bool(((x + r >= tx * 16 - 1) & (x - r <= tx * 16 + 16) & (y + r >= ty * 16 - 1) & (y - r <= ty * 16 + 16)).all())
