"""Gaussian-splatting family: encodings, PLY formats, densification surgery and short training runs."""
import os

import numpy as np
import pytest
import torch

from landmarksystem_b200.components.fields.encodings.gaussian_encoding import GaussianEncoding
from landmarksystem_b200.components.fields.encodings.octreegs_encoding import OctreeGSEncoding
from landmarksystem_b200.components.fields.encodings.scaffoldgs_encoding import ScaffoldGSEncoding, voxel_keys
from landmarksystem_b200.components.utils.graphics_utils import BasicPointCloud
from landmarksystem_b200.components.utils.ply_utils import read_ply
from landmarksystem_b200.configs import BaseConfig
from landmarksystem_b200.ops.knn import distCUDA2, knn_mean_dist2_reference

ROOT = os.path.join(os.path.dirname(__file__), "..", "landmarksystem_b200", "models")


def _pcd(n=200, seed=0):
    rng = np.random.default_rng(seed)
    return BasicPointCloud(rng.random((n, 3), dtype=np.float32) * 2 - 1, rng.random((n, 3), dtype=np.float32),
                           np.zeros((n, 3), np.float32))


def test_gaussian_encoding_ply_roundtrip_and_properties(tmp_path):
    enc = GaussianEncoding(3, device="cpu")
    enc.create_from_pcd(_pcd())
    path = str(tmp_path / "point_cloud.ply")
    enc.save_ply(path)
    names = read_ply(path).dtype.names
    assert names[:6] == ("x", "y", "z", "nx", "ny", "nz") and "f_dc_2" in names and "f_rest_44" in names
    assert "opacity" in names and "scale_2" in names and "rot_3" in names
    other = GaussianEncoding(3, device="cpu")
    other.load_ply(path)
    for a, b in zip(enc.parameters(), other.parameters()):
        assert torch.allclose(a, b)
    cache = str(tmp_path / "cache.ply")
    enc.save_ply(cache, cache=True)
    assert "cache_opacity" in read_ply(cache).dtype.names
    third = GaussianEncoding(3, device="cpu")
    third.load_ply(cache)
    assert torch.allclose(third.get_opacity, enc.get_opacity, atol=1e-5)
    assert torch.allclose(third.get_scaling, enc.get_scaling, rtol=1e-4)


def test_gaussian_encoding_setters_follow_the_activation_cache():
    """Setters of the reference (gaussian_encoding.py:855-925): raw tensors in training, activated values through
    the cache when ``act_cache`` is on and the module evaluates."""
    enc = GaussianEncoding(1, act_cache=True, device="cpu")
    enc.create_from_pcd(_pcd(20))
    enc.train()
    raw = torch.full_like(enc._scaling, -2.0)
    enc.set_scaling(raw)
    assert torch.allclose(enc.get_scaling, torch.exp(raw))
    with pytest.raises(NotImplementedError):
        enc.set_features(enc.get_features)
    enc.eval()
    act = torch.full_like(enc._opacity, 0.25)
    enc.set_opacity(act)
    assert torch.equal(enc.get_opacity, act)                        # taken as the activated value
    feats = torch.zeros_like(enc.get_features)
    enc.set_features(feats)
    assert enc.get_features is feats
    moved = enc.get_xyz.detach() + 1
    enc.set_xyz(moved)
    assert torch.equal(enc.get_xyz, moved) and isinstance(enc._xyz, torch.nn.Parameter)
    opt = torch.optim.Adam([{"params": [enc._xyz], "name": "xyz"}], lr=1e-3)
    enc._xyz.grad = torch.ones_like(enc._xyz)
    opt.step()
    new = enc.cat_tensors_to_optimizer({"xyz": torch.zeros(3, 3)}, opt)
    assert new["xyz"].shape[0] == 23 and opt.state[new["xyz"]]["exp_avg"][-3:].abs().sum() == 0
    swapped = enc.replace_tensor_to_optimizer(torch.ones(23, 3), "xyz", opt)
    assert opt.param_groups[0]["params"][0] is swapped["xyz"] and opt.state[swapped["xyz"]]["exp_avg"].abs().sum() == 0


def test_rasterizer_component_renders_several_models_in_one_sort():
    """``GaussianSplattingRasterizer``: a list of models renders like one model that holds all their Gaussians."""
    from landmarksystem_b200.components.data.cameras import Camera
    from landmarksystem_b200.components.renderers import GassianSplattingRasterizer, GaussianSplattingRasterizer
    from landmarksystem_b200.synthetic import ring_cameras

    assert GassianSplattingRasterizer is GaussianSplattingRasterizer
    torch.manual_seed(0)
    parts = []
    for seed in (0, 1):
        enc = GaussianEncoding(1, device="cpu")
        enc.create_from_pcd(_pcd(40, seed=seed))
        enc._opacity.data.fill_(1.5)
        enc._scaling.data.fill_(-2.0)
        parts.append(enc)
    whole = GaussianEncoding(1, device="cpu")
    whole._set_params(*(torch.cat([getattr(p, n).detach() for p in parts]) for n in
                        ("_xyz", "_features_dc", "_features_rest", "_scaling", "_rotation", "_opacity")))
    cam = Camera.from_c2w(ring_cameras(4, 3.0)[0].numpy(), 24, 20, 30.0)
    renderer = GaussianSplattingRasterizer(white_background=True)
    both = renderer(parts, camera=cam)
    one = renderer(whole, camera=cam)
    assert both["counts"] == [len(parts[0]), len(parts[1])] and both["render"].shape == (3, 20, 24)
    assert torch.allclose(both["render"], one["render"], atol=1e-6) and torch.equal(both["radii"], one["radii"])
    assert both["visibility_filter"].any() and float(one["render"].detach().min()) < 0.99        # something was drawn
    first_only = renderer(parts[0], camera=cam)["render"]
    assert not torch.allclose(first_only, both["render"], atol=1e-3)
    both["render"].sum().backward()
    assert parts[1]._xyz.grad is not None and parts[1]._xyz.grad.abs().sum() > 0


@pytest.mark.parametrize("device", ["cpu", pytest.param("cuda", marks=pytest.mark.gpu)])
def test_hooks_on_the_rasteriser_see_one_tensor_of_coefficients(device):
    from landmarksystem_b200.components.data.cameras import Camera
    from landmarksystem_b200.models.origin_gs.gs_model import Gaussian3DConfig, GaussianModel
    from landmarksystem_b200.synthetic import ring_cameras
    from landmarksystem_b200.utils import Config

    cfg = Config(dict(Gaussian3DConfig()))
    cfg.update(device=device, debug=False)
    model = GaussianModel(cfg, None, 1.0).eval()
    model.gaussian_encoding.create_from_pcd(_pcd(40, seed=0))
    cam = Camera.from_c2w(ring_cameras(4, 3.0)[0].numpy(), 24, 20, 30.0)
    seen = []
    with torch.no_grad():
        want = model(cam)
        model.renderer.register_forward_pre_hook(lambda module, args, kwargs: seen.append(kwargs["shs"]), with_kwargs=True)
        got = model(cam)
    assert len(seen) == 1 and torch.equal(seen[0], model.gaussian_encoding.get_features) and torch.equal(got, want)


def test_densify_and_prune_keeps_optimizer_in_sync():
    torch.manual_seed(0)
    enc = GaussianEncoding(1, device="cpu")
    enc.create_from_pcd(_pcd(100))
    groups = [{"params": [getattr(enc, a)], "lr": 1e-3, "name": n} for n, a in
              (("xyz", "_xyz"), ("f_dc", "_features_dc"), ("f_rest", "_features_rest"), ("opacity", "_opacity"),
               ("scaling", "_scaling"), ("rotation", "_rotation"))]
    opt = torch.optim.Adam(groups, lr=0.0, eps=1e-15)
    for p in enc.parameters():
        p.grad = torch.randn_like(p)
    opt.step()
    enc.xyz_gradient_accum[:] = torch.rand(100, 1)
    enc.denom[:] = 1
    enc.densify_and_prune(0.5, 0.005, 4.0, None, opt)
    n = enc._xyz.shape[0]
    assert n != 100
    for g in opt.param_groups:
        p = g["params"][0]
        assert p.shape[0] == n and opt.state[p]["exp_avg"].shape == p.shape
    assert enc.denom.shape[0] == n and enc.max_radii2D.shape[0] == n
    enc.reset_opacity(opt)
    assert enc.get_opacity.max() <= 0.0101


def test_knn_reference_small():
    pts = torch.tensor([[0.0, 0, 0], [1, 0, 0], [0, 2, 0], [0, 0, 3], [5, 5, 5]])
    d = knn_mean_dist2_reference(pts)
    assert torch.allclose(d[0], torch.tensor((1 + 4 + 9) / 3.0))


@pytest.mark.gpu
def test_knn_cuda_matches_reference():
    torch.manual_seed(0)
    pts = torch.rand(20000, 3) * torch.tensor([10.0, 4.0, 1.0])
    ref = knn_mean_dist2_reference(pts)
    got = distCUDA2(pts.cuda()).cpu()
    assert torch.allclose(got, ref, rtol=1e-4, atol=1e-7)
    flat = pts.clone(); flat[:, 2] = 0
    assert torch.allclose(distCUDA2(flat.cuda()).cpu(), knn_mean_dist2_reference(flat), rtol=1e-4, atol=1e-7)


def test_scaffold_encoding_ply_and_growing(tmp_path):
    torch.manual_seed(0)
    enc = ScaffoldGSEncoding(feat_dim=8, n_offsets=4, voxel_size=0.25, device="cpu")
    enc.create_from_pcd(_pcd(400))
    n0 = len(enc)
    assert n0 > 0 and len(torch.unique(voxel_keys(torch.round(enc._anchor / 0.25)))) == n0
    path = str(tmp_path / "pc.ply")
    enc.save_ply(path)
    names = read_ply(path).dtype.names
    assert "f_offset_11" in names and "f_anchor_feat_7" in names and "scale_5" in names
    other = ScaffoldGSEncoding(feat_dim=8, n_offsets=4, voxel_size=0.25, device="cpu")
    other.load_ply(path)
    assert torch.allclose(other._offset, enc._offset) and torch.allclose(other._scaling, enc._scaling)
    groups = [{"params": [getattr(enc, a)], "lr": 1e-3, "name": n} for n, a in
              (("anchor", "_anchor"), ("offset", "_offset"), ("anchor_feat", "_anchor_feat"), ("opacity", "_opacity"),
               ("scaling", "_scaling"), ("rotation", "_rotation"))]
    opt = torch.optim.Adam(groups, lr=0.0, eps=1e-15)
    enc._offset.data.normal_(0, 3.0)            # push neural Gaussians into empty voxels
    enc.offset_gradient_accum[:] = 1.0
    enc.offset_denom[:] = 100
    enc.anchor_demon[:] = 100
    enc.opacity_accum[:] = 100
    enc.opacity_accum[:5] = 0                   # these anchors get pruned
    enc.adjust_anchor(check_interval=100, success_threshold=0.8, grad_threshold=0.0002, min_opacity=0.005, optimizer=opt)
    n1 = len(enc)
    assert n1 > n0 - 5
    assert enc.offset_denom.shape[0] == n1 * 4 and enc.opacity_accum.shape[0] == n1
    for g in opt.param_groups:
        assert g["params"][0].shape[0] == n1


def test_octree_levels_and_lod_mask():
    from landmarksystem_b200.components.data.cameras import Camera
    from landmarksystem_b200.synthetic import ring_cameras

    enc = OctreeGSEncoding(feat_dim=8, n_offsets=4, base_layer=3, device="cpu", visible_threshold=0.0)
    cams = [Camera.from_c2w(p.numpy(), 32, 32, 30.0, uid=i) for i, p in enumerate(ring_cameras(6, 3.0))]
    pcd = _pcd(500)
    enc.set_level(torch.from_numpy(pcd.points), cams, [1.0], dist_ratio=0.95, levels=3)
    enc.set_coarse_interval(300, 1.5)
    assert enc.levels == 3 and len(enc.coarse_intervals) == 3 - 1 - enc.init_level
    enc.create_from_pcd(pcd)
    assert set(enc.get_level.unique().tolist()) <= {0.0, 1.0, 2.0}
    enc.set_anchor_mask(torch.tensor([0.0, 0.0, 0.5]), 10 ** 6, 1.0, True)
    near = enc._anchor_mask.sum()
    enc.set_anchor_mask(torch.tensor([0.0, 0.0, 50.0]), 10 ** 6, 1.0, True)
    far = enc._anchor_mask.sum()
    assert near > far > 0          # a distant camera selects only coarse levels


@pytest.mark.gpu
def test_octree_lod_kernel_matches_torch():
    from landmarksystem_b200.components.data.cameras import Camera
    from landmarksystem_b200.synthetic import ring_cameras

    cams = [Camera.from_c2w(p.numpy(), 32, 32, 30.0, uid=i) for i, p in enumerate(ring_cameras(6, 3.0))]
    pcd = _pcd(3000)
    for mode in ("round", "floor", "progressive"):
        cpu = OctreeGSEncoding(feat_dim=8, n_offsets=4, base_layer=4, device="cpu", dist2level=mode)
        cpu.set_level(torch.from_numpy(pcd.points), cams, [1.0], levels=4)
        cpu.create_from_pcd(pcd)
        gpu = OctreeGSEncoding(feat_dim=8, n_offsets=4, base_layer=4, device="cuda", dist2level=mode)
        gpu.levels, gpu.standard_dist, gpu.init_level = cpu.levels, cpu.standard_dist, cpu.init_level
        gpu.voxel_size = cpu.voxel_size
        gpu.load_encoding_state({k: v.detach() for k, v in [("_anchor", cpu._anchor), ("_offset", cpu._offset),
                                 ("_anchor_feat", cpu._anchor_feat), ("_scaling", cpu._scaling),
                                 ("_rotation", cpu._rotation), ("_opacity", cpu._opacity), ("_level", cpu._level),
                                 ("_extra_level", cpu._extra_level)]})
        gpu.voxel_size, gpu.standard_dist, gpu.levels = cpu.voxel_size, cpu.standard_dist, cpu.levels
        c = torch.tensor([0.4, -0.3, 2.0])
        cpu.set_anchor_mask(c, 10 ** 6, 1.0, False)
        gpu.set_anchor_mask(c, 10 ** 6, 1.0, False)
        assert (cpu._anchor_mask != gpu._anchor_mask.cpu()).float().mean() < 1e-3


def test_anchor_encoding_accessors_and_octree_helpers(tmp_path):
    """Accessors the reference's encodings offer (scaffoldgs_encoding.py:307-760, octreegs_encoding.py:445-1101)."""
    from landmarksystem_b200.components.utils.general_utils import build_rotation

    torch.manual_seed(1)
    enc = OctreeGSEncoding(feat_dim=8, n_offsets=4, base_layer=3, device="cpu", visible_threshold=0.0)
    enc.levels, enc.init_level = 3, 0
    enc.create_from_pcd(_pcd(300))
    n = len(enc)
    enc._rotation.data = torch.nn.functional.normalize(torch.randn(n, 4), dim=-1)
    assert enc.get_anchor_feat is enc._anchor_feat and enc.get_offset is enc._offset
    cov = enc.get_covariance(2.0)                                   # upper triangle of R S S^T R^T, S = 2 * scales
    R, S = build_rotation(enc._rotation), 2.0 * enc.get_scaling[:, :3]
    full = R @ torch.diag_embed(S * S) @ R.transpose(1, 2)
    assert torch.allclose(cov, torch.stack((full[:, 0, 0], full[:, 0, 1], full[:, 0, 2], full[:, 1, 1], full[:, 1, 2],
                                            full[:, 2, 2]), -1), atol=1e-6)
    path = str(tmp_path / "pc.ply")
    enc.save_ply(path)
    assert list(read_ply(path).dtype.names) == enc.construct_list_of_attributes()
    rows = enc.plot_levels()
    assert sum(r[1] for r in rows) == n and abs(sum(r[2] for r in rows) - 1.0) < 1e-6
    grid = torch.tensor([[0, 0, 0], [1, 2, 3], [-4, 5, 6], [7, 7, 7]], dtype=torch.float32)
    sel = torch.tensor([[1, 2, 3], [7, 7, 7], [9, 9, 9]], dtype=torch.float32)
    assert enc.get_remove_duplicates(grid, sel).tolist() == [False, True, False, True]
    moved = enc.get_anchor + 1.0
    enc.set_anchor(moved)
    assert torch.equal(enc.get_anchor, moved)
    with pytest.raises(AssertionError):
        enc.set_anchor(moved[:-1])


def test_scaffold_model_helpers_cov_prefilter_and_mlp_file(tmp_path):
    """Model-level helpers of the reference (scaffold_gs/gs_model.py, octree_gs/gs_model.py:200-221, 428-443,
    base_model.py:266-304): the covariance route of the anchor pre-filter agrees with the scale / rotation route."""
    import importlib

    from landmarksystem_b200.components.data.cameras import Camera
    from landmarksystem_b200.synthetic import ring_cameras

    mod = importlib.import_module("landmarksystem_b200.models.octree_gs.gs_trainer")
    conf = os.path.join(ROOT, "octree_gs", "confs", "synthetic_train.py")
    cfg = BaseConfig.from_file(conf, {"basedir": str(tmp_path), "device": "cpu", "n_iters": "1",
                                      "datadir": "ring:3:16x16:18:3", "init_points_num": "80",
                                      "progress_refresh_rate": "100"})
    assert cfg.ratio == 1 and cfg.compute_cov3D_python is False
    model = mod.OctreeGSTrainer(cfg).model
    cam = [Camera.from_c2w(p.numpy(), 32, 32, 40.0, uid=i) for i, p in enumerate(ring_cameras(3, 3.0))][0]
    model.set_anchor_mask(cam.camera_center, 10 ** 6, 1.0)
    mask = model.gaussian_encoding._anchor_mask.clone()
    by_scales = model.prefilter_voxel(cam, anchor_mask=mask)
    cfg.compute_cov3D_python = True
    by_cov = model.prefilter_voxel(cam, anchor_mask=mask)
    cfg.compute_cov3D_python = False
    assert by_scales.any() and torch.equal(by_scales, by_cov)
    # the reference's extra forward arguments: an anchor filter and an explicit appearance code (eval only)
    model.eval()
    with torch.no_grad():
        base = model(cam)
        nothing = model(cam, 1.0, False, torch.zeros_like(mask), -1)
        assert torch.allclose(nothing, model.background[:, None, None].expand_as(nothing)) and not torch.allclose(base, nothing)
        if model.embedding_appearance is not None and model.embedding_appearance.num_embeddings > 1:
            model.embedding_appearance.weight.data.normal_(0, 2.0)
            own, other = model(cam, ape_code=-1), model(cam, ape_code=(int(cam.uid) + 1) % model.embedding_appearance.num_embeddings)
            assert not torch.allclose(own, other) and torch.allclose(own, model(cam, ape_code=int(cam.uid)))
    model.train()
    cam.c2w = None                                                  # adapters of the reference clear it before pickling
    assert cam.c2w is None
    assert len(model.plot_levels()) == model.gaussian_encoding.levels
    code = model.get_appearance_code(torch.tensor(0)) if model.embedding_appearance is not None else None
    assert code is None or code.shape == (cfg.appearance_dim,)

    with torch.no_grad():                                       # make the saved heads differ from a fresh initialisation
        for prm in model.anchor_decoder.mlp_color.parameters():
            prm.add_(0.37)
    model.save_mlp_checkpoints(str(tmp_path / "mlp" / "checkpoint.pth"))
    saved = torch.load(str(tmp_path / "mlp" / "checkpoint.pth"), weights_only=False)
    assert {"anchor_decoder.opacity_mlp", "anchor_decoder.cov_mlp", "anchor_decoder.color_mlp"} <= set(saved)
    assert ("anchor_decoder.embedding_appearance" in saved) == (model.embedding_appearance is not None)
    # the decoder file converts into the flat state dict a fresh model loads beside the point cloud
    from landmarksystem_b200.render.utils import transform_gs_mlp_checkpoint

    model.save_ply(str(tmp_path / "mlp"))
    flat = transform_gs_mlp_checkpoint(str(tmp_path / "mlp" / "checkpoint.pth"), out_dir=str(tmp_path / "converted"))
    assert os.path.exists(tmp_path / "converted" / "point_cloud.ply")
    fresh = mod.OctreeGSTrainer(cfg).build_model()
    if model.embedding_appearance is not None:
        fresh.set_appearance(model.embedding_appearance.num_embeddings)
    fresh.load_from_state_dict(fresh.get_state_dict_from_ckpt(str(tmp_path / "converted" / "point_cloud.ply"), "cpu"))
    assert flat.endswith("state_dict.th") and fresh.get_primitives_num == model.get_primitives_num
    for a, b in zip(fresh.anchor_decoder.mlp_color.parameters(), model.anchor_decoder.mlp_color.parameters()):
        assert torch.equal(a, b)
    model.save_ply(str(tmp_path / "out"), rank=1)
    model.save_state_dict(str(tmp_path / "out" / "state_dict-sub1.th"))
    assert os.path.exists(tmp_path / "out" / "point_cloud-sub1.ply")
    rest = torch.load(str(tmp_path / "out" / "state_dict-sub1.th"), weights_only=False)
    assert rest and not any(k.startswith("gaussian_encoding.") for k in rest)


@pytest.mark.parametrize("family,trainer_name", [("origin_gs", "Gaussian3DTrainer"), ("scaffold_gs", "ScaffoldGSTrainer"),
                                                  ("octree_gs", "OctreeGSTrainer")])
def test_cpu_smoke_training_and_checkpoint(family, trainer_name, tmp_path):
    import importlib

    mod = importlib.import_module(f"landmarksystem_b200.models.{family}.gs_trainer")
    conf = os.path.join(ROOT, family, "confs", "synthetic_train.py")
    cfg = BaseConfig.from_file(conf, {"basedir": str(tmp_path), "device": "cpu", "n_iters": "3",
                                      "datadir": "ring:3:16x16:18:3", "init_points_num": "60",
                                      "progress_refresh_rate": "100"})
    trainer = getattr(mod, trainer_name)(cfg)
    ps = trainer.train()
    assert np.isfinite(ps)
    folder = os.path.join(trainer.logfolder, "point_cloud", "iteration_3")
    assert os.path.exists(os.path.join(folder, "point_cloud.ply")) and os.path.exists(os.path.join(folder, "opt.th"))
    # checkpoint round trip through the model-level API
    fresh = trainer.build_model()
    fresh.load_from_state_dict(fresh.get_state_dict_from_ckpt(os.path.join(folder, "point_cloud.ply"), "cpu"))
    assert fresh.get_primitives_num == trainer.model.get_primitives_num


@pytest.mark.gpu
@pytest.mark.parametrize("family,trainer_name,gain", [("origin_gs", "Gaussian3DTrainer", 3.0),
                                                       ("scaffold_gs", "ScaffoldGSTrainer", 2.0),
                                                       ("octree_gs", "OctreeGSTrainer", 2.0)])
def test_gpu_training_improves_psnr(family, trainer_name, gain, tmp_path):
    import importlib

    mod = importlib.import_module(f"landmarksystem_b200.models.{family}.gs_trainer")
    conf = os.path.join(ROOT, family, "confs", "synthetic_train.py")
    cfg = BaseConfig.from_file(conf, {"basedir": str(tmp_path), "device": "cuda", "n_iters": "400",
                                      "datadir": "ring:12:64x64:75:3", "init_points_num": "3000",
                                      "progress_refresh_rate": "1000", "skip_save_imgs": "true"})
    trainer = getattr(mod, trainer_name)(cfg)
    before = trainer.evaluation(str(tmp_path / "before"), stride=1)
    after = trainer.train()
    assert after > before + gain, (before, after)


def test_camera_cells_and_positional_densification(tmp_path):
    """Per-block camera subsets of the data manager (``divide_dataset / switch_cell / use_all_data``, reference:
    data_manager.py:196-329) and the reference's positional form of ``densification_postfix``."""
    from landmarksystem_b200.components.data.data_manager import DatasetManager

    conf = os.path.join(ROOT, "origin_gs", "confs", "synthetic_train.py")
    cfg = BaseConfig.from_file(conf, {"basedir": str(tmp_path), "device": "cpu", "datadir": "ring:8:8x8:10:3"})
    mgr = DatasetManager(cfg)
    total = mgr.train_data_size
    counts = mgr.divide_dataset([2, 2], ((-4.0, -4.0), (4.0, 4.0)))
    assert sum(counts) == total == 8 and len(counts) == 4 and max(counts) < total
    mgr.switch_cell((1, 0))                                       # block coordinate -> cell 2
    assert mgr.train_data_size == counts[2]
    cam, image = mgr.get_camera("train")
    assert float(cam.camera_center[0]) >= 0.0 and float(cam.camera_center[1]) < 0.0
    mgr.switch_cell(3)
    assert mgr.train_data_size == counts[3]
    mgr.use_all_data()
    assert mgr.train_data_size == total

    enc = GaussianEncoding(1, device="cpu")
    enc.create_from_pcd(_pcd(10))
    groups = [{"params": [getattr(enc, a)], "lr": 1e-3, "name": n} for n, a in
              (("xyz", "_xyz"), ("f_dc", "_features_dc"), ("f_rest", "_features_rest"), ("opacity", "_opacity"),
               ("scaling", "_scaling"), ("rotation", "_rotation"))]
    opt = torch.optim.Adam(groups, lr=0.0, eps=1e-15)
    enc.densification_postfix(torch.ones(3, 3), torch.zeros(3, 1, 3), torch.zeros(3, 3, 3), torch.zeros(3, 1),
                              torch.zeros(3, 3), torch.tensor([[1.0, 0, 0, 0]]).repeat(3, 1), opt)
    assert len(enc) == 13 and torch.equal(enc.get_xyz[-3:], torch.ones(3, 3)) and enc.denom.shape[0] == 13
    assert all(g["params"][0].shape[0] == 13 for g in opt.param_groups)


@pytest.mark.gpu
@pytest.mark.parametrize("n,share,feat,dists", [(1, 1.0, 32, (0, 0, 0)), (700, 0.6, 32, (1, 0, 1)), (5001, 0.3, 32, (1, 1, 1)),
                                                (900, 0.5, 30, (0, 1, 0)), (300, 0.0, 32, (0, 0, 0))])
def test_anchors_decoded_by_index_equal_those_selected_by_mask(n, share, feat, dists, monkeypatch):
    """The rows of the heads written by one kernel against the selection by tensor operations: the same candidates survive and
    their attributes agree to the rounding of bf16 inputs, for every layout of the rows, without visible anchors too."""
    from landmarksystem_b200.components.fields.anchor_decoder import AnchorDecoder, FusedAnchorDecoder

    g = torch.Generator(device="cuda").manual_seed(n)
    torch.manual_seed(n)
    dec = FusedAnchorDecoder(False, *(bool(d) for d in dists), 3, feat, 10).cuda().eval()
    anchor, feats = torch.randn(n, 3, device="cuda", generator=g), torch.randn(n, feat, device="cuda", generator=g)
    offset, scaling = torch.randn(n, 10, 3, device="cuda", generator=g), torch.rand(n, 6, device="cuda", generator=g)
    visible = torch.rand(n, device="cuda", generator=g) < share
    centre = torch.tensor([0.3, -2.0, 5.0], device="cuda")
    with torch.no_grad():
        assert dec._rows_ok(centre, anchor, feats, offset, scaling, visible, None, None, None)
        got = dec(centre, anchor, feats, offset, scaling, visible)
        monkeypatch.setattr(AnchorDecoder, "_rows_ok", lambda *a: False)
        want = dec(centre, anchor, feats, offset, scaling, visible)
    assert len(got) == len(want) and got[5] is None and got[6] is None
    if int(visible.sum()) == 0:
        assert all(t.shape[0] == 0 for t in got[:5])
        return
    # the direction's last fp32 bit may differ and round to the other bf16 value: a candidate at zero opacity may change sides
    assert abs(got[0].shape[0] - want[0].shape[0]) <= max(2, want[0].shape[0] // 500)
    if got[0].shape == want[0].shape:
        for a, b in zip(got[:5], want[:5]):
            assert float((a - b).norm()) <= 4e-3 * float(b.norm()) + 1e-6


@pytest.mark.gpu
@pytest.mark.parametrize("n,share,feat,dists", [(1, 1.0, 32, (0, 0, 0)), (700, 0.6, 32, (1, 0, 1)), (5001, 0.3, 32, (1, 1, 1)),
                                                (900, 0.5, 30, (0, 1, 0)), (1201, 0.7, 64, (1, 1, 0))])
def test_attributes_of_anchors_decoded_by_index(n, share, feat, dists, monkeypatch):
    """Every candidate is kept by a bias far from zero, so that both ways return the same ones in the same order: positions to the rounding
    of one multiplication and addition, the outputs of the heads to that of the direction's bf16 value (2^-9 of inputs of order one
    through weights below 0.25).  The offsets tell the candidates apart."""
    from landmarksystem_b200.components.fields.anchor_decoder import AnchorDecoder, FusedAnchorDecoder

    g = torch.Generator(device="cuda").manual_seed(n)
    torch.manual_seed(n)
    dec = FusedAnchorDecoder(False, *(bool(d) for d in dists), 3, feat, 10).cuda().eval()
    with torch.no_grad():
        last = [m for m in dec.mlp_opacity if isinstance(m, torch.nn.Linear)][-1]
        last.weight.mul_(0.05)
        last.bias.fill_(0.7)
        last.bias[::3] = -0.7                                    # four of ten are dropped, for every anchor
    anchor, feats = torch.randn(n, 3, device="cuda", generator=g), torch.randn(n, feat, device="cuda", generator=g)
    offset, scaling = torch.randn(n, 10, 3, device="cuda", generator=g), torch.rand(n, 6, device="cuda", generator=g)
    visible = torch.rand(n, device="cuda", generator=g) < share
    centre = torch.tensor([0.3, -2.0, 5.0], device="cuda")
    with torch.no_grad():
        got = dec(centre, anchor, feats, offset, scaling, visible)
        monkeypatch.setattr(AnchorDecoder, "_rows_ok", lambda *a: False)
        want = dec(centre, anchor, feats, offset, scaling, visible)
    kept = int(visible.sum()) * 6
    assert all(a.shape == b.shape and a.shape[0] == kept for a, b in zip(got[:5], want[:5]))
    idx = visible.nonzero().squeeze(-1)
    keep = (torch.arange(10, device="cuda") % 3 != 0)
    xyz = (anchor[idx, None] + offset[idx] * scaling[idx, None, :3])[:, keep].reshape(-1, 3)
    assert torch.allclose(got[0], xyz, rtol=1e-6, atol=1e-6)
    for a, b in zip(got[1:5], want[1:5]):
        assert float((a - b).abs().max()) <= 0.02 and float((a - b).norm()) <= 4e-3 * float(b.norm())


@pytest.mark.gpu
def test_camera_centres_that_do_not_name_a_point_keep_the_general_path():
    """``[3]`` and ``[1, 3]`` are a point; a column would be read as one, but is subtracted row by row (and refused by its shape)."""
    from landmarksystem_b200.components.fields.anchor_decoder import FusedAnchorDecoder

    dec = FusedAnchorDecoder(False, False, False, False, 3, 32, 10).cuda().eval()
    anchor, feats, offset = torch.randn(4, 3).cuda(), torch.randn(4, 32).cuda(), torch.randn(4, 10, 3).cuda()
    scaling, visible, c = torch.rand(4, 6).cuda(), torch.ones(4, dtype=torch.bool).cuda(), torch.tensor([0.3, -2.0, 5.0]).cuda()
    with torch.no_grad():
        point, row = (dec(x, anchor, feats, offset, scaling, visible) for x in (c, c[None]))
        assert all(torch.equal(a, b) for a, b in zip(point[:5], row[:5]))
        for bad in (c[:, None], c[None, None]):
            assert not dec._rows_ok(bad, anchor, feats, offset, scaling, visible, None, None, None)
        with pytest.raises(RuntimeError):
            dec(c[:, None], anchor, feats, offset, scaling, visible)
