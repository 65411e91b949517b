"""The work whose speed is tracked: training steps, rendered frames and small interactive calls of the model families,
each through the entry point a user's program calls (a trainer's ``train_step``, a model in evaluation mode, the inference
engine), with random inputs and randomly initialised fields of the shapes that the shipped configurations, the tests and
``bench.py`` use.

Learning rates of the training cases are low (late in a schedule), so that the scene a pass sees stays the same however
many passes were made before it; the arithmetic of a step does not depend on the rate.
"""
from __future__ import annotations

import math
import os
import tempfile

import numpy as np
import torch

from landmarksystem_b200.components.data.cameras import Camera
from landmarksystem_b200.components.scene import SceneManager
from landmarksystem_b200.configs import BaseConfig
from landmarksystem_b200.models.gridnerf.gridnerf import GridNeRF, GridNeRFConfig
from landmarksystem_b200.models.gridnerf.gridnerf_trainer import GridNeRFTrainer
from landmarksystem_b200.models.instant_ngp.instant_ngp_trainer import NGPTrainer
from landmarksystem_b200.models.nerfacto.nerfacto_trainer import NerfactoTrainer
from landmarksystem_b200.models.origin_gs.gs_model import Gaussian3DConfig, GaussianModel
from landmarksystem_b200.models.origin_gs.gs_trainer import Gaussian3DTrainer
from landmarksystem_b200.models.scaffold_gs.gs_model import ScaffoldGS, ScaffoldGSConfig
from landmarksystem_b200.render.adapters import make_adapter
from landmarksystem_b200.render.inference_engine import InferenceEngine
from landmarksystem_b200.synthetic.scene import aerial_cameras, look_at
from landmarksystem_b200.utils import Config

_BLOCK = (1000.0, 1000.0, 300.0)     # metres: one spatial block of the large-scene GridNeRF configuration
_GS_BOX = (400.0, 400.0, 50.0)       # metres: the box of the 3DGS benchmark cloud
_BATCHES = 4                         # a training state cycles through this many device-resident batches


def listed():
    return [
        # the headline training step: one 4096^2 block, 16 + 48 channels, deferred Adam, no plane regularisers
        {"name": "gridnerf_train_block", "kind": "gridnerf_train", "plane": 4096, "line": 512, "rays": 8192, "samples": 128,
         "regularised": False},
        # the shipped regulariser set (L1 + TV on whole planes) at an odd intermediate resolution of the upsampling schedule
        {"name": "gridnerf_train_shipped", "kind": "gridnerf_train", "plane": 1371, "line": 203, "rays": 8192, "samples": 128,
         "regularised": True},
        # a 1080p frame of a flight through the engine
        {"name": "gridnerf_frame_1080p", "kind": "gridnerf_frame", "plane": 4096, "line": 512, "width": 1920, "height": 1080,
         "chunk": 1 << 18},
        # an interactive preview: one small chunk, where launches and host work count
        {"name": "gridnerf_preview", "kind": "gridnerf_frame", "plane": 1024, "line": 256, "width": 320, "height": 180,
         "chunk": 1 << 18},
        # evaluation render of a city-scale cloud
        {"name": "gs_frame_6m", "kind": "gs_frame", "count": 6_000_000, "width": 1920, "height": 1080},
        # viewer frame of an object-sized cloud at an odd size
        {"name": "gs_frame_60k", "kind": "gs_frame", "count": 60_001, "width": 801, "height": 603},
        # an optimisation step between two densifications
        {"name": "gs_train_1500k", "kind": "gs_train", "count": 1_500_000, "width": 1920, "height": 1080},
        # hash-grid field, large batch and table
        {"name": "ngp_train_128k_rays", "kind": "ngp_train", "rays": 1 << 17, "log2_table": 21},
        # hash-grid field, the batch and table of the low-quality configurations
        {"name": "ngp_train_4k_rays", "kind": "ngp_train", "rays": 4096, "log2_table": 19},
        # evaluation render of the hash-grid field, the trainer's chunk size
        {"name": "ngp_frame_800", "kind": "ngp_frame", "width": 800, "height": 800, "log2_table": 19, "chunk": 16384},
        # proposal-sampled field with the default heads and the shipped batch
        {"name": "nerfacto_train_16k_rays", "kind": "nerfacto_train", "rays": 16384},
        # anchors decoded per view on the kernel runtime
        {"name": "scaffold_frame_400k", "kind": "scaffold_frame", "anchors": 400_000, "width": 1920, "height": 1080},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["gridnerf_train", "gridnerf_frame", "gs_frame", "gs_train", "ngp_train", "ngp_frame", "nerfacto_train",
                       "scaffold_frame"])
    if kind == "gridnerf_train":
        regularised = rng.random() < 0.5
        return {"kind": kind, "plane": _log_uniform(rng, 500, 2048 if regularised else 4096), "line": rng.randint(100, 512),
                "rays": _log_uniform(rng, 2048, 8192), "samples": rng.randint(64, 128), "regularised": regularised}
    width = _log_uniform(rng, 240, 1920)
    height = max(int(width * rng.uniform(0.5, 0.75)), 120)
    if kind == "gridnerf_frame":
        return {"kind": kind, "plane": _log_uniform(rng, 800, 4096), "line": rng.randint(100, 512), "width": width,
                "height": height, "chunk": rng.choice([1 << 16, 1 << 18])}
    if kind == "gs_frame":
        return {"kind": kind, "count": _log_uniform(rng, 50_000, 6_000_000), "width": width, "height": height}
    if kind == "gs_train":
        return {"kind": kind, "count": _log_uniform(rng, 50_000, 2_000_000), "width": width, "height": height}
    if kind == "ngp_train":
        return {"kind": kind, "rays": _log_uniform(rng, 2048, 1 << 17), "log2_table": rng.randint(18, 21)}
    if kind == "ngp_frame":
        side = _log_uniform(rng, 200, 900)
        return {"kind": kind, "width": side, "height": int(side * rng.uniform(0.6, 1.0)), "log2_table": rng.randint(18, 21),
                "chunk": rng.choice([8192, 16384])}
    if kind == "nerfacto_train":
        return {"kind": kind, "rays": _log_uniform(rng, 1024, 16384)}
    return {"kind": kind, "anchors": _log_uniform(rng, 30_000, 500_000), "width": width, "height": height}


def _conf(family, name, **overrides):
    """A shipped configuration file with console-style overrides."""
    path = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "landmarksystem_b200", "models", family, "confs", name)
    base = {"basedir": os.path.join(tempfile.gettempdir(), "lmb_perf_cases"), "n_iters": "1000000",
            "progress_refresh_rate": "1000000"}
    return BaseConfig.from_file(path, {**base, **{k: str(v) for k, v in overrides.items()}})


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _optimiser_state(trainer):
    """Updated parameters, and the first moments that the optimiser keeps for them."""
    out = {}
    names = {id(p): n for n, p in trainer.model.named_parameters()}
    for group in trainer.optimizer.param_groups:
        for p in group["params"]:
            name = names[id(p)]
            out[name] = p.detach()
            moment = trainer.optimizer.state.get(p, {}).get("exp_avg")
            if moment is not None:
                out[name + ".exp_avg"] = moment
    return out


# -- GridNeRF -------------------------------------------------------------------------------------------------
def _aerial_batches(rays, seed):
    """``[_BATCHES, rays, 10]`` packed batches (origin, unit direction, colour, camera) of a nadir-ish capture 400 m above
    the block: random pixels of random 1920 x 1080 cameras, smooth ground colours."""
    g = _generator(seed)
    poses = aerial_cameras(64, (0.0, 0.0, 0.0), _BLOCK, 400.0, 30.0, seed=seed).cuda()
    n = rays * _BATCHES
    cam = torch.randint(0, 64, (n,), device="cuda", generator=g)
    pix = torch.rand(n, 2, device="cuda", generator=g) * torch.tensor([1920.0, 1080.0], device="cuda")
    local = torch.cat(((pix[:, :1] - 960.0) / 1662.8, (540.0 - pix[:, 1:]) / 1662.8, -torch.ones(n, 1, device="cuda")), -1)
    d = torch.nn.functional.normalize(torch.einsum("nij,nj->ni", poses[cam, :3, :3], local), dim=-1)
    o = poses[cam, :3, 3]
    hit = o + d * (-o[:, 2:] / d[:, 2:].clamp(max=-1e-3))
    rgb = 0.5 + 0.5 * torch.sin(torch.stack((hit[:, 0] * 0.01, hit[:, 1] * 0.013, (hit[:, 0] + hit[:, 1]) * 0.007), -1))
    return torch.cat((o, d, rgb, (cam % 8).float()[:, None]), -1).view(_BATCHES, rays, 10)


def _prepare_gridnerf_train(case, seed):
    cfg = _conf("gridnerf", "bench_branch_parallel.py", random_seed=seed, nSamples=case["samples"], lr_init=2e-3, lr_basis=1e-4,
                batch_size=case["rays"])
    cfg.init_grid_size = [case["plane"], case["plane"], case["line"]]
    if case["regularised"]:
        cfg.L1_weight_inital, cfg.L1_weight_rest, cfg.TV_weight_density, cfg.TV_weight_app = 8e-5, 4e-5, 0.1, 0.01
    trainer = GridNeRFTrainer(cfg)
    trainer.model.train()
    return {"trainer": trainer, "batches": _aerial_batches(case["rays"], seed), "step": 0}


class _FloatFrames(make_adapter(GridNeRF)):
    """Pose -> linear image and depth (the stock adapter quantises to 8 bits)."""

    def postprocess(self, rgb, depth=None):
        H, W = self._shape
        return rgb.reshape(H, W, 3), depth.reshape(H, W)


def _prepare_gridnerf_frame(case, seed):
    torch.manual_seed(seed)
    dev = torch.device("cuda", torch.cuda.current_device())
    cfg = Config(dict(GridNeRFConfig(resMode=[1], n_lamb_sigma=[16], n_lamb_sh=[48], nonlinear_density=True, view_pe=2,
                                     fea_pe=2, featureC=128, train_near_far=[10.0, 2000.0], step_ratio=10.0, nSamples=128,
                                     sampling_opt=True, n_importance=128, distance_scale=25, fea2denseAct="relu",
                                     grid_dtype="bf16", runtime="Kernel")))
    cfg.update(is_train=False, device=dev, lb=[0.0, 0.0, 0.0], ub=list(_BLOCK), plane_division=[1, 1], branch_parallel=False)
    scene = SceneManager(cfg)
    engine = InferenceEngine(_FloatFrames(aabb=scene.aabb, gridSize=[case["plane"], case["plane"], case["line"]], device=dev,
                                          near_far=[10.0, 2000.0], scene_manager=scene, config=cfg),
                             Config(runtime="Kernel", kernel_fusion=True))
    rng = np.random.default_rng(seed)
    tilt = math.radians(10.0 + 10.0 * rng.random())
    pose = np.eye(4, dtype=np.float32)
    pose[:3, :3] = [[1.0, 0.0, 0.0], [0.0, math.cos(tilt), -math.sin(tilt)], [0.0, math.sin(tilt), math.cos(tilt)]]
    pose[:3, 3] = [400.0 + 200.0 * rng.random(), 400.0 + 200.0 * rng.random(), 400.0]
    return {"engine": engine, "pose": torch.from_numpy(pose), "focal": 2317.645 * case["width"] / 1920.0}


# -- Gaussians --------------------------------------------------------------------------------------------------
def _cloud(count, seed):
    """Random Gaussians over a 400 m x 400 m x 50 m box; their size falls with their number, so that the overdraw of a
    view stays that of the 6 M cloud (log-scales around -3)."""
    g = _generator(seed)
    shs = torch.randn(count, 16, 3, device="cuda", generator=g) * 0.01
    shs[:, 0] = torch.rand(count, 3, device="cuda", generator=g)
    return {"_xyz": (torch.rand(count, 3, device="cuda", generator=g) - 0.5) * torch.tensor(_GS_BOX, device="cuda"),
            "_features_dc": shs[:, :1].contiguous(), "_features_rest": shs[:, 1:].contiguous(),
            "_scaling": torch.randn(count, 3, device="cuda", generator=g) * 0.5 - 3.0 + 0.5 * math.log(6e6 / count),
            "_rotation": torch.randn(count, 4, device="cuda", generator=g),
            "_opacity": torch.randn(count, 1, device="cuda", generator=g)}


def _orbit_camera(case, seed, k=0):
    angle = 2.0 * math.pi * np.random.default_rng(seed * 7 + k).random()
    eye = torch.tensor([260.0 * math.cos(angle), 260.0 * math.sin(angle), 120.0])
    return Camera.from_c2w(look_at(eye, torch.zeros(3)).numpy(), case["width"], case["height"],
                           focal_x=1400.0 * case["width"] / 1920.0, zfar=2000.0).to("cuda")


def _prepare_gs_frame(case, seed):
    cfg = Config(dict(Gaussian3DConfig(sh_degree=3)))
    cfg.update(device="cuda", debug=False, is_train=False)
    model = GaussianModel(cfg)
    model.gaussian_encoding.load_encoding_state(_cloud(case["count"], seed))
    return {"model": model.eval(), "camera": _orbit_camera(case, seed)}


def _prepare_gs_train(case, seed):
    cfg = _conf("origin_gs", "synthetic_train.py", random_seed=seed, device="cuda", datadir="ring:3:16x16:18:3",
                init_points_num=64, densify_from_iter=10_000_000, densify_until_iter=10_000_000,
                opacity_reset_interval=10_000_000, position_lr_init=1.6e-6, position_lr_final=1.6e-6, feature_lr=2.5e-5,
                opacity_lr=5e-4, scaling_lr=5e-5, rotation_lr=1e-5)
    cfg.lb, cfg.ub = [-0.5 * v for v in _GS_BOX], [0.5 * v for v in _GS_BOX]
    trainer = Gaussian3DTrainer(cfg)
    enc = trainer.model.gaussian_encoding
    enc.load_encoding_state(_cloud(case["count"], seed))
    trainer.optimizer = trainer.create_optimizer()
    cameras = [_orbit_camera(case, seed, k) for k in range(_BATCHES)]
    trainer.model.eval()
    with torch.no_grad():            # the views of a slightly brighter scene
        enc._features_dc.add_(0.05)
        targets = [trainer.model(cam).clone() for cam in cameras]
        enc._features_dc.sub_(0.05)
    trainer.model.train()
    return {"trainer": trainer, "cameras": cameras, "targets": targets, "step": 0}


def _prepare_scaffold_frame(case, seed):
    torch.manual_seed(seed)
    g = _generator(seed)
    n, k, f = case["anchors"], 10, 32
    cfg = Config(dict(ScaffoldGSConfig(feat_dim=f, n_offsets=k, runtime="Kernel", kernel_fusion=True)))
    cfg.update(device="cuda", debug=False, is_train=False)
    model = ScaffoldGS(cfg)
    size = 0.5 * math.log(6e5 / n) - 2.2
    rot = torch.zeros(n, 4, device="cuda")
    rot[:, 0] = 1.0
    model.gaussian_encoding.load_encoding_state({
        "_anchor": (torch.rand(n, 3, device="cuda", generator=g) - 0.5) * torch.tensor(_GS_BOX, device="cuda"),
        "_offset": torch.randn(n, k, 3, device="cuda", generator=g) * 0.5,
        "_anchor_feat": torch.randn(n, f, device="cuda", generator=g),
        "_scaling": torch.randn(n, 6, device="cuda", generator=g) * 0.3 + size,
        "_rotation": rot, "_opacity": torch.zeros(n, 1, device="cuda")})
    return {"model": model.eval(), "camera": _orbit_camera(case, seed)}


# -- hash-grid fields -----------------------------------------------------------------------------------------------
def _trained_like(model, g):
    """Table entries that fall with the level and a density head of wide output, so that rays cross empty and opaque
    regions as in a trained field instead of the uniform fog of a fresh one."""
    meta = model.mlp_base_grid.meta
    with torch.no_grad():
        for table in model.mlp_base_grid.tables():
            rows = table.params.view(-1, meta.n_features)
            for level in range(meta.n_levels):
                part = rows[meta.offsets[level]:meta.offsets[level + 1]]
                part.copy_(torch.randn(part.shape, device="cuda", generator=g) * 0.75 ** level)
        head = [m for m in model.mlp_base_mlp.modules() if isinstance(m, torch.nn.Linear)][-1]
        head.weight[0].mul_(25.0)


def _unit_box_batches(rays, seed):
    """Rays from a circle of radius 3 aimed at the unit scene box, random colours."""
    g = _generator(seed + 1)
    n = rays * _BATCHES
    angle = torch.rand(n, device="cuda", generator=g) * 2.0 * math.pi
    o = torch.stack((3.0 * torch.cos(angle), 3.0 * torch.sin(angle), torch.rand(n, device="cuda", generator=g) - 0.5), -1)
    aim = torch.rand(n, 3, device="cuda", generator=g) * 1.6 - 0.8
    d = torch.nn.functional.normalize(aim - o, dim=-1)
    rgb = torch.rand(n, 3, device="cuda", generator=g)
    return torch.cat((o, d, rgb, torch.randint(0, 3, (n, 1), device="cuda", generator=g).float()), -1).view(_BATCHES, rays, 10)


def _ngp_trainer(case, seed, rays):
    cfg = _conf("instant_ngp", "synthetic_tiny.py", random_seed=seed, device="cuda", runtime="Kernel", num_levels=16, base_res=16,
                max_res=4096, log2_hashmap_size=case["log2_table"], grid_resolution=128, batch_size=rays,
                datadir="ring:3:16x16:20:3", lr_init=1e-4, lr_final=1e-5, lr_decay_max_steps=100_000)
    trainer = NGPTrainer(cfg)
    _trained_like(trainer.model, _generator(seed))
    trainer.model.train()
    trainer.model.update_occupancy_grid(0)
    return trainer


def _prepare_ngp_train(case, seed):
    trainer = _ngp_trainer(case, seed, case["rays"])
    return {"trainer": trainer, "batches": _unit_box_batches(case["rays"], seed), "step": 0, "first_iteration": 1000}


def _prepare_ngp_frame(case, seed):
    model = _ngp_trainer(case, seed, case["chunk"]).model.eval()
    angle = 2.0 * math.pi * np.random.default_rng(seed).random()
    pose = look_at(torch.tensor([3.0 * math.cos(angle), 3.0 * math.sin(angle), 0.6]), torch.zeros(3)).cuda()
    H, W, focal = case["height"], case["width"], 1.2 * case["width"]
    y, x = torch.meshgrid(torch.arange(H, device="cuda") + 0.5, torch.arange(W, device="cuda") + 0.5, indexing="ij")
    local = torch.stack(((x - W / 2) / focal, -(y - H / 2) / focal, -torch.ones_like(x)), -1).view(-1, 3)
    d = torch.nn.functional.normalize(local @ pose[:3, :3].T, dim=-1)
    return {"model": model, "rays": torch.cat((pose[:3, 3].expand_as(d), d), -1).contiguous()}


def _prepare_nerfacto_train(case, seed):
    cfg = _conf("nerfacto", "synthetic_tiny.py", random_seed=seed, device="cuda", runtime="Kernel", num_levels=16, base_res=16,
                max_res=2048, log2_hashmap_size=19, num_nerf_samples_per_ray=48, disable_scene_contraction=False,
                background_color="last_sample", proposal_warmup=5000, proposal_weights_anneal_max_num_iters=1000,
                batch_size=case["rays"], datadir="ring:3:16x16:20:3", lr_init=1e-4, lr_final=1e-5, lr_decay_max_steps=50_000)
    cfg.num_proposal_samples_per_ray = (256, 96)
    cfg.proposal_net_args_list = [{"hidden_dim": 16, "log2_hashmap_size": 17, "num_levels": 5, "max_res": 128},
                                  {"hidden_dim": 16, "log2_hashmap_size": 17, "num_levels": 5, "max_res": 256}]
    cfg.train_near_far = [0.05, 1000.0]
    trainer = NerfactoTrainer(cfg)
    _trained_like(trainer.model, _generator(seed))
    trainer.model.train()
    return {"trainer": trainer, "batches": _unit_box_batches(case["rays"], seed), "step": 0, "first_iteration": 20_000}


# -- one pass --------------------------------------------------------------------------------------------------------
def prepare(case, seed):
    state = {"gridnerf_train": _prepare_gridnerf_train, "gridnerf_frame": _prepare_gridnerf_frame, "gs_frame": _prepare_gs_frame,
             "gs_train": _prepare_gs_train, "ngp_train": _prepare_ngp_train, "ngp_frame": _prepare_ngp_frame,
             "nerfacto_train": _prepare_nerfacto_train, "scaffold_frame": _prepare_scaffold_frame}[case["kind"]](case, seed)
    state["case"] = case
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("gridnerf_train", "ngp_train", "nerfacto_train"):
        trainer, k = state["trainer"], state["step"]
        batch = state["batches"][k % _BATCHES]
        trainer.iteration = state.get("first_iteration", 0) + k
        state["step"] = k + 1
        loss = trainer.train_step(batch[:, :6], batch[:, 6:9], batch[:, 9])
        return {"loss": loss, **_optimiser_state(trainer)}
    if kind == "gs_train":
        trainer, k = state["trainer"], state["step"]
        trainer.iteration = 1000 + k
        state["step"] = k + 1
        loss, l1, image = trainer.train_step(state["cameras"][k % _BATCHES], state["targets"][k % _BATCHES])
        return {"loss": loss, "l1": l1, "image": image, **_optimiser_state(trainer)}
    if kind == "gridnerf_frame":
        image, depth = state["engine"](state["pose"], case["chunk"], case["height"], case["width"], state["focal"])
        return {"image": image, "depth": depth}
    with torch.no_grad():
        if kind == "ngp_frame":
            return state["model"].render_all_rays(state["rays"], chunk_size=case["chunk"])
        return {"image": state["model"](state["camera"])}


# -- what a pass cannot do without ----------------------------------------------------------------------------------
def _gridnerf_work(samples, texels, coloured, train):
    """``samples`` inside the block read 4 plane texels of 16 bf16 channels each, ``coloured`` of them 4 texels of 48; distinct
    texels count once.  Training also reads and writes the fp32 value and both moments of every touched channel."""
    density, colour = min(4 * samples, texels) * 16, min(4 * coloured, texels) * 48
    flops = samples * 16 * 10 + coloured * 2 * (48 * 48 + 159 * 128 + 128 * 128 + 128 * 3)
    return {"bytes": (density + colour) * (2 + (26 if train else 0)), "flops": flops * (3 if train else 1)}


def work(case):
    kind = case["kind"]
    if kind == "gridnerf_train":
        w = _gridnerf_work(0.6 * case["rays"] * case["samples"], case["plane"] ** 2, 8.0 * case["rays"], True)
        if case["regularised"]:      # every texel of the planes is updated: value and moments read and written, bf16 copy written
            w["bytes"] = case["plane"] ** 2 * 64 * 26
        return w
    pixels = case.get("width", 0) * case.get("height", 0)
    if kind == "gridnerf_frame":
        # a view from 400 m covers about 7 % of the block's footprint
        w = _gridnerf_work(100.0 * pixels, 0.07 * case["plane"] ** 2, 8.0 * pixels, False)
        return {"bytes": w["bytes"] + 16 * pixels, "flops": w["flops"]}
    if kind in ("gs_frame", "gs_train"):
        # 59 floats per Gaussian (three quarters of the cloud in view), some 40 blended Gaussians per pixel
        read, blend = case["count"] * 0.75 * 59 * 4, pixels * 40 * 25.0
        if kind == "gs_frame":
            return {"bytes": read + 12 * pixels, "flops": blend}
        return {"bytes": case["count"] * 59 * 4 * 6 + read + 24 * pixels, "flops": 4 * blend}
    if kind == "scaffold_frame":
        return {"bytes": case["anchors"] * (3 + 32 + 30 + 6) * 4.0 + 12 * pixels,
                "flops": case["anchors"] * 0.75 * 2 * (3 * 36 * 32 + 32 * 110) + pixels * 40 * 25.0}
    table = 16 * 2 * 2.0 ** case.get("log2_table", 19)
    head = 2 * (32 * 64 + 64 * 16 + 64 * 64 + 64 * 64 + 64 * 3)
    if kind == "ngp_frame":
        return {"bytes": table * 2 + 16 * pixels, "flops": pixels * 60.0 * head}
    if kind == "ngp_train":
        return {"bytes": table * 26, "flops": case["rays"] * 25.0 * head * 3}
    return {"bytes": table * 24, "flops": case["rays"] * (48 * head * 3 + (256 + 96) * 2 * (10 * 16 + 16) * 1.4)}


def tolerance(case):
    """About four times the difference that was measured between the kernels and the same path compiled with IEEE division
    and library transcendentals (Gaussians: 9e-6 and 0.004 for a frame, 2e-3 and a single value at about its size for the
    moments of a step, where a blend may stop one Gaussian earlier), or evaluated by fp32 tensor operations (hash-grid
    frame 5e-4 and 0.02, moments of its training 1e-2 and 0.5: bf16 features and heads with fp32 sums)."""
    kind = case["kind"]
    if kind == "gs_frame":
        return {"rel": 5e-5, "max": 0.02}
    if kind == "gs_train":
        return {"rel": 8e-3, "max": 0.99}
    if kind == "ngp_frame":
        return {"rel": 2e-3, "max": 0.08}
    if kind in ("gridnerf_frame", "scaffold_frame"):
        return {"rel": 1e-2, "max": 0.5}
    return {"rel": 1e-2, "max": 0.9}
