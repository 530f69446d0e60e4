"""The workloads that this library's speed is measured on.

Every case is one pass through the public entry points of one renderer, as a training or a
reconstruction program calls it: mostly forward and backward of a frame, and of a batch of
frames, with the sizes of this repository's configurations (64 to 512 pixels a side, 2 thousand
to 1 million Gaussians, B-mode frames of 512 scanlines by 1024 samples) and ragged ones between.

``listed()`` names the cases, ``draw(rng)`` gives further ones of the same ranges,
``prepare(case, seed)`` makes what a program has in hand before the call, ``run(state)`` is one
pass, ``work(case)`` what the pass cannot do without, ``exact(case, seed)`` the same outputs
from plain torch in 64 bits. Where the renderers' published conventions are not the
derivative of their image (finite-difference shape gradients, pose entries, screen-space and
quaternion gradients of the surfels), an output has no such value and ``exact`` has None there.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path
from types import SimpleNamespace

import torch

ROOT = Path(__file__).resolve().parents[1]
PACKAGE = ROOT / "ultrasound-3d-reconstruction_b200"
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

CHI2, BETA, BG_ALPHA = 7.815, 1.0e-4, 1.0e-6
CUBE_MM = 64.0


# ------------------------------------------------------------------------------------
# The cases
# ------------------------------------------------------------------------------------

def listed():
    return [
        # A preview frame of a small model, image and gradients: the smallest call there is, where
        # launches and host work count.
        dict(name="ug_frame_small", kind="ug_frame", gauss=2048, height=64, width=64, fov_mm=64.0, scene="cube"),
        # One frame of a freehand sweep through a tissue-like model, as the reference's training loop
        # calls the renderer (one frame per step).
        dict(name="ug_frame", kind="ug_frame", gauss=200_000, height=256, width=256, fov_mm=51.2, scene="clustered"),
        # Evaluation of one frame with the per-pixel candidate lists, at a ragged size: forward only.
        dict(name="ug_inspect_ragged", kind="ug_inspect", gauss=100_000, height=203, width=157, fov_mm=48.0,
             scene="cube"),
        # The headline batch: sixteen 512x512 frames of a sweep through a million Gaussians.
        dict(name="ug_batch", kind="ug_batch", gauss=1_000_000, frames=16, height=512, width=512, fov_mm=64.0,
             scene="cube"),
        # Independent patients' sweeps with their own models and frame sizes in one call.
        dict(name="ug_sweeps", kind="ug_sweeps", sweeps=8, gauss_min=10_000, gauss_max=200_000, frames_min=2,
             frames_max=8),
        # A whole training step (loss, backward, Adam) on a fixed batch, late in a decayed schedule.
        dict(name="ug_train_step", kind="ug_train", gauss=300_000, frames=8, height=192, width=192, fov_mm=57.6,
             scene="clustered"),
        # The projected-slice renderer on one frame, pose refinement included.
        dict(name="gp_frame", kind="gp", gauss=200_000, height=256, width=256, fov_mm=51.2, pose=True),
        # The slice-adapted renderer on one frame: projection, cull, splat and their gradients.
        dict(name="sa_frame", kind="sa", gauss=200_000, height=256, width=256, fov_mm=51.2),
        # The same renderer on a small ragged frame.
        dict(name="sa_frame_small", kind="sa", gauss=12_000, height=101, width=133, fov_mm=30.0),
        # The surfel rasteriser on one frame, colour and the seven auxiliary maps.
        dict(name="gs_frame", kind="gs", gauss=200_000, height=256, width=256, fov_mm=51.2, degree=0),
        # A linear-array frame of the scanline renderer.
        dict(name="ugr_frame", kind="ugr", gauss=100_000, width=128, height=512, scene="probe"),
        # A full B-mode frame of the scanline renderer: the largest single call.
        dict(name="ugr_bmode", kind="ugr", gauss=1_000_000, width=512, height=1024, scene="bmode"),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ug_frame", "ug_frame", "ug_inspect", "ug_batch", "ug_sweeps", "ug_train", "gp", "gp", "sa",
                       "sa", "gs", "gs", "ugr", "ugr"])
    side = lambda lo=48, hi=512: _log_int(rng, lo, hi)  # noqa: E731
    fov = round(rng.uniform(30.0, 60.0), 2)
    scene = rng.choice(["cube", "clustered"])
    if kind in ("ug_frame", "ug_inspect"):
        return dict(kind=kind, gauss=_log_int(rng, 2_000, 1_000_000 if kind == "ug_frame" else 200_000),
                    height=side(), width=side(), fov_mm=fov, scene=scene)
    if kind == "ug_batch":
        return dict(kind=kind, gauss=_log_int(rng, 20_000, 1_000_000), frames=rng.randint(2, 16),
                    height=side(96, 400), width=side(96, 400), fov_mm=fov, scene=scene)
    if kind == "ug_sweeps":
        return dict(kind=kind, sweeps=rng.randint(2, 10), gauss_min=_log_int(rng, 5_000, 20_000),
                    gauss_max=_log_int(rng, 50_000, 200_000), frames_min=rng.randint(1, 3),
                    frames_max=rng.randint(4, 8))
    if kind == "ug_train":
        return dict(kind=kind, gauss=_log_int(rng, 20_000, 500_000), frames=rng.randint(2, 8),
                    height=side(96, 224), width=side(96, 224), fov_mm=fov, scene=scene)
    if kind == "gp":
        return dict(kind=kind, gauss=_log_int(rng, 3_000, 250_000), height=side(64, 320), width=side(64, 320),
                    fov_mm=fov, pose=rng.random() < 0.5)
    if kind == "sa":
        return dict(kind=kind, gauss=_log_int(rng, 5_000, 400_000), height=side(64, 400), width=side(64, 400),
                    fov_mm=fov)
    if kind == "gs":
        return dict(kind=kind, gauss=_log_int(rng, 3_000, 250_000), height=side(64, 400), width=side(64, 400),
                    fov_mm=fov, degree=rng.choice([0, 0, 1]))
    return dict(kind="ugr", gauss=_log_int(rng, 3_000, 200_000), width=_log_int(rng, 48, 256),
                height=_log_int(rng, 96, 768), scene=rng.choice(["probe", "bmode"]))


# ------------------------------------------------------------------------------------
# Inputs
# ------------------------------------------------------------------------------------

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(1_000_003 * int(seed) + 17)
    return g


def _scene(n, scene, g):
    """Means, scales, unit quaternions, opacities, intensities and raw precision factors of n
    Gaussians: "cube" uniform in a 64 mm cube (1 mm median scales, opacity sigmoid(N(0,1))),
    "clustered" twenty ellipsoidal clusters in a 100 x 60 x 80 mm box with a tenth of background
    (0.8 mm median scales, opacity sigmoid(N(-1,1)))."""
    from us3d_b200 import scenes

    dev = _device()
    rand = lambda *s: torch.rand(s, generator=g, device=dev, dtype=torch.float64)  # noqa: E731
    randn = lambda *s: torch.randn(s, generator=g, device=dev, dtype=torch.float64)  # noqa: E731
    if scene == "cube":
        means = rand(n, 3) * CUBE_MM
        scales = torch.exp(0.3 * randn(n, 3))
        opac = torch.sigmoid(randn(n))
    else:
        ext = torch.tensor([100.0, 60.0, 80.0], dtype=torch.float64, device=dev)
        centre = (0.1 + 0.8 * rand(20, 3)) * ext
        semi = 3.0 + 9.0 * rand(20, 3)
        q = randn(20, 4)
        rot = scenes.quat_to_rot(q / q.norm(dim=1, keepdim=True))
        which = (rand(n) * 20).long().clamp_max(19)
        d = randn(n, 3)
        local = d / d.norm(dim=1, keepdim=True) * rand(n, 1).pow(1.0 / 3.0) * semi[which]
        pts = centre[which] + (rot[which] * local[:, None, :]).sum(-1)
        means = torch.where(rand(n, 1) < 0.1, rand(n, 3) * ext, pts).clamp_min(0.0).minimum(ext)
        scales = torch.exp(math.log(0.8) + 0.4 * randn(n, 3))
        opac = torch.sigmoid(randn(n) - 1.0)
    q = randn(n, 4)
    q = q / q.norm(dim=1, keepdim=True).clamp_min(1e-12)
    inten = rand(n)
    tril = scenes.precision_tril_from_scales_quats(scales, q, BETA)
    f = lambda t: t.float().contiguous()  # noqa: E731
    return SimpleNamespace(means=f(means), scales=f(scales), quats=f(q), opacities=f(opac), intensities=f(inten),
                           tril=tril.contiguous())


def _sweep(case, seed, n_frames=1):
    """Frames of the case's size: a linear sweep through the cube or a freehand random walk."""
    from us3d_b200 import scenes

    H, W = case["height"], case["width"]
    spacing = case["fov_mm"] / max(H, W)
    if case["scene"] == "cube":
        return scenes.linear_sweep(n_frames, H, W, spacing, seed=seed)
    return scenes.random_walk_sweep(n_frames + 3, H, W, spacing, seed=seed)[3:]


def _leaf(*tensors):
    return [t.detach().clone().requires_grad_(True) for t in tensors]


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=_device())


def _pose(fr, dev):
    P = torch.eye(4)
    P[:3, 0], P[:3, 1], P[:3, 2], P[:3, 3] = fr.axis_lat, fr.axis_ax, fr.axis_ele, fr.origin
    return P.to(dev)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state.call(state)


def _grads(out, params, adjoint):
    return torch.autograd.grad(out, params, adjoint)


# UltraGauss, one frame ---------------------------------------------------------------

def _prepare_ug_frame(case, seed):
    from ultragauss_renderer import SliceGeometry, UltraGaussRenderConfig, UltraGaussRenderer

    g = _generator(seed)
    sc = _scene(case["gauss"], case["scene"], g)
    fr = _sweep(case, seed)[0].to(_device())
    cfg = UltraGaussRenderConfig(H=fr.height, W=fr.width, lateral_spacing_mm_per_pix=fr.lateral_spacing,
                                 axial_spacing_mm_per_pix=fr.axial_spacing, axial_near_mm=fr.axial_near,
                                 chi2_threshold=CHI2, diag_beta=BETA, fixed_bg_alpha=BG_ALPHA,
                                 lateral_col_offset=fr.lateral_col_offset)
    params = _leaf(sc.means, sc.tril, sc.opacities, sc.intensities)
    return SimpleNamespace(call=_run_ug_frame if case["kind"] == "ug_frame" else _run_ug_inspect, frames=[fr],
                           sets=[(0, case["gauss"])], renderer=UltraGaussRenderer(cfg), params=params,
                           pixels=fr.pixels.contiguous(),
                           geometry=SliceGeometry(fr.origin, fr.axis_lat, fr.axis_ax, fr.axis_ele),
                           adjoint=_randn(g, fr.height, fr.width))


def _run_ug_frame(s):
    image, alpha, depth, _ = s.renderer(*s.params, s.pixels, s.geometry)
    return [image.detach(), alpha.detach(), depth.detach(), *_grads(image, s.params, s.adjoint)]


def _run_ug_inspect(s):
    with torch.no_grad():
        image, alpha, depth, inter = s.renderer(*s.params, s.pixels, s.geometry, True)
        # reading the offsets builds the candidate lists too; their length hangs on the scene
        return [image, alpha, depth, inter["pixel_gauss_counts"], inter["pixel_gauss_offsets"]]


# UltraGauss, batches of frames -------------------------------------------------------

def _spec(fr, gaussian_set=None):
    from us3d_b200 import ultragauss as UG

    return UG.SliceSpec(fr.height, fr.width, fr.lateral_spacing, fr.axial_spacing, fr.axial_near,
                        fr.lateral_col_offset, fr.origin, fr.axis_lat, fr.axis_ax, fr.axis_ele, gaussian_set)


def _prepare_ug_batch(case, seed):
    from us3d_b200.batch import UltraGaussBatchRenderer

    g = _generator(seed)
    sc = _scene(case["gauss"], case["scene"], g)
    frames = _sweep(case, seed, case["frames"])
    dev = _device()
    pixels = torch.cat([f.pixels for f in frames]).to(dev).contiguous()
    return SimpleNamespace(call=_run_ug_batch, frames=frames, sets=[(0, case["gauss"])] * len(frames),
                           renderer=UltraGaussBatchRenderer([_spec(f) for f in frames], dev),
                           params=_leaf(sc.means, sc.tril, sc.opacities, sc.intensities), pixels=pixels,
                           adjoint=_randn(g, pixels.shape[0]))


def _prepare_ug_sweeps(case, seed):
    from us3d_b200 import scenes
    from us3d_b200.batch import UltraGaussBatchRenderer

    g, dev = _generator(seed), _device()
    frames, sets, parts, first = [], [], [], 0
    for k in range(case["sweeps"]):
        u = (k + 0.5) / case["sweeps"]
        n = int(round(case["gauss_min"] * (case["gauss_max"] / case["gauss_min"]) ** u))
        size = (128, 200, 256, 131)[k % 4]
        count = case["frames_min"] + (k * 5) % (case["frames_max"] - case["frames_min"] + 1)
        parts.append(_scene(n, "cube", g))
        fr = scenes.linear_sweep(count, size, size, CUBE_MM / size, seed=seed + k, step_mm=4.0)
        frames += fr
        sets += [(first, n)] * count
        first += n
    cat = lambda name: torch.cat([getattr(p, name) for p in parts]).contiguous()  # noqa: E731
    pixels = torch.cat([f.pixels for f in frames]).to(dev).contiguous()
    return SimpleNamespace(call=_run_ug_batch, frames=frames, sets=sets,
                           renderer=UltraGaussBatchRenderer([_spec(f, s) for f, s in zip(frames, sets)], dev),
                           params=_leaf(cat("means"), cat("tril"), cat("opacities"), cat("intensities")),
                           pixels=pixels, adjoint=_randn(g, pixels.shape[0]))


def _run_ug_batch(s):
    image, alpha, depth = s.renderer(*s.params, s.pixels)
    return [image.detach(), alpha.detach(), depth.detach(), *_grads(image, s.params, s.adjoint)]


def _prepare_ug_train(case, seed):
    from us3d_b200.train import TrainConfig, UltraGaussParameters, UltraGaussTrainer

    g, dev = _generator(seed), _device()
    sc = _scene(case["gauss"], case["scene"], g)
    frames = _sweep(case, seed, case["frames"])
    logit = lambda x: torch.log(x / (1.0 - x))  # noqa: E731
    params = UltraGaussParameters(sc.means, sc.tril, logit(sc.opacities.clamp(1e-4, 1 - 1e-4)),
                                  logit(sc.intensities.clamp(1e-4, 1 - 1e-4)))
    pixels = torch.cat([f.pixels for f in frames]).to(dev).contiguous()
    targets = torch.rand(pixels.shape[0], generator=g, device=dev)
    trainer = UltraGaussTrainer(params, [([_spec(f) for f in frames], pixels, targets)],
                                TrainConfig(lr=1.0e-5, ssim_weight=0.2), margin=1.5)
    return SimpleNamespace(call=_run_ug_train, trainer=trainer)


def _run_ug_train(s):
    s.trainer.step()
    return [*s.trainer.grads, s.trainer.params.means]


# GaussianPile ------------------------------------------------------------------------

def _prepare_gp(case, seed):
    from gaussianplie_renderer import GaussianPlieRenderConfig, GaussianPlieRenderer, build_slice_grid_pack

    g, dev = _generator(seed), _device()
    sc = _scene(case["gauss"], "clustered", g)
    fr = _sweep(dict(case, scene="clustered"), seed)[0]
    H, W, sp = fr.height, fr.width, fr.lateral_spacing
    renderer = GaussianPlieRenderer(GaussianPlieRenderConfig(
        H=H, W=W, lateral_spacing_mm_per_pix=sp, axial_spacing_mm_per_pix=sp, axial_near_mm=0.0, sigma_z_mm=1.0))
    renderer.set_slice_grid_geometry(build_slice_grid_pack(SimpleNamespace(
        H=H, W=W, delta_lateral_mm=sp, delta_axial_mm=sp, near_mm=0.0, center_lateral=True), dev))
    # rotations around the identity that training starts from: the renderer's R D R is a covariance
    # near it, and singular to rounding for some rotations far from it
    quats = torch.tensor([1.0, 0.0, 0.0, 0.0], device=dev) + 0.02 * _randn(g, case["gauss"], 4)
    params = _leaf(sc.means, sc.scales, quats / quats.norm(dim=1, keepdim=True), sc.opacities)
    pose = _pose(fr, dev).requires_grad_(bool(case["pose"]))
    return SimpleNamespace(call=_run_gp, renderer=renderer, params=params, pose=pose, spacing=sp,
                           adjoint=_randn(g, H, W))


def _run_gp(s):
    image = s.renderer(*s.params, s.pose)
    return [image.detach(), *_grads(image, s.params + ([s.pose] if s.pose.requires_grad else []), s.adjoint)]


# slice-adapted 3DGS ------------------------------------------------------------------

def _prepare_sa(case, seed):
    from slice_adapted_3dgs_renderer.fused import (SliceAdapted3DGSInput, SliceAdaptedRenderSettings,
                                                   SliceCameraInput)

    g, dev = _generator(seed), _device()
    sc = _scene(case["gauss"], "clustered", g)
    fr = _sweep(dict(case, scene="clustered"), seed)[0]
    hw, hh = fr.width * fr.lateral_spacing / 2, fr.height * fr.axial_spacing / 2
    view = torch.eye(4)
    rot = torch.stack([fr.axis_lat, fr.axis_ax, fr.axis_ele])
    view[:3, :3] = rot
    view[:3, 3] = -(rot @ (fr.origin + fr.axis_ax * hh))
    colors = sc.intensities[:, None] * (0.6 + 0.4 * torch.rand((case["gauss"], 3), generator=g, device=dev))
    params = _leaf(sc.means, sc.scales, sc.quats, sc.opacities[:, None], colors)
    return SimpleNamespace(
        call=_run_sa, params=params, gaussians=SliceAdapted3DGSInput(*params),
        camera=SliceCameraInput(fr.height, fr.width, hw, hh, 0.0, view.t().contiguous().to(dev)),
        settings=SliceAdaptedRenderSettings(output_grayscale=False, clamp_output=False),
        adjoint=_randn(g, 3, fr.height, fr.width))


def _run_sa(s):
    from slice_adapted_3dgs_renderer import render_slice_adapted_3dgs

    out = render_slice_adapted_3dgs(s.gaussians, s.camera, s.settings)
    return [out.image.detach(), out.extras["alpha_image"].detach(), out.extras["visibility_filter"],
            *_grads(out.image, s.params, s.adjoint)]


# UltraGS surfels ---------------------------------------------------------------------

CAMERA_MM = 60.0


def _prepare_gs(case, seed):
    from ultrags_baseline_renderer import GaussianRasterizationSettings, GaussianRasterizer

    g, dev = _generator(seed), _device()
    sc = _scene(case["gauss"], "clustered", g)
    fr = _sweep(dict(case, scene="clustered"), seed)[0]
    H, W, sp = fr.height, fr.width, fr.lateral_spacing
    rot = torch.stack([fr.axis_lat, fr.axis_ax, fr.axis_ele]).double()
    cam = fr.origin.double() + fr.axis_ax.double() * (H * sp / 2) - CAMERA_MM * fr.axis_ele.double()
    view = torch.eye(4, dtype=torch.float64)
    view[:3, :3] = rot
    view[:3, 3] = -(rot @ cam)
    tx, ty = (W * sp / 2) / CAMERA_MM, (H * sp / 2) / CAMERA_MM
    near, far = 0.01, 1000.0
    proj = torch.zeros((4, 4), dtype=torch.float64)
    proj[0, 0], proj[1, 1], proj[3, 2] = 1.0 / tx, 1.0 / ty, 1.0
    proj[2, 2], proj[2, 3] = far / (far - near), -(far * near) / (far - near)
    d = lambda t: t.float().to(dev).contiguous()  # noqa: E731
    settings = GaussianRasterizationSettings(H, W, tx, ty, torch.zeros(3, device=dev), 1.0, d(view.t()),
                                             d((proj @ view).t()), int(case["degree"]), d(cam), False, False)
    sh = 0.1 * _randn(g, case["gauss"], (case["degree"] + 1) ** 2, 3)
    sh[:, 0, :] = ((sc.intensities - 0.5) / 0.28209479177387814)[:, None]
    params = _leaf(sc.means, torch.zeros_like(sc.means), sc.opacities[:, None], sh, sc.scales[:, :2].contiguous(),
                   sc.quats)
    return SimpleNamespace(call=_run_gs, renderer=GaussianRasterizer(settings), settings=settings, params=params,
                           adjoint=[_randn(g, 3, H, W), 0.1 * _randn(g, 7, H, W)])


def _run_gs(s):
    means, means2d, opac, sh, scales, quats = s.params
    color, radii, allmap = s.renderer(means, means2d, opac, shs=sh, scales=scales, rotations=quats)
    return [color.detach(), allmap.detach(), radii, *_grads([color, allmap], s.params, s.adjoint)]


# UltraGray scanlines -----------------------------------------------------------------

def _prepare_ugr(case, seed):
    from us3d_b200 import scenes
    from ultragray_renderer import ProbeGeometry, UltragrayRenderConfig, UltragrayRenderer

    g, dev = _generator(seed), _device()
    n, W, H = case["gauss"], case["width"], case["height"]
    rand = lambda *s: torch.rand(s, generator=g, device=dev)  # noqa: E731
    quats = _randn(g, n, 4)
    quats = quats / quats.norm(dim=1, keepdim=True).clamp_min(1e-12)
    if case["scene"] == "bmode":
        # tissue attenuating 0.5 dB/cm/MHz at 5 MHz in a 40 x 60 x 64 mm box, 5 % strong reflectors
        width, near, depth, off = 40.0, 0.0, 60.0, 0.5
        box = torch.tensor([40.0, 60.0, 64.0], device=dev)
        means = rand(n, 3) * box
        scales = torch.exp(0.3 * _randn(g, n, 3))
        sh = torch.zeros((n, 4), device=dev)
        sh[:, 0] = torch.where(rand(n) < 0.05, 5.0 + 5.0 * rand(n), rand(n))
        att = torch.full((n,), scenes.bmode_attenuation_logit(n, 40.0 * 60.0 * 64.0), device=dev)
        fr = scenes.bmode_sweep(1, W, H)[0]
        origin, lat, ele, ax = fr.origin, fr.axis_lat, fr.axis_ele, fr.axis_ax
        rays, dirs, pixels = fr.ray_origins, fr.ray_dirs, fr.pixels
    else:
        # a slab of 5 mm thickness under a 38 mm linear array
        width, near, depth, off = 38.0, 2.0, 40.0, 0.5
        u, v, w = (rand(n) - 0.5) * 1.1 * width, (rand(n) - 0.5) * 5.0, rand(n) * (depth + 4.0)
        means = torch.stack([u, v, w], 1)
        scales = torch.exp(math.log(0.25) + rand(n, 3) * math.log(1.2 / 0.25))
        sh = torch.cat([0.2 + 0.8 * rand(n, 1), 0.15 * _randn(g, n, 3)], 1)
        att = 0.5 + 1.2 * _randn(g, n)
        lat, ele, ax = torch.eye(3)
        origin = torch.zeros(3)
        xs = (torch.arange(W, dtype=torch.float64) - (W - 1) * 0.5) * (width / W)
        zs = near + (torch.arange(H, dtype=torch.float64) + 0.5) * (depth / H)
        rays = (xs[:, None] * lat.double()).float()
        dirs = ax.repeat(W, 1)
        pixels = (xs[:, None, None] * lat.double() + zs[None, :, None] * ax.double()).float()
    d = lambda t: t.float().to(dev).contiguous()  # noqa: E731
    cfg = UltragrayRenderConfig(image_width=W, image_height=H, width_mm=width, near_mm=near, ops_max_offset_mm=off)
    params = _leaf(means.contiguous(), scales.contiguous(), quats.contiguous(), att, sh.contiguous())
    return SimpleNamespace(call=_run_ugr, renderer=UltragrayRenderer(cfg), cfg=cfg, params=params, pixels=d(pixels),
                           rays=d(rays), dirs=d(dirs), geometry=ProbeGeometry(d(origin), d(lat), d(ele), d(ax)),
                           seed=int(seed), adjoint=_randn(g, H, W))


def _run_ugr(s):
    torch.cuda.manual_seed(s.seed)  # the renderer draws each ray's elevational offset
    image = s.renderer(*s.params, s.pixels, s.rays, s.dirs, s.geometry)
    return [image.detach(), *_grads(image, s.params, s.adjoint)]


_PREPARE = dict(ug_frame=_prepare_ug_frame, ug_inspect=_prepare_ug_frame, ug_batch=_prepare_ug_batch,
                ug_sweeps=_prepare_ug_sweeps, ug_train=_prepare_ug_train, gp=_prepare_gp, sa=_prepare_sa,
                gs=_prepare_gs, ugr=_prepare_ugr)


# ------------------------------------------------------------------------------------
# Work
# ------------------------------------------------------------------------------------

def _ug_pairs(gauss, pixels_per_mm2, box_mm=CUBE_MM, sigma=1.0):
    """(Gaussian, pixel) pairs inside the chi-square ellipsoids of one frame: an ellipsoid of
    half-width sqrt(chi2) sigma meets the slice with probability 2 sqrt(chi2) sigma / box, in a
    disc of 2/3 pi chi2 sigma^2 on average."""
    return gauss * (2 * math.sqrt(CHI2) * sigma / box_mm) * (2.0 / 3.0 * math.pi * CHI2 * sigma ** 2) * pixels_per_mm2


def work(case):
    kind = case["kind"]
    f = 4.0
    if kind == "ug_sweeps":
        n = case["sweeps"]
        mean_g = (case["gauss_max"] - case["gauss_min"]) / math.log(case["gauss_max"] / case["gauss_min"])
        frames = n * (case["frames_min"] + case["frames_max"]) / 2
        px = 178.0 ** 2
        return dict(bytes=n * mean_g * 22 * f + frames * px * 7 * f,
                    flops=frames * _ug_pairs(mean_g, px / CUBE_MM ** 2) * 75)
    G, px = case["gauss"], case["height"] * case["width"]
    if kind in ("ug_frame", "ug_inspect", "ug_batch", "ug_train"):
        F = case.get("frames", 1)
        sp = case["fov_mm"] / max(case["height"], case["width"])
        cube = case["scene"] == "cube"
        seen = min(1.0, px * sp * sp / (CUBE_MM ** 2 if cube else 6000.0))
        pairs = F * _ug_pairs(G * seen, 1.0 / sp ** 2, CUBE_MM if cube else 80.0, 1.0 if cube else 0.85)
        if kind == "ug_inspect":
            return dict(bytes=G * 11 * f + px * 8 * f + pairs * f, flops=pairs * 40)
        back = 22 + (33 if kind == "ug_train" else 0)
        return dict(bytes=G * back * f + F * px * 7 * f, flops=pairs * 75)
    sp = case.get("fov_mm", 0.0) / max(case["height"], case["width"])
    if kind == "gp":
        pairs = G * 0.25 * min(1.0, px * sp * sp / 6000.0) * 18.0 / sp ** 2
        return dict(bytes=G * 22 * f + px * 2 * f, flops=pairs * 60 + G * 14 * 200)
    if kind == "sa":
        pairs = G * 0.07 * min(1.0, px * sp * sp / 6000.0) * 18.0 / sp ** 2
        return dict(bytes=G * 28 * f + G + px * 7 * f, flops=pairs * 60 + G * 300)
    if kind == "gs":
        sh = 3 * (case["degree"] + 1) ** 2
        return dict(bytes=G * (2 * (13 + sh) + 1) * f + px * 20 * f, flops=px * 60 * 250 + G * 600)
    # scanlines: every sample past a Gaussian is attenuated by it
    area = 40.0 * 60.0 * 64.0 if case["scene"] == "bmode" else 41.8 * 5.0 * 44.0
    radius = 3.0 * (1.3 if case["scene"] == "bmode" else 0.8)
    width = 40.0 if case["scene"] == "bmode" else 38.0
    slab = min(1.0, 2 * radius * (60.0 if case["scene"] == "bmode" else 44.0) * width / area)
    instances = G * slab * min(1.0, 2 * radius / width) * case["width"]
    near = case["height"] * min(1.0, 2 * radius / 60.0)
    return dict(bytes=G * 30 * f + px * 6 * f, flops=instances * near * 100)


# ------------------------------------------------------------------------------------
# The same outputs in 64 bits, plain torch
# ------------------------------------------------------------------------------------

PAIR_CHUNK = 8_000_000


def exact(case, seed):
    fn = _EXACT.get(case["kind"])
    return None if fn is None else fn(case, prepare(case, seed))


def _box_chunks(x0, x1, y0, y1):
    """Chunks (element ids, x, y) over all pixels of the elements' boxes [x0, x1] x [y0, y1]."""
    w, h = (x1 - x0 + 1).clamp_min(0), (y1 - y0 + 1).clamp_min(0)
    area = w * h
    ends = torch.cumsum(area, 0)
    n, i0, done = int(area.numel()), 0, 0
    while i0 < n:
        i1 = min(n, max(i0 + 1, int(torch.searchsorted(ends, done + PAIR_CHUNK))))
        part = area[i0:i1]
        total = int(part.sum())
        if total:
            ids = torch.repeat_interleave(torch.arange(i0, i1, device=area.device), part)
            k = torch.arange(total, device=area.device) + (done - (ends - area)[ids])
            yield ids, x0[ids] + k % w[ids], y0[ids] + k // w[ids]
        done = int(ends[i1 - 1])
        i0 = i1


def _splat(values, chunks, contribution, n_pixels, n_sums):
    """(n_pixels, n_sums) sums over pairs of contribution(gathered values, x, y) -> (pixel index,
    list of contributions), and a function taking d/dsums to d/dvalues (values: (n, k) tensor)."""
    chunks = list(chunks) if not callable(chunks) else chunks
    each = lambda: chunks() if callable(chunks) else chunks  # noqa: E731
    sums = torch.zeros((n_pixels, n_sums), dtype=torch.float64, device=values.device)
    for ids, x, y in each():
        p, c = contribution(values[ids], x, y)
        sums.index_add_(0, p, torch.stack(c, 1))

    def backward(d_sums):
        grad = torch.zeros_like(values)
        for ids, x, y in each():
            with torch.enable_grad():
                v = values[ids].detach().requires_grad_(True)
                p, c = contribution(v, x, y)
                loss = sum((ck * d_sums[p, k]).sum() for k, ck in enumerate(c))
            grad.index_add_(0, ids, torch.autograd.grad(loss, v)[0])
        return grad

    return sums, backward


def _exact_ug(case, s):
    """Every pair with d^T Lambda d <= chi2 contributes alpha = o exp(-q/2): image = (sum alpha c +
    bg) / (sum alpha + bg), depth the alpha-weighted elevation."""
    if case["kind"] != "ug_inspect" and work(case)["flops"] > 4e11:
        return None
    dev = _device()
    means, tril, opac, inten = (p.detach().double() for p in s.params)
    l11, l22, l33 = (tril[:, k] ** 2 + BETA for k in (0, 3, 5))
    raw = torch.cat([means, tril, opac[:, None], inten[:, None]], 1)
    total = torch.zeros_like(raw)
    images, alphas, depths, off = [], [], [], 0
    for fr, (first, count) in zip(s.frames, s.sets):
        H, W = fr.height, fr.width
        pix = s.pixels[off:off + H * W].double()
        adj = s.adjoint.reshape(-1)[off:off + H * W].double()
        off += H * W
        o, lat, ax, ele = (t.double().to(dev) for t in (fr.origin, fr.axis_lat, fr.axis_ax, fr.axis_ele))
        sl = slice(first, first + count)
        d = means[sl] - o

        def half(a):  # sqrt(chi2) |L^-1 a|
            y0 = a[0] / l11[sl]
            y1 = (a[1] - tril[sl, 1] * y0) / l22[sl]
            y2 = (a[2] - tril[sl, 2] * y0 - tril[sl, 4] * y1) / l33[sl]
            return (CHI2 * (y0 * y0 + y1 * y1 + y2 * y2)).sqrt()

        u, v = d @ lat / fr.lateral_spacing + fr.lateral_col_offset, (d @ ax - fr.axial_near) / fr.axial_spacing
        ru, rv = half(lat) / fr.lateral_spacing + 1.0, half(ax) / fr.axial_spacing + 1.0
        lo = lambda c, r: (c - r).floor().long().clamp_min(0)  # noqa: E731
        hi = lambda c, r, n: (c + r).ceil().long().clamp_max(n - 1)  # noqa: E731
        x0, x1, y0, y1 = lo(u, ru), hi(u, ru, W), lo(v, rv), hi(v, rv, H)
        keep = ((d @ ele).abs() <= half(ele)) & (x0 <= x1) & (y0 <= y1)
        idx = torch.nonzero(keep).reshape(-1)
        boxes = [t[idx] for t in (x0, x1, y0, y1)]

        def pair(g, x, y):
            p = y * W + x
            e = pix[p] - g[:, :3]
            a, b, c = g[:, 3] ** 2 + BETA, g[:, 6] ** 2 + BETA, g[:, 8] ** 2 + BETA
            z0 = a * e[:, 0] + g[:, 4] * e[:, 1] + g[:, 5] * e[:, 2]
            z1 = b * e[:, 1] + g[:, 7] * e[:, 2]
            z2 = c * e[:, 2]
            q = z0 * z0 + z1 * z1 + z2 * z2
            al = g[:, 9] * torch.exp(-0.5 * q) * (q.detach() <= CHI2)
            return p, [al, al * g[:, 10], al * ((g[:, :3] - o) @ ele)]

        sums, back = _splat(raw[sl][idx], lambda b=boxes: _box_chunks(*b), pair, H * W, 3)
        leaf = sums.clone().requires_grad_(True)
        with torch.enable_grad():
            img = leaf[:, 1] / (leaf[:, 0] + BG_ALPHA).clamp_min(1e-8)
        images.append(img.detach().clamp(0.0, 1.0))
        alphas.append(sums[:, 0] + BG_ALPHA)
        depths.append(sums[:, 2] / sums[:, 0].clamp_min(1e-8))
        if case["kind"] != "ug_inspect":
            g = back(torch.autograd.grad(img, leaf, adj)[0])
            total.index_add_(0, idx + first, g)
    out = [torch.cat(t) for t in (images, alphas, depths)]
    if case["kind"] in ("ug_frame", "ug_inspect"):
        out = [t.reshape(case["height"], case["width"]) for t in out]
    if case["kind"] == "ug_inspect":
        return out + [None, None]
    return out + [total[:, :3], total[:, 3:9], total[:, 9], total[:, 10]]


def _rotation(q):
    w, x, y, z = (q / q.norm(dim=1, keepdim=True)).unbind(-1)
    rows = [1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
            2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
            2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)]
    return torch.stack(rows, -1).reshape(-1, 3, 3)


def _exact_gp(case, s):
    """The Gaussian conditioned on the slice by an elevational beam of sigma_z = 1 mm, splatted as
    its 2D marginal inside a box of 3 sqrt(S_ii + |S_01|); the world covariance is R D R, the
    renderer's convention. Scale, quaternion and pose gradients follow published conventions
    that are not derivatives: None."""
    H, W, sp = case["height"], case["width"], s.spacing
    P = s.pose.detach().double()
    A = P[:3, :3] / P[:3, :3].norm(dim=0, keepdim=True)
    eps = 1e-6

    def project(means, scales, quats, opac):
        R = _rotation(quats)
        cov = A.T @ ((R * (scales ** 2)[:, None, :]) @ R) @ A + 1e-6 * torch.eye(3, dtype=torch.float64, device=P.device)
        mu = (means - P[:3, 3]) @ A
        prec = torch.linalg.inv(cov)
        cond = prec.clone()
        cond[:, 2, 2] = cond[:, 2, 2] + 1.0
        Se = torch.linalg.inv(cond)
        m2 = (Se @ (prec @ mu[:, :, None]))[:, :2, 0]
        s00, s11, s01 = Se[:, 0, 0], Se[:, 1, 1], 0.5 * (Se[:, 0, 1] + Se[:, 1, 0])
        det = s00 * s11 - s01 * s01
        w0 = opac * torch.exp(-0.5 * mu[:, 2] ** 2 / (cov[:, 2, 2] + 1.0 + eps)) / (det + eps).sqrt()
        vals = torch.stack([m2[:, 0], m2[:, 1], s11 / det, -s01 / det, s00 / det, w0], 1)
        radii = [3.0 * (v + s01.abs()).detach().clamp_min(1e-12).sqrt() for v in (s00, s11)]
        ok = (torch.linalg.det(cov) > 1e-12) & (torch.linalg.det(cond) > 1e-12) & (det > eps) & (w0 >= 1e-6)
        return vals, radii, ok & torch.isfinite(vals).all(1)

    raw = [p.detach().double() for p in s.params]
    idx = torch.nonzero(project(*raw)[2]).reshape(-1)
    with torch.enable_grad():
        part = [p[idx].requires_grad_(True) for p in raw]
        vals, (rl, ra), _ = project(*part)
    c = vals.detach()
    off = (W - 1) * 0.5
    lo = lambda v: v.ceil().long().clamp_min(0)  # noqa: E731
    box = [lo((c[:, 0] - rl) / sp + off), ((c[:, 0] + rl) / sp + off).floor().long().clamp_max(W - 1),
           lo((c[:, 1] - ra) / sp), ((c[:, 1] + ra) / sp).floor().long().clamp_max(H - 1)]

    def pair(g, x, y):
        dl, da = (x - off) * sp - g[:, 0], y * sp - g[:, 1]
        q = dl * (g[:, 2] * dl + g[:, 3] * da) + da * (g[:, 3] * dl + g[:, 4] * da)
        w = g[:, 5] * torch.exp(-0.5 * q)
        return y * W + x, [w * ((w >= 1e-6) & (q >= 0)).detach()]

    sums, back = _splat(c, lambda: _box_chunks(*box), pair, H * W, 1)
    grads = torch.autograd.grad(vals, [part[0], part[3]], back(s.adjoint.reshape(-1, 1).double()))
    dm, do = (torch.zeros_like(r).index_add_(0, idx, gr) for r, gr in zip((raw[0], raw[3]), grads))
    return [sums.reshape(H, W), dm, None, None, do] + ([None] if case["pose"] else [])


def _exact_sa(case, s):
    """Projection onto the slice, cull at three slice sigmas, additive splat with q <= 9."""
    cam, st = s.camera, s.settings
    H, W, hw, hh = cam.image_height, cam.image_width, cam.half_width_mm, cam.half_height_mm
    mc = st.min_covariance
    with torch.enable_grad():
        means, scales, quats, opac, colors = leaves = [p.detach().double().requires_grad_(True) for p in s.params]
        V = cam.world_view_transform.double()
        r = V[:3, :3]
        c = means @ r + V[3, :3]
        R = _rotation(quats)
        C = r.T @ ((R * (scales ** 2)[:, None, :]) @ R.transpose(1, 2)) @ r
        a, b, d = C[:, 0, 0] + mc, C[:, 0, 1], C[:, 1, 1] + mc
        sig = (C[:, 2, 2].clamp_min(mc) + st.slice_thickness_mm ** 2).sqrt()
        z = c[:, 2] - cam.focal_depth_mm
        keep = (z.abs() <= st.cull_std * sig * st.thickness_scale).detach()
        det = (a * d - b * b).clamp_min(mc)
        w = opac[:, 0] * torch.exp(-0.5 * (z / sig) ** 2) / det.sqrt()
        vals = torch.cat([c[:, :2], torch.stack([d / det, -b / det, a / det, w], 1), colors], 1)
    v = vals.detach()
    inv_det = (v[:, 2] * v[:, 4] - v[:, 3] ** 2).clamp_min(1e-8)
    rx, ry = (3.0 * (v[:, k] / inv_det).clamp_min(1e-8).sqrt() for k in (4, 2))
    kx, ky = (W - 1) / (2 * hw), (H - 1) / (2 * hh)
    idx = torch.nonzero(keep).reshape(-1)
    box = [((v[:, 0] - rx + hw) * kx).floor().long().clamp_min(0)[idx],
           ((v[:, 0] + rx + hw) * kx).ceil().long().clamp_max(W - 1)[idx],
           ((v[:, 1] - ry + hh) * ky).floor().long().clamp_min(0)[idx],
           ((v[:, 1] + ry + hh) * ky).ceil().long().clamp_max(H - 1)[idx]]

    def pair(g, x, y):
        dx, dy = -hw + x / kx - g[:, 0], -hh + y / ky - g[:, 1]
        q = dx * (g[:, 2] * dx + g[:, 3] * dy) + dy * (g[:, 3] * dx + g[:, 4] * dy)
        wt = g[:, 5] * torch.exp(-0.5 * q) * (q.detach() <= st.cull_std ** 2)
        return y * W + x, [wt * g[:, 6], wt * g[:, 7], wt * g[:, 8], wt]

    sums, back = _splat(v[idx], lambda: _box_chunks(*box), pair, H * W, 4)
    adj = torch.zeros_like(sums)
    adj[:, :3] = s.adjoint.double().reshape(3, -1).T
    g = torch.zeros_like(v).index_add_(0, idx, back(adj))
    grads = torch.autograd.grad(vals, leaves, g)
    return [sums[:, :3].T.reshape(3, H, W) + st.bg_color, sums[:, 3].reshape(1, H, W), None, *grads]


def _exact_gs(case, s):
    """Front-to-back compositing of ray-surfel hits per 16 x 16 tile, for the colour and the maps;
    gradients of opacities and degree-0 coefficients. The other gradients follow the published
    rasteriser's conventions (screen-space means, unnormalised quaternions): None."""
    st = s.settings
    H, W = st.image_height, st.image_width
    dev = _device()
    means, _, opac, sh, scales, quats = (p.detach().double() for p in s.params)
    view, proj, cam = st.viewmatrix.double(), st.projmatrix.double(), st.campos.double()
    one = torch.ones((means.shape[0], 1), dtype=torch.float64, device=dev)
    pv = torch.cat([means, one], 1) @ view[:, :3]
    R = _rotation(quats)
    lu, lv, n = R[:, :, 0] * scales[:, :1], R[:, :, 1] * scales[:, 1:], R[:, :, 2]
    n = n @ view[:3, :3]
    cos = -(pv * n).sum(1)
    n = n * torch.where(cos > 0, 1.0, -1.0)[:, None]
    ndc = torch.tensor([[W / 2, 0, 0, (W - 1) / 2], [0, H / 2, 0, (H - 1) / 2], [0, 0, 0, 1.0]], dtype=torch.float64,
                       device=dev)
    M = proj @ ndc.T  # world (4) -> pixel (3)
    zero = torch.zeros_like(one)
    T = torch.stack([torch.cat([lu, zero], 1) @ M, torch.cat([lv, zero], 1) @ M, torch.cat([means, one], 1) @ M], 2)
    Tu, Tv, Tw = T[:, 0], T[:, 1], T[:, 2]
    t = torch.tensor([9.0, 9.0, -1.0], dtype=torch.float64, device=dev)
    f = t / (t * Tw * Tw).sum(1, keepdim=True)
    px, py = (f * Tu * Tw).sum(1), (f * Tv * Tw).sum(1)
    ext = torch.maximum((px * px - (f * Tu * Tu).sum(1)).clamp_min(1e-4).sqrt(),
                        (py * py - (f * Tv * Tv).sum(1)).clamp_min(1e-4).sqrt()).clamp_min(3 * 0.707106)
    rad = ext.ceil()
    valid = (pv[:, 2] > 0.2) & (cos != 0) & torch.isfinite(rad)
    gx, gy = (W + 15) // 16, (H + 15) // 16
    tile = lambda v, hi: torch.nan_to_num(v).div(16).trunc().long().clamp(0, hi)  # noqa: E731
    x0, y0, x1, y1 = tile(px - rad, gx), tile(py - rad, gy), tile(px + rad + 15, gx), tile(py + rad + 15, gy)
    basis = [0.28209479177387814 * sh[:, 0]]
    if case["degree"] > 0:
        d = means - cam
        d = d / d.norm(dim=1, keepdim=True)
        c1 = 0.4886025119029199
        basis += [-c1 * d[:, 1:2] * sh[:, 1], c1 * d[:, 2:3] * sh[:, 2], -c1 * d[:, 0:1] * sh[:, 3]]
    rgb_raw = sum(basis) + 0.5
    rgb = rgb_raw.clamp_min(0.0)
    order = torch.argsort(pv[:, 2].float(), stable=True)
    color = torch.zeros((3, H, W), dtype=torch.float64, device=dev)
    maps = torch.zeros((7, H, W), dtype=torch.float64, device=dev)
    color += st.bg.double()[:, None, None]
    d_op, d_rgb = torch.zeros_like(opac[:, 0]), torch.zeros_like(rgb)
    near, far = 0.2, 100.0
    for ty in range(gy):
        row = order[(valid & (y0 <= ty) & (y1 > ty))[order]]
        for tx in range(gx):
            ids = row[(x0[row] <= tx) & (x1[row] > tx)]
            if ids.numel() == 0:
                continue
            X, Y = torch.meshgrid(torch.arange(16 * tx, min(W, 16 * tx + 16), device=dev),
                                  torch.arange(16 * ty, min(H, 16 * ty + 16), device=dev), indexing="xy")
            fx, fy = X.reshape(-1, 1).double(), Y.reshape(-1, 1).double()
            # chunks of the list, carrying the transmittance and the running sums; a tile whose
            # pixels have all stopped is done
            Tp = torch.ones((fx.shape[0], 1), dtype=torch.float64, device=dev)
            live = torch.ones_like(Tp, dtype=torch.bool)
            rec = []
            for k0 in range(0, ids.numel(), 2048):
                g = ids[k0:k0 + 2048]
                k = fx[..., None] * Tw[g] - Tu[g]
                l = fy[..., None] * Tw[g] - Tv[g]
                p = torch.cross(k, l, dim=2)
                sx, sy = p[..., 0] / p[..., 2], p[..., 1] / p[..., 2]
                rho = torch.minimum(sx * sx + sy * sy, 2 * ((px[g] - fx) ** 2 + (py[g] - fy) ** 2))
                depth = sx * Tw[g][:, 0] + sy * Tw[g][:, 1] + Tw[g][:, 2]
                G = torch.exp(-0.5 * rho)
                al = (opac[g, 0] * G).clamp_max(0.99)
                al = torch.where((p[..., 2] != 0) & (depth >= near) & (al >= 1.0 / 255.0), al, 0.0)
                after = Tp * torch.cumprod(1 - al, 1)
                on = live & (torch.cummin(torch.where(al > 0, after, 1.0), 1)[0] >= 1e-4) & (al > 0)
                before = torch.cat([Tp, after[:, :-1]], 1)
                rec.append((g, torch.where(on, al, 0.0), before, torch.where(on, depth, 1.0), on, G))
                Tp = Tp * torch.prod(1 - rec[-1][1], 1, keepdim=True)
                live = live & ~((al > 0) & ~on).any(1, keepdim=True)
                if not live.any():
                    break
            g = torch.cat([r[0] for r in rec])
            al, before, depth, on, G = (torch.cat([r[j] for r in rec], 1) for j in (1, 2, 3, 4, 5))
            w = al * before
            m = far / (far - near) * (1 - near / depth)
            m1, m2 = torch.cumsum(m * w, 1) - m * w, torch.cumsum(m * m * w, 1) - m * m * w
            Xi, Yi = X.reshape(-1), Y.reshape(-1)
            color[:, Yi, Xi] = (w @ rgb[g]).T + Tp[:, 0] * st.bg.double()[:, None]
            maps[0, Yi, Xi] = (depth * w).sum(1)
            maps[1, Yi, Xi] = 1 - Tp[:, 0]
            maps[2:5, Yi, Xi] = (w @ n[g]).T
            last = torch.where(on & (before > 0.5), torch.arange(g.numel(), device=dev), -1).amax(1)
            maps[5, Yi, Xi] = torch.where(last >= 0, depth.gather(1, last.clamp_min(0)[:, None])[:, 0], 0.0)
            maps[6, Yi, Xi] = ((m * m * (1 - before) + m2 - 2 * m * m1) * w).sum(1)
            # opacity and colour gradients of the sums above
            dc, da = s.adjoint[0].double()[:, Yi, Xi].T, s.adjoint[1].double()[:, Yi, Xi]
            d_rgb.index_add_(0, g, w.T @ dc)
            al_ = al.detach().requires_grad_(True)
            with torch.enable_grad():
                bf = torch.cumprod(torch.cat([torch.ones_like(al_[:, :1]), 1 - al_], 1), 1)
                w_, Tf = al_ * bf[:, :-1], bf[:, -1]
                a1, a2 = torch.cumsum(m * w_, 1) - m * w_, torch.cumsum(m * m * w_, 1) - m * m * w_
                loss = ((w_ @ rgb[g] + Tf[:, None] * st.bg.double()) * dc).sum() + ((depth * w_).sum(1) * da[0]).sum() \
                    + ((1 - Tf) * da[1]).sum() + ((w_ @ n[g]) * da[2:5].T).sum() \
                    + (((m * m * (1 - bf[:, :-1]) + a2 - 2 * m * a1) * w_).sum(1) * da[6]).sum()
            d_al = torch.autograd.grad(loss, al_)[0]
            d_op.index_add_(0, g, (torch.where(on, d_al, 0.0) * G).sum(0))
    d_rgb = torch.where(rgb_raw < 0, 0.0, d_rgb)
    d_sh = [0.28209479177387814 * d_rgb]
    if case["degree"] > 0:
        d_sh += [-c1 * d[:, 1:2] * d_rgb, c1 * d[:, 2:3] * d_rgb, -c1 * d[:, 0:1] * d_rgb]
    return [color, maps, None, None, None, d_op[:, None], torch.stack(d_sh, 1), None, None]


def _exact_ugr(case, s):
    """Per ray: every Gaussian in reach multiplies the transmission of the samples past it by
    tau + (1 - tau) exp(-psi), psi its three-point quadrature over a window of 2 mm around the
    closest point (limits held fixed in the gradient), and echoes at the samples within three
    of its largest scales."""
    if case["gauss"] * case["width"] * case["height"] > 2e10:
        return None
    c = s.cfg
    W, H = c.image_width, c.image_height
    dev = _device()
    means, scales, quats, att, sh = raw = [p.detach().double() for p in s.params]
    torch.cuda.manual_seed(s.seed)
    u = torch.rand(W, device=dev, dtype=torch.float32)
    pert = (torch.asin(2.0 * u - 1.0) / (math.pi / 2.0) * c.ops_max_offset_mm).double()
    o, lat, ele, ax = (t.double() for t in (s.geometry.origin_world, s.geometry.axis_lateral_world,
                                            s.geometry.axis_elevational_world, s.geometry.axis_axial_world))
    d = means - o
    radius = scales.amax(1) * c.k_sigma
    spacing = c.width_mm / W
    centre, rad = d @ lat / spacing + c.lateral_col_offset, radius / spacing
    first, last = (centre - rad).floor(), (centre + rad).ceil()
    ok = (d @ ax + radius >= c.near_mm) & ((d @ ele).abs() <= radius + c.elev_cutoff_margin_mm)
    nodes = torch.tensor([-0.7745966692, 0.0, 0.7745966692], dtype=torch.float64, device=dev)
    weights = torch.tensor([0.5555555556, 0.8888888889, 0.5555555556], dtype=torch.float64, device=dev)
    wr = c.quadrature_window_radius_mm
    image = torch.zeros((H, W), dtype=torch.float64, device=dev)
    grads = [torch.zeros_like(t) for t in raw]
    for x in range(W):
        idx = torch.nonzero(ok & (first <= x) & (last >= x)).reshape(-1)
        if idx.numel() == 0:
            continue
        ro, rd = s.rays[x].double() + ele * pert[x], s.dirs[x].double()
        pix = s.pixels[x].double()
        tp = ((pix - ro) @ rd).clamp_min(0.0)
        adj = s.adjoint[:, x].double()
        adj = torch.where(adj.abs() < 1e-6, 0.0, adj)

        def rays_of(part):
            m, sc, q, a, h = part
            R = _rotation(q)
            dr = sc.detach().amax(1) * c.k_sigma
            tg = ((m - ro) @ rd).detach()
            og = ((ro - m)[:, None, :] @ R)[:, 0] / sc
            dg = (rd @ R) / sc
            tc = (-(og * dg).sum(1) / ((dg * dg).sum(1) + 1e-8)).detach()
            t0 = (tc - wr).clamp_min(0.0)[:, None].expand(-1, H)
            t1 = torch.minimum(tp[None, :], (tc + wr)[:, None])
            half, mid = 0.5 * (t1 - t0), 0.5 * (t1 + t0)
            aa, bb, cc = (og * og).sum(1)[:, None], (og * dg).sum(1)[:, None], (dg * dg).sum(1)[:, None]
            psi = 0.0
            for k in range(3):
                t = half * nodes[k] + mid
                psi = psi + weights[k] * torch.exp(-0.5 * (aa + 2 * bb * t + cc * t * t))
            psi = torch.where(t1 > t0, half * psi, 0.0)
            tau = torch.sigmoid(a)[:, None]
            logt = torch.where(tg[:, None] < tp[None, :], torch.log(tau + (1 - tau) * torch.exp(-psi)), 0.0)
            e = ((pix[None] - m[:, None]) @ R) / sc[:, None]
            wt = torch.exp(-0.5 * (e * e).sum(2)) * ((tg[:, None] - tp[None, :]).abs() <= dr[:, None])
            echo = (h[:, 0] + h[:, 1:] @ rd)[:, None]
            return logt.sum(0), (echo * wt).sum(0), wt.sum(0)

        step = max(1, 4_000_000 // H)
        parts = [idx[k:k + step] for k in range(0, idx.numel(), step)]
        sums = [torch.zeros(H, dtype=torch.float64, device=dev) for _ in range(3)]
        with torch.no_grad():
            for p in parts:
                for acc, v in zip(sums, rays_of([t[p] for t in raw])):
                    acc += v
        leaf = [t.requires_grad_(True) for t in sums]
        with torch.enable_grad():
            img = torch.exp(leaf[0]) * (1 - torch.exp(-leaf[2])) * (leaf[1] / (leaf[2] + 1e-6))
        image[:, x] = img.detach()
        d_sums = torch.autograd.grad(img, leaf, adj)
        for p in parts:
            with torch.enable_grad():
                part = [t[p].requires_grad_(True) for t in raw]
                out = rays_of(part)
            for acc, gpart in zip(grads, torch.autograd.grad(out, part, d_sums)):
                acc.index_add_(0, p, gpart)
    return [image, *grads]


_EXACT = dict(ug_frame=_exact_ug, ug_inspect=_exact_ug, ug_batch=_exact_ug, ug_sweeps=_exact_ug, gp=_exact_gp,
              sa=_exact_sa, gs=_exact_gs, ugr=_exact_ugr)
