"""The slice-adapted 3DGS frame render with the projection fused on the GPU.

``render_slice_adapted_3dgs(gaussians, camera, settings)`` has the signature, inputs and
outputs of the reference adapter baselines/slice_adapted_3dgs/render.py:60-129 (any objects
with the fields of its dataclasses are accepted; the same dataclasses are defined here).
The reference projects the 3D Gaussians with about thirty PyTorch operations and boolean-mask
gathers; here one library call projects, culls and compacts them in index order and one
computes the projection's vector-Jacobian product, around the bounded splat. Gradients reach
means, scales_3d, quats, opacities and colors (not the view transform).
"""

from dataclasses import dataclass, field
from typing import Dict, Optional

import torch

from us3d_b200 import slice_adapted as _sa

from .api import _check_bounded_inputs


@dataclass
class SliceCameraInput:
    image_height: int
    image_width: int
    half_width_mm: float
    half_height_mm: float
    focal_depth_mm: float
    world_view_transform: torch.Tensor


@dataclass
class SliceAdapted3DGSInput:
    means: torch.Tensor
    scales_3d: torch.Tensor
    quats: torch.Tensor
    opacities: torch.Tensor
    colors: torch.Tensor


@dataclass
class SliceAdaptedRenderSettings:
    slice_thickness_mm: float = 0.3
    cull_std: float = 3.0
    thickness_scale: float = 1.0
    min_covariance: float = 1.0e-4
    normalize_by_footprint: bool = True
    clamp_output: bool = True
    bg_color: float = 0.0
    output_grayscale: bool = True


@dataclass
class RenderOutput:
    image: torch.Tensor
    depth: Optional[torch.Tensor] = None
    extras: Dict[str, torch.Tensor] = field(default_factory=dict)


class _SliceRender(torch.autograd.Function):
    """Image and alpha image (H*W, 1) of the Gaussians whose projection ``projected`` holds, as one node: the bounded
    splat with the background added (H*W, 3), or the grey image (H*W,) with the clamp applied."""

    @staticmethod
    def forward(ctx, means, scales, quats, opacities, colors, inputs, projected, settings, frame):
        H, W, half_w, half_h, sigma, bg, gray, clamp = frame
        m2, inv, w, colk, idx = projected
        _check_bounded_inputs(H, W, half_w, half_h, m2, inv, w, colk, sigma)
        image, alpha, b = _sa.bounded_forward(H, W, half_w, half_h, m2, inv, w, colk, sigma)
        ctx.set_materialize_grads(False)
        ctx.b, ctx.settings, ctx.frame, ctx.opacity_shape = b, settings, frame, opacities.shape
        if gray:
            ctx.save_for_backward(*inputs, idx, m2, inv, w, colk, image)
            return _sa.finish(image, bg, clamp), alpha
        ctx.save_for_backward(*inputs, idx, m2, inv, w, colk)
        return image.add_(bg), alpha

    @staticmethod
    def backward(ctx, d_out, d_alpha):
        m, s, q, o, v, idx, m2, inv, w, colk, *image = ctx.saved_tensors
        H, W, half_w, half_h, sigma, bg, gray, clamp = ctx.frame
        if d_out is None:
            d_out = torch.zeros((H * W, 3), device=m.device)
        elif gray:
            d_out = _sa.finish_backward(image[0], bg, clamp, d_out.contiguous())
        g = _sa.bounded_backward(ctx.b, half_w, half_h, m2, inv, w, colk, d_out, d_alpha, sigma, absent_zero=True)
        dm, ds, dq, dop, dc = _sa.project_backward(idx, m, s, q, o, v, ctx.settings, *g)
        return dm, ds, dq, dop.reshape(ctx.opacity_shape), dc, None, None, None, None


def _finalize(image, alpha, keep, settings):
    if settings.output_grayscale:
        image = (0.299 * image[0] + 0.587 * image[1] + 0.114 * image[2]).unsqueeze(0)
    return RenderOutput(image=image, depth=None, extras={"visibility_filter": keep, "alpha_image": alpha})


def render_slice_adapted_3dgs(gaussians, camera, settings) -> RenderOutput:
    device = gaussians.means.device
    if device.type != "cuda" or gaussians.means.dtype != torch.float32:
        raise RuntimeError("This simplified delivery renderer expects CUDA float32 tensors for additive_splat_bounded.")
    view = camera.world_view_transform.to(device=device, dtype=gaussians.means.dtype)
    ps = _sa.ProjectionSettings(focal_depth=float(camera.focal_depth_mm),
                                slice_thickness=float(settings.slice_thickness_mm), cull_std=float(settings.cull_std),
                                thickness_scale=float(settings.thickness_scale),
                                min_covariance=float(settings.min_covariance),
                                normalize_by_footprint=bool(settings.normalize_by_footprint))
    c = lambda t: t.detach().to(dtype=torch.float32).contiguous()  # noqa: E731
    inputs = (c(gaussians.means), c(gaussians.scales_3d), c(gaussians.quats), c(gaussians.opacities).reshape(-1),
              c(view))
    *projected, keep = _sa.project(*inputs[:4], c(gaussians.colors), inputs[4], ps)
    H, W = int(camera.image_height), int(camera.image_width)
    if projected[0].shape[0] == 0:
        image = torch.full((3, H, W), float(settings.bg_color), device=device, dtype=gaussians.means.dtype)
        return _finalize(image, None, keep, settings)
    gray, clamp = bool(settings.output_grayscale), bool(settings.clamp_output)
    frame = (H, W, float(camera.half_width_mm), float(camera.half_height_mm), float(settings.cull_std),
             float(settings.bg_color), gray, clamp)
    image, alpha = _SliceRender.apply(gaussians.means, gaussians.scales_3d, gaussians.quats, gaussians.opacities,
                                      gaussians.colors, inputs, projected, ps, frame)
    if gray:
        image = image.view(1, H, W)
    else:
        if clamp:
            image = image.clamp(0.0, 1.0)
        image = image.transpose(0, 1).reshape(3, H, W)
    return RenderOutput(image=image, depth=None,
                        extras={"visibility_filter": keep, "alpha_image": alpha.view(1, H, W)})
