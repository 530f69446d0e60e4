"""The slice-adapted renderer's grey output as one node against the colour output followed by the same tensor
operations: images and gradients bit for bit, for every option, any combination of outputs used, and NaN."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def _inputs(dev, n, seed, nan=False):
    g = torch.Generator().manual_seed(seed)
    r = lambda *s: torch.rand(s, generator=g)  # noqa: E731
    means = (r(n, 3) - 0.5) * torch.tensor([20.0, 16.0, 1.5])
    quats = torch.tensor([1.0, 0.0, 0.0, 0.0]) + 0.3 * torch.randn(n, 4, generator=g)
    colors = 2.5 * r(n, 3) - 0.4
    if nan:
        colors[n // 2] = float("nan")
    t = [means, 0.4 + r(n, 3), quats, r(n), colors]
    return [x.to(dev).requires_grad_(True) for x in t]


def _render(t, gray, H, W, **options):
    from slice_adapted_3dgs_renderer import render_slice_adapted_3dgs
    from slice_adapted_3dgs_renderer.fused import (SliceAdapted3DGSInput, SliceAdaptedRenderSettings,
                                                   SliceCameraInput)

    cam = SliceCameraInput(H, W, 10.0, 8.0, 0.0, torch.eye(4, device=t[0].device))
    out = render_slice_adapted_3dgs(SliceAdapted3DGSInput(*t), cam,
                                    SliceAdaptedRenderSettings(output_grayscale=gray, **options))
    image = out.image
    if not gray:
        image = (0.299 * image[0] + 0.587 * image[1] + 0.114 * image[2]).unsqueeze(0)
    return image, out.extras["alpha_image"], out.extras["visibility_filter"]


@pytest.mark.parametrize("clamp,bg", [(True, 0.0), (True, 0.05), (True, -0.3), (False, 0.2), (True, 1.2)])
@pytest.mark.parametrize("H,W,use", [(1, 1, "image"), (16, 16, "both"), (37, 70, "image"), (64, 51, "alpha")])
def test_grey_output(clamp, bg, H, W, use, cuda_device):
    res = []
    for gray in (True, False):
        t = _inputs(cuda_device, 400, 5)
        image, alpha, keep = _render(t, gray, H, W, clamp_output=clamp, bg_color=bg)
        assert image.shape == (1, H, W) and alpha.shape == (1, H, W) and keep.dtype == torch.bool
        w = torch.linspace(-1.0, 2.0, H * W, device=cuda_device).reshape(1, H, W)
        loss = 0.0
        if use != "alpha":
            loss = loss + (image * w).sum()
        if use != "image":
            loss = loss + (alpha * w.flip(1)).sum()
        grads = torch.autograd.grad(loss, t, allow_unused=True)
        res.append([image.detach(), alpha.detach(), keep, *grads])
    for a, b in zip(*res):
        assert (a is None and b is None) or torch.equal(a if a is not None else torch.zeros_like(b), b)


def test_grey_output_with_nan(cuda_device):
    a, b = (_render(_inputs(cuda_device, 200, 6, nan=True), gray, 20, 24)[0].detach() for gray in (True, False))
    assert torch.isnan(b).any() and torch.equal(torch.isnan(a), torch.isnan(b))
    assert torch.equal(a.nan_to_num(), b.nan_to_num())


def test_nothing_in_the_slice(cuda_device):
    t = _inputs(cuda_device, 50, 7)
    with torch.no_grad():
        t[0][:, 2] += 500.0
    from slice_adapted_3dgs_renderer import render_slice_adapted_3dgs
    from slice_adapted_3dgs_renderer.fused import (SliceAdapted3DGSInput, SliceAdaptedRenderSettings,
                                                   SliceCameraInput)

    cam = SliceCameraInput(9, 10, 10.0, 8.0, 0.0, torch.eye(4, device=cuda_device))
    out = render_slice_adapted_3dgs(SliceAdapted3DGSInput(*t), cam, SliceAdaptedRenderSettings(bg_color=0.25))
    assert out.extras["alpha_image"] is None and not out.extras["visibility_filter"].any()
    assert torch.allclose(out.image, torch.full((1, 9, 10), 0.25, device=cuda_device)) and not out.image.requires_grad
