"""Projected-slice calls with depth keys (sort_by_v): few Gaussians sort their buckets, many order all Gaussians once.
The lists and the image are the same, and a small call makes no more launches than the bucket sort needs."""

from __future__ import annotations

from types import SimpleNamespace

import pytest
import torch

pytestmark = pytest.mark.gpu


def _call(n, pad, H, W, sort_by_v, dev, seed=4):
    from gaussianplie_renderer import GaussianPlieRenderConfig, build_slice_grid_pack
    from gaussianplie_renderer.autograd import _us_focus_params_vector

    from us3d_b200 import _lib, scenes
    from us3d_b200 import gaussianpile as GP

    sp = 40.0 / max(H, W)
    sc = scenes.make_scene(n, seed=seed, cube_mm=40.0, opacity_mu=-1.0)
    far = torch.full((pad, 3), 1e6)
    tail = lambda t: torch.cat([t, t[:1].expand(pad, *t.shape[1:])])  # noqa: E731
    pose = torch.eye(4)
    pose[:3, 3] = torch.tensor([20.0, 0.0, 20.0])
    cfg = GaussianPlieRenderConfig(H=H, W=W, lateral_spacing_mm_per_pix=sp, axial_spacing_mm_per_pix=sp,
                                   axial_near_mm=0.0)
    grid = build_slice_grid_pack(SimpleNamespace(H=H, W=W, delta_lateral_mm=sp, delta_axial_mm=sp, near_mm=0.0,
                                                 center_lateral=True), dev)
    t = [x.to(dev).float().contiguous() for x in (torch.cat([sc.means, far]), tail(sc.scales), tail(sc.quats),
                                                  tail(sc.opacities), torch.ones(n + pad))]
    args = (*t, pose.to(dev).reshape(16), grid, _us_focus_params_vector(cfg, dev), H, W, sp, sp, 0.0, 16, 3.0, sort_by_v)
    GP.forward(*args)  # the capacity is known from here on
    n0 = _lib.call("us3d_launch_count")
    image, b = GP.forward(*args)
    return [image, *GP.export_bins(b)[:3]], _lib.call("us3d_launch_count") - n0


@pytest.mark.parametrize("n", [900, 6000, 65535])
@pytest.mark.parametrize("H,W", [(64, 80), (250, 130)])
def test_small_keyed_calls(n, H, W, cuda_device):
    small, launches = _call(n, 0, H, W, True, cuda_device)
    large, _ = _call(n, 66000, H, W, True, cuda_device)
    assert int((small[1] >= 0).sum()) > n // 2
    for a, b in zip(small, large):
        assert torch.equal(a, b)
    _, plain = _call(n, 0, H, W, False, cuda_device)
    assert launches <= plain + 3  # the sort's four kernels at most in place of the fill's three
