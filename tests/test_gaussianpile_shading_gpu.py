"""GaussianPile shading where its loops change form: lists that end within, at and after a staged batch and its
warp-wide tests, images and tiles that end within a pixel block, Gaussians of one class only, and a
weight threshold that is not positive. Against the CPU oracle: images and opacity gradients are sums of a few
hundred products formed in fp32 in another order, which 1e-5 (relative, l2) bounds. The boxes end at eight standard deviations, so that a
test decided the other way by rounding changes nothing either."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from ug_helpers import rel_l2

pytestmark = pytest.mark.gpu


def _case(n, H, W, seed, spread):
    """n overlapping Gaussians around an H x W slice of 0.5 mm pixels (plane y = 0 of the world)."""
    rng = np.random.default_rng(seed)
    f = lambda a: np.ascontiguousarray(a, np.float32)  # noqa: E731
    means = rng.uniform([0.0, -0.6, 0.0], [0.5 * W, 0.6, 0.5 * H], (n, 3))
    quats = np.array([1.0, 0.0, 0.0, 0.0]) + 0.05 * rng.standard_normal((n, 4))
    pose = np.eye(4)[:, [0, 2, 1, 3]]  # lateral = x, axial = z, elevational = y
    pose[0, 3] = 0.25 * (W - 1)
    grid = [0.0, H, W, 0.5, 0.5, 0.0, (W - 1) * 0.5, 1.0] + [0.0] * 8
    params = [1.0, 0.0, 1.0, 1.0, 1.0, 0.0, 0.5, 8.0, 0.5, 1e-12, 1e-12, 0.0, 0.0, 0.0]
    return dict(means=f(means), scales=f(spread * rng.uniform(0.5, 1.5, (n, 3))), quats=f(quats),
                opac=f(rng.uniform(0.1, 0.9, n)), inten=f(rng.uniform(0.2, 1.0, n)), pose=f(pose), grid=f(grid),
                params=f(params), H=H, W=W, grad=f(rng.standard_normal((H, W))))


def _check(c, dev, tile=16):
    from oracle import gaussianpile_oracle as GO
    from us3d_b200 import gaussianpile as GP

    keys = ("means", "scales", "quats", "opac", "inten", "pose", "grid", "params")
    t = [torch.as_tensor(c[k]).to(dev) for k in keys]
    t[5] = t[5].reshape(16)
    img, b = GP.forward(*t, c["H"], c["W"], 0.5, 0.5, 0.0, tile, 8.0, False)
    g = GP.backward(b, torch.as_tensor(c["grad"]).to(dev), True)
    st = GO.render(*(c[k] for k in keys), c["H"], c["W"], 0.5, 0.5, 0.0, tile, 8.0)
    og = GO.backward(st, c["grad"], pose_grad=True)
    assert np.abs(st["image"]).max() > 1e-3
    assert rel_l2(img.cpu().numpy(), st["image"]) <= 1e-5
    assert rel_l2(g[3].cpu().numpy(), og["d_opacity"]) <= 1e-5
    assert rel_l2(g[4].cpu().numpy(), og["d_intensity"]) <= 1e-5
    assert rel_l2(g[0].cpu().numpy(), og["d_means"]) <= 1e-4  # the existing bound for position gradients
    return img


@pytest.mark.parametrize("n", [1, 31, 32, 33, 127, 129, 255, 256, 257, 700])
def test_list_lengths(n, cuda_device):
    _check(_case(n, 16, 16, n, 0.4), cuda_device)


@pytest.mark.parametrize("H,W,tile", [(1, 1, 16), (5, 9, 16), (17, 33, 16), (40, 23, 1), (21, 30, 3), (33, 31, 20),
                                      (70, 65, 32)])
def test_ragged_images_and_tiles(H, W, tile, cuda_device):
    _check(_case(300, H, W, 7 * H + W, 0.3), cuda_device, tile)


def test_one_class_only(cuda_device):
    """Only Gaussians whose index is 5 mod 16 reach the slice: one queue takes whole batches."""
    c = _case(16 * 300, 16, 16, 3, 0.4)
    out = np.arange(16 * 300) % 16 != 5
    c["means"][out, 1] = 500.0
    _check(c, cuda_device)


@pytest.mark.parametrize("weight_min", [0.0, -1.0, 1e-7])
def test_weight_thresholds(weight_min, cuda_device):
    c = _case(200, 24, 40, 11, 0.4)
    c["params"][10] = weight_min
    _check(c, cuda_device)
