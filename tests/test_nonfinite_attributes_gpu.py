"""A Gaussian with an infinite or NaN amplitude, or an infinite or NaN upstream gradient at one sample, shows only
where it reaches: everything else keeps every bit."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
ODD = [float("inf"), float("-inf"), float("nan")]


def _bits(a, b):
    return np.testing.assert_array_equal(a.cpu().numpy().view(np.int32), b.cpu().numpy().view(np.int32))


def _slice_case(dev, centre, t, opacity):
    """A 32x32 frame (1 mm pixels) of 300 Gaussians and one more, of precision t^4 at `centre`, in the middle of the
    list."""
    from us3d_b200 import ultragauss as UG

    rng = np.random.default_rng(11)
    n, k = 301, 150
    means = np.stack([rng.uniform(-16, 16, n), rng.uniform(0, 32, n), rng.uniform(-0.5, 0.5, n)], 1)
    tril = np.tile([0.9, 0.1, -0.1, 1.0, 0.05, 1.1], (n, 1))
    opac, inten = rng.uniform(0.05, 0.9, n), rng.uniform(0.1, 1.0, n)
    means[k], tril[k], opac[k] = [*centre, 0.0], [t, 0, 0, t, 0, t], opacity
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32)).to(dev)  # noqa: E731
    eye = torch.eye(3)
    spec = UG.SliceSpec(32, 32, 1.0, 1.0, 0.0, 15.5, torch.zeros(3), eye[0], eye[1], eye[2])
    y, x = torch.meshgrid(torch.arange(32.0), torch.arange(32.0), indexing="ij")
    pix = torch.stack([x - 15.5, y, torch.zeros(32, 32)], -1).reshape(-1, 3).to(dev)
    return [f(means), f(tril), f(opac), f(inten)], k, spec, pix


def _slice_render(params, spec, pix, cull, dev):
    from us3d_b200 import ultragauss as UG

    b = UG.bin_gaussians(*params, UG.build_frame_table([spec], dev), 7.815, 1e-4, True,
                         slice_cull_pixels=pix if cull else None)
    img, alp, dep, _ = UG.forward(b, pix, 1e-6, 0.1, want_counts=False)
    return b, img, alp, dep


@pytest.mark.parametrize("value", ODD)
@pytest.mark.parametrize("cull", [False, True])
@pytest.mark.parametrize("opacity", [0.7, 3e-8])  # 3e-8: some of its pairs are left out of the image
def test_slice_intensity_stays_where_it_reaches(value, cull, opacity, cuda_device):
    dev = cuda_device
    params, k, spec, pix = _slice_case(dev, (3.2, 14.3), 0.9, opacity)
    want = _slice_render(params, spec, pix, cull, dev)[1:]
    odd = [p.clone() for p in params]
    odd[3][k] = value
    got = _slice_render(odd, spec, pix, cull, dev)[1:]
    # precision (t^2 + beta)^2 = 0.656: it reaches 3.451 mm
    d = (pix - params[0][k]).double().norm(dim=1)
    out = d > 3.46
    assert 20 < int((~out).sum()) < 60
    for a, b in zip(got, want):
        _bits(a[out], b[out])
    for a, b in zip(got[1:], want[1:]):  # alpha and depth don't depend on it anywhere
        _bits(a, b)


@pytest.mark.parametrize("value", ODD)
@pytest.mark.parametrize("cull", [False, True])
def test_slice_intensity_between_the_pixels(value, cull, cuda_device):
    """It is in the lists (a rectangle is a pixel wide at least) and reaches no pixel centre."""
    from us3d_b200 import ultragauss as UG

    dev = cuda_device
    params, k, spec, pix = _slice_case(dev, (3.0, 14.5), 4.0, 0.7)
    odd = [p.clone() for p in params]
    odd[3][k] = value
    others = torch.arange(params[0].shape[0], device=dev) != k
    up = torch.linspace(-1, 1, pix.shape[0], device=dev)
    res = []
    for p in (params, odd):
        b, img, alp, dep = _slice_render(p, spec, pix, cull, dev)
        grads = UG.backward(b, pix, up, up.flip(0), up, alp, 1e-6, 0.1)
        res.append([img, alp, dep] + [g[others] for g in grads])
    for a, b in zip(*res):
        assert torch.isfinite(a).all()
        _bits(b, a)


def _scanline_case(G, W, H, seed):
    from ugr_helpers import make_scene

    return make_scene(G, W, H, seed, scale_range=(0.3, 0.6), width_mm=4.0)


def _depths(scene):
    """Depth of every Gaussian along the (parallel) scanlines, its echo radius, and the samples' depths."""
    t = (scene["means"].astype(np.float64) - scene["origin"]) @ scene["ax"].astype(np.float64)
    z = (scene["pixels"][0].astype(np.float64) - scene["ray_o"][0]) @ scene["ray_d"][0].astype(np.float64)
    return t, scene["scales"].max(1).astype(np.float64) * scene["k_sigma"], z


@pytest.mark.parametrize("value", ODD)
@pytest.mark.parametrize("G,W,H", [(40, 3, 64), (41, 1, 97), (400, 2, 300)])
def test_scanline_amplitude_stays_where_it_echoes(value, G, W, H, cuda_device):
    from ugr_helpers import run_b200_ugr

    scene = _scanline_case(G, W, H, 5 + G)
    t, radius, z = _depths(scene)
    k = int(np.argmin(np.abs(t - z[H // 2])))
    want = run_b200_ugr(scene, cuda_device, backward=False)
    scene["sh"][k, 0] = value
    got = run_b200_ugr(scene, cuda_device, backward=False)
    out = np.abs(z - t[k]) > radius[k] + 1e-3
    assert want["counts"].min() > 10 and 0 < out.sum() < H
    np.testing.assert_array_equal(got["image"].reshape(H, W)[out].view(np.int32),
                                  want["image"].reshape(H, W)[out].view(np.int32))
    assert not np.array_equal(got["image"], want["image"])


@pytest.mark.parametrize("value", ODD)
@pytest.mark.parametrize("y0", [20, 21])  # either half of a pair of samples
def test_scanline_gradient_stays_with_its_sample(value, y0, cuda_device):
    """Gaussians whose echo begins at the sample after the odd one, and all deeper ones, get the gradients that they
    get when that sample's gradient is zero."""
    from ugr_helpers import run_b200_ugr

    scene = _scanline_case(300, 2, 120, 9)
    t, radius, z = _depths(scene)
    # every other Gaussian from just behind the sample on
    step = z[1] - z[0]
    deep = t - radius > z[y0] + 1e-3
    edge = np.nonzero(deep)[0][:20]
    shift = z[y0] + np.linspace(0.1, 0.9, edge.size) * step - (t - radius)[edge]
    scene["means"][edge] += (shift[:, None] * scene["ax"]).astype(np.float32)
    t, radius, _ = _depths(scene)
    deep = t - radius > z[y0] + 1e-3
    assert ((t - radius)[edge] < z[y0] + step).all() and deep[edge].all() and 100 < deep.sum() < 290
    scene["grad_image"][y0] = 0.0
    want = run_b200_ugr(scene, cuda_device)
    scene["grad_image"][y0] = value
    got = run_b200_ugr(scene, cuda_device)
    for k in ("d_means", "d_scales", "d_quats", "d_attens", "d_sh"):
        assert want[k][edge].any()
        np.testing.assert_array_equal(got[k][deep].view(np.int32), want[k][deep].view(np.int32), err_msg=k)
