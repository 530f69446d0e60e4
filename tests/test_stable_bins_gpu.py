"""Bucket lists filled in element order (small bucket grids) against their definition and against the
per-bucket sort: grids around the limits of one word of a bitmap, of a chunk and of the path
itself, element counts around chunks and radix blocks. Everything here is exact."""

from __future__ import annotations

from types import SimpleNamespace

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _gp_lists(n, H, W, seed, dev, tile=16, sort_by_v=False):
    from gaussianplie_renderer import GaussianPlieRenderConfig, build_slice_grid_pack
    from gaussianplie_renderer.autograd import _us_focus_params_vector

    from us3d_b200 import gaussianpile as GP
    from us3d_b200 import scenes

    sp = 40.0 / max(H, W)
    sc = scenes.make_scene(n, seed=seed, cube_mm=40.0, opacity_mu=-1.0)
    pose = torch.eye(4)
    pose[:3, 3] = torch.tensor([20.0, 0.0, 20.0])
    cfg = GaussianPlieRenderConfig(H=H, W=W, lateral_spacing_mm_per_pix=sp, axial_spacing_mm_per_pix=sp,
                                   axial_near_mm=0.0)
    grid = build_slice_grid_pack(SimpleNamespace(H=H, W=W, delta_lateral_mm=sp, delta_axial_mm=sp, near_mm=0.0,
                                                 center_lateral=True), dev)
    t = [x.to(dev).float().contiguous() for x in (sc.means, sc.scales, sc.quats, sc.opacities, torch.ones(n))]
    image, b = GP.forward(*t, pose.to(dev).reshape(16), grid, _us_focus_params_vector(cfg, dev), H, W, sp, sp, 0.0,
                          tile, 3.0, sort_by_v)
    ids, rs, re, rects = (x.cpu().numpy() for x in GP.export_bins(b))
    return ids, rs, re, rects, image


@pytest.mark.parametrize("n,H,W,tile,seed", [
    (1, 16, 16, 16, 0), (127, 16, 48, 16, 1), (129, 100, 70, 16, 2), (40000, 250, 130, 16, 3), (3000, 64, 64, 2, 4),
    (700, 512, 1024, 16, 5),    # exactly 2048 buckets
    (700, 512, 1040, 16, 6),    # more: the per-bucket sort
])
def test_lists_hold_every_rectangle_in_order(n, H, W, tile, seed, cuda_device):
    ids, rs, re, rects, _ = _gp_lists(n, H, W, seed, cuda_device, tile)
    tx = (W + tile - 1) // tile
    for t in range(rs.size):
        x, y = t % tx, t // tx
        want = np.nonzero((rects[:, 0] <= x) & (x < rects[:, 2]) & (rects[:, 1] <= y) & (y < rects[:, 3]))[0]
        got = ids[rs[t]:re[t]] if rs[t] >= 0 else ids[:0]
        np.testing.assert_array_equal(got, want)


def test_depth_keys_on_a_small_call(cuda_device):
    """Without a minimum count (the projected slice): the same members, in one order for all tiles."""
    a = _gp_lists(900, 64, 80, 7, cuda_device)
    b = _gp_lists(900, 64, 80, 7, cuda_device, sort_by_v=True)
    place = {}
    for t in range(a[1].size):
        la, lb = a[0][a[1][t]:a[2][t]], b[0][b[1][t]:b[2][t]]
        np.testing.assert_array_equal(np.sort(la), np.sort(lb))
        for i, j in zip(lb[:-1], lb[1:]):
            assert (j, i) not in place
            place[(i, j)] = True
    assert any(i > j for i, j in place)  # not the element order
    assert (a[4] - b[4]).abs().max() <= 1e-5 * a[4].abs().max()


@pytest.mark.parametrize("n,pad,W", [(32000, 768, 40), (32000, 1000, 3), (32767, 33000, 130), (20000, 20001, 257)])
def test_scanline_lists_match_the_sort(n, pad, W, cuda_device):
    """Culled Gaussians after the others change nothing but the path."""
    from ugr_helpers import make_scene, run_b200_ugr

    scene = make_scene(n, W, 40, 70 + W)
    big = dict(scene)
    for k, v in dict(means=(0.0, 0.0, -50.0), scales=(1.0, 1.0, 1.0), quats=(1.0, 0.0, 0.0, 0.0), attenuations=0.0,
                     sh=(1.0, 0.0, 0.0, 0.0)).items():
        extra = np.broadcast_to(np.float32(v), (pad,) + scene[k].shape[1:])
        big[k] = np.ascontiguousarray(np.concatenate([scene[k], extra]))
    a, b = run_b200_ugr(scene, cuda_device), run_b200_ugr(big, cuda_device)
    for k in ("counts", "offsets", "indices", "depths", "image"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for k in ("d_means", "d_scales", "d_quats", "d_attens", "d_sh"):
        np.testing.assert_array_equal(a[k], b[k][:n], err_msg=k)
        assert not b[k][n:].any()


def test_surfel_lists_match_the_sort(cuda_device):
    from gs_helpers import make_scene, run_b200_gs

    n, pad = 30000, 5000
    scene = make_scene(n, 150, 90, 8)
    big = dict(scene)
    behind = scene["campos"] - 5.0 * scene["viewmatrix"][:3, 2]  # behind the camera: culled
    for k in ("means", "scales", "quats", "opacities", "shs"):
        extra = np.repeat(scene[k][:1], pad, 0) if k != "means" else np.repeat(behind[None].astype(np.float32), pad, 0)
        big[k] = np.ascontiguousarray(np.concatenate([scene[k], extra]))
    a, b = run_b200_gs(scene, cuda_device), run_b200_gs(big, cuda_device)
    for k in ("point_list", "keys", "ranges", "n_contrib", "color", "others"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    for k in ("d_means3D", "d_opacity", "d_sh", "d_scales", "d_rot"):
        np.testing.assert_array_equal(a[k], b[k][:n], err_msg=k)
