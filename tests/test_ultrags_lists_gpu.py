"""Surfels that are in the tiles' lists but too faint for any pixel (opacity below 1/255) must change nothing, however
they move the others through the 32-entry steps and the batches of the warps' own lists: images, final
transmittances and gradients bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,faint", [(1, 0), (1, 31), (31, 1), (32, 32), (33, 31), (64, 1), (65, 63), (130, 200),
                                     (700, 900)])
@pytest.mark.parametrize("W,H", [(8, 4), (17, 33), (64, 50)])
def test_faint_surfels_change_nothing(n, faint, W, H, cuda_device):
    from gs_helpers import make_scene, run_b200_gs

    scene = make_scene(n + faint, W, H, 100 + n, mode="colors", scale_range=(0.1, 0.6))
    rng = np.random.default_rng(n + faint)
    order = rng.permutation(n + faint)
    keep, pale = np.sort(order[:n]), order[n:]
    scene["opacities"][pale] = rng.uniform(0.0, 0.0039, (faint, 1)).astype(np.float32)
    few = dict(scene)
    for k in ("means", "scales", "quats", "opacities", "colors"):
        few[k] = np.ascontiguousarray(scene[k][keep])
    a, b = run_b200_gs(few, cuda_device), run_b200_gs(scene, cuda_device)
    assert n < 30 or (a["accum"][0] < 0.9).any()
    assert faint < 30 or b["num"] > a["num"] or W * H < 100
    for k in ("color", "others", "accum"):
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)
    np.testing.assert_array_equal(a["n_contrib"] > 0, b["n_contrib"] > 0)
    for k in ("d_means2D", "d_colors", "d_opacity", "d_means3D", "d_transmat", "d_scales", "d_rot"):
        np.testing.assert_array_equal(a[k], b[k][keep], err_msg=k)
        assert not b[k][pale].any(), k
