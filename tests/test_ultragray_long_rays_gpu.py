"""Rays of as many samples as the searches for an instance's ranges hold in shared memory (4,096), and of more (they
search global memory), against the FP64 oracle. Tolerances as for the shorter rays: image 1e-4, gradients 1e-3
relative L2 (fp32 places a window's end to 2^-18 mm on rays of 42 mm: 2e-6 of a 2 mm window, and a product of
dozens of such factors is good to some 4e-5; the gradients sum the two sides of a mean, one digit less)."""

from __future__ import annotations

import numpy as np
import pytest

from ug_helpers import rel_l2
from ugr_helpers import make_scene, run_b200_ugr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [4095, 4096, 4097, 6001])
@pytest.mark.parametrize("G,W", [(40, 3), (120, 1)])
def test_long_rays_match_oracle(G, W, H, cuda_device):
    from oracle import ultragray_oracle as UO

    scene = make_scene(G, W, H, 80 + W, width_mm=6.0, scale_range=(0.4, 2.0))
    out = run_b200_ugr(scene, cuda_device)
    st = UO.render(scene, "f64")
    assert out["total"] == st["total"]
    assert rel_l2(out["image"], st["image"]) <= 1e-4, rel_l2(out["image"], st["image"])
    g = UO.backward(st, scene["grad_image"])
    for k in ("d_means", "d_scales", "d_quats", "d_attens", "d_sh"):
        assert np.isfinite(out[k]).all()
        assert rel_l2(out[k], g[k]) <= 1e-3, (k, rel_l2(out[k], g[k]))
