"""The checkpointed scanline kernels at the edges of their tiles against the C oracle: ray lists
around a chunk of 128 instances and odd counts (pairs of instances), sample counts around a tile
of 32 and odd ones (pairs of samples), echo ranges longer than the samples a block stages, and
transmittance that is used up before the ray ends.

Tolerances: image 1e-4 and gradients 1e-3 relative L2 against the FP64 oracle. A ray's depths
reach 42 mm, so fp32 places a window's end to 2^-18 mm: 2e-6 of a 2 mm window, and a product of up
to a few hundred such factors is good to some 4e-5; gradients divide by single factors and sum the
two sides of a mean, one digit less."""

from __future__ import annotations

import numpy as np
import pytest

from ug_helpers import rel_l2
from ugr_helpers import make_scene, run_b200_ugr

pytestmark = pytest.mark.gpu

CASES = [
    # G, W, H, seed, make_scene arguments, attenuation logit (None: the scene's)
    (3, 1, 1, 60, dict(scale_range=(6.0, 9.0)), None),
    (127, 3, 33, 61, dict(scale_range=(1.5, 3.0), width_mm=4.0), None),
    (128, 2, 32, 62, dict(scale_range=(1.5, 3.0), width_mm=4.0), None),
    (129, 2, 31, 63, dict(scale_range=(1.5, 3.0), width_mm=4.0, tilted=True), None),
    (400, 5, 97, 64, dict(scale_range=(0.2, 1.0)), None),
    (60, 2, 1501, 65, dict(scale_range=(4.0, 6.0), elev_mm=4.0), 2.0),  # echo ranges of ~1,200 samples
    (900, 4, 200, 66, dict(scale_range=(0.5, 1.5)), -9.0),              # transmittance underflows
]


@pytest.mark.parametrize("G,W,H,seed,kw,logit", CASES)
def test_checkpointed_kernels_match_oracle(G, W, H, seed, kw, logit, cuda_device):
    from oracle import ultragray_oracle as UO

    scene = make_scene(G, W, H, seed, **kw)
    if logit is not None:
        scene["attenuations"] = np.full(G, logit, np.float32)
    out = run_b200_ugr(scene, cuda_device)
    st = UO.render(scene, "f64")
    assert out["total"] == st["total"]
    if G in (127, 128, 129):
        assert (out["counts"] == G).all()  # every ray lists every Gaussian
    assert rel_l2(out["image"], st["image"]) <= 1e-4, rel_l2(out["image"], st["image"])
    g = UO.backward(st, scene["grad_image"])
    for k in ("d_means", "d_scales", "d_quats", "d_attens", "d_sh"):
        assert np.isfinite(out[k]).all()
        assert rel_l2(out[k], g[k]) <= 1e-3, (k, rel_l2(out[k], g[k]))
