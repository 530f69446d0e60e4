"""Binning calls with more (Gaussian, frame) pairs than their instances alone leave room for: the capacity that the
first call finds out serves all later ones."""

from __future__ import annotations

import pytest
import torch

pytestmark = pytest.mark.gpu


def test_repeated_binning_does_not_retry(cuda_device):
    from us3d_b200 import _lib, scenes
    from us3d_b200 import ultragauss as UG

    dev = cuda_device
    sc = scenes.make_scene(60001, seed=6).to(dev)
    params = [sc.means, sc.precision_tril.contiguous(), sc.opacities, sc.intensities]
    specs, pix = [], []
    for f in scenes.linear_sweep(24, 16, 16, 4.0, seed=6):
        f = f.to(dev)
        specs.append(UG.SliceSpec(16, 16, 4.0, 4.0, 0.25, f.lateral_col_offset, f.origin, f.axis_lat, f.axis_ax,
                                  f.axis_ele))
        pix.append(f.pixels)
    table, pix = UG.build_frame_table(specs, dev), torch.cat(pix).contiguous()
    launches, caps = [], []
    for _ in range(5):
        n0 = _lib.call("us3d_launch_count")
        b = UG.bin_gaussians(*params, table, 7.815, 1e-4, True, slice_cull_pixels=pix)
        launches.append(_lib.call("us3d_launch_count") - n0)
        caps.append(b.capacity)
        assert UG.read_status(b) == (b.total, 0)
    assert b.total * 1.25 + 1024 < caps[-1]  # the pairs ask for more than the instances do
    assert launches[1:] == [min(launches)] * 4 and len(set(caps[1:])) == 1
