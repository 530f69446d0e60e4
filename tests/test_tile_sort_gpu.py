"""Order within a tile's list for depth distributions that the distribution sort spreads well, badly (many keys in
a bin: the comparison network takes over) and not at all (equal depths), at the sizes where the path
changes: exact."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _depths(kind, n, rng):
    if kind == "even":
        return rng.permutation(np.linspace(1.0, 14.0, n))
    if kind == "equal":
        return np.full(n, 7.0)
    if kind == "steps":  # five depths
        return rng.choice([1.0, 2.0, 7.5, 7.501, 14.0], n)
    if kind == "outlier":  # all but one within a fiftieth of a bin
        return np.where(np.arange(n) == n // 2, 0.5, 14.0 + 2e-4 * rng.random(n))
    return np.where(rng.random(n) < 0.5, 3.0, rng.uniform(1.0, 14.0, n))  # "half"


@pytest.mark.parametrize("kind", ["even", "equal", "steps", "outlier", "half"])
@pytest.mark.parametrize("n", [1, 64, 65, 300, 1024, 1025, 4096])
def test_order_within_a_tile(kind, n, cuda_device):
    from us3d_b200 import ultragauss as UG

    dev = cuda_device
    rng = np.random.default_rng(n)
    eye = torch.eye(3)
    spec = UG.SliceSpec(16, 16, 1.0, 1.0, 0.0, 7.5, torch.zeros(3), eye[0], eye[1], eye[2])
    means = np.stack([rng.uniform(-3, 3, n), _depths(kind, n, rng), rng.uniform(-0.2, 0.2, n)], 1)
    tril = torch.tensor([1.0, 0.0, 0.0, 1.0, 0.0, 1.0], device=dev).repeat(n, 1)
    t = lambda a: torch.as_tensor(np.asarray(a, np.float32)).to(dev)  # noqa: E731
    for by_depth in (True, False):
        b = UG.bin_gaussians(t(means), tril, t(np.full(n, 0.5)), t(rng.random(n)), UG.build_frame_table([spec], dev),
                             7.815, 1e-4, by_depth)
        keys, vals, rs, re = (x.cpu().numpy() for x in UG.export_bins(b, 0))
        assert rs[0] == 0 and re[0] == n and b.total == n
        np.testing.assert_array_equal(np.sort(vals), np.arange(n))
        np.testing.assert_array_equal(np.lexsort((vals, keys)), np.arange(n))
        depth = keys & 0xFFFFFFFF
        want = ((means[vals, 1].astype(np.float32) + np.float32(500.0)) * np.float32(1000.0)) if by_depth else 0.0 * vals
        assert np.abs(depth - want).max() <= 1.0  # the key's own truncation
