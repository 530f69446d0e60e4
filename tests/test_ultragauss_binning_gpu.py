"""UltraGauss binning at the sizes where its scans and its frame masks change form: Gaussian counts around
one block's scan, around the largest scan of two launches and beyond, and more frames than a mask word holds.
Gaussians that reach no frame must change nothing (the others keep the parity of their index: a pixel sums
its Gaussians of even and of odd index apart), and a batch must give its frames' own results:
everything here is exact."""

from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _scene(dev, n, seed):
    from us3d_b200 import scenes

    sc = scenes.make_scene(n, seed=seed).to(dev)
    return [sc.means, sc.precision_tril.contiguous(), sc.opacities, sc.intensities]


def _frames(n, H, W, s, seed):
    from us3d_b200 import scenes
    from us3d_b200 import ultragauss as UG

    sweep = scenes.linear_sweep(n, H, W, s, seed=seed)
    return [(UG.SliceSpec(H, W, s, s, 0.0, f.lateral_col_offset, f.origin, f.axis_lat, f.axis_ax, f.axis_ele),
             f.pixels) for f in sweep]


def _render(params, frames, dev, cull):
    from us3d_b200 import ultragauss as UG

    pix = torch.cat([p for _, p in frames]).to(dev)
    table = UG.build_frame_table([s for s, _ in frames], dev)
    b = UG.bin_gaussians(*params, table, 7.815, 1e-4, True, slice_cull_pixels=pix if cull else None)
    img, alp, dep, _ = UG.forward(b, pix, 1e-6, 0.0, want_counts=not cull)
    g = torch.linspace(-1.0, 1.0, 3 * pix.shape[0], device=dev).reshape(3, -1)
    grads = UG.backward(b, pix, g[0].contiguous(), g[1].contiguous(), g[2].contiguous(), alp, 1e-6, 0.0)
    return (img, alp, dep), grads


@pytest.mark.parametrize("n,total", [(4096, 4096), (4094, 4097), (5000, 16383), (5000, 16384), (5000, 16385),
                                     (9000, 4096 * 1024), (9000, 4096 * 1024 + 1)])
def test_gaussians_out_of_reach_change_nothing(n, total, cuda_device):
    params = _scene(cuda_device, n, 11)
    frames = _frames(2, 70, 90, 0.7, 11)
    pairs = np.sort(np.random.default_rng(total).choice(total // 2, n // 2, replace=False))
    place = torch.as_tensor(np.stack([2 * pairs, 2 * pairs + 1], 1).reshape(-1)).to(cuda_device)
    many = []
    for p, far in zip(params, (1e4, 1.0, 0.5, 0.5)):
        x = torch.full((total,) + p.shape[1:], far, device=cuda_device)
        x[place] = p
        many.append(x)
    for cull in (False, True):
        out, grads = _render(params, frames, cuda_device, cull)
        out2, grads2 = _render(many, frames, cuda_device, cull)
        assert (out[1] > 1e-3).any()
        for a, b in zip(out, out2):
            assert torch.equal(a, b)
        for a, b in zip(grads, grads2):
            assert torch.equal(a, b[place]) and torch.count_nonzero(b) == torch.count_nonzero(a)


@pytest.mark.parametrize("n_frames", [31, 32, 33, 70])
def test_more_frames_than_a_mask_word(n_frames, cuda_device):
    params = _scene(cuda_device, 3000, 12)
    frames = _frames(n_frames, 40, 33, 1.3, 12)
    for cull in (False, True):
        out, grads = _render(params, frames, cuda_device, cull)
        off = 0
        for f in frames:
            one, _ = _render(params, [f], cuda_device, cull)
            m = one[0].shape[0]
            for a, b in zip(out, one):
                assert torch.equal(a[off:off + m], b)
            off += m
        assert all(torch.isfinite(g).all() for g in grads)


@pytest.mark.parametrize("use", [12, 20, 27])
def test_gradients_do_not_depend_on_the_blocks_per_tile(use, cuda_device):
    """Forty frames (2,560 tiles, one block each in the backward) with an adjoint on one of them against that
    frame alone (64 tiles, four blocks each): the same bits."""
    from us3d_b200 import ultragauss as UG

    params = _scene(cuda_device, 6000, 13)
    frames = _frames(40, 128, 128, 0.5, 13)
    grads = []
    for sel in (frames, frames[use:use + 1]):
        pix = torch.cat([p for _, p in sel]).to(cuda_device)
        b = UG.bin_gaussians(*params, UG.build_frame_table([s for s, _ in sel], cuda_device), 7.815, 1e-4, True,
                             slice_cull_pixels=pix)
        assert (b.frames.n_tiles < 4 * 4 * 148) == (len(sel) == 1)
        alpha = UG.forward(b, pix, 1e-6, 0.0, want_counts=False)[1]
        g = torch.zeros((2, pix.shape[0]), device=cuda_device)
        at = use * 128 * 128 if len(sel) > 1 else 0
        g[:, at:at + 128 * 128] = torch.linspace(-1.0, 1.0, 2 * 128 * 128, device=cuda_device).reshape(2, -1)
        zero = torch.zeros_like(g[0])
        grads.append(UG.backward(b, pix, g[0].contiguous(), g[1].contiguous(), zero, alpha, 1e-6, 0.0))
    for a, b in zip(*grads):
        assert torch.count_nonzero(b) > 0 and torch.equal(a, b)
