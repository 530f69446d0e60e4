"""UltraGauss shading of one tile against plain torch in 64 bits where its loops change form: list lengths around a
staged batch, a warp-wide step and a round of the backward, lists of one parity only, with and without a depth
gradient, and on frames few and many. The chi-square cut lies where a pair weighs less than 1e-8, so no
rounding of the test shows, and every pixel has weight from many; sums of up to a thousand products in fp32 then agree to 1e-5, and the
gradients, which partly cancel, to 1e-4 (relative, l2)."""

from __future__ import annotations

import numpy as np
import pytest
import torch

from ug_helpers import rel_l2

pytestmark = pytest.mark.gpu
CHI2, BETA = 45.0, 1e-4


def _case(dev, n, seed, parity=None):
    rng = np.random.default_rng(seed)
    total = n if parity is None else 2 * n
    means = np.stack([rng.uniform(-4, 4, total), rng.uniform(0, 8, total), rng.uniform(-0.5, 0.5, total)], 1)
    tril = np.concatenate([rng.uniform(0.8, 1.3, (total, 1)), 0.2 * rng.standard_normal((total, 2)),
                           rng.uniform(0.8, 1.3, (total, 1)), 0.2 * rng.standard_normal((total, 1)),
                           rng.uniform(0.8, 1.3, (total, 1))], 1)
    if parity is not None:
        means[np.arange(total) % 2 != parity, 0] = 900.0
    f = lambda a: torch.as_tensor(np.ascontiguousarray(a, np.float32)).to(dev)  # noqa: E731
    return [f(means), f(tril), f(rng.uniform(0.05, 0.9, total)), f(rng.uniform(0.1, 1.0, total))]


def _exact(params, pix, adj, bg):
    p = [x.double().detach().requires_grad_(True) for x in params]
    m, t, o, c = p
    z = torch.zeros_like(t[:, 0])
    L = torch.stack([t[:, 0] ** 2 + BETA, z, z, t[:, 1], t[:, 3] ** 2 + BETA, z, t[:, 2], t[:, 4],
                     t[:, 5] ** 2 + BETA], 1).reshape(-1, 3, 3)
    v = torch.einsum("gji,pgj->pgi", L, pix.double()[:, None] - m[None])  # L^T d
    a = o * torch.exp(-0.5 * (v ** 2).sum(-1))
    s = a.sum(1)
    out = ((a * c).sum(1) + bg * 0.25) / (s + bg), s + bg, (a * m[:, 2]).sum(1) / s
    loss = sum((x * y.double()).sum() for x, y in zip(out, adj))
    return [x.detach() for x in out], torch.autograd.grad(loss, p)


@pytest.mark.parametrize("n", [31, 33, 127, 129, 255, 256, 257, 511, 513, 1023, 1025])
@pytest.mark.parametrize("depth", [True, False])
def test_one_tile(n, depth, cuda_device):
    _check(_case(cuda_device, n, n), depth, cuda_device)


@pytest.mark.parametrize("parity", [0, 1])
def test_one_parity(parity, cuda_device):
    _check(_case(cuda_device, 300, 7, parity), True, cuda_device)


def test_many_tiles(cuda_device):
    """The same tile in a batch of 2,400 frames (one block per tile): the same bits as alone."""
    _check(_case(cuda_device, 300, 9), True, cuda_device, copies=2400)


def _check(params, depth, dev, copies=1):
    from us3d_b200 import ultragauss as UG

    eye = torch.eye(3)
    spec = UG.SliceSpec(16, 16, 0.5, 0.5, 0.0, 7.5, torch.zeros(3), eye[0], eye[1], eye[2])
    y, x = torch.meshgrid(torch.arange(16.0), torch.arange(16.0), indexing="ij")
    one = torch.stack([(x - 7.5) * 0.5, y * 0.5, torch.zeros(16, 16)], -1).reshape(-1, 3).to(dev)
    bg = 1e-3
    g = torch.Generator().manual_seed(len(params[0]))
    adj = torch.randn(3, 256, generator=g).to(dev)
    if not depth:
        adj[2] = 0.0
    res = []
    for k in sorted({1, copies}):
        pix = one.repeat(k, 1)
        b = UG.bin_gaussians(*params, UG.build_frame_table([spec] * k, dev), CHI2, BETA, True, slice_cull_pixels=pix)
        img, alp, dep, _ = UG.forward(b, pix, bg, 0.25, want_counts=False)
        full = torch.zeros((3, 256 * k), device=dev)
        full[:, -256:] = adj
        grads = UG.backward(b, pix, *(a.contiguous() for a in full), alp, bg, 0.25)
        res.append(([x[-256:] for x in (img, alp, dep)], grads))
    out, grads = _exact(params, one, adj, bg)
    for a, e in zip(res[0][0], out):
        assert rel_l2(a.cpu().numpy(), e.cpu().numpy()) <= 1e-5
    for a, e in zip(res[0][1], grads):
        assert rel_l2(a.cpu().numpy(), e.cpu().numpy()) <= 1e-4
    for a, b in zip(res[0][0] + list(res[0][1]), res[-1][0] + list(res[-1][1])):
        assert torch.equal(a, b)
