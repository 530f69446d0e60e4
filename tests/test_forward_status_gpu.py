"""Calls that bin and shade before the host has read the instance total: their results are those of the separate
calls, a too small capacity is noticed and retried, absent gradients count as zeros, threads and
streams don't share status words, and a captured stream is refused as before. All exact."""

from __future__ import annotations

import threading

import pytest
import torch

pytestmark = pytest.mark.gpu


def _params(dev, n, seed):
    from us3d_b200 import scenes

    sc = scenes.make_scene(n, seed=seed).to(dev)
    return [sc.means, sc.precision_tril.contiguous(), sc.opacities, sc.intensities]


def _specs(dev, n, H, W, s, seed):
    from us3d_b200 import scenes
    from us3d_b200 import ultragauss as UG

    out = []
    for f in scenes.linear_sweep(n, H, W, s, seed=seed):
        f = f.to(dev)
        out.append((UG.SliceSpec(H, W, s, s, 0.25, f.lateral_col_offset, f.origin, f.axis_lat, f.axis_ax, f.axis_ele),
                    f.pixels.contiguous()))
    return out


@pytest.mark.parametrize("H,W", [(1, 1), (16, 17), (33, 250)])
def test_one_frame_table(H, W, cuda_device):
    from us3d_b200 import ultragauss as UG

    spec = _specs(cuda_device, 1, H, W, 0.4, 3)[0][0]
    assert UG._on_device(spec, cuda_device)
    a = UG.build_frame_table([spec], cuda_device)
    host = UG.SliceSpec(*[x.cpu() if isinstance(x, torch.Tensor) else x for x in vars(spec).values()])
    b = UG.build_frame_table([host], cuda_device)
    assert torch.equal(a.table.view(torch.int32), b.table.view(torch.int32))
    a.table = b.table = None
    assert a == b


@pytest.mark.parametrize("cull,capacity", [(True, None), (False, None), (True, 0), (False, 4096)])
def test_bin_forward_matches_separate_calls(cull, capacity, cuda_device):
    from us3d_b200 import ultragauss as UG

    params = _params(cuda_device, 20000, 5)
    frames = _specs(cuda_device, 2, 100, 130, 0.5, 5)
    table = UG.build_frame_table([s for s, _ in frames], cuda_device)
    pix = torch.cat([p for _, p in frames])
    b0 = UG.bin_gaussians(*params, table, 7.815, 1e-4, True, slice_cull_pixels=pix if cull else None)
    want = UG.forward(b0, pix, 1e-6, 0.1)
    b, *got = UG.bin_forward(*params, table, 7.815, 1e-4, True, pix, 1e-6, 0.1, cull, True, capacity=capacity)
    assert b.total == b0.total and b.capacity >= b.total and (capacity is None or b.capacity > capacity)
    for x, y in zip(got, want):
        assert (x is None and y is None) or torch.equal(x, y)
    g = torch.linspace(-1, 1, pix.shape[0], device=cuda_device)
    zero = torch.zeros_like(g)
    a = UG.backward(b, pix, g, None, None, got[1], 1e-6, 0.1, absent_zero=True)
    z = UG.backward(b0, pix, g, zero, zero, want[1], 1e-6, 0.1)
    for x, y in zip(a, z):
        assert torch.equal(x, y)
    with pytest.raises(ValueError):
        UG.backward(b, pix, g, None, None, got[1], 1e-6, 0.1)


def test_many_small_frames_bin_once_when_repeated(cuda_device):
    """More (Gaussian, frame) pairs than the instance total alone leaves room for."""
    from us3d_b200 import _lib
    from us3d_b200.batch import UltraGaussBatchRenderer

    params = _params(cuda_device, 60000, 6)
    frames = _specs(cuda_device, 24, 16, 16, 4.0, 6)
    r = UltraGaussBatchRenderer([s for s, _ in frames], cuda_device)
    pix = torch.cat([p for _, p in frames])
    r(*params, pix)
    n0 = _lib.call("us3d_launch_count")
    r(*params, pix)
    n1 = _lib.call("us3d_launch_count")
    r(*params, pix)
    assert _lib.call("us3d_launch_count") - n1 == n1 - n0 <= 25


def test_threads_and_streams(cuda_device):
    from us3d_b200.batch import UltraGaussBatchRenderer

    jobs = []
    for i in range(4):
        params = _params(cuda_device, 3000 * (i + 1), 20 + i)
        frames = _specs(cuda_device, i + 1, 40, 50 + i, 0.9, 20 + i)
        r = UltraGaussBatchRenderer([s for s, _ in frames], cuda_device)
        pix = torch.cat([p for _, p in frames])
        jobs.append((r, params, pix, [x.clone() for x in r(*params, pix)]))
    torch.cuda.synchronize()
    bad = []

    def work(i):
        r, params, pix, want = jobs[i]
        with torch.cuda.stream(torch.cuda.Stream(cuda_device)):
            for _ in range(20):
                out = r(*params, pix)
                torch.cuda.current_stream().synchronize()
                if not all(torch.equal(a, b) for a, b in zip(out, want)):
                    bad.append(i)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad


def test_refused_while_captured(cuda_device):
    from us3d_b200.batch import UltraGaussBatchRenderer

    params = _params(cuda_device, 2000, 9)
    spec, pix = _specs(cuda_device, 1, 32, 32, 1.0, 9)[0]
    r = UltraGaussBatchRenderer([spec], cuda_device)
    want = r(*params, pix)
    torch.cuda.synchronize()
    with pytest.raises(RuntimeError):
        with torch.cuda.graph(torch.cuda.CUDAGraph()):
            r(*params, pix)
    torch.cuda.synchronize()
    for a, b in zip(r(*params, pix), want):
        assert torch.equal(a, b)
