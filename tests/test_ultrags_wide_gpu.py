"""Frames with a side beyond 32,768 pixels: surfels near the far end are drawn, and receive gradients, exactly as in a
small frame that shows the same pixels. The homographies are parallel to the image and their entries chosen such
that moving them by 32,768 pixels rounds nowhere (centres and axes whose squares are whole multiples of the
spacing of floats there), so everything is compared bit for bit."""

from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SHIFT, SIDE = 32768, 32


def _scene(tall, shift, n=14):
    rng = np.random.default_rng(3)
    far = rng.choice([0.0, 16.0, 32.0], n)
    axis = rng.choice([8.0, 16.0], (n, 1)) * rng.choice([-1.0, 1.0], (n, 2))
    near, other = rng.uniform(2, 14, n), rng.uniform(-6, 6, (n, 2))
    along = np.concatenate([axis, (far + shift)[:, None]], 1)
    across = np.concatenate([other, near[:, None]], 1)
    rows = (across, along) if tall else (along, across)
    transmat = np.concatenate([*rows, np.tile([0.0, 0.0, 1.0], (n, 1))], 1)
    H, W = (shift + SIDE, 16) if tall else (16, shift + SIDE)
    g = rng.normal(size=(10, SIDE, 16) if tall else (10, 16, SIDE))
    grad = np.zeros((10, H, W))
    grad[:, H - g.shape[1]:, W - g.shape[2]:] = g
    f = lambda a: np.ascontiguousarray(a, dtype=np.float32)  # noqa: E731
    e = f(np.zeros((0,)))
    means = np.stack([np.zeros(n), np.zeros(n), rng.permutation(np.linspace(1, 5, n))], 1)
    return dict(means=f(means), scales=f(np.ones((n, 2))), quats=f(np.ones((n, 4))),
                opacities=f(rng.uniform(0.1, 0.9, (n, 1))), shs=e, colors=f(rng.uniform(0, 1, (n, 3))),
                transmat=f(transmat), viewmatrix=f(np.eye(4)), projmatrix=f(np.eye(4)), campos=f(np.zeros(3)),
                bg=f([0.1, 0.2, 0.3]), grad_color=f(grad[:3]), grad_others=f(grad[3:]), W=W, H=H, tanfovx=1.0,
                tanfovy=1.0, scale_modifier=1.0, sh_degree=0)


@pytest.mark.parametrize("tall", [False, True])
def test_the_far_end_is_drawn(tall, cuda_device):
    from gs_helpers import run_b200_gs

    small, large = (run_b200_gs(_scene(tall, s), cuda_device) for s in (0, SHIFT))
    assert (small["accum"][0] < 0.5).any()
    for k in ("color", "others", "accum", "n_contrib"):
        a, b = small[k], large[k]
        np.testing.assert_array_equal(b[:, b.shape[1] - a.shape[1]:, b.shape[2] - a.shape[2]:], a, err_msg=k)
    for k in ("d_opacity", "d_colors"):
        assert small[k].any()
        np.testing.assert_array_equal(large[k], small[k], err_msg=k)
