"""A batch whose bricks are mostly empty takes each ray's domains one by one, any
other walks them in one loop: both give the images of the views rendered alone."""
import numpy as np
import pytest
import torch

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("first", [0.0, 0.3, 0.55, 0.99])   # the opaque entries start here
def test_batch_equals_views(first):
    n, rng = 33, np.random.default_rng(8)
    sc = S.Scene(0)
    h = 1.0 / (2 * (n - 1))
    for k in range(8):
        at = [(k >> a & 1) * 0.5 for a in range(3)]
        x, y, z = (at[a] + np.arange(n) * h for a in range(3))
        f = (z[:, None, None] + y[None, :, None] + x[None, None, :]) / 3.0
        sc.add_uniform((f + 0.002 * rng.random(f.shape)).astype(np.float32), tuple(at), (h, h, h))
    u = np.linspace(0, 1, 256)
    lut = np.stack([u, 1 - u, 0.5 + 0 * u, np.where(u >= first, 0.05, 0.0)], 1).astype(np.float32)
    cams = S.cinema_cameras(sc.bounds(), np.array([[20, 30], [100, 60], [-150, 110]], np.float32))
    p = N.make_params(50, 37, S.sample_distance(sc.bounds(), 120), (0.0, 1.0), lut)
    rgba, depth = (t.cpu() for t in sc.render_batch(cams, p, device_out=True)[:2])
    for i, c in enumerate(cams):
        one = sc.render(c, p, device_out=True)
        assert torch.equal(rgba[i], one[0].cpu()) and torch.equal(depth[i], one[1].cpu())
    # the last case hides all but a corner that no sample lies in
    assert (rgba[..., 3].max() > 0.05) == (first < 0.9)
