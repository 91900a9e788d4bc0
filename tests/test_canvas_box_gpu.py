"""An opaque canvas among domains that lie apart, where the box around all of
them, which decides whose rays the canvas can end, is mostly empty: canvas
depths swept from before the first domain to behind the last, rays through one,
through several and past all of them. Against the FP64 oracle at the bar of
test_canvas_end_gpu.py.
"""
import numpy as np
import pytest

from ascent_gb300 import scene as S
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W
from oracle import oracle as O

from conftest import assert_parity
from test_canvas_end_gpu import image_depth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("domains", [1, 2, 5, 40])
@pytest.mark.parametrize("mixed", [False, True])
def test_domains_apart(domains, mixed):
    wl = W.plain_small(n=12, width=96, height=72, samples=300)
    rng = np.random.default_rng(domains)
    cam = V.workload_camera(wl)
    p = V.workload_params(wl, lut=V.workload_renderer(wl).lut(True))
    osc = O.OracleScene(64)
    h, w = wl.height, wl.width
    dist = np.linalg.norm(np.array(cam.position[:]) - 0.5)
    depth = np.tile([image_depth(cam, dist + t) for t in np.linspace(-1.2, 1.2, w)], (h, 1)).astype(np.float32)
    rgba = np.zeros((h, w, 4), np.float32)
    rgba[..., 1], rgba[..., 3] = 0.25, 1.0
    field = wl.domains[0].field
    n = field.shape[0]
    with S.Scene(0) as sc:
        cells = [(x, y, z) for z in range(4) for y in range(4) for x in range(4)]
        for k, c in enumerate(rng.permutation(len(cells))[:domains]):
            # boxes of a tenth in a raster of a quarter
            lo = 0.25 * np.array(cells[c]) + 0.07
            if mixed and k % 2:
                xs = [np.linspace(a, a + 0.1, n) for a in lo]
                sc.add_rectilinear(field, *xs)
                osc.add_rectilinear(*xs, field)
            else:
                sc.add_uniform(field, lo, (0.1 / (n - 1),) * 3)
                osc.add_uniform((n, n, n), lo, (0.1 / (n - 1),) * 3, field)
        g, _, gn = sc.render_over(cam, p, rgba, depth, count_samples=True)
    o, _, on = osc.render_over(cam, p, rgba, depth)
    assert_parity(g, o)
    assert abs(gn - on) <= 2e-3 * on + 4, (gn, on)
    assert gn > 0
