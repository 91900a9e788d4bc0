"""Where an opaque canvas ends a ray, against the FP64 oracle: canvas depths
swept across the image through the volume, in front of it, behind it, at and
beyond the clip planes, for clip planes that put the volume at very different
image depths, and for vertex, cell-centred and several domains.

Bar: that of test_render_gpu.py (2/255 on 99.9% of the pixels, mean error 1e-3;
for the cell-centred field 99% and 2e-3), with the sample counts within 2e-3.
"""
import numpy as np
import pytest

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W
from oracle import oracle as O

from conftest import assert_parity, image_error

pytestmark = pytest.mark.gpu


def image_depth(cam, dist):
    n, f = float(cam.near_plane), float(cam.far_plane)
    return 0.5 * ((f + n) / (f - n) - 2 * f * n / ((f - n) * dist)) + 0.5


@pytest.mark.parametrize("near,far", [(0.01, 100.0), (1e-4, 1e4), (1.0, 4.0), (2.5, 2.9)])
@pytest.mark.parametrize("kind", ["vertex", "cells", "domains"])
def test_canvas_depths(near, far, kind):
    wl = W.plain_small(n=28, width=96, height=72, samples=90, parts=(2, 1, 2) if kind == "domains" else None)
    cam = V.workload_camera(wl)
    cam.near_plane, cam.far_plane = near, far
    p = V.workload_params(wl, lut=V.workload_renderer(wl).lut(True))
    osc = O.OracleScene(64)
    h, w = wl.height, wl.width
    dist = np.linalg.norm(np.array(cam.position[:]) - 0.5)
    # image depths of distances from in front of the volume to behind it, along x
    depth = np.tile([image_depth(cam, dist + t) for t in np.linspace(-1.2, 1.2, w)], (h, 1)).astype(np.float32)
    for row, d in enumerate((1.0, 0.0, 1.5, -0.5, np.nextafter(np.float32(1), np.float32(0)), 0.5)):
        depth[6 * row] = d
    rgba = np.zeros((h, w, 4), np.float32)
    rgba[..., 1], rgba[..., 3] = 0.25, 1.0
    with S.Scene(0) as sc:
        for d in wl.domains:
            if kind == "cells":
                f = np.ascontiguousarray(d.field[:-1, :-1, :-1])
                sc.add_uniform(f, d.origin, d.spacing, association=N.ASSOC_ELEMENT)
                osc.add_uniform(d.dims, d.origin, d.spacing, f, assoc=N.ASSOC_ELEMENT)
            else:
                sc.add_uniform(d.field, d.origin, d.spacing)
                osc.add_uniform(d.dims, d.origin, d.spacing, d.field)
        g, gd, gn = sc.render_over(cam, p, rgba, depth, count_samples=True)
    o, od, on = osc.render_over(cam, p, rgba, depth)
    if kind == "cells":
        e = image_error(g, o)
        assert e["frac_within_2"] >= 0.99 and e["mae"] <= 2e-3, e
    else:
        assert_parity(g, o)
    assert abs(gn - on) <= 2e-3 * on + 4, (gn, on)
    assert gn > 0
