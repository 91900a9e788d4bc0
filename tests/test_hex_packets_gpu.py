"""The packet width that a hexahedral frame takes until one is set, on both sides
of the tile count at which it changes: the image, depths and sample count are
those of either width that is set.
"""
import numpy as np
import pytest

from ascent_gb300 import scene as S
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height", [(33, 17), (752, 512), (753, 512), (768, 513)])
def test_images_do_not_depend_on_the_width(width, height):
    wl = W.hex_mesh(n_cells=12, width=width, height=height)
    cam, p = V.workload_camera(wl), V.workload_params(wl)
    with S.Scene(0) as sc:
        V.load_workload(sc, wl)
        rgba, depth, count = sc.render(cam, p, count_samples=True)
        assert count > 0 and rgba[..., 3].max() > 0
        for packet in (4, 8):
            sc.set_tuning(packet_w=packet, unroll=1, min_blocks=4)
            a, d, n = sc.render(cam, p, count_samples=True)
            np.testing.assert_array_equal(a, rgba)
            np.testing.assert_array_equal(d, depth)
            assert n == count
