"""The forward render from corner quads: a launch with few samples per node
reads the field as it is, one with more a copy of its corner quads along x, one
with many a copy along the longer edge of each view's packets. The three read
the same corners, so a view's image is the same bits whichever its launch took."""
import numpy as np
import pytest
import torch

from ascent_gb300 import diff as D
from ascent_gb300 import scene as S

pytestmark = pytest.mark.gpu


# dims are (z, y, x); about 33,600 nodes, 128 samples per ray at most: 851
# rays are 3.2 samples per node, four views of them 13, sixteen 52
@pytest.mark.parametrize("dims", [(35, 29, 33), (96, 70, 5), (5, 70, 96), (5600, 2, 3), (2, 3, 5600), (33, 32, 31)])
def test_images_do_not_depend_on_the_launch(dims):
    rng = np.random.default_rng(sum(dims))
    field = torch.from_numpy(rng.random(dims, dtype=np.float32)).cuda()
    spacing = [1.0 / (n - 1) * s for n, s in zip(dims[::-1], (1.0, 1.3, 0.8))]
    bounds = np.array([0.0, 1.0, 0.0, 1.3, 0.0, 0.8])
    lut = torch.from_numpy(rng.random((33, 4), dtype=np.float32)).cuda() * 0.3
    sd = S.sample_distance(bounds, 120)
    points = np.array([[90.0 * (i % 4) + 5 * (i // 4), 3 + 45 * (i // 4)] for i in range(16)], np.float32)
    cams = S.cinema_cameras(bounds, points)

    def render(cameras):
        return D.render(field, lut, cameras, (0.0, 0.0, 0.0), spacing, 37, 23, sd, (0.0, 1.0)).cpu().numpy()

    alone = np.concatenate([render([c]) for c in cams])
    fours = np.concatenate([render(cams[i:i + 4]) for i in range(0, 16, 4)])
    assert alone[..., 3].max() > 0.5
    assert np.array_equal(alone, fours)
    assert np.array_equal(alone, render(cams))
