"""The forward's corner quads at the sizes from which they are copied: about
33,600 nodes and 122 samples per ray at most, one view of 208 x 160 reads the
field as it is, twelve a copy along x, sixteen a copy per axis. A view's image is
the same bits whichever its launch took.
"""
import numpy as np
import pytest
import torch

from ascent_gb300 import diff as D
from ascent_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(35, 29, 33), (96, 70, 5), (5, 70, 96), (5600, 2, 3), (2, 3, 5600), (33, 32, 31)])
@pytest.mark.parametrize("width", [208, 205])
def test_images_do_not_depend_on_the_launch(dims, width):
    rng = np.random.default_rng(sum(dims))
    field = torch.from_numpy(rng.random(dims, dtype=np.float32)).cuda()
    spacing = [1.0 / (n - 1) * s for n, s in zip(dims[::-1], (1.0, 1.3, 0.8))]
    bounds = np.array([0.0, 1.0, 0.0, 1.3, 0.0, 0.8])
    lut = torch.from_numpy(rng.random((33, 4), dtype=np.float32)).cuda() * 0.3
    sd = S.sample_distance(bounds, 120)
    points = np.array([[90.0 * (i % 4) + 5 * (i // 4), 3 + 45 * (i // 4)] for i in range(16)], np.float32)
    cams = S.cinema_cameras(bounds, points)

    def render(cameras):
        return D.render(field, lut, cameras, (0.0, 0.0, 0.0), spacing, width, 160, sd, (0.0, 1.0)).cpu().numpy()

    alone = np.concatenate([render([c]) for c in cams])
    assert alone[..., 3].max() > 0.5
    assert np.array_equal(alone, np.concatenate([render(cams[:12]), render(cams[12:])]))
    assert np.array_equal(alone, render(cams))
