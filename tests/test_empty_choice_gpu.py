"""What a frame does at empty bricks depends on how many there are and on the
step: at each combination, for one domain, several, and a large one beside small
ones, a frame and a batch (whose limits differ) give the same image, and the FP64
oracle's at the bar of test_render_gpu.py with the sample counts within 2e-3.
"""
import numpy as np
import pytest

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S
from oracle import oracle as O

from conftest import assert_parity

pytestmark = pytest.mark.gpu


def field(shape, lo):
    """Rises from 0 to 1 along x over the box, so that a threshold hides that share of it."""
    x = np.linspace(lo[0], lo[1], shape[2])
    return np.broadcast_to(x, shape).astype(np.float32) + 1e-3 * np.sin(np.arange(shape[1]))[None, :, None].astype(np.float32)


def domains(kind):
    if kind == "one":
        return [((65, 49, 57), (0.0, 0.0, 0.0), (1 / 56, 1 / 48, 1 / 64), (0.0, 1.0))]
    if kind == "eight":
        return [((33, 25, 29), (0.5 * i, 0.5 * j, 0.5 * k), (1 / 56, 1 / 48, 1 / 64), (0.5 * i, 0.5 * i + 0.5))
                for k in range(2) for j in range(2) for i in range(2)]
    # the large one first in x, seven slabs of one brick each behind it
    return [((65, 49, 57), (0.0, 0.0, 0.0), (1 / 56, 1 / 48, 1 / 64), (0.0, 1.0))] + \
           [((9, 9, 9), (1.0, j / 7, 0.0), (1 / 8, 1 / 56, 1 / 8), (0.0, 0.2)) for j in range(7)]


@pytest.mark.parametrize("kind", ["one", "eight", "uneven"])
@pytest.mark.parametrize("share", [0.1, 0.35, 0.8, 0.9, 0.97])
@pytest.mark.parametrize("step", [0.5, 1.0, 1.6, 3.0, 6.0])
def test_frames_batches_and_the_oracle(kind, share, step):
    x = np.linspace(0.0, 1.0, 257, dtype=np.float32)
    alpha = np.where(x <= share, 0.0, 1.0 - 0.8 ** step).astype(np.float32)
    lut = np.stack([x, 1 - x, 0.5 + 0 * x, alpha], 1)
    p = N.make_params(60, 44, step / 60, (0.0, 1.0), lut)
    osc = O.OracleScene(64)
    with S.Scene(0) as sc:
        for shape, origin, spacing, span in domains(kind):
            f = field(shape, span)
            sc.add_uniform(f, origin, spacing)
            osc.add_uniform(shape[::-1], origin, spacing, f)
        cam = S.camera_reset_to_bounds(sc.bounds())
        S.camera_azimuth(cam, 200.0)
        S.camera_elevation(cam, 25.0)
        g, gd, gn = sc.render(cam, p, count_samples=True)
        images, depths = sc.render_batch([cam, cam], p)
    assert np.array_equal(images[0], g) and np.array_equal(depths[1], gd)
    o, _, on = osc.render(cam, p)
    assert_parity(g, o)
    assert abs(gn - on) <= 2e-3 * on + 4, (gn, on)
    assert share > 0.9 or o[..., 3].max() > 0.1
