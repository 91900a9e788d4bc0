"""The emptiness pass over several domains against the FP64 oracle: LUT sizes
around the 256 threads that tabulate it and at its limits, transfer functions
with hidden ranges at either end and in the middle, both filters, domains of one
brick and of several, one domain without any hidden brick, and a field update
between two renders. A brick wrongly called empty loses its samples' colour.

Bar: that of test_render_gpu.py (2/255 on 99.9% of the pixels, mean error 1e-3).
"""
import numpy as np
import pytest

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S
from ascent_gb300 import workloads as W
from oracle import oracle as O

from conftest import assert_parity

pytestmark = pytest.mark.gpu

SIZES = [2, 3, 255, 256, 257, 1024, 4095, 4096]
HIDDEN = {"low": (0.0, 0.3), "high": (0.6, 1.01), "middle": (0.35, 0.7), "all": (-1.0, 2.0), "none": (2.0, 3.0)}


def domains(rng):
    """A (41, 9, 18)-node grid as three domains, the second of one brick."""
    nodes = (41, 9, 18)
    xs = [np.linspace(0, 1, n) for n in nodes]
    f = W.blob_field(xs, *W.blob_params(rng))
    h = tuple(1.0 / (n - 1) for n in nodes)
    return [(np.ascontiguousarray(f[:, :, a:b + 1]), (a * h[0], 0.0, 0.0), h) for a, b in ((0, 17), (17, 24), (24, 40))], f


@pytest.mark.parametrize("size", SIZES)
@pytest.mark.parametrize("hidden", sorted(HIDDEN))
@pytest.mark.parametrize("filt", [N.LUT_NEAREST, N.LUT_LINEAR])
def test_hidden_ranges(size, hidden, filt):
    rng = np.random.default_rng(size)
    doms, f = domains(rng)
    x = np.linspace(0, 1, size)
    lo, hi = HIDDEN[hidden]
    lut = np.stack([x, 1 - x, 0.5 + 0 * x, np.where((x >= lo) & (x <= hi), 0.0, 0.08)], 1).astype(np.float32)
    b = np.array([0, 1, 0, 1, 0, 1.0])
    cam = S.camera_reset_to_bounds(b)
    S.camera_azimuth(cam, 50)
    S.camera_elevation(cam, 30)
    p = N.make_params(61, 47, S.sample_distance(b, 120), (float(f.min()), float(f.max())), lut, lut_filter=filt)
    osc, osc2 = O.OracleScene(64), O.OracleScene(64)
    with S.Scene(0) as sc:
        for d, o, h in doms:
            sc.add_uniform(d, o, h)
            osc.add_uniform((d.shape[2], d.shape[1], d.shape[0]), o, h, d)
            osc2.add_uniform((d.shape[2], d.shape[1], d.shape[0]), o, h, np.ascontiguousarray(d[::-1]))
        g, _, n = sc.render(cam, p, count_samples=True)
        sc.update_fields(range(3), [np.ascontiguousarray(d[::-1]) for d, _, _ in doms])
        g2, _ = sc.render(cam, p)
    o, _, on = osc.render(cam, p)
    assert_parity(g, o)
    assert abs(n - on) <= 1e-3 * on + 4
    assert_parity(g2, osc2.render(cam, p)[0])
    if hidden == "all":
        assert g.max() == 0.0
