"""Rectilinear and cell-centred domains against the FP64 oracle where their
march can go wrong: grids of one cell and of one node more or less than a
brick, cells whose widths differ by orders of magnitude, steps over many cells
and many steps in a cell, rays along either direction of every axis, the camera
inside the grid, and transfer functions that leave whole bricks empty.

Bars: for vertex fields the one of test_render_gpu.py (2/255 on 99.9% of the
pixels, mean error 1e-3); for cell-centred fields, whose values jump at the
cells' faces, where FP32 and FP64 positions fall on different sides, 99% and
2e-3, as there.
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

NODES = [(2, 2, 2), (3, 9, 10), (8, 17, 18), (33, 25, 40)]
VIEWS = [(40.0, 25.0, False), (-130.0, -50.0, False), (75.0, 10.0, True)]


def axes_of(nodes, rng, spread):
    out = []
    for n in nodes:
        w = np.exp(rng.uniform(-spread, spread, n - 1))
        x = np.concatenate([[0.0], np.cumsum(w)]).astype(np.float32).astype(np.float64)
        out.append(x / x[-1])
    return out


def case(nodes, view, hidden, samples, assoc, rng, spread):
    xs = axes_of(nodes, rng, spread)
    at = xs if assoc == N.ASSOC_VERTEX else [0.5 * (x[1:] + x[:-1]) for x in xs]
    f = W.blob_field(at, *W.blob_params(rng))
    vr = V.VolumeRenderer()
    rp, rgb, ap, al = W.linear_ramp_tf(alpha_max=0.6)
    if hidden:
        ap, al = np.array([0.0, 0.45, 1.0]), np.array([0.0, 0.0, 0.8])
    vr.set_color_table(V.TransferFunction(rp, rgb, ap, al))
    vr.set_num_samples(samples)
    b = np.array([0, 1, 0, 1, 0, 1.0])
    cam = S.camera_reset_to_bounds(b)
    az, el, inside = view
    S.camera_azimuth(cam, az)
    S.camera_elevation(cam, el)
    if inside:
        for a in range(3):
            cam.position[a] = 0.5 + 0.1 * (cam.position[a] - 0.5)
        cam.fov_y = 70.0
    p = N.make_params(67, 53, S.sample_distance(b, samples), (float(f.min()), float(f.max())), vr.lut(True))
    return xs, f, cam, p


def check(g, gn, o, on, assoc):
    if assoc == N.ASSOC_VERTEX:
        assert_parity(g, o)
    else:
        e = image_error(g, o)
        assert e["frac_within_2"] >= 0.99 and e["mae"] <= 2e-3, e
    assert abs(gn - on) <= 2e-3 * on + 4, (gn, on)


@pytest.mark.parametrize("nodes", NODES)
@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("assoc", [N.ASSOC_VERTEX, N.ASSOC_ELEMENT])
@pytest.mark.parametrize("hidden,samples", [(False, 30), (True, 400)])
def test_rectilinear(nodes, view, assoc, hidden, samples):
    rng = np.random.default_rng(sum(nodes) + samples)
    xs, f, cam, p = case(nodes, view, hidden, samples, assoc, rng, 1.5)
    with S.Scene(0) as sc:
        sc.add_rectilinear(f, *xs, association=assoc)
        g, _, gn = sc.render(cam, p, count_samples=True)
        batch, _ = sc.render_batch([cam, cam], p)
    assert np.array_equal(batch[0], g) and np.array_equal(batch[1], g)
    osc = O.OracleScene(64)
    osc.add_rectilinear(*xs, f, assoc=assoc)
    o, _, on = osc.render(cam, p)
    check(g, gn, o, on, assoc)


@pytest.mark.parametrize("nodes", NODES)
@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("samples", [30, 400])
def test_uniform_cells(nodes, view, samples):
    rng = np.random.default_rng(sum(nodes) + samples)
    xs, f, cam, p = case(nodes, view, False, samples, N.ASSOC_ELEMENT, rng, 0.0)
    spacing = [1.0 / (n - 1) for n in nodes]
    with S.Scene(0) as sc:
        sc.add_uniform(f, (0, 0, 0), spacing, association=N.ASSOC_ELEMENT)
        g, _, gn = sc.render(cam, p, count_samples=True)
    osc = O.OracleScene(64)
    osc.add_uniform(nodes, (0, 0, 0), spacing, f, assoc=N.ASSOC_ELEMENT)
    o, _, on = osc.render(cam, p)
    check(g, gn, o, on, N.ASSOC_ELEMENT)
