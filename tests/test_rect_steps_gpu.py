"""Rectilinear domains sampled in steps of many cells, where the march passes
over nodes four at a time: axes of fewer cells than that and of hundreds, steps
from a third of an axis down to a few cells, rays along either direction, bricks
that are empty, at steps that jump over them and at steps that do not. Against
the FP64 oracle, with the bars of test_march_fields_gpu.py.
"""
import numpy as np
import pytest

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S
from oracle import oracle as O

from test_march_fields_gpu import VIEWS, case, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nodes", [(2, 3, 4), (5, 6, 7), (10, 71, 301), (120, 9, 64)])
@pytest.mark.parametrize("view", VIEWS)
@pytest.mark.parametrize("assoc", [N.ASSOC_VERTEX, N.ASSOC_ELEMENT])
@pytest.mark.parametrize("hidden", [False, True])
@pytest.mark.parametrize("samples", [5, 17, 90])
def test_long_steps(nodes, view, assoc, hidden, samples):
    rng = np.random.default_rng(sum(nodes) + samples)
    xs, f, cam, p = case(nodes, view, hidden, samples, assoc, rng, 0.8)
    with S.Scene(0) as sc:
        sc.add_rectilinear(f, *xs, association=assoc)
        g, _, gn = sc.render(cam, p, count_samples=True)
        batch, _ = sc.render_batch([cam], p)
    assert np.array_equal(batch[0], g)
    osc = O.OracleScene(64)
    osc.add_rectilinear(*xs, f, assoc=assoc)
    o, _, on = osc.render(cam, p)
    check(g, gn, o, on, assoc)
