"""The tuner's candidates: each runs a kernel that no other does, by what
gvr_scene_set_tuning says of them, and every shape that is accepted, candidate or
not, gives the same image.
"""
import itertools

import numpy as np
import pytest

from ascent_gb300 import scene as S
from ascent_gb300 import tune
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W


def kernel(packet_w, unroll, min_blocks):
    """3 and 4 samples run as 4 at 3 CTAs per SM and as 2 otherwise."""
    if unroll >= 3:
        unroll = 4 if min_blocks == 3 and packet_w != 16 else 2
    return packet_w, unroll, min_blocks


SHAPES = [(p, u, m) for p, u, m in itertools.product((4, 8, 16), (1, 2, 3, 4), (3, 4))
          if p != 16 or u < 3 or (u, m) == (3, 4)]


def test_candidates_run_kernels_of_their_own():
    ran = [kernel(**c) for c in tune.CANDIDATES]
    assert len(set(ran)) == len(ran)
    assert set(ran) == {kernel(*s) for s in SHAPES}
    batch = [kernel(**c) for c in tune.BATCH_CANDIDATES]
    assert len(set(batch)) == len(batch) and all(u <= 2 for _, u, _ in batch)


@pytest.mark.gpu
@pytest.mark.parametrize("parts", [None, (2, 1, 2)])
def test_every_accepted_shape_gives_the_same_image(parts):
    wl = W.plain_small(n=41, width=100, height=84, parts=parts)
    cam, p = V.workload_camera(wl), V.workload_params(wl)
    with S.Scene(0) as sc:
        V.load_workload(sc, wl)
        want, depth = sc.render(cam, p)
        for shape in SHAPES:
            sc.set_tuning(*shape)
            got, gd = sc.render(cam, p)
            assert np.array_equal(got, want) and np.array_equal(gd, depth), shape
