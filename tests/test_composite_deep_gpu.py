"""Pixels deeper than their places, against the FP32 restatement byte for byte:
every pixel of a frame with the same number of records around the limits of the
insertion, the warps and the CTA (32, 33, 1024, 1025), frames on either side of
the size from which a CTA takes 1024 pixels instead of 256, and both kinds of
deep pixels side by side.
"""
import numpy as np
import pytest

from ascent_gb300 import compositing as CP
from oracle import oracle as O

from test_composite_slots_gpu import records

pytestmark = pytest.mark.gpu


def check(counts, seed, ties):
    a = records(counts, seed, ties)
    want = O.composite_partials_f32([a])
    d = CP.to_device(a)
    assert CP.from_device(CP.composite_partials_device(d)).tobytes() == want.tobytes()
    out, n = CP.composite_partials_device_async(d, -17, len(counts) - 18)
    assert CP.from_device(out[:int(n)]).tobytes() == want.tobytes()


@pytest.mark.parametrize("depth", [8, 9, 16, 31, 32, 33, 40, 64, 65, 1024, 1025, 2500])
@pytest.mark.parametrize("ties", [False, True])
def test_even_depths(depth, ties):
    check(np.full(300 if depth < 100 else 40, depth), depth, ties)


@pytest.mark.parametrize("pixels", [152 * 4 * 1024 - 1, 152 * 4 * 1024, 152 * 4 * 1024 + 1025])
def test_uneven_depths(pixels):
    rng = np.random.default_rng(pixels)
    counts = rng.choice([0, 1, 2, 8, 9], pixels, p=[0.5, 0.2, 0.2, 0.05, 0.05])
    crowd = rng.integers(0, pixels - 2048)
    counts[crowd:crowd + 2048] = rng.choice([12, 32, 33, 47], 2048)
    counts[[crowd + 3, crowd + 4, crowd + 1500, 0, pixels - 1]] = [1024, 1025, 4000, 33, 1100]
    check(counts, pixels, False)
