"""The histogram path on its own ground since the slots took the denser ranges:
ranges of more than twice the records, below and above the 1024^2 pixels that its
fused scan covers, against the FP32 restatement byte for byte.
"""
import numpy as np
import pytest

from ascent_gb300 import compositing as CP
from oracle import oracle as O

from test_composite_slots_gpu import records

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pixels", [70_000, 1024 * 1024, 1024 * 1024 + 1, 2_200_000])
@pytest.mark.parametrize("deep", [1, 8, 9, 40])
def test_wide_ranges(pixels, deep):
    rng = np.random.default_rng(pixels + deep)
    counts = (rng.random(pixels) < 0.3).astype(np.int64)
    counts[rng.integers(0, pixels, 100)] = deep
    counts[[0, -1]] = 1
    a = records(counts, pixels, False)
    assert pixels > 2 * len(a)
    want = O.composite_partials_f32([a])
    out, n = CP.composite_partials_device_async(CP.to_device(a), -17, pixels - 18)
    assert CP.from_device(out[:int(n)]).tobytes() == want.tobytes()
    assert CP.from_device(CP.composite_partials_device(CP.to_device(a))).tobytes() == want.tobytes()
