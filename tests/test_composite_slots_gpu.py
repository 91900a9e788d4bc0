"""The compositor's slot path against the FP32 restatement, byte for byte: pixel
ranges around its tiles of 1024 and blocks of 256 pixels, pixels with none, one,
the eight records a pixel has places for, nine, the 32 that are ordered in local
arrays, 33 and hundreds, in shuffled input order, with equal, negative, signed
zero and infinite depths; records aligned to 4 bytes only; ranges on either side
of twice the records, past which the histogram path takes over; records outside
the caller's range.
"""
import numpy as np
import pytest
import torch

from ascent_gb300 import compositing as CP
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def records(counts, seed, ties):
    rng = np.random.default_rng(seed)
    pid = np.repeat(np.arange(len(counts)), counts)
    rng.shuffle(pid)
    a = np.zeros(len(pid), CP.PARTIAL_DTYPE)
    a["pixel_id"] = pid - 17
    a["depth"] = (rng.choice(np.array([-0.0, 0.0, 1.5, -2.5, np.inf, -np.inf, 3e38], np.float32), len(pid)) if ties
                  else rng.uniform(-4, 4, len(pid)))
    a["alpha"] = rng.choice(np.array([0.0, 0.02, 0.3, 0.9, 1.0], np.float32), len(pid))
    a["rgb"] = rng.uniform(0, 1, (len(pid), 3)) * a["alpha"][:, None]
    return a


def device(a, lead):
    """The records as an (n, 6) tensor `lead` words into its buffer."""
    buf = torch.zeros(6 * len(a) + lead, dtype=torch.int32, device="cuda")
    buf[lead:] = CP.to_device(a).reshape(-1)
    return buf[lead:].reshape(-1, 6)


@pytest.mark.parametrize("pixels", [1, 2, 255, 256, 1023, 1024, 1025, 4097])
@pytest.mark.parametrize("deep", [0, 9, 33, 700])
@pytest.mark.parametrize("lead,ties", [(0, False), (1, True), (3, False)])
def test_counts(pixels, deep, lead, ties):
    rng = np.random.default_rng(pixels + deep)
    counts = rng.choice([0, 1, 1, 2, 5, 8, 9, 31, 32], pixels)
    counts[rng.integers(0, pixels)] = max(deep, 1)
    counts[[0, -1]] = np.maximum(counts[[0, -1]], 1)
    a = records(counts, pixels, ties)
    want = O.composite_partials_f32([a])
    d = device(a, lead)
    assert CP.from_device(CP.composite_partials_device(d)).tobytes() == want.tobytes()
    out, n = CP.composite_partials_device_async(d, -17, pixels - 18)
    assert int(n) == len(want)
    assert CP.from_device(out[:int(n)]).tobytes() == want.tobytes()
    # a range wider than the records, below and above the slots' limit
    for extra in (len(a) // 2, 2 * len(a) + 5000):
        out, n = CP.composite_partials_device_async(d, -17 - extra, pixels - 18)
        assert CP.from_device(out[:int(n)]).tobytes() == want.tobytes()
    if pixels > 1:
        assert int(CP.composite_partials_device_async(d, -16, pixels - 18)[1]) == -1
        assert int(CP.composite_partials_device_async(d, -17, pixels - 19)[1]) == -1
