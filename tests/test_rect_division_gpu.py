"""The rectilinear march's quotients by a kept reciprocal: equal to CUDA's
division bit for bit over the widths that use them, and a domain of widths that do
not, from subnormal to huge ones, renders like the same domain at an ordinary size.

The scaled domain is the ordinary one times a power of two, camera and step too,
so that every operation scales exactly but for what subnormal numbers round: 2^-149
against a box of 2^-126, the resolution of a float at the box. The bar is the one
of test_render_gpu.py for FP32 against FP64 positions.
"""
import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from ascent_gb300 import _native as N
from ascent_gb300 import build as B
from ascent_gb300 import scene as S
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W

from conftest import assert_parity

pytestmark = pytest.mark.gpu

HERE = Path(__file__).resolve().parent


def test_quotients(tmp_path):
    so = tmp_path / "rect_division.so"
    subprocess.run([B._nvcc(), *B.ARCH, *B.COMMON, "-shared", str(HERE / "rect_division.cu"), "-o", str(so),
                    "-lcudart_static", "-lrt", "-ldl", "-lpthread"], check=True)
    differing = C.CDLL(str(so)).differing
    differing.argtypes = [C.c_uint64, C.c_int64, C.c_int, C.c_int]
    differing.restype = C.c_int64
    assert differing(1, 1 << 30, 0, 0) == 0
    assert differing(2, 1 << 30, -64, 63) == 0


def image(scale, hidden):
    xs = [scale * np.cumsum(np.r_[0.0, w]) / 64 for w in
          ([4, 1, 1, 2, 8, 16, 32], [32, 8, 8, 2, 1, 1, 12], [1, 3, 60])]
    rng = np.random.default_rng(3)
    f = rng.random([len(x) for x in xs][::-1]).astype(np.float32)
    vr = V.VolumeRenderer()
    rp, rgb, ap, al = W.linear_ramp_tf(alpha_max=0.6)
    if hidden:
        ap, al = np.array([0.0, 0.45, 1.0]), np.array([0.0, 0.0, 0.8])
    vr.set_color_table(V.TransferFunction(rp, rgb, ap, al))
    vr.set_num_samples(200)
    b = np.array([0, 1, 0, 1, 0, 1.0])
    cam = S.camera_reset_to_bounds(b)
    S.camera_azimuth(cam, 40.0)
    S.camera_elevation(cam, 25.0)
    for a in range(3):
        cam.position[a] *= scale
        cam.look_at[a] *= scale
    p = N.make_params(67, 53, 2.0 ** -7 * scale, (0.0, 1.0), vr.lut(True))
    with S.Scene(0) as sc:
        sc.add_rectilinear(f, *xs)
        return sc.render(cam, p, count_samples=True)


@pytest.mark.parametrize("exponent", [-126, -100, -59, -57, 60, 70])
@pytest.mark.parametrize("hidden", [False, True])
def test_widths(exponent, hidden):
    want, _, n = image(1.0, hidden)
    got, _, m = image(2.0 ** exponent, hidden)
    assert want[..., 3].max() > 0.5
    assert_parity(got, want)
    assert abs(n - m) <= 2e-3 * n + 4
