"""A cell-centred uniform domain whose one z layer holds more than 2^31 cells:
32768 x 70000 x 1, whose rows from 65536 on lie past a 32-bit index. The field
is constant over blocks of 16384 x 2000 cells, so a domain of 2 x 35 x 1 cells
over the same box is the same function and its image the reference.

Bars: those of test_march_fields_gpu.py for cell-centred fields (99% of the
pixels within 2/255, mean error 2e-3): the two grids place a sample within
rounding of a block's face on different sides.
"""
import numpy as np
import pytest
import torch

from ascent_gb300 import _native as N
from ascent_gb300 import scene as S
from ascent_gb300 import volume as V
from ascent_gb300 import workloads as W

from conftest import image_error

pytestmark = pytest.mark.gpu


def test_layer_beyond_32_bits():
    coarse = torch.rand((35, 2), generator=torch.Generator().manual_seed(5)).cuda()
    fine = coarse[:, None, :, None].expand(35, 2000, 2, 16384).reshape(1, 70000, 32768)
    vr = V.VolumeRenderer()
    rp, rgb, ap, al = W.linear_ramp_tf(alpha_max=0.6)
    vr.set_color_table(V.TransferFunction(rp, rgb, ap, al))
    vr.set_num_samples(60)
    b = np.array([0, 1, 0, 1, 0, 0.25])
    lo, hi = float(coarse.min()), float(coarse.max())
    p = N.make_params(96, 96, S.sample_distance(b, 60), (lo, hi), vr.lut(True))
    cams = []
    for az, el in ((0.0, 0.0), (20.0, 35.0)):
        cam = S.camera_reset_to_bounds(b)
        S.camera_azimuth(cam, az)
        S.camera_elevation(cam, el)
        cams.append(cam)
    images = []
    for f, spacing in ((coarse[None], (1 / 2, 1 / 35, 0.25)), (fine, (1 / 32768, 1 / 70000, 0.25))):
        with S.Scene(0) as sc:
            sc.add_uniform(f.contiguous(), (0, 0, 0), spacing, association=N.ASSOC_ELEMENT)
            images.append([sc.render(cam, p)[0] for cam in cams])
    del fine, f
    torch.cuda.empty_cache()
    for want, got in zip(*images):
        assert (want[..., 3] > 0.05).mean() > 0.2     # the box is in view
        e = image_error(got, want)
        assert e["frac_within_2"] >= 0.99 and e["mae"] <= 2e-3, e
