"""The adjoint's transmittances lie in shared memory up to 512 transfer-function
entries and in local memory beyond: gradients on both sides of the line against
FP64 autograd, with rays of several 64-sample segments and some of one."""
import numpy as np
import pytest
import torch

from ascent_gb300 import diff as D
from ascent_gb300 import scene as S
from oracle import torch_reference as TR

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lut_n", [2, 512, 513])
def test_gradients_at_lut_sizes(lut_n):
    rng = np.random.default_rng(lut_n)
    n, size = (20, 23, 17), (19, 13)
    z, y, x = np.meshgrid(*[np.linspace(0, 1, k) for k in n], indexing="ij")
    field = (0.2 + 0.5 * np.exp(-6 * ((x - 0.4) ** 2 + (y - 0.6) ** 2 + (z - 0.5) ** 2)) + 0.1 * x).astype(np.float32)
    u = np.linspace(0, 1, lut_n)
    lut = np.stack([u, 0.5 + 0.3 * np.sin(6 * u), 1 - u, 0.02 + 0.05 * u], 1).astype(np.float32)
    spacing = [1.0 / (k - 1) for k in n[::-1]]
    cams = S.cinema_cameras(np.array([0.0, 1.0] * 3), np.array([[30, 40], [100, 70]], np.float32))
    sd = S.sample_distance(np.array([0.0, 1.0] * 3), 150)
    target = torch.from_numpy(rng.uniform(0, 0.5, (2, size[1], size[0], 4)).astype(np.float32))
    f = torch.from_numpy(field).cuda().requires_grad_(True)
    lt = torch.from_numpy(lut).cuda().requires_grad_(True)
    img = D.render(f, lt, cams, (0.0, 0.0, 0.0), spacing, *size, sd, (0.0, 1.0))
    ((img - target.cuda()) ** 2).sum().backward()
    fr = torch.from_numpy(field).double().requires_grad_(True)
    lr = torch.from_numpy(lut).double().requires_grad_(True)
    ref = TR.render(fr, lr, cams, (0.0, 0.0, 0.0), spacing, *size, sd, (0.0, 1.0))
    ((ref - target.double()) ** 2).sum().backward()
    ef = (f.grad.cpu().double() - fr.grad).norm() / fr.grad.norm()
    el = (lt.grad.cpu().double() - lr.grad).norm() / lr.grad.norm()
    # the tolerance of the adjoint's other comparison with FP64 autograd: a
    # sample at a kink of the transfer function takes the other interval's slope
    assert fr.grad.norm() > 0 and ef < 2e-3 and el < 2e-3, (float(ef), float(el))
