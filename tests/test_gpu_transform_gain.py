"""The mean gain of the transforms: roundings that all point the same way, which a
comparison of single voxels does not see."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# line lengths (x halved) whose constants are all rational products: what the
# inverse's constants leave is under 1e-8 per axis, 2^-24 in all with the twiddle tables
@pytest.mark.parametrize('size', [(96, 96, 96), (384, 192, 96), (192, 288, 192)])
def test_convolution_with_an_impulse(gpu, size):
    from gbkfit_b200.driver import DriverB200
    fft = DriverB200(0).backends().fft(np.float32)
    gen = torch.Generator(device='cuda').manual_seed(6)
    a = torch.randn(size[::-1], generator=gen, device='cuda')
    impulse = torch.zeros_like(a)
    impulse[0, 0, 0] = 1.0
    out = a.clone()
    fft.fft_convolve_cached(out, impulse)
    # the scale 1 / N in fp32 is part of the interface
    n = float(np.prod(size))
    scale = float(np.float32(1.0) / np.float32(n)) * n
    x, y = a.double() * scale, out.double()
    assert abs(float((x * y).sum() / (x * x).sum()) - 1) < 2.0 ** -24
