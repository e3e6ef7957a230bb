"""The two-factor line transforms of the FFT convolution (mode 0) and the
mixed-radix passes at compile-time lengths (mode 1) against numpy's 64-bit
transforms, at every instantiated length and on grids whose rows do
not fill a block's 16 columns or 16 rows."""

import numpy as np
import pytest
import torch

from gbkfit_b200 import _native
from gbkfit_b200.driver import DriverB200

pytestmark = pytest.mark.gpu

# error of an fp32 transform of n points: a few roundings (2^-24 each) per
# butterfly level, growing like sqrt(log2 n) in the 2-norm; 4 levels per axis
# and three axes forward and back stay below 32 roundings
TOL = 32 * 2.0 ** -24


def _rel(a, b):
    return np.linalg.norm(a - b) / np.linalg.norm(b)


# every line length once per axis (x: nx / 2), beside lengths that take the
# mixed-radix passes (2, 24, 20 and odd) and ragged row counts
@pytest.mark.parametrize('size', [
    (32, 32, 64), (64, 64, 32), (96, 96, 96), (128, 128, 128), (160, 160, 2), (192, 192, 1),
    (224, 224, 2), (256, 256, 2), (288, 288, 3), (320, 320, 2), (352, 352, 1), (384, 384, 1),
    (32, 3, 160), (64, 5, 192), (32, 1, 224), (32, 3, 256), (96, 1, 288), (32, 2, 320),
    (32, 1, 352), (34, 2, 384), (24, 32, 20), (31, 64, 32), (416, 32, 32)])
@pytest.mark.parametrize('mode', [0, 1])
def test_transforms_and_convolution(size, mode):
    nx, ny, nz = size
    rng = np.random.default_rng(nx + 1000 * ny + 1000000 * nz)
    a = rng.standard_normal((nz, ny, nx)).astype(np.float32)
    k = rng.standard_normal((nz, ny, nx)).astype(np.float32)
    fft = DriverB200(0).backends().fft(np.float32)
    fft._ctx.set_fft(mode)
    spec = np.fft.rfftn(a.astype(np.float64))
    ar = torch.from_numpy(a).cuda()
    ac = torch.zeros((nz, ny, nx // 2 + 1), dtype=torch.complex64, device='cuda')
    fft.fft_r2c(ar, ac)
    assert _rel(ac.cpu().numpy(), spec) < TOL
    back = torch.empty_like(ar)
    fft.fft_c2r(ac, back)
    assert _rel(back.cpu().numpy() / a.size, a) < TOL
    want = np.fft.irfftn(spec * np.fft.rfftn(k.astype(np.float64)), s=a.shape, axes=(0, 1, 2))
    kr = torch.from_numpy(k).cuda()
    # the cached form (its own padded spectra), twice with the cached spectrum
    for _ in range(2):
        got = torch.from_numpy(a).cuda()
        fft.fft_convolve_cached(got, kr)
        assert _rel(got.cpu().numpy(), want) < TOL
    # the form on the caller's dense spectra
    kc = torch.empty_like(ac)
    fft.fft_r2c(kr, kc)
    got = torch.from_numpy(a).cuda()
    fft.fft_convolve(got, ac, kc)
    assert _rel(got.cpu().numpy(), want) < TOL


def test_mode_keeps_the_mixed_radix_passes():
    """Both modes agree within the tolerance, and mode 1 takes other kernels
    (other last bits) on a grid that has two-factor lengths."""
    rng = np.random.default_rng(5)
    a = torch.from_numpy(rng.standard_normal((96, 64, 160)).astype(np.float32)).cuda()
    out = []
    for mode in (0, 1):
        fft = DriverB200(0).backends().fft(np.float32)
        fft._ctx.set_fft(mode)
        c = torch.zeros((96, 64, 81), dtype=torch.complex64, device='cuda')
        fft.fft_r2c(a, c)
        out.append(c.cpu().numpy())
    assert _rel(out[0], out[1]) < 2 * TOL
    assert not np.array_equal(out[0], out[1])
    with pytest.raises(_native.NativeError):
        fft._ctx.set_fft(2)
