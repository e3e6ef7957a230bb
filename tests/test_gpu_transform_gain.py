"""The mean gain of the transforms and of the plane-wise FFT mode: roundings that
all point the same way, which a comparison of single voxels does not see."""

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


def test_flux_of_the_planewise_mode(gpu):
    """Without PSF and LSF, on 64 x 64 point planes, the transforms keep the
    planes' sums up to the rounding of their additions: the flux is that of the
    drop-in disk's lines."""
    from gbkfit_b200 import _native, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    from gbkfit_b200.driver import DriverB200
    from tests.helpers import gpu_smdisk, upload
    n, size = 8, (64, 60, 160)
    w = workloads.smdisk_batch128(nsets=n, size=size, nnodes=16)
    w.geom = g = workloads.Geometry(size, (1, 1, 10), (0, 0, 79.5), (0, 0, 0), None, None)
    w.params.update(xpos=np.full(n, 32.0), ypos=np.full(n, 30.0))
    ev = BatchedSMDisk(w.disk, g, np.zeros(size[::-1], np.float32), max_sets=n, conv='fft')
    assert _native.lib().gbkb200_batch_planewise(ev.handle) == 1
    bufs = ev.alloc_inputs(n)
    ev.upload(ev.pack(w.params, n), bufs, n)
    model = torch.empty((n,) + size[::-1], device='cuda')
    ev.evaluate_device(bufs, n, model=model)
    geo = dict(loose=False, tilted=False, spat_size=(64, 60, 1), spat_step=(1, 1, 0.0),
               spat_zero=(g.zero[0], g.zero[1], 0.0), spec_size=160, spec_step=g.step[2],
               spec_zero=g.zero[2])
    gm = DriverB200(0).backends().gmodel(np.float32)
    ratio = []
    for i in range(n):
        cube = torch.zeros(size[::-1], device='cuda')
        gpu_smdisk(gm, upload(w.disk.pack(workloads.set_params(w, i)), 'cuda'), geo,
                   dict(scube=cube))
        assert float(cube.max()) > 0
        ratio.append(float(model[i].double().sum() / cube.double().sum()) - 1)
    # a plane's sum: a few additions of 2^-25 each, some hundred planes a set
    assert abs(np.mean(ratio)) < 2.0 ** -26, ratio
