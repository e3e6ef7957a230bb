"""Automatic waves of very small cubes: sets are a grid dimension of at most
65535, which 256 MB of scratch could exceed."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# W at most 16 x 32 on one channel: 4 KB of spectra, or 2.6 KB of planes, a set
@pytest.mark.parametrize('conv', ['fft', 'direct'])
def test_more_sets_than_a_grid_dimension(gpu, conv):
    from gbkfit_b200 import psflsf, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    n, size = 70000, (10, 8, 1)
    w = workloads.smdisk_batch128(nsets=4, size=size, nnodes=4)
    psf = psflsf.PSFGauss(psflsf.gauss_fwhm_to_sigma(1.0))
    lsf = psflsf.LSFGauss(psflsf.gauss_fwhm_to_sigma(10.0))
    w.geom = workloads.Geometry(size, (1, 1, 10), (0, 0, 0), (0, 0, 0), psf, lsf)
    w.params = {k: np.tile(np.asarray(v), (n // 4,) + (1,) * (np.ndim(v) - 1))
                for k, v in w.params.items()}
    w.params.update(xpos=np.random.default_rng(0).uniform(3, 7, n), ypos=np.full(n, 4.0))
    data = np.random.default_rng(1).standard_normal(size[::-1]).astype(np.float32)
    out = []
    for chunk in (0, 1000):
        ev = BatchedSMDisk(w.disk, w.geom, data, max_sets=n, chunk=chunk, conv=conv)
        assert ev.chunk <= 65535
        bufs = ev.alloc_inputs(n)
        ev.upload(ev.pack(w.params, n), bufs, n)
        out.append(ev.evaluate_device(bufs, n).cpu().numpy().copy())
        ev.close()
    assert np.array_equal(out[0], out[1]) and len(np.unique(out[0])) > 1000
