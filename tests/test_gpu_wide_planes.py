"""Planes too large for one pass of the PSF kernel (several passes, bands where
a launch has few blocks) against a band given explicitly and the FFT mode."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


# (size, sets, fwhm): over the 180 KB of the rule with 1, 2 and 3 bands chosen
# (blocks = sets x planes), ragged rows, and just below it
@pytest.mark.parametrize('size,n,fwhm', [((256, 200, 6), 2, 3.0), ((251, 203, 16), 20, 2.0),
                                         ((240, 240, 64), 40, 1.5), ((150, 150, 6), 2, 3.0)])
def test_wide_planes(gpu, size, n, fwhm):
    from gbkfit_b200 import psflsf, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    w = workloads.smdisk_batch128(nsets=n, size=size, nnodes=20)
    psf = psflsf.PSFGauss(psflsf.gauss_fwhm_to_sigma(fwhm))
    w.geom = workloads.Geometry(size, (1, 1, 10), (0, 0, (size[2] - 1) / 2), (0, 0, 0), psf,
                                w.geom.lsf)
    w.params.update(xpos=np.full(n, size[0] / 2), ypos=np.full(n, size[1] / 2))
    rng = np.random.default_rng(2)
    data = rng.standard_normal(size[::-1]).astype(np.float32)
    err = rng.uniform(0.5, 1.5, size[::-1]).astype(np.float32)
    out = []
    for cfg in (dict(conv='direct'), dict(conv='direct', band=24), dict(conv='fft')):
        ev = BatchedSMDisk(w.disk, w.geom, data, err, max_sets=n, chunk=n, **cfg)
        bufs = ev.alloc_inputs(n)
        ev.upload(ev.pack(w.params, n), bufs, n)
        k = min(n, 2)
        model = torch.full((k,) + size[::-1], float('nan'), device='cuda')
        chi2 = ev.evaluate_device(bufs, n).cpu().numpy().copy()
        ev.evaluate_device(bufs, k, model=model)
        out.append((chi2, model.cpu().numpy()))
        ev.close()
    # bands change no model value, only the grouping of chi^2's partial sums
    assert np.array_equal(out[0][1], out[1][1])
    assert np.max(np.abs(out[0][0] / out[1][0] - 1)) < 1e-6
    # the FFT mode's rounding: a few 2^-24 of the plane's peak
    assert np.max(np.abs(out[0][1] - out[2][1])) < 3e-6 * np.max(out[0][1])
    assert np.max(np.abs(out[0][0] / out[2][0] - 1)) < 1e-5
