"""The plane-wise FFT mode of the batched evaluator (PSFs that are not
separable) against the oracle's chain, at the edges of its tiles: windows that
fill a 16-row group or a 32-column chunk exactly and by one, odd and not
4-aligned rows, empty planes, and what stays with the 3-D form."""

import numpy as np
import pytest

from tests.helpers import rel_err

pytestmark = pytest.mark.gpu


def _workload(size, nsets, fwhm, lsf_fwhm, seed):
    from gbkfit_b200 import psflsf, workloads
    w = workloads.smdisk_batch128(nsets=nsets, size=size, nnodes=12, seed=seed)
    nx, ny, nz = size
    psf = psflsf.PSFMoffat(psflsf.moffat_fwhm_beta_to_alpha(fwhm, 2.5), 2.5)
    lsf = psflsf.LSFGauss(psflsf.gauss_fwhm_to_sigma(lsf_fwhm * 10.0))
    w.geom = workloads.Geometry(size, (1, 1, 10), (0, 0, (nz - 1) / 2), (0, 0, 0), psf, lsf)
    w.params.update(xpos=np.full(nsets, nx / 2), ypos=np.full(nsets, ny / 2))
    return w


# (size, PSF FWHM, LSF FWHM, plane-wise?); the 1.15 px PSF has 17 taps (W = N +
# 16), the 3 px one 43; 40 channels of 10 km/s around 0 leave empty planes at
# 200; the last two have an LSF of more than 33 taps and a window over 384
@pytest.mark.parametrize('size,fwhm,lsf,planes', [
    ((48, 48, 20), 1.15, 1.5, 1), ((49, 47, 20), 1.15, 1.5, 1), ((80, 16, 12), 1.15, 1.5, 1),
    ((33, 64, 200), 1.15, 1.0, 1), ((54, 35, 16), 3.0, 2.0, 1), ((150, 150, 9), 3.0, 1.5, 1),
    # every transform length of 16 N1 points with N1 > 12 along x and along y
    *[((16 * n1 - 16, 18, 5), 1.15, 1.5, 1) for n1 in (14, 15, 16, 18, 20, 22, 24)],
    *[((18, 16 * n1 - 16, 5), 1.15, 1.5, 1) for n1 in (14, 15, 16, 18, 20, 22, 24)],
    ((342, 20, 8), 3.0, 1.5, 1), ((20, 341, 8), 3.0, 1.5, 1),
    ((40, 36, 24), 1.5, 6.0, 0), ((343, 24, 6), 3.0, 1.5, 0)])
def test_planewise_vs_oracle(gpu, oracle_built, size, fwhm, lsf, planes):
    import torch
    from oracle.oracle import scube_pipeline
    from gbkfit_b200 import _native, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    n = 3
    w = _workload(size, n, fwhm, lsf, seed=size[0] + size[1])
    rng = np.random.default_rng(1)
    shape = size[::-1]
    data = rng.standard_normal(shape).astype(np.float32)
    err = rng.uniform(0.5, 1.5, shape).astype(np.float32)
    mask = (rng.uniform(size=shape) > 0.1).astype(np.float32)
    ev = BatchedSMDisk(w.disk, w.geom, data, err, mask, weight=0.5, max_sets=n, chunk=2)
    assert ev.conv_mode == 'fft'
    assert _native.lib().gbkb200_batch_planewise(ev.handle) == planes
    bufs = ev.alloc_inputs(n)
    ev.upload(ev.pack(w.params, n), bufs, n)
    # planes that hold no emission must come out as zeros whatever was there
    model = torch.full((n,) + shape, float('nan'), device='cuda')
    got = ev.evaluate_device(bufs, n, model=model).cpu().numpy()
    again = ev.evaluate_device(bufs, n).cpu().numpy()
    assert np.array_equal(got, again)
    model = model.cpu().numpy()
    for i in range(n):
        p = w.disk.pack(workloads.set_params(w, i))
        ref64 = scube_pipeline(p, w.geom, precision='f64')
        cpu = rel_err(scube_pipeline(p, w.geom, precision='f32'), ref64)
        assert rel_err(model[i], ref64) <= max(1e-5, 1.5 * cpu)
        c = np.sum(((ref64 - data) / err * mask * 0.5) ** 2)
        assert abs(got[i] - c) / c < 1e-4
