"""Launches whose dynamic shared memory is just below 48 KB: the default limit
holds for static and dynamic bytes together.  A raised limit stays for the
process, so the sizes run in a fresh one, in ascending order."""

import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def _thick():
    import numpy as np
    import torch
    from gbkfit_b200.driver import DriverB200
    from oracle.oracle import Oracle
    from tests import trait_catalogue as C
    from tests.helpers import gpu_smdisk, rel_err, upload
    from tests.test_gpu_disk_kernels import _disk, _geo
    disk, p = _disk(True)
    gm = DriverB200(0).backends().gmodel(np.float32)
    # 128 bytes a channel beside 12 KB: exactly 48 KB at 288
    for spec in (288, 289, 320, 352, 384):
        geo, packed = _geo(20, 3, 9, spec), disk.pack(p)
        cube = torch.zeros((spec, 3, 20), device='cuda')
        gpu_smdisk(gm, upload(packed, 'cuda'), geo, dict(scube=cube))
        out = {}
        for prec, dt in (('f64', np.float64), ('f32', np.float32)):
            o = C.host_outputs(geo, dt)
            Oracle(prec).smdisk_evaluate(packed, geo, o)
            out[prec] = o['scube']
        assert out['f64'].max() > 0
        cpu = rel_err(out['f32'], out['f64'])
        assert rel_err(cube.cpu().numpy(), out['f64']) <= max(1e-5, 1.5 * cpu), spec


def _psf():
    import numpy as np
    import torch
    from gbkfit_b200 import psflsf, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    n, size = 2, (147, 39, 6)
    w = workloads.smdisk_batch128(nsets=n, size=size, nnodes=12)
    psf = psflsf.PSFGauss(psflsf.gauss_fwhm_to_sigma(2.5))      # 15 taps: 49096 bytes
    w.geom = workloads.Geometry(size, (1, 1, 10), (0, 0, (size[2] - 1) / 2), (0, 0, 0), psf,
                                w.geom.lsf)
    w.params.update(xpos=np.full(n, size[0] / 2), ypos=np.full(n, size[1] / 2))
    data = np.random.default_rng(1).standard_normal(size[::-1]).astype(np.float32)
    out = []
    for conv in ('direct', 'fft'):
        ev = BatchedSMDisk(w.disk, w.geom, data, max_sets=n, conv=conv)
        bufs = ev.alloc_inputs(n)
        ev.upload(ev.pack(w.params, n), bufs, n)
        model = torch.full((n,) + size[::-1], float('nan'), device='cuda')
        chi2 = ev.evaluate_device(bufs, n, model=model).cpu().numpy().copy()
        out.append((chi2, model.cpu().numpy()))
    # the FFT mode's rounding: a few 2^-24 of the plane's peak
    assert np.max(np.abs(out[0][1] - out[1][1])) < 3e-6 * np.max(out[1][1])
    assert np.max(np.abs(out[0][0] / out[1][0] - 1)) < 1e-5


@pytest.mark.parametrize('what', ['_thick', '_psf'])
def test_launches_below_the_default_limit(gpu, oracle_built, what):
    r = subprocess.run([sys.executable, '-c', 'from tests.test_gpu_shared_memory import ' + what +
                        ' as f; f()'], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-2000:]
