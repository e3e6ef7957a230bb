"""Grids much taller than they are wide."""

import numpy as np
import pytest
import torch

from tests import trait_catalogue as C
from tests.helpers import gpu_smdisk, rel_err, upload
from tests.test_gpu_disk_kernels import _disk, _geo

pytestmark = pytest.mark.gpu


def test_thin_disk_of_many_rows(gpu, oracle_built):
    """More row pairs than a grid dimension has blocks: the row after the last
    whole round, and a disk at the last rows."""
    from gbkfit_b200.driver import DriverB200
    from oracle.oracle import Oracle
    disk, p = _disk(False)
    sx, sy, spec = 3, 2 * 65535 + 37, 5
    gm = DriverB200(0).backends().gmodel(np.float32)
    for ypos in (sy / 2 - 20.0, -sy / 2 + 3.0):
        geo, packed = _geo(sx, sy, 1, spec), disk.pack(dict(p, ypos=ypos))
        cube = torch.zeros((spec, sy, sx), device='cuda')
        gpu_smdisk(gm, upload(packed, 'cuda'), geo, dict(scube=cube))
        out = {}
        for prec, dt in (('f64', np.float64), ('f32', np.float32)):
            o = C.host_outputs(geo, dt)
            Oracle(prec).smdisk_evaluate(packed, geo, o)
            out[prec] = o['scube']
        assert out['f64'].max() > 0
        cpu = rel_err(out['f32'], out['f64'])
        assert rel_err(cube.cpu().numpy(), out['f64']) <= max(1e-5, 1.5 * cpu)


@pytest.mark.parametrize('size', [(512, 2790, 1), (510, 2371, 1)])
def test_direct_mode_of_many_rows(gpu, size):
    """A band whose range entries leave no room for its rows is divided; the
    model is that of small bands."""
    from gbkfit_b200 import psflsf, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    n = 2
    w = workloads.smdisk_batch128(nsets=n, size=size, nnodes=30)
    # 5 and 17 taps
    psf = psflsf.PSFGauss(psflsf.gauss_fwhm_to_sigma(1.0 if size[0] == 512 else 3.0))
    w.geom = workloads.Geometry(size, (1, 1, 10), (0, 0, 0), (0, 0, 0), psf, w.geom.lsf)
    w.params.update(xpos=np.full(n, size[0] / 2), ypos=np.full(n, size[1] - 250.0))
    data = np.random.default_rng(2).standard_normal(size[::-1]).astype(np.float32)
    out = []
    for band in (size[1], 256):
        ev = BatchedSMDisk(w.disk, w.geom, data, max_sets=n, conv='direct', band=band)
        bufs = ev.alloc_inputs(n)
        ev.upload(ev.pack(w.params, n), bufs, n)
        model = torch.full((n,) + size[::-1], float('nan'), device='cuda')
        out.append((ev.evaluate_device(bufs, n, model=model).cpu().numpy().copy(),
                    model.cpu().numpy()))
        ev.close()
    assert np.max(out[0][1]) > 0 and np.array_equal(out[0][1], out[1][1])
    # the grouping of chi^2's partial sums
    assert np.max(np.abs(out[0][0] / out[1][0] - 1)) < 1e-6
