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
