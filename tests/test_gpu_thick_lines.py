"""The thick-disk kernel's lines are the thin-disk kernel's: a thin disk on a grid
of two spatial z adds every line twice, which is exact in fp32."""

import numpy as np
import pytest
import torch

from tests.helpers import gpu_smdisk, upload
from tests.test_gpu_disk_kernels import _disk, _geo

pytestmark = pytest.mark.gpu


# columns in shared memory (also past the default 48 KB) and straight in the cube
@pytest.mark.parametrize('spec', [33, 400, 1650])
def test_lines_of_both_kernels(gpu, spec):
    from gbkfit_b200.driver import DriverB200
    disk, p = _disk(False)
    gm, packed = DriverB200(0).backends().gmodel(np.float32), upload(disk.pack(p), 'cuda')
    cubes = []
    for sz in (1, 2):
        cubes.append(torch.zeros((spec, 31, 35), device='cuda'))
        gpu_smdisk(gm, packed, _geo(35, 31, sz, spec), dict(scube=cubes[-1]))
    assert float(cubes[0].max()) > 0
    assert torch.equal(cubes[1], 2 * cubes[0])
