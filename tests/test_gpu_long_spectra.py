"""Spectra of more planes than the tile kernel's shared memory holds (2048): the
model kernel on a warp per 32-column chunk, with planes that nothing reaches, a
window that is no multiple of 32 wide and the generic trait path."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nz,nodewise', [(2049, True), (2060, False)])
def test_long_spectra(gpu, oracle_built, nz, nodewise):
    from gbkfit_b200 import traits as T
    from gbkfit_b200 import workloads
    from gbkfit_b200.batched import BatchedSMDisk
    from gbkfit_b200.disk import Disk
    from oracle.oracle import chi2, scube_pipeline
    from tests.helpers import rel_err
    n, size = 2, (20, 18, nz)
    w = workloads.smdisk_batch128(nsets=n, size=size, nnodes=6)
    if not nodewise:
        w.disk = Disk(False, False, w.disk.rnodes, traits=dict(
            rpt=[T.bpt('nw_uniform')], vpt=[T.vpt('nw_tan_uniform')], dpt=[T.dpt('nw_uniform')],
            spt=[T.spt('azrange')]))
        w.params.update(spt_p=np.full(n, 30.0), spt_s=np.full(n, 300.0))
    w.params.update(xpos=np.full(n, 10.0), ypos=np.full(n, 9.0),
                    vsys=np.array([-10300.0, 9000.0]))   # cut off by the end, and inside
    rng = np.random.default_rng(3)
    data = rng.standard_normal(size[::-1]).astype(np.float32) * 0.01
    err = rng.uniform(0.5, 1.5, size[::-1]).astype(np.float32)
    ev = BatchedSMDisk(w.disk, w.geom, data, err, max_sets=n, conv='direct')
    bufs = ev.alloc_inputs(n)
    ev.upload(ev.pack(w.params, n), bufs, n)
    model = torch.full((n,) + size[::-1], 7.0, device='cuda')
    got = ev.evaluate_device(bufs, n, model=model).cpu().numpy()
    model = model.cpu().numpy()
    for i in range(n):
        p = w.disk.pack(workloads.set_params(w, i))
        ref = scube_pipeline(p, w.geom, precision='f64')
        ref32 = scube_pipeline(p, w.geom, precision='f32')
        assert ref.max() > 0
        assert rel_err(model[i], ref) <= max(1e-5, 1.5 * rel_err(ref32, ref)), i
        assert not np.any(model[i] == 7.0) and np.count_nonzero(model[i]) < model[i].size
        c = chi2(ref, data, err)
        assert abs(got[i] - c) / c < 1e-4
