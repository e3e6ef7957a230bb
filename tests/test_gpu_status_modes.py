"""The status of calls made in asynchronous mode, after the context has gone to
synchronous mode: reported once, by the first call that waits."""

import numpy as np
import pytest
import torch

from tests.helpers import gpu_smdisk, upload
from tests.test_gpu_disk_kernels import _disk, _geo

pytestmark = pytest.mark.gpu


class _Calls:
    """One smooth-disk call with and without an unknown trait uid."""

    def __init__(self):
        from gbkfit_b200.driver import DriverB200
        disk, p = _disk(False)
        self.gm = DriverB200(0).backends().gmodel(np.float32)
        self.ctx = self.gm._ctx
        self.cube = torch.zeros((8, 16, 16), device='cuda')
        good = upload(disk.pack(p), 'cuda')
        bad = dict(good, dpt=dict(good['dpt'], uids=torch.full_like(good['dpt']['uids'], 77)))
        geo = _geo(16, 16, 1, 8)
        self.good = lambda: gpu_smdisk(self.gm, good, geo, dict(scube=self.cube))
        self.bad = lambda: gpu_smdisk(self.gm, bad, geo, dict(scube=self.cube))


def test_status_after_an_evaluator_is_made(gpu, monkeypatch):
    """Making an evaluator of the 3-D FFT form waits inside; the context stays
    asynchronous, and so does the status of what follows."""
    from gbkfit_b200 import _native, batched, psflsf, workloads
    c = _Calls()
    c.ctx.set_sync(False)
    monkeypatch.setattr(batched._native, 'Context', lambda **kw: c.ctx)
    w = workloads.smdisk_batch128(nsets=1, size=(32, 30, 16), nnodes=8)
    lsf = psflsf.LSFGauss(psflsf.gauss_fwhm_to_sigma(70.0))     # over 33 taps
    w.geom = workloads.Geometry(w.geom.size, (1, 1, 10), (0, 0, 7.5), (0, 0, 0), w.geom.psf, lsf)
    ev = batched.BatchedSMDisk(w.disk, w.geom, np.ones((16, 30, 32), np.float32), max_sets=1,
                               conv='fft')
    assert _native.lib().gbkb200_batch_planewise(ev.handle) == 0
    c.bad()
    c.ctx.set_sync(True)
    with pytest.raises(_native.NativeError):
        c.good()
    c.good()


def test_status_of_a_replayed_graph(gpu):
    from gbkfit_b200 import _native
    c = _Calls()
    s = torch.cuda.Stream()
    c.ctx.set_stream(s)
    c.ctx.set_sync(False)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        c.bad()
    c.ctx.set_sync(True)
    c.good()
    with torch.cuda.stream(s):
        g.replay()
    with pytest.raises(_native.NativeError):
        c.good()
    c.good()


def test_status_of_both_modes_at_once(gpu):
    from gbkfit_b200 import _native
    c = _Calls()
    c.ctx.set_sync(False)
    c.bad()
    c.ctx.set_sync(True)
    with pytest.raises(_native.NativeError):
        c.bad()
    c.good()
