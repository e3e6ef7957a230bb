"""The FFT mode reads error and mask when it is called, as it reads the data: an
evaluator made from device tensors follows their edits in place, also in a
captured graph.  Widths with and without whole 16-byte rows, and arrays that
start off a 16-byte boundary."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('nx,shift,mask', [(40, 0, True), (37, 0, True), (40, 1, True),
                                           (40, 0, False)])
def test_error_and_mask_are_read_at_the_call(gpu, nx, shift, mask):
    from gbkfit_b200 import _native, workloads
    from gbkfit_b200.batched import BatchedSMDisk
    n, size = 3, (nx, 33, 9)
    w = workloads.smdisk_batch128(nsets=n, size=size, nnodes=10)
    w.params.update(xpos=np.full(n, nx / 2), ypos=np.full(n, 16.0))
    gen = torch.Generator(device='cuda').manual_seed(4)
    shape = size[::-1]

    def cube(lo):
        flat = torch.empty(int(np.prod(shape)) + shift, device='cuda')
        t = flat[shift:].view(shape)
        t.copy_(lo + torch.rand(shape, generator=gen, device='cuda'))
        return t

    data, err, msk = cube(0.0), cube(0.5), cube(0.0) if mask else None

    def chi2(e):
        bufs = e.alloc_inputs(n)
        e.upload(e.pack(w.params, n), bufs, n)
        return e.evaluate_device(bufs, n).cpu().numpy().copy(), bufs

    make = lambda: BatchedSMDisk(w.disk, w.geom, data, err, msk, weight=0.7, max_sets=n,
                                 conv='fft')
    ev = make()
    assert _native.lib().gbkb200_batch_planewise(ev.handle) == 1
    before, bufs = chi2(ev)
    ev.capture(bufs, n)
    err.mul_(1.5)
    if mask:
        msk[:, ::2] = 0.0
    after, _ = chi2(ev)
    want, _ = chi2(make())
    assert np.array_equal(after, want) and not np.any(after == before)
    ev.chi2.zero_()
    ev.replay()
    torch.cuda.synchronize()
    assert np.array_equal(ev.chi2.cpu().numpy(), want)
