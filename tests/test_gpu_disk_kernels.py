"""Edges of the disk, data-model and context kernels: thick disks whose z, x and
spectral sizes do not fill a round or tile (and a spectrum beyond shared
memory), thin columns whose windows straddle the batches of eight channels,
crops of ragged sizes, the Monte Carlo transpose-add at partial tiles, and the
status word across the synchronous and asynchronous modes."""

import numpy as np
import pytest
import torch

from tests import trait_catalogue as C
from tests.helpers import gpu_mcdisk, gpu_smdisk, rel_err, upload

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def backends(gpu):
    from gbkfit_b200.driver import DriverB200
    return DriverB200(0).backends()


def _disk(thick, mc=False):
    from gbkfit_b200 import traits as T
    from gbkfit_b200.disk import Disk
    tr = dict(rpt=[T.bpt('exponential')], vpt=[T.vpt('tan_arctan')], dpt=[T.dpt('uniform')])
    if thick:
        tr.update(rht=[T.bht('sech2')], vht=[T.vht_one()], dht=[T.dht_one()])
    d = Disk(False, False, np.linspace(0, 14, 15), traits=tr)
    p = dict(vsys=3.0, xpos=0.4, ypos=-0.3, posa=33.0, incl=57.0, bpt_a=1.0, bpt_s=5.0,
             vpt_rt=3.0, vpt_vt=140.0, dpt_a=17.0)
    if thick:
        p['bht_s'] = 2.0
    return d, p


def _geo(sx, sy, sz, spec):
    half = lambda n: -(n / 2 - 0.5)
    return dict(loose=False, tilted=False, opacity=None, spat_size=(sx, sy, sz),
                spat_step=(1, 1, 1), spat_zero=(half(sx), half(sy), half(sz) if sz > 1 else 0.0),
                spec_size=spec, spec_step=400.0 / spec, spec_zero=half(spec) * 400.0 / spec)


# bound of the reference comparisons: 1e-5 normwise, or 1.5 x the fp32 oracle's
# own distance from the fp64 one
@pytest.mark.parametrize('sx,sy,sz,spec', [(32, 2, 16, 32), (33, 3, 17, 31), (31, 5, 15, 33),
                                           (1, 1, 40, 1), (40, 2, 33, 97), (20, 2, 9, 1650)])
def test_thick_disk_edges(backends, oracle_built, sx, sy, sz, spec):
    from oracle.oracle import Oracle
    disk, p = _disk(True)
    geo, packed = _geo(sx, sy, sz, spec), disk.pack(p)
    cube = torch.full((spec, sy, sx), 0.25, device='cuda')
    gpu_smdisk(backends.gmodel(np.float32), upload(packed, 'cuda'), geo, dict(scube=cube))
    again = torch.full((spec, sy, sx), 0.25, device='cuda')
    gpu_smdisk(backends.gmodel(np.float32), upload(packed, 'cuda'), geo, dict(scube=again))
    assert torch.equal(cube, again)
    out = {}
    for prec, dt in (('f64', np.float64), ('f32', np.float32)):
        o = C.host_outputs(geo, dt)
        o['scube'][:] = 0.25
        Oracle(prec).smdisk_evaluate(packed, geo, o)
        out[prec] = o['scube']
    assert out['f64'].max() > 0.25
    cpu = rel_err(out['f32'], out['f64'])
    assert rel_err(cube.cpu().numpy(), out['f64']) <= max(1e-5, 1.5 * cpu)


@pytest.mark.parametrize('sx,sy,spec', [(32, 2, 8), (33, 3, 7), (65, 1, 9), (30, 31, 64)])
def test_thin_disk_edges(backends, oracle_built, sx, sy, spec):
    from oracle.oracle import Oracle
    disk, p = _disk(False)
    geo, packed = _geo(sx, sy, 1, spec), disk.pack(p)
    cube = torch.full((spec, sy, sx), -0.5, device='cuda')
    gpu_smdisk(backends.gmodel(np.float32), upload(packed, 'cuda'), geo, dict(scube=cube))
    out = {}
    for prec, dt in (('f64', np.float64), ('f32', np.float32)):
        o = C.host_outputs(geo, dt)
        o['scube'][:] = -0.5
        Oracle(prec).smdisk_evaluate(packed, geo, o)
        out[prec] = o['scube']
    cpu = rel_err(out['f32'], out['f64'])
    assert rel_err(cube.cpu().numpy(), out['f64']) <= max(1e-5, 1.5 * cpu)


@pytest.mark.parametrize('dst,scale,off,extra', [
    ((1, 1, 1), (1, 1, 1), (0, 0, 0), 0), ((33, 9, 5), (1, 1, 1), (3, 2, 1), 2),
    ((31, 7, 4), (2, 3, 1), (1, 0, 2), 1), ((64, 8, 3), (1, 1, 2), (0, 5, 0), 3)])
def test_downscale_edges(backends, dst, scale, off, extra):
    src = [off[i] + dst[i] * scale[i] + extra for i in range(3)]
    a = np.random.default_rng(3).standard_normal(src[::-1]).astype(np.float32)
    out = torch.zeros(dst[::-1], device='cuda')
    backends.dmodel(np.float32).dcube_downscale(scale, off, torch.from_numpy(a).cuda(), out)
    c = a[off[2]:off[2] + dst[2] * scale[2], off[1]:off[1] + dst[1] * scale[1],
          off[0]:off[0] + dst[0] * scale[0]].astype(np.float64)
    want = c.reshape(dst[2], scale[2], dst[1], scale[1], dst[0], scale[0]).mean(axis=(1, 3, 5))
    if scale == (1, 1, 1):
        assert np.array_equal(out.cpu().numpy(), want.astype(np.float32))
    else:       # at most 6 summands: 6 roundings of 2^-24
        assert np.abs(out.cpu().numpy() - want).max() <= 8 * 2.0 ** -24 * np.abs(a).max()


# nx ny on both sides of the 64-spaxel tile, channels on both sides of 32
@pytest.mark.parametrize('sx,sy,spec', [(8, 8, 32), (13, 5, 33), (16, 9, 31), (7, 3, 66)])
def test_mcdisk_transpose_add_edges(backends, sx, sy, spec):
    disk, p = _disk(True, mc=True)
    geo, packed = _geo(sx, sy, 8, spec), disk.pack(p)
    total = np.sum(disk.traits['rpt'][0].integrate(dict(a=1.0, s=5.0), disk.subrnodes[1:-1]))
    csum = disk.ncloudscsum(p, float(total / 20000))
    gm = backends.gmodel(np.float32)
    cubes = []
    for mode in (0, 3):
        gm.set_mcdisk(7, mode)
        cube = torch.full((spec, sy, sx), 0.125, device='cuda')
        gpu_mcdisk(gm, float(total / 20000), int(csum[-1]), torch.from_numpy(csum).cuda(),
                   torch.from_numpy(disk.hasordint()).cuda(), upload(packed, 'cuda'), geo,
                   dict(scube=cube))
        cubes.append(cube.cpu().numpy())
    assert cubes[1].max() > 0.125
    # the same clouds in another order of fp32 additions
    assert rel_err(cubes[0], cubes[1]) < 1e-5


def test_status_word_across_modes(backends):
    """An unknown trait uid is reported by the call that met it, in both modes,
    once, and an asynchronous call's by the next wait in sync mode."""
    from gbkfit_b200 import _native
    disk, p = _disk(False)
    geo = _geo(16, 16, 1, 8)
    good = upload(disk.pack(p), 'cuda')
    bad = dict(good, dpt=dict(good['dpt'], uids=torch.full_like(good['dpt']['uids'], 77)))
    gm = backends.gmodel(np.float32)
    cube = torch.zeros((8, 16, 16), device='cuda')
    run = lambda d: gpu_smdisk(gm, d, geo, dict(scube=cube))
    run(good)
    with pytest.raises(_native.NativeError):
        run(bad)
    run(good)
    gm._ctx.set_sync(False)
    run(bad)
    with pytest.raises(_native.NativeError):
        gm._ctx.synchronize()
    run(bad)
    gm._ctx.set_sync(True)
    with pytest.raises(_native.NativeError):
        run(good)
    run(good)
