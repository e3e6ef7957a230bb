"""Performance cases of the model-evaluation path.

Each case is one call that a fitter, sampler or server makes through the
package's public entry points, over the sizes its configurations, tests and
benchmark use:

* ``batch``: ``BatchedSMDisk``, chi^2 of many parameter sets of one thin disk
  against one data cube (sampler walkers, coalesced serving requests), with
  host parameter dicts (``evaluate``) or device-resident rows
  (``evaluate_device``), a separable PSF (direct convolution) or a Moffat one
  (FFT convolution), optionally with the model cubes (posterior predictive);
* ``scube``: ``Model.evaluate_d`` of ``DModelSCube``, the drop-in call chain
  (disk -> FFT convolution -> crop), thin, thick or Monte Carlo disk;
* ``loglike``: ``Objective.log_likelihood`` on top of it;
* ``mmaps``: ``Model.evaluate_h`` of ``DModelMMaps`` (moment maps to the host);
* ``grad``: ``SMDiskChi2.value_and_grad`` (chi^2 and its gradient).

``exact`` restates each of them in 64-bit torch, without the package.
"""

import math

import numpy as np
import torch

from gbkfit_b200 import psflsf, traits
from gbkfit_b200.adjoint import SMDiskChi2, to_vector
from gbkfit_b200.batched import BatchedSMDisk
from gbkfit_b200.disk import Disk
from gbkfit_b200.driver import DriverB200
from gbkfit_b200.model import (DModelMMaps, DModelSCube, GModelKinematics2D, GModelKinematics3D,
                               Model, Objective, SpectralMCDisk3D, SpectralSMDisk2D,
                               SpectralSMDisk3D)
from gbkfit_b200.workloads import Geometry, dcube_geometry

DZ = 10.0            # channel width, km/s


def listed():
    return [
        # one ensemble step of a small sampler on a small cutout: host
        # parameters in, chi^2 out, the evaluator's defaults; launches and
        # latency count
        dict(name='walkers48', kind='batch', nx=48, ny=44, nz=32, nsets=32, nnodes=12, chunk=0,
             psf='gauss', fwhm=3.0, lsf=1.5, host=True, mask=False, model=False),
        # an ensemble step on an odd-sized cube with masked voxels
        dict(name='walkers97', kind='batch', nx=97, ny=83, nz=61, nsets=100, nnodes=20,
             chunk=100, psf='gauss', fwhm=2.3, lsf=2.0, host=True, mask=True, model=False),
        # the benchmark's batch: 512 resident parameter sets in one wave
        dict(name='batch128', kind='batch', nx=128, ny=128, nz=96, nsets=512, nnodes=30,
             chunk=512, psf='gauss', fwhm=3.0, lsf=1.5, host=False, mask=False, model=False),
        # posterior-predictive cubes of 16 samples on the largest served side
        dict(name='predict256', kind='batch', nx=256, ny=240, nz=128, nsets=16, nnodes=30,
             chunk=16, psf='gauss', fwhm=3.6, lsf=2.4, host=False, mask=False, model=True),
        # a sampler's batch with a PSF that is not separable (FFT convolution)
        dict(name='moffat128', kind='batch', nx=128, ny=128, nz=96, nsets=64, nnodes=30,
             chunk=16, psf='moffat', fwhm=3.0, lsf=1.5, host=False, mask=False, model=False),
        # a large thin-disk cube through the drop-in chain
        dict(name='scube256', kind='scube', disk='thin', nx=256, ny=256, nz=128, scale=1,
             psf='moffat', fwhm=3.0, lsf=2.0),
        # a supersampled likelihood on an odd-sized cube (a fitter's inner call)
        dict(name='loglike101', kind='loglike', disk='thin', nx=101, ny=75, nz=47, scale=2,
             psf='gauss', fwhm=2.5, lsf=2.0),
        # the plain moment-map configuration, host maps out
        dict(name='mmaps64', kind='mmaps', disk='thin', nx=64, ny=64, nz=64, scale=1,
             psf='gauss', fwhm=2.5, lsf=2.0),
        # 1e7 clouds of a thick Monte Carlo disk, fast accumulation
        dict(name='mcdisk256', kind='scube', disk='mc', nx=256, ny=256, nz=128, scale=1,
             psf='moffat', fwhm=3.0, lsf=2.0, clouds=10_000_000, mode=0),
        # a small Monte Carlo disk, reproducible accumulation
        dict(name='mcdisk64', kind='scube', disk='mc', nx=64, ny=61, nz=40, scale=1,
             psf='gauss', fwhm=2.5, lsf=2.0, clouds=300_000, mode=1),
        # chi^2 and the gradient of 66 parameters
        dict(name='grad96', kind='grad', nx=96, ny=96, nz=64, nnodes=20, psf='gauss', fwhm=2.5,
             lsf=2.0),
        # a thick smooth disk: every voxel of the 3-D spatial grid emits
        dict(name='thick64', kind='scube', disk='thick', nx=64, ny=64, nz=64, scale=1,
             psf='gauss', fwhm=2.5, lsf=2.0),
    ]


def draw(rng):
    def lu(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(['batch', 'batch', 'batch', 'fft', 'thin', 'loglike', 'mmaps', 'mc',
                       'grad', 'thick'])
    c = dict(nx=lu(32, 256), ny=lu(32, 256), nz=lu(32, 192), psf='gauss',
             fwhm=round(rng.uniform(1.5, 4.0), 2), lsf=round(rng.uniform(1.0, 3.0), 2))
    if what in ('batch', 'fft'):
        fft = what == 'fft'
        # no more voxels than a third of the largest listed batch of the kind
        vox = c['nx'] * c['ny'] * c['nz']
        top = max(1, min(512, int((512 if not fft else 64) * 128 * 128 * 96 / 3 / vox)))
        n = lu(1, top)
        c.update(kind='batch', nsets=n, nnodes=rng.randint(8, 30),
                 chunk=rng.choice([0, n]) if not fft else min(n, 16),
                 psf='moffat' if fft else 'gauss', host=rng.random() < 0.5,
                 mask=rng.random() < 0.3, model=n <= 16 and rng.random() < 0.3)
        if fft:
            c['fwhm'] = round(rng.uniform(1.5, 3.0), 2)
    elif what == 'mc':
        c.update(kind='scube', disk='mc', clouds=lu(100_000, 5_000_000),
                 mode=rng.choice([0, 0, 1]), scale=1)
    elif what == 'thick':
        c.update(kind='scube', disk='thick', nx=lu(32, 80), ny=lu(32, 80), nz=lu(32, 96), scale=1)
    elif what == 'grad':
        c.update(kind='grad', nx=lu(32, 128), ny=lu(32, 128), nz=lu(32, 96),
                 nnodes=rng.randint(8, 30))
    elif what == 'loglike':
        s = rng.choice([1, 2])
        c.update(kind='loglike', disk='thin', nx=lu(32, 200 // s), ny=lu(32, 200 // s), scale=s)
    else:
        c.update(kind='scube' if what == 'thin' else 'mmaps', disk='thin', scale=1,
                 psf=rng.choice(['gauss', 'moffat']))
        if c['psf'] == 'moffat':
            c['fwhm'] = round(rng.uniform(1.5, 3.0), 2)
    return c


# ---- inputs ---------------------------------------------------------------------

def _gauss_sigma(fwhm):
    return fwhm / math.sqrt(8 * math.log(2))


def _moffat_alpha(fwhm, beta=2.5):
    return fwhm / (2 * math.sqrt(2 ** (1 / beta) - 1))


def _psf_lsf(case):
    psf = (psflsf.PSFGauss(_gauss_sigma(case['fwhm'])) if case['psf'] == 'gauss'
           else psflsf.PSFMoffat(_moffat_alpha(case['fwhm']), 2.5))
    return psf, psflsf.LSFGauss(_gauss_sigma(case['lsf'] * DZ))


def _centred(case):
    """True where the world coordinates are centred on the cube."""
    return case['kind'] in ('scube', 'loglike', 'mmaps')


def _rnodes(case):
    side = min(case['nx'], case['ny'])
    if 'nnodes' in case:                       # node-wise disks
        return np.linspace(0, 0.47 * side, case['nnodes'])
    return np.linspace(0, 0.47 * side, 61 if case['disk'] == 'mc' else 20)


def _params(case, seed):
    """The parameters of one call, per set (batch) or for one disk."""
    rng = np.random.default_rng([seed, 11])
    side = min(case['nx'], case['ny'])
    if case['kind'] == 'batch':
        # walkers around the disk's centre, as smdisk_batch128
        n, nn = case['nsets'], case['nnodes']
        return dict(
            vsys=rng.uniform(-5, 5, n), xpos=case['nx'] / 2 + rng.uniform(-1, 1, n),
            ypos=case['ny'] / 2 + rng.uniform(-1, 1, n), posa=rng.uniform(0, 360, n),
            incl=rng.uniform(20, 80, n), bpt_a=np.exp(rng.normal(0, 0.5, (n, nn))),
            vpt_vt=rng.uniform(50, 300, (n, nn)), dpt_a=rng.uniform(5, 40, (n, nn)))
    if case['kind'] == 'grad':
        rn = _rnodes(case)
        nn = len(rn)
        taper = 1 - (rn / rn[-1]) ** 4         # the disk's edge does not cut emission off
        return dict(
            vsys=rng.uniform(-8, 8), xpos=case['nx'] / 2 + rng.uniform(-1, 1),
            ypos=case['ny'] / 2 + rng.uniform(-1, 1), posa=rng.uniform(20, 70),
            incl=rng.uniform(40, 65),
            bpt_a=np.exp(-rn / (0.125 * side)) * (1 + 0.1 * rng.standard_normal(nn)) * taper,
            vpt_vt=200 * np.tanh(rn / (0.0625 * side)) + 5 * rng.standard_normal(nn),
            dpt_a=20 + 3 * rng.standard_normal(nn))
    p = dict(vsys=rng.uniform(-20, 20), xpos=rng.uniform(-2, 2), ypos=rng.uniform(-2, 2),
             posa=rng.uniform(0, 360), bpt_a=1.0, bpt_s=rng.uniform(0.08, 0.13) * side,
             vpt_vt=rng.uniform(150, 250))
    if case['disk'] == 'thin':
        p.update(incl=rng.uniform(40, 70), vpt_rt=rng.uniform(3, 6), dpt_a=rng.uniform(15, 30))
    else:
        p.update(incl=rng.uniform(50, 75), vpt_rt=0.04 * side, dpt_a=rng.uniform(12, 25),
                 bht_s=rng.uniform(1.5, 3.0))
    return p


def _nw_disk(case):
    return Disk(False, False, _rnodes(case), traits=dict(
        rpt=[traits.bpt('nw_uniform')], vpt=[traits.vpt('nw_tan_uniform')],
        dpt=[traits.dpt('nw_uniform')]))


def _gmodel(case, params):
    rn = _rnodes(case)
    if case['disk'] == 'thin':
        return GModelKinematics2D([SpectralSMDisk2D(
            False, False, traits.bpt('exponential'), traits.vpt('tan_arctan'),
            traits.dpt('uniform'), rnodes=rn)])
    tr = (traits.bpt('exponential'), traits.vpt('tan_lramp'), traits.dpt('uniform'),
          traits.bht('sech2'))
    if case['disk'] == 'thick':
        return GModelKinematics3D([SpectralSMDisk3D(False, False, *tr, rnodes=rn)])
    sub = _subnodes(rn)
    mid, h = sub[1:-1], sub[2] - sub[1]        # ring integrals of the density
    total = np.sum(np.exp(-mid / params['bpt_s']) * math.pi * 2 * mid * h)
    comp = SpectralMCDisk3D(float(total / case['clouds']), False, False, *tr, rnodes=rn)
    comp.set_mcdisk(42, case['mode'])
    return GModelKinematics3D([comp])


def _geometry(case):
    psf, lsf = _psf_lsf(case)
    size = (case['nx'], case['ny'], case['nz'])
    return Geometry(size, (1, 1, DZ), (0, 0, (case['nz'] - 1) / 2), (0, 0, 0), psf, lsf)


def _data(case, seed, truth):
    """Data, error and mask cubes: the model of ``truth`` plus noise."""
    gen = torch.Generator(device='cuda').manual_seed(1000003 * (seed + 1))
    cube = _convolved(case, truth)
    sigma = 0.02 * float(cube.max())
    noise = torch.randn(cube.shape, generator=gen, device='cuda', dtype=torch.float64)
    data = (cube + sigma * noise).float()
    err = (sigma * (0.8 + 0.4 * torch.rand(cube.shape, generator=gen, device='cuda'))).float()
    mask = (torch.rand(cube.shape, generator=gen, device='cuda') > 0.05).float()
    return data, err, mask


def _truth(case, seed):
    p = _params(case, seed + 7919)
    if case['kind'] == 'batch':
        p = {k: v[0] for k, v in p.items()}
    return p


def prepare(case, seed):
    params = _params(case, seed)
    st = dict(case=case, params=params)
    if case['kind'] in ('batch', 'grad', 'loglike'):
        data, err, mask = _data(case, seed, _truth(case, seed))
    if case['kind'] == 'batch':
        n = case['nsets']
        ev = BatchedSMDisk(_nw_disk(case), _geometry(case), data, err,
                           mask if case['mask'] else None, max_sets=n, chunk=case['chunk'])
        st['ev'] = ev
        if not case['host']:
            st['bufs'] = ev.alloc_inputs(n)
            ev.upload(ev.pack(params, n), st['bufs'], n)
        if case['model']:
            st['model'] = torch.empty((n, case['nz'], case['ny'], case['nx']), device='cuda')
            if case['host']:
                st['bufs'] = ev.alloc_inputs(n)
    elif case['kind'] == 'grad':
        st['model'] = SMDiskChi2(_nw_disk(case), _geometry(case), data.cpu().numpy(),
                                 err.cpu().numpy())
        st['theta'] = to_vector(params, 1.1)
    else:
        psf, lsf = _psf_lsf(case)
        s = case['scale']
        if case['kind'] == 'mmaps':
            # a cutoff at about a percent of the peak: the emission that is measured
            dmodel = DModelMMaps((case['nx'], case['ny'], case['nz']), (1, 1, DZ), psf=psf,
                                 lsf=lsf, mask_cutoff=1e-2, orders=(0, 1, 2))
        else:
            dmodel = DModelSCube((case['nx'], case['ny'], case['nz']), (1, 1, DZ),
                                 scale=(s, s, 1), psf=psf, lsf=lsf)
        st['model'] = Model(DriverB200(0), dmodel, _gmodel(case, params))
        if case['kind'] == 'loglike':
            st['objective'] = Objective(st['model'], data.cpu().numpy(), err.cpu().numpy(),
                                        mask.cpu().numpy())
    return st


def run(state):
    case, params = state['case'], state['params']
    if case['kind'] == 'batch':
        ev, n = state['ev'], case['nsets']
        if case['model']:
            if case['host']:
                ev.upload(ev.pack(params, n), state['bufs'], n)
            return ev.evaluate_device(state['bufs'], n, model=state['model']), state['model']
        if case['host']:
            return ev.evaluate(params, n)
        return ev.evaluate_device(state['bufs'], n)
    if case['kind'] == 'grad':
        return state['model'].value_and_grad(state['theta'])
    if case['kind'] == 'loglike':
        return state['objective'].log_likelihood(params)
    if case['kind'] == 'mmaps':
        out = state['model'].evaluate_h(params)
        return [out[k]['d'] for k in ('mmap0', 'mmap1', 'mmap2')] + [out['mmap0']['m']]
    return state['model'].evaluate_d(params)['scube']['d']


# ---- the work of a pass ------------------------------------------------------------

def _padded(case):
    """The padded grid of the FFT convolution (x, y, z)."""
    psf, lsf = _psf_lsf(case)
    s = case.get('scale', 1)
    return dcube_geometry((case['nx'], case['ny'], case['nz']), (1, 1, DZ), (0, 0, 0), (0, 0, 0),
                          (s, s, 1), psf, lsf)[1]


def _emission(case):
    """(spaxels, channels per line) of one disk: its ellipse at 60 degrees."""
    r = 0.47 * min(case['nx'], case['ny']) * case.get('scale', 1)
    return math.pi * r * r * 0.5, min(case['nz'], 2 * 5 * 20 / DZ + 1)


def work(case):
    vox = case['nx'] * case['ny'] * case['nz']
    spaxels, chan = _emission(case)
    px, py, pz = _padded(case)
    v = px * py * pz
    fft = 5.0 * v * math.log2(v) + 6.0 * (px // 2 + 1) * py * pz
    if case['kind'] == 'batch':
        n = case['nsets']
        flops = n * (spaxels * (60 + 8 * chan) + 3.0 * spaxels * chan)
        if case['psf'] == 'gauss':
            ks = 2 * math.ceil(7 * _gauss_sigma(case['fwhm'])) + 1
            kz = 2 * math.ceil(7 * _gauss_sigma(case['lsf'])) + 1
            flops += n * spaxels * chan * 2.0 * (2 * ks + kz)
        else:
            flops += n * fft
        nbytes = 4 * (vox * (2 + case['mask']) + n * (6 + 3 * case['nnodes']))
        if case['model']:
            nbytes += 4 * n * vox
        return dict(bytes=nbytes, flops=flops)
    if case['kind'] == 'grad':
        return dict(bytes=4 * (2 * vox + v) + 8 * 70, flops=2 * fft + spaxels * (160 + 26 * chan))
    flops = fft + spaxels * (80 + 10 * chan)
    # the kernel's spectrum is read, the cube (or the maps, or the sum) written
    nbytes = 8 * (px // 2 + 1) * py * pz
    if case['disk'] == 'thick':
        flops += spaxels * 8 * (80 + 10 * chan)
    if case['disk'] == 'mc':
        flops += case['clouds'] * (200 + 10.0 * chan)
    if case['kind'] == 'mmaps':
        nbytes += 4 * 4 * case['nx'] * case['ny']
    elif case['kind'] == 'loglike':
        nbytes += 4 * 3 * vox
    else:
        nbytes += 4 * vox
    return dict(bytes=nbytes, flops=flops)


# ---- the same in 64 bits, in plain torch -------------------------------------------

def _odd_up(x):
    e = 2 * math.ceil(0.5 * x)
    return int(e + 1 if e - 1 < x else e - 1)


def _subnodes(rn):
    h = min(1.0, float(np.min(np.diff(rn))) / 2)
    sub = np.arange(rn[0] + h / 2, rn[-1], h)
    sub = np.insert(sub, 0, rn[0])
    return np.append(sub, sub[-1] + h / 2)


def _kernels(case):
    """PSF image and LSF on their own boxes, normalised."""
    s = case.get('scale', 1)
    if case['psf'] == 'gauss':
        width = _gauss_sigma(case['fwhm'])
        prof = lambda r: np.exp(-r * r / (2 * width * width))
    else:
        width = _moffat_alpha(case['fwhm'])
        prof = lambda r: (1 + (r / width) ** 2) ** -2.5
    k = _odd_up(16 * width * s)
    a = (np.arange(k) - k // 2) / s
    r = np.hypot(a[None, :], a[:, None])
    psf = np.where(r > 8 * width, 0.0, prof(r))
    w = _gauss_sigma(case['lsf'] * DZ)
    kz = _odd_up(16 * w / DZ)
    z = (np.arange(kz) - kz // 2) * DZ
    lsf = np.where(z > 8 * w, 0.0, np.exp(-z * z / (2 * w * w)))
    return psf / psf.sum(), lsf / lsf.sum()


def _lerp(r, sub, vals):
    """Linear interpolation on the sub-nodes; r inside them."""
    k = torch.searchsorted(sub, r.detach().contiguous(), right=True).clamp(1, len(sub) - 1)
    x1, x2 = sub[k - 1], sub[k]
    return vals[k - 1] + (r - x1) / (x2 - x1) * (vals[k] - vals[k - 1])


def _fields(case, p, x, y, z=None):
    """Brightness, velocity, dispersion of the spaxels (0 brightness outside)."""
    dev = 'cuda'
    rad = math.pi / 180
    sub = torch.as_tensor(_subnodes(_rnodes(case)), device=dev)
    t = lambda v: torch.as_tensor(v, dtype=torch.float64, device=dev)
    pa, inc = t(p['posa']) * rad, t(p['incl']) * rad
    sp, cp, si, ci = torch.sin(pa), torch.cos(pa), torch.sin(inc), torch.cos(inc)
    dx, dy = x - t(p['xpos']), y - t(p['ypos'])
    xd, yd = -dx * sp + dy * cp, -dx * cp - dy * sp
    if z is None:
        yd = yd / ci
    else:
        yd, zd = yd * ci + z * si, -yd * si + z * ci
    r = torch.sqrt(xd * xd + yd * yd)
    cos = xd / torch.where(r == 0, torch.ones_like(r), r)
    inside = (r >= sub[0]) & (r < sub[-1])
    rc = torch.where(inside, r, torch.full_like(r, float(0.5 * (sub[0] + sub[-1]))))
    if 'nnodes' in case:
        rn = _rnodes(case)
        idx = np.clip(np.searchsorted(rn, _subnodes(rn), side='right') - 1, 0, len(rn) - 2)
        w = t(np.clip((_subnodes(rn) - rn[idx]) / (rn[idx + 1] - rn[idx]), 0, 1))
        idx = torch.as_tensor(idx, device=dev)
        onsub = lambda v: t(v)[idx] * (1 - w) + t(v)[idx + 1] * w
        b, v, d = (_lerp(rc, sub, onsub(p[k])) for k in ('bpt_a', 'vpt_vt', 'dpt_a'))
    else:
        b = p['bpt_a'] * torch.exp(-rc / p['bpt_s'])
        if case['disk'] == 'thin':
            v = p['vpt_vt'] * (2 / math.pi) * torch.atan(rc / p['vpt_rt'])
        else:
            v = p['vpt_vt'] * torch.clamp(rc / p['vpt_rt'], max=1.0)
        d = torch.full_like(rc, p['dpt_a'])
    if z is None:
        b = b / ci
    else:
        b = b * (0.5 / p['bht_s']) / torch.cosh(zd.abs() / p['bht_s']) ** 2
    return torch.where(inside, b, torch.zeros_like(b)), v * cos * si + t(p['vsys']), d.abs()


def _convolved(case, p, dtype=torch.float64):
    """The convolved cube (nz, ny, nx) of one parameter set."""
    s = case.get('scale', 1)
    psf, lsf = _kernels(case)
    kx, kz = psf.shape[0], lsf.shape[0]
    n = (case['nx'] * s, case['ny'] * s, case['nz'])
    w = (n[0] + kx - 1, n[1] + kx - 1, n[2] + kz - 1)
    lo = (-(case['nx'] / 2 - 0.5), -(case['ny'] / 2 - 0.5)) if _centred(case) else (0.0, 0.0)
    axis = lambda m, zero, edge, h: zero + (torch.arange(m, device='cuda',
                                                         dtype=dtype) - edge) * h
    # a supersampled grid starts half a coarse pixel before the first centre
    sub = lambda c: c - 0.5 + 0.5 / s
    x = axis(w[0], sub(lo[0]), kx // 2, 1.0 / s)[None, :]
    y = axis(w[1], sub(lo[1]), kx // 2, 1.0 / s)[:, None]
    v0 = -(case['nz'] - 1) / 2 * DZ
    # the spectral grid of the evaluation ends with its padding; its lines'
    # windows are clamped to it
    zc = torch.arange(w[2], device='cuda', dtype=dtype)[:, None, None]
    vz = v0 + (zc - kz // 2) * DZ
    vbase = v0 - (kz // 2) * DZ

    def lines(b, v, d):
        zlo = torch.round((v.detach() - 5 * d.detach() - vbase) / DZ).clamp(min=0)
        zhi = torch.round((v.detach() + 5 * d.detach() - vbase) / DZ)
        on = (zc >= zlo) & (zc <= zhi)
        g = torch.exp(-(vz - v) ** 2 / (2 * d * d)) * (b / (d * math.sqrt(2 * math.pi)))
        return torch.where(on, g, torch.zeros_like(g))

    if case.get('disk') == 'thick':
        # the spatial z grid of the padded cube: as long as its longer side
        px, py, _ = _padded(case)
        sz = px if px >= py else py
        cube = torch.zeros((w[2], w[1], w[0]), device='cuda', dtype=dtype)
        for i in range(sz):
            z = torch.tensor(-(sz / 2 - 0.5) + i, device='cuda', dtype=dtype)
            cube += lines(*_fields(case, p, x, y, z))
    else:
        cube = lines(*_fields(case, p, x, y))
    f = [(m + 7) // 8 * 8 for m in w]
    kern = torch.as_tensor(psf[None] * lsf[:, None, None], device='cuda')
    spec = torch.fft.rfftn(cube, s=f[::-1]) * torch.fft.rfftn(kern, s=f[::-1])
    out = torch.fft.irfftn(spec, s=f[::-1])[kz - 1:w[2], kx - 1:w[1], kx - 1:w[0]]
    if s > 1:
        out = out.reshape(n[2], case['ny'], s, case['nx'], s).mean(dim=(2, 4))
    return out


def _chi2(cube, data, err, mask=None, scale=1.0):
    r = (scale * cube - data.double()) / err.double()
    if mask is not None:
        r = r * mask.double()
    return (r * r).sum()


def exact(case, seed):
    if case.get('disk') == 'mc':
        # clouds are assigned to voxels by rounding 32-bit positions that come
        # from 32-bit random numbers: there is no 64-bit value
        return None
    params = _params(case, seed)
    if case['kind'] in ('batch', 'grad', 'loglike'):
        data, err, mask = _data(case, seed, _truth(case, seed))
    if case['kind'] == 'batch':
        chi2, cubes = [], []
        for i in range(case['nsets']):
            m = _convolved(case, {k: v[i] for k, v in params.items()})
            chi2.append(_chi2(m, data, err, mask if case['mask'] else None))
            if case['model']:
                cubes.append(m.cpu())
        chi2 = torch.stack(chi2).cpu()
        if case['model']:
            return chi2, torch.stack(cubes)
        return chi2.numpy() if case['host'] else chi2
    if case['kind'] == 'grad':
        names = ('vsys', 'xpos', 'ypos', 'posa', 'incl', 'bpt_a', 'vpt_vt', 'dpt_a')
        p = {k: torch.tensor(np.asarray(params[k]), dtype=torch.float64, device='cuda',
                             requires_grad=True) for k in names}
        scale = torch.tensor(1.1, dtype=torch.float64, device='cuda', requires_grad=True)
        c = _chi2(_convolved(case, p), data, err, None, scale)
        g = torch.autograd.grad(c, [p[k] for k in names] + [scale])
        return float(c), torch.cat([v.reshape(-1) for v in g]).cpu().numpy()
    cube = _convolved(case, params)
    if case['kind'] == 'loglike':
        return -0.5 * float(_chi2(cube, data, err, mask))
    if case['kind'] == 'mmaps':
        v = ((torch.arange(case['nz'], device='cuda', dtype=torch.float64)
              - (case['nz'] / 2 - 0.5)) * DZ)[:, None, None]
        m0 = cube.sum(0) * DZ
        m1 = (cube * v).sum(0) * DZ / m0
        m2 = torch.sqrt((cube * (v - m1) ** 2).sum(0) * DZ / m0)
        on = m0.abs() > 1e-2
        nan = torch.full_like(m0, float('nan'))
        return [torch.where(on, m, nan).cpu().numpy() for m in (m0, m1, m2)] + \
               [on.double().cpu().numpy()]
    return cube.cpu()
