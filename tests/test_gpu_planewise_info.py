"""What an evaluator of the plane-wise FFT mode says about itself, and what the
tuner tries on it."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(nsets):
    from gbkfit_b200 import psflsf, workloads
    w = workloads.smdisk_batch128(nsets=nsets, size=(70, 44, 24), nnodes=8)
    w.geom = workloads.Geometry(w.geom.size, (1, 1, 10), (0, 0, 11.5), (0, 0, 0),
                                psflsf.PSFMoffat(1.2, 2.5), w.geom.lsf)
    return w, np.ones((24, 44, 70), np.float32)


@pytest.mark.parametrize('nsets,chunk', [(3, 0), (400, 0), (400, 7)])
def test_info(gpu, nsets, chunk):
    from gbkfit_b200.batched import BatchedSMDisk
    w, data = _workload(nsets)
    ev = BatchedSMDisk(w.disk, w.geom, data, max_sets=nsets, chunk=chunk, fft_size=(128, 81, 50))
    assert ev.conv_mode == 'fft' and ev.planewise
    win = [w.geom.size[i] + w.geom.kernel_size[i] - 1 for i in range(2)]
    # the shortest lines of 16 points times an instantiated factor
    assert all(win[i] <= ev.fft_size[i] < win[i] + 16 for i in range(2)) and ev.fft_size[2] == 1
    lines = 24 * -(-win[1] // 16) * 16 * -(-(ev.fft_size[0] // 2 + 1) // 16) * 16 * 8
    wave = min(nsets, (256 << 20) // lines)
    assert ev.chunk == (min(chunk, wave) if chunk else wave)
    # the work of a wave: row spectra, crop rows, planes with their masks and flags; then
    # the tables and partials
    rows = ev.chunk * 24 * win[1] * -(-win[0] // 32)
    crop = 24 * 44 * -(-(ev.fft_size[0] // 2 + 1) // 16) * 16 * 8
    fixed = 8 * (ev.fft_size[0] + ev.fft_size[1] * (1 + crop // (24 * 44 * 8)))
    assert ev.work_bytes == ev.chunk * (lines + crop + 24 * 32) + rows * 132 + fixed + \
        nsets * 24 * -(-44 // 16) * 8
    assert ev.chunk * lines <= 256 << 20 and crop <= lines and 132 * rows <= ev.chunk * lines
    ev.close()


def test_tuner_leaves_the_3d_knobs_alone(gpu, monkeypatch):
    from gbkfit_b200 import autotune
    w, data = _workload(6)
    tried, orig = [], autotune.time_config

    def time_config(w, data, err, nsets, cfg, *a, **kw):
        if cfg['conv'] == 'fft':
            tried.append(cfg)
        return orig(w, data, err, nsets, cfg, *a, **kw)

    monkeypatch.setattr(autotune, 'time_config', time_config)
    autotune.tune_batched(w, data, None, 6, use_cache=False)
    assert len(tried) > 1 and len({(c['fft_size'], c['rows_k1']) for c in tried}) == 1
    assert len({c['chunk'] for c in tried}) == len(tried)
