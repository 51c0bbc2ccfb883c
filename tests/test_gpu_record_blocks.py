"""The recorded loop's blocks of 16 samples (csrc/bif_device.cuh: record_loop)
against the oracle where they can go wrong: records that end just before, at and
after a block's edge, every recorded variable, more than one step per sample,
divergence bounds that fire inside a block, trajectories that stop being numbers,
and equilibria whose last bits wobble (peaks and plateaus every few samples).
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import CHEN, LORENZ, MEMRISTIVE, ROSSLER, both

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 15, 16, 17, 18, 31, 32, 33, 47, 48, 49, 64, 65, 479]


def _peaks_equal(cbf, orc, kw):
    j, o = both(cbf, orc, task=cbf.TASK_PEAKS, **kw)
    peaks, counts = cbf.run_host(j)
    n = kw["nPts"] ** len(kw["idxMut"])
    wp, _, wc = orc.map_peaks(o, 0, n, max(peaks.shape[1], 1))
    assert np.array_equal(counts, wc), np.nonzero(counts != wc)
    for k in range(n):
        assert np.array_equal(peaks[k, :counts[k]], wp[k, :wc[k]]), k
    return counts


@pytest.mark.parametrize("record", LENGTHS)
def test_record_lengths_around_the_blocks(cbf, orc, gpu_ok, record):
    # long steps, so that short records hold peaks; (record + 0.5) h truncates to `record`
    h = 0.02
    kw = dict(LORENZ, nPts=11, ranges=[8, 12, 20, 60], idxMut=[1, 2], h=h, tMax=(record + 0.5) * h,
              transientTime=10.0, maxValue=1e4)
    _peaks_equal(cbf, orc, kw)


@pytest.mark.parametrize("system_kw,extra", [
    (ROSSLER, dict(ranges=[0.05, 0.40, 0.05, 0.35], idxMut=[1, 2], h=0.01, tMax=60.3)),   # some points diverge
    (LORENZ, dict(ranges=[5, 20, 20, 200], idxMut=[1, 2], h=0.005, tMax=30.1)),
    (dict(CHEN, values=[0.3, 35.0, 3.0, 28.0]), dict(ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.002, tMax=12.0)),
    (CHEN, dict(ranges=[-3, 45, 20, 30], idxMut=[1, 3], h=0.002, tMax=12.0)),             # a through 0: plain form
    (MEMRISTIVE, dict(ranges=[-6, 6, -15, 15], idxMut=[4, 3], h=0.005, tMax=20.0)),
])
@pytest.mark.parametrize("pre", [1, 3])
@pytest.mark.parametrize("bound", [0.0, 14.0, 1e4])
def test_variables_samplings_and_bounds(cbf, orc, gpu_ok, system_kw, extra, pre, bound):
    for wv in range(len(system_kw["ic"])):
        kw = dict(system_kw, nPts=7, transientTime=5.0, writableVar=wv, preScaller=pre, maxValue=bound, **extra)
        _peaks_equal(cbf, orc, kw)


def test_wobbling_equilibria(cbf, orc, gpu_ok):
    # rho from 0.2 to 24: fixed points reached to the last bit, samples rise, fall
    # and stay by single ulps
    kw = dict(LORENZ, nPts=16, ranges=[9, 11, 0.2, 24], idxMut=[1, 2], h=0.01, tMax=20.0, transientTime=400.0,
              maxValue=1e4)
    counts = [_peaks_equal(cbf, orc, dict(kw, writableVar=wv)) for wv in range(3)]
    assert max(c.max() for c in counts) > 100  # the wobble shows as peaks


@pytest.mark.parametrize("bound", [0.0, 1e4])
def test_cluster_and_mode_counts_of_short_and_diverging_records(cbf, orc, gpu_ok, bound):
    kw = dict(ROSSLER, nPts=12, ranges=[0.05, 0.45, 0.05, 0.35], idxMut=[1, 2], h=0.01, tMax=80.0,
              transientTime=30.0, maxValue=bound, maxAmountOfPeaks=400)
    j, o = both(cbf, orc, task=cbf.TASK_DBSCAN, dbscanEps=0.05, **kw)
    assert np.array_equal(cbf.run_host(j)[0], orc.map_dbscan(o, 0, 144))
    j, o = both(cbf, orc, task=cbf.TASK_KDE, kdeSampling=4, kdeI1=-20.0, kdeI2=20.0, kdeH=0.5, **kw)
    assert np.array_equal(cbf.run_host(j)[0], orc.map_kde(o, 0, 144))
