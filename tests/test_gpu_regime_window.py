"""The regime window's blocks (csrc/lle_regime.cu: window_loop) against the oracle:
windows that end before, at and after a block's or an interval's edge, or past the
record; every recorded variable; intervals that are no multiple of a block; bounds
that fire in the window; the amplitude rule, whose extremes come from the block
masks; and point counts that leave the last tile ragged.
"""
import numpy as np
import pytest

from test_gpu_parity import CHEN, LORENZ, MEMRISTIVE, ROSSLER, assert_lle_close, both

pytestmark = pytest.mark.gpu

BASE = dict(CHEN, nPts=9, ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.002, NT=0.5, tMax=12.0, transientTime=6.0,
            lleEps=1e-8, maxValue=1e4, seedChunk=200000, maxAmountOfPeaks=512, dbscanEps=0.02, regimeTime=6.0)


def _check(cbf, orc, kw):
    n = kw["nPts"] ** len(kw["idxMut"])
    j, o = both(cbf, orc, task=cbf.TASK_LLE_REGIME, **kw)
    lle, cls = cbf.run_host(j)
    want_l, want_c = orc.map_lle_regime(o, np.arange(n), cbf.lle_seeds(j))
    assert np.array_equal(cls, want_c), np.nonzero(cls != want_c)
    assert_lle_close(lle, want_l)
    return cls


@pytest.mark.parametrize("steps", [0, 1, 2, 15, 16, 17, 249, 250, 251, 266, 1000, 5999, 6000, 6001, 50000])
def test_window_lengths(cbf, orc, gpu_ok, steps):
    # steps + 0.5 truncates to `steps`; 6000 steps is the whole record
    _check(cbf, orc, dict(BASE, regimeTime=(steps + 0.5) * 0.002, regimeMinAmp=1e-6))


@pytest.mark.parametrize("nt", [0.002, 0.03, 0.034, 0.1])  # 1, 15, 17 and 50 steps an interval
@pytest.mark.parametrize("wv", [0, 1, 2])
def test_intervals_and_variables(cbf, orc, gpu_ok, nt, wv):
    _check(cbf, orc, dict(BASE, NT=nt, tMax=4.0, regimeTime=3.0, writableVar=wv, regimeMinAmp=1e-6))


@pytest.mark.parametrize("amp", [0.0, 1e-6, 5.0, 25.0, 40.0])
@pytest.mark.parametrize("bound", [0.0, 20.0, 1e4])
def test_amplitude_and_bounds(cbf, orc, gpu_ok, amp, bound):
    # the amplitude thresholds cut through the map, so the extremes decide classes
    _check(cbf, orc, dict(BASE, nPts=13, regimeMinAmp=amp, maxValue=bound))


@pytest.mark.parametrize("system_kw,extra", [
    (LORENZ, dict(ranges=[5, 20, 0.5, 200], idxMut=[1, 2], h=0.005)),
    (ROSSLER, dict(ranges=[0.05, 0.45, 0.05, 0.35], idxMut=[1, 2], h=0.01)),     # part of the map diverges
    (dict(CHEN, values=[0.3, 35.0, 3.0, 28.0]), dict(ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.002)),
    (CHEN, dict(ranges=[-3, 45, 20, 30], idxMut=[1, 3], h=0.002)),
    (MEMRISTIVE, dict(ranges=[-6, 6, -15, 15], idxMut=[4, 3], h=0.005, maxValue=1e7, writableVar=4)),
])
def test_systems(cbf, orc, gpu_ok, system_kw, extra):
    kw = dict(BASE, **system_kw)
    kw.update(extra, nPts=11, tMax=20.0, regimeTime=10.0, regimeMinAmp=1e-6, regimeChaosLle=0.05)
    _check(cbf, orc, kw)
