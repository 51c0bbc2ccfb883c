"""Regime windows in which a trajectory stops being a number (csrc/lle_regime.cu:
window_loop, `lost`): from the start, in the window, or only the offset one (an offset
of 0 makes the first renormalisation 0 / 0); without a bound and with one; classes
against the oracle, and which exponents are numbers.
"""
import numpy as np
import pytest

from test_gpu_parity import CHEN, MEMRISTIVE, ROSSLER, both

pytestmark = pytest.mark.gpu

BASE = dict(nPts=11, NT=0.5, tMax=12.0, transientTime=0.0, seedChunk=200000, maxAmountOfPeaks=512, dbscanEps=0.02,
            regimeTime=8.0)
SYSTEMS = [
    dict(CHEN, ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.002),
    dict(CHEN, ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.1),                    # leaves the numbers
    dict(CHEN, ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.002, ic=[float("nan"), 0.1, 0.1]),
    dict(ROSSLER, ranges=[0.05, 0.6, 0.05, 0.35], idxMut=[1, 2], h=0.05, tMax=200.0, regimeTime=150.0),
    dict(MEMRISTIVE, ranges=[-6, 6, -15, 15], idxMut=[4, 3], h=0.005),
]


@pytest.mark.parametrize("kw", SYSTEMS)
@pytest.mark.parametrize("eps", [0.0, 1e-8])
@pytest.mark.parametrize("bound", [0.0, 1e4])
@pytest.mark.parametrize("wv", [0, 2])
def test_classes(cbf, orc, gpu_ok, kw, eps, bound, wv):
    kw = dict(BASE, **kw)
    kw.update(lleEps=eps, maxValue=bound, writableVar=wv, regimeMinAmp=1e-6)
    j, o = both(cbf, orc, task=cbf.TASK_LLE_REGIME, **kw)
    lle, cls = cbf.run_host(j)
    want_l, want_c = orc.map_lle_regime(o, np.arange(121), cbf.lle_seeds(j))
    assert np.array_equal(cls, want_c), np.nonzero(cls != want_c)
    assert np.array_equal(np.isnan(lle), np.isnan(want_l))
