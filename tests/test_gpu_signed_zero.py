"""Trajectories that start on zeros of either sign: a step from -0 to +0 is no rise
(csrc/peak_stream.cuh: RiseMask).  Rossler at s = 1 from y = -0 takes that step at
the start of the record; peaks, counts and classes against the oracle.
"""
import numpy as np
import pytest

from test_gpu_parity import ROSSLER, both

pytestmark = pytest.mark.gpu

START = dict(ROSSLER, values=[1.0, 0.2, 0.2, 5.7], nPts=5, ranges=[0.1, 0.3], idxMut=[1], h=0.01,
             transientTime=0.0, maxValue=1e4)


@pytest.mark.parametrize("ic", [[0.0, -0.0, 0.0], [0.0, 0.0, 0.0], [-0.0, -0.0, -0.0], [-0.0, 0.0, 0.0]])
@pytest.mark.parametrize("wv", [0, 1, 2])
def test_peaks_of_a_start_on_zero(cbf, orc, gpu_ok, ic, wv):
    j, o = both(cbf, orc, task=cbf.TASK_PEAKS, **dict(START, ic=ic, writableVar=wv, tMax=60.0))
    peaks, counts = cbf.run_host(j)
    wp, _, wc = orc.map_peaks(o, 0, 5, peaks.shape[1])
    assert np.array_equal(counts, wc) and counts.min() > 1
    for k in range(5):
        assert peaks[k, :counts[k]].tobytes() == wp[k, :wc[k]].tobytes(), k


def test_the_sign_of_a_starting_zero_adds_no_peak(cbf, gpu_ok):
    # two points, both at a = 0.2 (a sweep of one point has no step: 0 / 0)
    for y in (-0.0, 0.0):
        counts = cbf.bifurcation1D(60.0, 2, 0.01, 3, [0.0, y, 0.0], [0.2, 0.2], [1], 1, 1e4, 0.0, [1.0, 0.2, 0.2, 5.7],
                                   4, 1, system="rossler")[1]
        assert counts.tolist() == [8, 8], y


@pytest.mark.parametrize("ic", [[0.0, -0.0, 0.0], [0.0, 0.0, 0.0]])
def test_regime_window_of_a_start_on_zero(cbf, orc, gpu_ok, ic):
    kw = dict(START, ic=ic, writableVar=1, NT=0.5, tMax=80.0, lleEps=1e-8, seedChunk=200000, maxAmountOfPeaks=512,
              dbscanEps=1e-3, regimeTime=60.0, regimeMinAmp=1e-6)
    j, o = both(cbf, orc, task=cbf.TASK_LLE_REGIME, **kw)
    cls = cbf.run_host(j)[1]
    assert np.array_equal(cls, orc.map_lle_regime(o, np.arange(5), cbf.lle_seeds(j))[1])
