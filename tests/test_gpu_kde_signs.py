"""The KDE epilogue's FP32 sums with an error bound (csrc/bif_device.cuh: kde_warp)
against the oracle's exact sums, where the bound, the windows or the sort can go
wrong: peak counts around a sort's sizes and past the shared-memory keys (1024,
then keys in global memory), thousands of peaks of one value but for its last bits
(one weighted key), samples far from every peak (sums of exactly 0), sums that
underflow, dense sampling (neighbouring sums that differ by their last bits), a
reversed interval, negative and extreme bandwidths, and one or two samples.
"""
import ctypes as C

import numpy as np
import pytest

from test_gpu_parity import CHEN, LORENZ, LORENZ_MAP, ROSSLER, SPLIT_MAP, both

pytestmark = pytest.mark.gpu


def _check(cbf, orc, kw, flags=0):
    j, o = both(cbf, orc, task=cbf.TASK_KDE, flags=flags, **kw)
    got, _ = cbf.run_host(j)
    n = kw["nPts"] ** 2
    if flags & cbf.FLAG_KDE_FIXED:
        peaks, _, counts = orc.map_peaks(o, 0, n, cbf.lib().cbf_peak_capacity(C.byref(j)))
        want = np.array([orc.kde_fixed(peaks[k, :counts[k]], kw["maxAmountOfPeaks"], kw["kdeSampling"],
                                       kw["kdeI1"], kw["kdeI2"], kw["kdeH"]) for k in range(n)], np.int32)
    else:
        want = orc.map_kde(o, 0, n)
    assert np.array_equal(got, want), np.nonzero(got != want)
    return want


@pytest.mark.parametrize("tMax", [4.0, 12.0, 25.0, 26.5, 51.0])  # from 3 to about 70 peaks: P = 32, 64, 128
@pytest.mark.parametrize("h", [0.02, 0.5, 6.0])
def test_few_peaks(cbf, orc, gpu_ok, tMax, h):
    kw = dict(LORENZ_MAP, nPts=9, tMax=tMax, maxAmountOfPeaks=10000, kdeSampling=12, kdeI1=-25.0, kdeI2=70.0, kdeH=h)
    _check(cbf, orc, kw)


@pytest.mark.parametrize("samp,i1,i2,h", [(1, -60.0, 60.0, 0.3), (2, 60.0, -60.0, 0.05), (1, 0.0, 40.0, -0.5),
                                          (1, -60.0, 60.0, 1e-3), (1, -20.0, 60.0, 20.0)])
def test_more_peaks_than_the_shared_keys(cbf, orc, gpu_ok, samp, i1, i2, h):
    # 985 to 2849 peaks a point, those past 1024 in the second pass
    _check(cbf, orc, dict(SPLIT_MAP, kdeSampling=samp, kdeI1=i1, kdeI2=i2, kdeH=h))


@pytest.mark.parametrize("h", [0.5, 0.05])
def test_wobbling_fixed_points(cbf, orc, gpu_ok, h):
    # rho below the onset of chaos: thousands of peaks within some ulps
    kw = dict(LORENZ, nPts=8, ranges=[9, 11, 2, 20], idxMut=[1, 2], h=0.01, tMax=60.0, transientTime=400.0,
              maxValue=1e4, maxAmountOfPeaks=3000, kdeSampling=2, kdeI1=-20.0, kdeI2=20.0, kdeH=h)
    _check(cbf, orc, kw)


@pytest.mark.parametrize("samp,i1,i2,h", [
    (4, 200.0, 300.0, 0.5),      # no peak in reach of any sample
    (4, 30.0, 300.0, 0.5),       # the sums fall through the underflow to 0
    (200, 10.0, 12.0, 0.5),      # neighbouring samples 1e-4 bandwidths apart
    (40, -20.0, 60.0, 1e-4),     # spikes between zeros
    (10, 5.0, 5.0, 0.5),         # an empty interval
])
def test_ends_of_the_range(cbf, orc, gpu_ok, samp, i1, i2, h):
    kw = dict(LORENZ_MAP, nPts=6, tMax=40.0, maxAmountOfPeaks=10000, kdeSampling=samp, kdeI1=i1, kdeI2=i2, kdeH=h)
    _check(cbf, orc, kw)


@pytest.mark.parametrize("samp,h", [(1, 1e5), (2, 300.0), (1, 0.3)])
def test_sums_that_differ_by_their_last_bits(cbf, gpu_ok, samp, h):
    """A bandwidth far beyond the interval: neighbouring sums differ by their last
    bits, which FP32 expf decides (CUDA's and the C library's are not the same), so
    the map is compared with the batch kernel, whose epilogue keeps no more than
    1024 keys and computes the exact sums of points with more peaks."""
    torch = pytest.importorskip("torch")
    kw = dict(SPLIT_MAP, kdeSampling=samp, kdeI1=-20.0, kdeI2=60.0, kdeH=h)
    n = kw["nPts"] ** 2
    got, _ = cbf.run_host(cbf.make_job(task=cbf.TASK_KDE, **kw))
    out = torch.zeros(n, dtype=torch.int32, device="cuda")
    b = cbf.Batch([cbf.make_job(task=cbf.TASK_KDE, **kw)], [out.data_ptr()])
    s = torch.cuda.Stream()
    b.run(s.cuda_stream)
    s.synchronize()
    b.check()
    b.close()
    assert np.array_equal(got, out.cpu().numpy())


@pytest.mark.parametrize("samples", [1, 2, 3, 4, 32, 33, 34, 63, 64])
def test_fixed_sample_counts(cbf, orc, gpu_ok, samples):
    kw = dict(LORENZ_MAP, nPts=6, tMax=30.0, maxAmountOfPeaks=10000, kdeSampling=samples, kdeI1=-20.0, kdeI2=60.0,
              kdeH=1.0)
    _check(cbf, orc, kw, flags=cbf.FLAG_KDE_FIXED)


@pytest.mark.parametrize("side", [3, 49, 70])  # tiles of 1, 2 and 3 points
def test_small_maps_and_their_tiles(cbf, orc, gpu_ok, side):
    kw = dict(ROSSLER, nPts=side, ranges=[0.05, 0.40, 0.05, 0.35], idxMut=[1, 2], h=0.02, tMax=60.0,
              transientTime=10.0, maxValue=1e4, maxAmountOfPeaks=200, kdeSampling=4, kdeI1=-20.0, kdeI2=20.0, kdeH=0.5)
    _check(cbf, orc, kw)
    kw = dict(CHEN, nPts=side, ranges=[30, 45, 20, 30], idxMut=[1, 3], h=0.004, tMax=6.0, transientTime=4.0,
              maxValue=1e4, maxAmountOfPeaks=200, dbscanEps=0.05)
    j, o = both(cbf, orc, task=cbf.TASK_DBSCAN, **kw)
    assert np.array_equal(cbf.run_host(j)[0], orc.map_dbscan(o, 0, side * side))
