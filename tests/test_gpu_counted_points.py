"""Points whose number of peaks alone decides their result are written by their lanes
and not shared (csrc/bif_device.cuh: kde_by_count, dbscan_by_count): maps where all,
some or none of a tile's points are such -- none, one, two or three peaks, and more
than the maximum, zero and negative ones among the maxima -- against the oracle, alone
and as jobs of a batch.
"""
import numpy as np
import pytest

from test_gpu_parity import LORENZ, both

pytestmark = pytest.mark.gpu

KW = dict(LORENZ, ranges=[5, 20, 20, 200], idxMut=[1, 2], h=0.01, transientTime=1.0, maxValue=1e4)
KDE = dict(kdeSampling=3, kdeI1=-20.0, kdeI2=20.0, kdeH=0.5)
RECORDS = [0.01, 0.5, 1.0, 1.5, 2.0, 8.0]


def _jobs(cbf, orc, side, record, most):
    kw = dict(KW, nPts=side, tMax=record, maxAmountOfPeaks=most)
    j, o = both(cbf, orc, task=cbf.TASK_DBSCAN, dbscanEps=0.05, **kw)
    yield j, orc.map_dbscan(o, 0, side * side)
    j, o = both(cbf, orc, task=cbf.TASK_KDE, **KDE, **kw)
    yield j, orc.map_kde(o, 0, side * side)


@pytest.mark.parametrize("most", [-3, -1, 0, 1, 2, 3, 5, 1000])
@pytest.mark.parametrize("side", [1, 9, 50])
def test_maps(cbf, orc, gpu_ok, side, most):
    for record in RECORDS:
        for j, want in _jobs(cbf, orc, side, record, most):
            assert np.array_equal(cbf.run_host(j)[0], want), record


@pytest.mark.parametrize("most", [2, 5])
def test_batches(cbf, orc, gpu_ok, most):
    torch = pytest.importorskip("torch")
    jobs, wants = zip(*[jw for side in (1, 50) for record in RECORDS for jw in _jobs(cbf, orc, side, record, most)])
    outs = [torch.full((w.size,), -7, dtype=torch.int32, device="cuda") for w in wants]
    b = cbf.Batch(list(jobs), [t.data_ptr() for t in outs])
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    b.run(s.cuda_stream)
    s.synchronize()
    b.check()
    for t, w in zip(outs, wants):
        assert np.array_equal(t.cpu().numpy(), w)
    b.close()
