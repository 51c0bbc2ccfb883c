"""Epilogues shared between warps (csrc/bif_device.cuh: epilogue_own, epilogue_help)
against the oracle, on maps where few points have almost all of the work: fixed
points whose last bits wobble beside others without a peak.  One point, one tile,
ragged tiles, and more tiles than warps; every map several times, as which warp
takes which point differs from run to run; alone, and as jobs of one batch.
"""
import numpy as np
import pytest

from test_gpu_parity import LORENZ, both

pytestmark = pytest.mark.gpu

KW = dict(LORENZ, ranges=[9, 11, 0.5, 30.0], idxMut=[1, 2], h=0.01, tMax=25.0, transientTime=80.0, maxValue=1e4,
          maxAmountOfPeaks=1500)
KDE = dict(kdeSampling=2, kdeI1=-20.0, kdeI2=20.0, kdeH=0.5)


@pytest.mark.parametrize("side", [1, 5, 33, 63])
def test_uneven_maps_repeat(cbf, orc, gpu_ok, side):
    kw = dict(KW, nPts=side)
    j, o = both(cbf, orc, task=cbf.TASK_DBSCAN, dbscanEps=0.05, **kw)
    want = orc.map_dbscan(o, 0, side * side)
    for _ in range(4):
        assert np.array_equal(cbf.run_host(j)[0], want)
    j, o = both(cbf, orc, task=cbf.TASK_KDE, **KDE, **kw)
    want = orc.map_kde(o, 0, side * side)
    for _ in range(4):
        assert np.array_equal(cbf.run_host(j)[0], want)


def test_more_tiles_than_warps(cbf, gpu_ok):
    # 400^2 points: 5000 tiles of 32, more than the GPU holds at once
    kw = dict(KW, nPts=400, tMax=8.0, transientTime=20.0)
    for task, extra in ((cbf.TASK_DBSCAN, dict(dbscanEps=0.05)), (cbf.TASK_KDE, KDE)):
        first, _ = cbf.run_host(cbf.make_job(task=task, **kw, **extra))
        for _ in range(2):
            assert np.array_equal(cbf.run_host(cbf.make_job(task=task, **kw, **extra))[0], first)
        # the same points as jobs of their own: tiles of one point each
        for p in (0, 31, 32, 159_999, 80_123):
            one, _ = cbf.run_host(cbf.make_job(task=task, firstPoint=p, nPoints=1, **kw, **extra))
            assert one[0] == first[p]


def test_batch_of_uneven_jobs(cbf, orc, gpu_ok):
    torch = pytest.importorskip("torch")
    jobs, wants, outs = [], [], []
    for side in (1, 7, 40):
        kw = dict(KW, nPts=side)
        for task, extra, oracle in ((cbf.TASK_DBSCAN, dict(dbscanEps=0.05), orc.map_dbscan),
                                    (cbf.TASK_KDE, KDE, orc.map_kde)):
            j, o = both(cbf, orc, task=task, **extra, **kw)
            jobs.append(j)
            wants.append(oracle(o, 0, side * side))
            outs.append(torch.zeros(side * side, dtype=torch.int32, device="cuda"))
    b = cbf.Batch(jobs, [t.data_ptr() for t in outs])
    s = torch.cuda.Stream()
    for _ in range(4):
        for t in outs:
            t.fill_(-7)
        torch.cuda.synchronize()
        b.run(s.cuda_stream)
        s.synchronize()
        b.check()
        for t, w in zip(outs, wants):
            assert np.array_equal(t.cpu().numpy(), w)
    b.close()
