"""Warps that have run out of tiles and find nothing to help with leave their SMs
(csrc/bif_device.cuh: epilogue_help): while a batch works on a few long points, a
kernel on another stream runs and ends.
"""
import time

import pytest

from test_gpu_parity import LORENZ

pytestmark = pytest.mark.gpu

KW = dict(LORENZ, ranges=[5, 20, 20, 200], idxMut=[1, 2], h=0.005, maxValue=1e4)


def _kde(cbf, side, record):
    return cbf.make_job(task=cbf.TASK_KDE, nPts=side, tMax=record, transientTime=1.0, maxAmountOfPeaks=1000,
                        kdeSampling=2, kdeI1=-60.0, kdeI2=60.0, kdeH=0.5, **KW)


# 16 points of 8 000 000 samples (some 0.4 s): alone, with as many short points as
# warps, with many tiles of short points
@pytest.mark.parametrize("short", [None, (48, 5.0), (200, 50.0)])
def test_another_stream_runs_beside_a_batchs_last_points(cbf, gpu_ok, short):
    torch = pytest.importorskip("torch")
    jobs = [_kde(cbf, 4, 40000.0)] + ([_kde(cbf, *short)] if short else [])
    outs = [torch.zeros(j.nPts ** 2, dtype=torch.int32, device="cuda") for j in jobs]
    batch = cbf.Batch(jobs, [o.data_ptr() for o in outs])
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    other = cbf.make_job(task=cbf.TASK_LLE, nPts=200, tMax=20.0, NT=0.5, transientTime=5.0, lleEps=1e-8,
                         seedChunk=200000, **KW)
    lle = torch.zeros(200 * 200, dtype=torch.float64, device="cuda")
    batch.capture(s1.cuda_stream)
    for _ in range(2):  # the first launch of either kernel may wait for its code
        torch.cuda.synchronize()
        batch.launch(s1.cuda_stream)
        time.sleep(0.05)
        cbf.run_device(other, lle.data_ptr(), 0, s2.cuda_stream)
        s2.synchronize()
        running = not s1.query()
    s1.synchronize()
    batch.check()
    assert running
    assert (outs[0] == 1000).all()  # more peaks than the maximum
    batch.close()
