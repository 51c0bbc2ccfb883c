"""The host entry points' packed copy of peak rows (csrc/capi.cu: copy_packed_peaks)
against the device rows: rows with no peak, with few, with more than the capacity,
and jobs whose rows are more than half full (copied whole).
"""
import numpy as np
import pytest

from test_gpu_parity import LORENZ, ROSSLER

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kw,cap", [
    (dict(ROSSLER, nPts=1, ranges=[0.2, 0.2], idxMut=[1], h=0.01, tMax=100.0), 0),
    (dict(ROSSLER, nPts=65, ranges=[0.05, 0.45], idxMut=[1], h=0.01, tMax=200.0), 0),      # diverged rows are empty
    (dict(ROSSLER, nPts=33, ranges=[0.05, 0.30], idxMut=[1], h=0.01, tMax=200.0), 20),     # rows past their capacity
    (dict(ROSSLER, nPts=33, ranges=[0.05, 0.30], idxMut=[1], h=0.01, tMax=200.0), 60),     # about half full
    (dict(LORENZ, nPts=7, ranges=[9, 11, 2, 24], idxMut=[1, 2], h=0.01, tMax=100.0), 0),   # thousands and none
    (dict(ROSSLER, nPts=5, ranges=[0.1, 0.2], idxMut=[1], h=0.01, tMax=0.0), 0),           # no sample
])
def test_packed_rows_equal_the_device_rows(cbf, gpu_ok, kw, cap):
    torch = pytest.importorskip("torch")
    job = cbf.make_job(task=cbf.TASK_PEAKS, transientTime=60.0, maxValue=1e4, peakCapacity=cap, **kw)
    peaks, counts = cbf.run_host(job)
    n, width = peaks.shape
    out = torch.zeros(n * width, dtype=torch.float64, device="cuda")
    aux = torch.zeros(n, dtype=torch.int32, device="cuda")
    cbf.run_device(job, out.data_ptr(), aux.data_ptr())
    torch.cuda.synchronize()
    rows = out.cpu().numpy().reshape(n, width)
    assert np.array_equal(counts, aux.cpu().numpy())
    for p in range(n):
        m = min(counts[p], width)
        assert np.array_equal(peaks[p, :m], rows[p, :m]), p
