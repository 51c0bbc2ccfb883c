"""A trajectory of no samples through run_host (__init__.py): the library's rows have
one slot at least (csrc/capi.cu: lower_job), so the buffer it fills must too.  The
library itself is replaced by one that looks at the buffer: no device is needed.
"""
import ctypes as C

import numpy as np
import pytest


class _Library:
    """The library, except that cbf_run_host only notes its output buffer."""

    def __init__(self, lib):
        self._lib = lib

    def __getattr__(self, name):
        return getattr(self._lib, name)

    def cbf_run_host(self, job, out, aux):
        self.out = out.value
        return 0


@pytest.mark.parametrize("record", [0.0, 0.005, 0.01, 0.05])
def test_rows_hold_what_the_library_writes(cbf, monkeypatch, record):
    fake = _Library(cbf.lib())
    monkeypatch.setattr(cbf, "lib", lambda: fake)
    job = cbf.make_job(task=cbf.TASK_TRAJECTORY, system="rossler", nPts=7, ranges=[0.1, 0.3], idxMut=[1],
                       ic=[0.1, 0.1, 0.1], values=[0.5, 0.2, 0.2, 5.7], h=0.01, tMax=record, maxValue=1e4)
    out, aux = cbf.run_host(job)
    samples = fake.cbf_record_length(C.byref(job))
    assert out.shape == (7, samples) and aux.shape == (7,)
    rows = out if out.base is None else out.base
    assert rows.ctypes.data == fake.out and rows.nbytes == 7 * max(samples, 1) * 8
    assert not np.any(rows)
