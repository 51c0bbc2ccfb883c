"""The peak rows that the host entry points return (__init__.py: _peak_rows) are
arrays like any other: zeros, private to the process, owning their data, and too many
of them are a MemoryError.  On either side of the sizes where the allocation changes.
"""
import os

import numpy as np
import pytest


@pytest.mark.parametrize("n,cap", [(1, 1), (3, 70000), (4, 65536), (61, 12500), (1000, 25000)])
def test_rows_are_ordinary_arrays(cbf, n, cap):
    for _ in range(3):  # a freed block of that size before the next one
        rows = cbf._peak_rows(n, cap)
        assert rows.shape == (n, cap) and rows.dtype == np.float64 and rows.flags.c_contiguous
        assert rows.flags.owndata and rows.flags.writeable and rows.base is None
        assert not rows[0].any() and not rows[-1].any() and not rows[:, -1].any()
        rows[:, 0] = rows[-1, -1] = 5.0
        assert rows.sum() == 5.0 * (n + (cap > 1))
        rows.resize((n, cap + 1))
        assert rows.shape == (n, cap + 1)
        del rows


@pytest.mark.parametrize("n,cap", [(4, 1000), (61, 12500), (1000, 25000)])
def test_a_forked_child_writes_its_own_copy(cbf, n, cap):
    rows = cbf._peak_rows(n, cap)
    rows[0, 0] = 1.0
    pid = os.fork()
    if pid == 0:
        rows[0, 0] = rows[n - 1, cap - 1] = 7.0
        os._exit(0 if rows[n - 1, cap - 1] == 7.0 else 1)
    assert os.waitpid(pid, 0)[1] == 0
    assert rows[0, 0] == 1.0 and rows[n - 1, cap - 1] == 0.0


def test_rows_that_no_memory_holds(cbf):
    with pytest.raises(MemoryError):
        cbf._peak_rows(1 << 20, 1 << 37)
