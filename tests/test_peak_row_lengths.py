"""Which peak rows get small pages (__init__.py: _peak_rows): long ones; short rows of
any number are numpy's zeros, whose large pages cost less there.  Ordinary arrays on
either side of the line.
"""
import numpy as np
import pytest


@pytest.mark.parametrize("n,cap,small_pages", [(3249, 250, False), (600, 3999, False), (600, 4000, True),
                                               (65, 4000, False), (66, 4000, True), (40000, 1000, False)])
def test_row_lengths(cbf, monkeypatch, n, cap, small_pages):
    rows = cbf._peak_rows(n, cap)
    assert rows.shape == (n, cap) and rows.flags.owndata and rows.flags.writeable
    assert not rows[0].any() and not rows[-1].any()
    monkeypatch.setattr(cbf, "_OWN_MAPPING", None)  # what only small pages need
    if small_pages:
        with pytest.raises(TypeError):
            cbf._peak_rows(n, cap)
    else:
        assert not np.any(cbf._peak_rows(n, cap)[:, 0])
