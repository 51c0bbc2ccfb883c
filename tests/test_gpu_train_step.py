"""The training step's two kernels (csrc/mlp_step.cuh) at the edges of their tiles.

A batch of up to as many 128-row tiles as clusters are resident goes through the
cluster kernel, a larger one through the one-CTA kernel; the weight gradients split
the rows into slices that need not end on a tile.  The CPU oracle rounds to BF16 at
the same places, so what is left is the order of FP32 sums: the bounds are those of
the gradient test of the network (1e-4 of the loss, 1e-2 of a parameter block).
"""
import numpy as np
import pytest

import mlp_oracle as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 127, 128, 129, 4097, 5000])
def test_gradients_at_tile_edges(cbf, gpu_ok, n):
    """n = 5000: more tiles than clusters, weight-gradient slices of 2.5 tiles."""
    rng = np.random.default_rng(n)
    net = cbf.Mlp(5000, seed=9)
    big = rng.uniform(-1, 1, (5000, 4)).astype(np.float32)
    net.forward_backward(big, np.zeros(5000, np.float32), np.zeros(5000, np.int32), 0.5)  # other rows before
    p = net.get_params()
    x = rng.uniform(-1, 1, (n, 4)).astype(np.float32)
    yl = rng.normal(size=n).astype(np.float32)
    yc = rng.integers(0, 16, n).astype(np.int32)
    loss, g, out = net.forward_backward(x, yl, yc, 0.5)
    wl, wg, wout = M.forward_backward(p.astype(np.float64), x, yl, yc, 0.5, bf16_round=True, scale=1.0)
    assert abs(loss - wl) <= 1e-4 * abs(wl)
    assert np.linalg.norm(out - wout) < 1e-3 * np.linalg.norm(wout)
    for name, (o, shape) in M.offsets().items():
        k = int(np.prod(shape))
        err = np.linalg.norm(g[o:o + k] - wg[o:o + k]) / max(np.linalg.norm(wg[o:o + k]), 1e-30)
        assert err < 1e-2, (name, err)
    net.close()
