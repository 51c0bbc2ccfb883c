"""Training on drawn rows through both step kernels (csrc/mlp_step.cuh): 4096 rows go
through the cluster kernel, 8192 and 20 000 through the one-CTA kernel, which draws
the rows a second time for their labels.  The rows of a step follow from the seed and
the step's number alone, so the oracle can take the same ones.

Bounds: the loss 1e-4 and the gradient 1e-2 of a parameter block's norm, as for given
rows.  The first Adam step moves every parameter by lr g / (|g| + 1e-8), so where the
oracle's |g| is above twice that bound the step's sign is known.
"""
import numpy as np
import pytest

import mlp_oracle as M

pytestmark = pytest.mark.gpu

ROWS, SEED, LR = 30011, 77, 1e-3


def _mix64(z):
    z = z + np.uint64(0x9E3779B97F4A7C15)
    z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
    z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
    return z ^ (z >> np.uint64(31))


def _drawn(step, batch):
    r = np.arange(batch, dtype=np.uint64)
    with np.errstate(over="ignore"):
        h = _mix64(np.uint64(SEED) ^ _mix64(np.uint64(step) * np.uint64(0x100000001B3) + r))
    return (h % np.uint64(ROWS)).astype(np.int64)


@pytest.mark.parametrize("batch", [4096, 8192, 20000])
def test_steps_on_drawn_rows(cbf, gpu_ok, batch):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(5)
    x = rng.uniform(-1, 1, (ROWS, 4)).astype(np.float32)
    yl = rng.normal(size=ROWS).astype(np.float32)
    yc = rng.integers(0, 16, ROWS).astype(np.int32)
    d = [torch.from_numpy(a).cuda() for a in (x, yl, yc)]
    stream = torch.cuda.Stream()
    net = cbf.Mlp(batch, seed=SEED)
    torch.cuda.synchronize()

    def train(steps, lr):
        return net.train(*(a.data_ptr() for a in d), ROWS, steps, lr, w_lle=0.5, stream=stream.cuda_stream, losses=True)

    def oracle(p, step):
        i = _drawn(step, batch)
        return M.forward_backward(p.astype(np.float64), x[i], yl[i], yc[i], 0.5, bf16_round=True, scale=1.0)[:2]

    p0 = net.get_params()
    losses = train(1, LR)
    p1 = net.get_params()
    loss, grad = oracle(p0, 0)
    assert abs(losses[0] - loss) <= 1e-4 * abs(loss)
    for name, (o, shape) in M.offsets().items():
        k = int(np.prod(shape))
        g = grad[o:o + k]
        sure = np.abs(g) > 2e-2 * np.linalg.norm(g)
        assert sure.any(), name
        assert np.array_equal(np.sign(p0[o:o + k] - p1[o:o + k])[sure], np.sign(g)[sure]), name
    # with lr 0 the parameters stay: the replayed graph draws other rows each step
    losses = train(3, 0.0)
    assert np.array_equal(net.get_params(), p1)
    for step in (1, 2, 3):
        loss, _ = oracle(p1, step)
        assert abs(losses[step - 1] - loss) <= 1e-4 * abs(loss), step
    net.close()
