"""GPU: the network kernels at the edges of their tiles -- one sample, one
short of and one past a 128-sample tile and a whole wave of tiles -- and host
arrays that start off the 16-byte boundary of the conversion's wide loads.
Gradients and outputs against the numpy restatement with the bars of
test_mlp.py (BF16 operands: 3e-2 relative norm, 2e-2 of the largest output);
training must not depend on where the host arrays start."""
import numpy as np
import pytest

import lsgb300
import mlp_ref

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, (n, 128)).astype(np.float32)
    return x, (0.5 * x[:, 3] + 0.25 * np.tanh(x[:, 7])).astype(np.float32)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 152 * 128 + 1])
def test_tile_edges(n):
    m = lsgb300.MLP(0)
    p = mlp_ref.init_params(n)
    m.set_params(p)
    x, t = _data(n, n)
    y, (yr, _) = m.predict(x), mlp_ref.forward(p, x)
    assert np.abs(y - yr).max() <= 2e-2 * (np.abs(yr).max() + 1e-3)
    g, loss = m.gradients(x, t)
    gr, lr = mlp_ref.gradients(p, x, t)
    assert abs(loss - lr) <= 1e-2 * lr + 1e-6
    assert np.linalg.norm(g - gr) <= 3e-2 * np.linalg.norm(gr)


def test_unaligned_host_arrays_and_repeats():
    n = 1000
    x, t = _data(n, 3)
    raw = np.zeros(n * 128 + 4, np.float32)
    out = []
    for offset in (0, 1, 3):
        xo = raw[offset:offset + n * 128]
        xo[:] = x.ravel()
        m = lsgb300.MLP(7)
        p0 = m.params()
        loss = m.train(xo.reshape(n, 128), t, epochs=2, batch=300)
        y = m.predict(xo.reshape(n, 128))
        out.append((m.params(), y, loss))
        # from the same parameters again: the optimiser starts over
        m.set_params(p0)
        assert m.train(x, t, epochs=2, batch=300) == loss
        assert np.array_equal(m.params(), out[-1][0])
    for p, y, loss in out[1:]:
        assert np.array_equal(p, out[0][0]) and np.array_equal(y, out[0][1]) and loss == out[0][2]
