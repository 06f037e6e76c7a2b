"""GPU: the paths that stage host arrays, which a GPU with access to pageable
host memory takes only when asked to, give the same bits as the direct ones;
and training whose rows arrive in pieces of several batches equals training
batch by batch."""
import numpy as np
import pytest

import lsgb300
import synth

pytestmark = pytest.mark.gpu


def _data(n, seed):
    rng = np.random.default_rng(seed)
    x = rng.normal(0, 1, (n, 128)).astype(np.float32)
    return x, (0.5 * x[:, 3] + 0.25 * np.tanh(x[:, 7])).astype(np.float32)


def _network_results(n, batch, staging):
    m = lsgb300.MLP(5)
    m.set_host_staging(staging)
    x, t = _data(n, n)
    out = [m.predict(x), *m.gradients(x, t)]
    out += [m.train(x, t, epochs=2, batch=batch), m.params(), m.predict(x[: n // 2 + 1])]
    m.set_host_staging(not staging)  # the other way on the same network
    out += [m.predict(x), m.train(x, t, epochs=1, batch=batch), m.params()]
    return out


# one batch, eight (one a piece), nine (two a piece), sixteen, seventeen, with
# a short last batch or piece
@pytest.mark.parametrize("n,batch", [(1, 64), (500, 512), (1024, 128), (1025, 128), (2048, 128), (2060, 128), (5000, 97)])
def test_network_staging_gives_the_same_bits(n, batch):
    a, b = _network_results(n, batch, False), _network_results(n, batch, True)
    assert a[3] == b[3]
    for u, v in zip(a, b):
        assert np.array_equal(np.asarray(u, np.float32).view(np.uint32), np.asarray(v, np.float32).view(np.uint32))


@pytest.mark.parametrize("staging", [False, True])
@pytest.mark.parametrize("n,batch", [(1025, 128), (2060, 128), (5000, 97), (3000, 300)])
def test_training_in_pieces_equals_batch_by_batch(n, batch, staging):
    x, t = _data(n, 2)
    whole, single = lsgb300.MLP(4), lsgb300.MLP(4)
    whole.set_host_staging(staging)
    whole.train(x, t, epochs=1, batch=batch)
    for i in range(0, n, batch):
        single.train(x[i:i + batch], t[i:i + batch], epochs=1, batch=batch)
    assert np.array_equal(whole.params().view(np.uint32), single.params().view(np.uint32))


def test_staged_batch_gives_the_same_bits():
    ws = synth.workload_batch(seed=3, nmesh=5, nmin=6, nmax=12)
    out = []
    for flags in (0, lsgb300.HOST_STAGING):
        b = lsgb300.LevelSetBatch()
        members = [lsgb300.from_workload(w, setup=False, flags=flags) for w in ws]
        for m in members:
            b.add(m)
        b.setup()
        out.append([b.phi(i) for i in range(5)])
        b.solve(2)
        out.append([b.phi(i) for i in (4, 0, 2, 1, 3)])
    for a, c in zip(out[:2], out[2:]):
        for u, v in zip(a, c):
            assert np.array_equal(u.view(np.uint32), v.view(np.uint32))
    for w, u in zip(ws, out[0]):
        assert np.array_equal(u, w["phi0"])
