"""GPU: max_fim_iters is the number of iterations that a step may take: a step
of exactly that many is done, one more is LS_DEVICE_TIMEOUT -- in the
persistent loop for any number, in the step graph and launch by launch in
whole loop bodies -- also when nothing follows the last iteration."""
import numpy as np
import pytest

import lsgb300
import synth

pytestmark = pytest.mark.gpu

WORKLOADS = [("c3", 8), ("c3", 12), ("c3", 16), ("c2", 8), ("c2", 12), ("c1", 16), ("c1", 24), ("c1", 40)]


@pytest.mark.parametrize("name,n", WORKLOADS)
@pytest.mark.parametrize("kw", [dict(), dict(bit_exact=True)])
@pytest.mark.parametrize("flags", [lsgb300.PERSISTENT, 0, lsgb300.NO_GRAPH])
def test_the_cap_is_exact(name, n, kw, flags):
    w = synth.workload(name, n=n)
    free = lsgb300.from_workload(w, flags=flags, **kw)
    free.step(1)
    iters = free.stats()["fim_iters"]
    assert iters > 2
    for cap in (iters - 1, iters):
        # bodies of two iterations: the cap counts up to the next even number
        allowed = cap if flags == lsgb300.PERSISTENT else cap + cap % 2
        ls = lsgb300.from_workload(w, flags=flags, max_fim_iters=cap, graph_chunk=2, **kw)
        if iters <= allowed:
            assert ls.step(1) == 1
            assert np.array_equal(ls.phi().view(np.uint32), free.phi().view(np.uint32))
        else:
            with pytest.raises(lsgb300.LevelSetError) as e:
                ls.step(1)
            assert e.value.code == lsgb300.LS_DEVICE_TIMEOUT


def test_each_support_round_has_the_whole_cap():
    # an untrained network's warm start takes several FIM loops per step: the
    # cap is each loop's, not their sum's
    w = synth.workload("c3", n=16)
    net = lsgb300.MLP(99)

    def run(cap):
        ls = lsgb300.from_workload(w, graph_chunk=2, max_fim_iters=cap)
        ls.set_learned(net)
        assert ls.step(1) == 1  # the first step has no narrowband to warm
        ls.reset_stats()
        assert ls.step(1) == 1
        return ls.phi(), ls.stats()

    phi, st = run(0)
    assert st["support_rounds"] > 2 and st["fim_iters"] > 16
    plain = lsgb300.from_workload(w)
    plain.step(1)
    least = plain.stats()["fim_iters"] + 2  # what the cold first step needs
    cap = max(least + least % 2, (st["fim_iters"] // 2 + 1) // 2 * 2)
    assert cap < st["fim_iters"] - 1
    phi2, st2 = run(cap)
    # (the support checks read values that other checks reset: the rounds, and
    # values within the check's tolerance, can differ from run to run)
    assert st2["support_rounds"] > 2
    band = np.abs(phi) <= w["bandwidth"]
    assert np.max(np.abs(phi - phi2)[band]) <= 1e-2 * w["h"]
