"""GPU: several inside iterations of the update per step (the reference's
insideIterations_), each reading the previous one's result: the bit-exact
build against the oracle, bit for bit, for each update kernel."""
import numpy as np
import pytest

import lsgb300
import lsoracle
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("name,n,update,ref", [("c1", 16, "advect", False), ("c1", 20, "curvature", False),
                                               ("c2", 9, "advect", True), ("c3", 10, "curvature", False),
                                               ("c3", 10, "curvature", True)])
@pytest.mark.parametrize("inside", [1, 2, 3])
def test_inside_iterations_equal_oracle(name, n, update, ref, inside):
    w = dict(synth.workload(name, n=n), update=update)
    w["dt"] /= inside
    ol = lsoracle.OracleLayout(w["dim"], w["xyz"], w["elems"], w["npart"], w["nparts"])
    p = ol.params(update_kind=lsoracle.UPDATE[update], dt=w["dt"], bandwidth=w["bandwidth"], curv_coeff=1.0,
                  ref_compat=1 if ref else 0)
    p.inside_niter = inside
    want, _, _, ost = ol.solve(p, w["phi0"], w["vel"], 3)
    ls = lsgb300.from_workload(w, bit_exact=True, ref_compat=ref, inside_iterations=inside)
    hist, done = ls.solve(3)
    assert done == ost["steps_run"]
    assert np.array_equal(hist.view(np.uint32), want[: done + 1].view(np.uint32))
