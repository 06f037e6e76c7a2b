"""GPU: handles side by side.  The dynamic shared memory that a kernel may
have is an attribute of the function, shared by every handle of the process:
setting up a mesh of small patches must leave an earlier handle of large
patches able to launch everything that it launches directly (not through its
step graph)."""
import numpy as np
import pytest

import lsgb300
import synth

pytestmark = pytest.mark.gpu


def _large(n=9, block=3, **kw):
    w = synth.workload("c2", n=n)
    w["npart"], w["nparts"] = synth.structured_partition(3, n + 1, block)
    return w, lsgb300.from_workload(w, **kw)


def _small(**kw):
    w = synth.workload("c2", n=6)
    w["npart"], w["nparts"] = synth.structured_partition(3, 7, 1)
    ls = lsgb300.from_workload(w, **kw)
    ls.step(1)
    return ls


def _results(w, ls):
    out = [ls.eikonal([3, 77], [0.0, 0.01])]
    ls.set_phi(w["phi0"])
    assert ls.step(2) == 2
    out.append(ls.phi())
    ls.set_phi(w["phi0"])
    ls.set_profile(True)
    assert ls.step(1) == 1
    ls.set_profile(False)
    out.append(ls.phi())
    return out


# the two-copies sweep (5, 7) and the one-copy sweeps, both builds, the
# precision form, the persistent loop, and the reference's curvature update
# on patches of more than 384 copies
@pytest.mark.parametrize("kw", [dict(), dict(fim_ctas_per_sm=7), dict(fim_ctas_per_sm=3), dict(fim_ctas_per_sm=2),
                                dict(bit_exact=True), dict(bit_exact=True, ref_compat=True), dict(fp64_flagged=True),
                                dict(flags=lsgb300.PERSISTENT), dict(flags=lsgb300.NO_GRAPH),
                                dict(block=4), dict(block=4, n=11, bit_exact=True, ref_compat=True, update_kind=1)])
def test_large_patches_after_a_setup_of_small_ones(kw):
    extra = {k: v for k, v in kw.items() if k not in ("n", "block", "update_kind")}
    w, ls = _large(kw.get("n", 9), kw.get("block", 3), **extra)
    if "update_kind" in kw:
        p = ls.get_params()
        p.update_kind, p.time_step = kw["update_kind"], 0.5 * w["h"] ** 2
        ls.set_params(p)
        ls.setup()
    before = _results(w, ls)
    other = _small(**extra)
    for a, b in zip(before, _results(w, ls)):
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    assert other.step(1) == 1
