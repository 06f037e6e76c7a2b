"""GPU: a step whose FIM loop is abandoned (every wait gives up at its first
check) ends there: the launches behind the abandoned one visit nothing, and
phi and the rest of a run's history stay what they were before the step."""
import ctypes

import numpy as np
import pytest

import lsgb300
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("flags", [0, lsgb300.NO_GRAPH, lsgb300.PERSISTENT, lsgb300.HOST_STAGING])
@pytest.mark.parametrize("kw", [dict(), dict(bit_exact=True), dict(fim_ctas_per_sm=7), dict(inside_iterations=2)])
@pytest.mark.parametrize("update", ["curvature", "none"])
def test_abandoned_step_changes_nothing(flags, kw, update):
    w = dict(synth.workload("c3", n=12), update=update)
    ls = lsgb300.from_workload(w, flags=flags, barrier_wait_limit=-1, **kw)
    hist = np.full((4, ls.nv), 7.0, np.float32)
    done = ctypes.c_int(-1)
    rc = lsgb300.lib().ls_solve(ls._h, 3, hist.ctypes.data_as(ctypes.c_void_p), ctypes.byref(done))
    assert rc == lsgb300.LS_DEVICE_TIMEOUT
    assert np.array_equal(hist[0], w["phi0"]) and np.all(hist[1:] == 7.0)
    assert np.array_equal(ls.phi(), w["phi0"])
    out = np.full_like(w["phi0"], 7.0)
    with pytest.raises(lsgb300.LevelSetError) as e:
        ls.step_host(w["phi0"], out)
    assert e.value.code == lsgb300.LS_DEVICE_TIMEOUT and np.all(out == 7.0)
    assert np.array_equal(ls.phi(), w["phi0"])
    st = ls.stats()
    for k in ("patch_visits", "check_visits", "fim_iters", "nb_patches", "nb_vertex_updates", "sweep_slab_bytes"):
        assert st[k] == 0, k
