"""GPU: ls_solve enqueues each step behind the previous one before it knows
how that one ended.  A run must equal the same steps called one by one -- also
when the interface vanishes in the middle (the step behind it does nothing,
and history rows past the last step stay as the caller left them), when a step
hits the iteration cap, across restarts of the stamps, and with the
persistent FIM loop -- and the handle must go on from there as before."""
import ctypes

import numpy as np
import pytest

import lsgb300
import lsoracle
import synth

pytestmark = pytest.mark.gpu

FLAGS = [0, lsgb300.PERSISTENT, lsgb300.NO_GRAPH, lsgb300.HOST_STAGING]


def _vanishing(n=10, r=0.14, f=2.0):
    w = synth.workload("c3", n=n)
    w["phi0"] = synth.phi_spheres(w["xyz"], [(0.5, 0.5, 0.5)], [r])
    w["dt"] *= f
    return w


def _raw_solve(ls, nsteps, fill):
    hist = np.full((nsteps + 1, ls.nv), fill, np.float32)
    done = ctypes.c_int(-1)
    rc = lsgb300.lib().ls_solve(ls._h, nsteps, hist.ctypes.data_as(ctypes.c_void_p), ctypes.byref(done))
    return rc, hist, done.value


@pytest.mark.parametrize("flags", FLAGS)
@pytest.mark.parametrize("extra", [0, 1, 7])
def test_run_ends_where_the_interface_vanishes(flags, extra):
    w = _vanishing()
    ol = lsoracle.OracleLayout(3, w["xyz"], w["elems"], w["npart"], w["nparts"])
    p = ol.params(update_kind=1, dt=w["dt"], bandwidth=w["bandwidth"], curv_coeff=1.0)
    ref, _, _, ost = ol.solve(p, w["phi0"], w["vel"], 40)
    n = ost["steps_run"]
    assert 2 < n < 40
    ls = lsgb300.from_workload(w, bit_exact=True, flags=flags)
    rc, hist, done = _raw_solve(ls, n + extra, 7.0)
    assert rc == 0 and done == n
    assert np.array_equal(hist[: n + 1].view(np.uint32), ref[: n + 1].view(np.uint32))
    assert np.all(hist[n + 1 :] == 7.0)
    st = ls.stats()
    assert st["steps_run"] == n
    # a run from a new phi on the same handle
    ls.set_phi(w["phi0"])
    h2, d2 = ls.solve(3)
    assert d2 == 3 and np.array_equal(h2.view(np.uint32), ref[:4].view(np.uint32))


@pytest.mark.parametrize("flags", FLAGS)
def test_run_equals_single_steps(flags):
    w = synth.workload("c2", n=9)
    a = lsgb300.from_workload(w, flags=flags)
    b = lsgb300.from_workload(w, flags=flags)
    ha, da = a.solve(9)  # the stamps of a new handle restart within these
    hb = [b.phi()]
    for _ in range(9):
        assert b.step(1) == 1
        hb.append(b.phi())
    assert da == 9 and np.array_equal(ha.view(np.uint32), np.array(hb).view(np.uint32))
    sa, sb = a.stats(), b.stats()
    for k in ("steps_run", "fim_iters", "patch_visits", "check_visits", "nb_vertex_updates", "nb_patches",
              "kernel_launches"):
        assert sa[k] == sb[k], k


@pytest.mark.parametrize("flags", FLAGS[:3])
def test_run_ends_at_the_iteration_cap(flags):
    w = synth.workload("c3", n=12)
    ls = lsgb300.from_workload(w, max_fim_iters=2, graph_chunk=2, flags=flags)
    rc, hist, _ = _raw_solve(ls, 5, 7.0)
    assert rc == lsgb300.LS_DEVICE_TIMEOUT
    assert np.array_equal(hist[0], w["phi0"]) and np.all(hist[2:] == 7.0)
    p = ls.get_params()
    p.max_fim_iters = 0
    ls.set_params(p)
    ls.setup()
    ls.set_phi(w["phi0"])
    h1, d1 = ls.solve(3)
    h0, d0 = lsgb300.from_workload(w, flags=flags).solve(3)
    assert d0 == d1 == 3 and np.array_equal(h0.view(np.uint32), h1.view(np.uint32))
