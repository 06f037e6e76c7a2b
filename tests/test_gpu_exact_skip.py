"""GPU: the bit-exact build leaves out the tet solves that cannot lower their
target; what it leaves out must not change a bit.  Against the oracle on
meshes from well shaped to nearly flat (one axis squeezed, where the bound
switches itself off), with large jitter, in both semantics."""
import numpy as np
import pytest

import lsgb300
import lsoracle
import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("squeeze", [1.0, 0.3, 0.05, 0.01, 1e-3])
@pytest.mark.parametrize("jitter,ref,update", [(0.15, False, "none"), (0.4, False, "none"), (0.3, True, "none"),
                                               (0.3, False, "advect")])
def test_left_out_solves_change_nothing(squeeze, jitter, ref, update):
    n = 10
    xyz, el = synth.cube_mesh(n, jitter, 5)
    xyz = (xyz * np.array([1, 1, squeeze])).astype(np.float32)
    npart, nparts = synth.structured_partition(3, n + 1, 3)
    phi = (np.sqrt(((xyz - np.array([0.4, 0.5, 0.5 * squeeze])) ** 2).sum(1)) - 0.27).astype(np.float32)
    vel = synth.velocity_rotation(xyz, el, 2.0)
    dt, bw = 0.01 * squeeze, 0.45
    ol = lsoracle.OracleLayout(3, xyz, el, npart, nparts)
    p = ol.params(update_kind=lsoracle.UPDATE[update], dt=dt, bandwidth=bw, curv_coeff=1.0, ref_compat=1 if ref else 0)
    want, nbs, _, ost = ol.solve(p, phi, vel, 3)
    kind = {"advect": lsgb300.UPDATE_ADVECT, "none": lsgb300.UPDATE_NONE}[update]
    flags = lsgb300.BITEXACT | (lsgb300.REF_COMPAT if ref else 0)
    ls = lsgb300.LevelSet(False, lsgb300.default_params(time_step=dt, bandwidth=bw, update_kind=kind, flags=flags))
    ls.set_mesh(xyz, el)
    ls.set_partition(npart, nparts)
    ls.set_phi(phi)
    ls.set_velocity(vel)
    ls.setup()
    hist, done = ls.solve(3)
    assert done == ost["steps_run"]
    assert np.array_equal(hist.view(np.uint32), want[: done + 1].view(np.uint32))
    st = ls.stats()
    for k in ("fim_iters", "patch_visits", "check_visits"):
        assert st[k] == ost[k], k
