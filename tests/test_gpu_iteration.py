"""GPU: the one-launch FIM iteration at the edges of its kernels' ranges.

The bit-exact build must equal the oracle bit for bit, with equal work
counters, whatever the patches look like: single-vertex patches, patches in
each block-size class, patches with more than 32 neighbours (the publishing
warp then loops), and steps on both sides of the restart of the stamps (a new
handle's first steps).  The fast build's triangle sweep is held to the FP64
oracle with the bar of the other fast kernels, 1e-3 h, over the same patches.
"""
import numpy as np
import pytest

import lsgb300
import lsoracle
import synth

pytestmark = pytest.mark.gpu

COUNTERS = ("fim_iters", "patch_visits", "check_visits", "nb_vertex_updates", "nb_patches")


def _workload(dim, n, block):
    w = synth.workload("c1" if dim == 2 else "c2", n=n)
    if block > 0:
        w["npart"], w["nparts"] = synth.structured_partition(dim, n + 1, block)
    else:
        # one patch in the middle, every other vertex a patch of its own
        x = w["xyz"][:, :dim]
        own = np.abs(x - 0.5).max(1) > 0.2
        npart = np.zeros(len(x), np.int32)
        npart[own] = 1 + np.arange(own.sum())
        w["npart"], w["nparts"] = npart, int(own.sum()) + 1
    return w


def _oracle(w, nsteps, precision=32):
    ol = lsoracle.OracleLayout(w["dim"], w["xyz"], w["elems"], w["npart"], w["nparts"])
    p = ol.params(update_kind=lsoracle.UPDATE[w["update"]], dt=w["dt"], bandwidth=w["bandwidth"], curv_coeff=1.0,
                  precision=precision)
    return ol.solve(p, w["phi0"], w["vel"], nsteps)


# 2D: blocks of 1 (6 copies) to 20 (880 copies: the 1024-thread class); 3D: 1
# (24 copies) to 4 (672 copies), and the uneven partition of both
CASES = [(2, 13, 1), (2, 24, 9), (2, 24, 12), (2, 45, 15), (2, 43, 20), (2, 24, 0), (3, 7, 1), (3, 9, 2), (3, 11, 4),
         (3, 8, 0)]


@pytest.mark.parametrize("dim,n,block", CASES)
def test_exact_iteration_equals_oracle(dim, n, block):
    w = _workload(dim, n, block)
    nsteps = 6  # the stamps restart after the first few
    ref, nbs, _, ost = _oracle(w, nsteps)
    ls = lsgb300.from_workload(w, bit_exact=True)
    hist, done = ls.solve(nsteps)
    assert done == ost["steps_run"]
    assert np.array_equal(hist.view(np.uint32), ref[: done + 1].view(np.uint32))
    assert np.array_equal(ls.narrowband(w["nparts"]), nbs[-1])
    st = ls.stats()
    for k in COUNTERS:
        assert st[k] == ost[k], k


@pytest.mark.parametrize("dim,n,block", [c for c in CASES if c[0] == 2])
def test_fast_triangles_stay_at_fp64(dim, n, block):
    w = dict(_workload(dim, n, block), update="none")
    ref, _, _, ost = _oracle(w, 2, precision=64)
    hist, done = lsgb300.from_workload(w).solve(2)
    assert done == ost["steps_run"] == 2
    for s in (1, 2):
        band = (np.abs(ref[s]) <= w["bandwidth"]) & (np.abs(hist[s]) <= w["bandwidth"])
        assert band.sum() > 0
        assert np.max(np.abs(hist[s][band] - ref[s][band])) <= 1e-3 * w["h"]
