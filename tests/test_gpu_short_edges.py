"""GPU: tetrahedra with edges so short that products of four lengths are
denormal numbers (reference semantics, or a caller's length scale: lengths
are then not brought to about 1).  The distance from a vertex is, in exact
arithmetic, no less than the straight line (linear interpolation of a convex
function lies above it) and no more than the shortest path along edges; FP32
with denormals kept stays within 1e-3 of that down to edges of 3e-11, where a
squared face area keeps about ten bits."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import dijkstra

import lsgb300
import synth

pytestmark = pytest.mark.gpu


def _edge_paths(x, elems, s):
    pairs = np.concatenate([elems[:, [a, b]] for a in range(4) for b in range(a + 1, 4)])
    pairs = np.unique(np.sort(pairs, axis=1), axis=0)
    length = np.linalg.norm(x[pairs[:, 0]] - x[pairs[:, 1]], axis=1)
    g = coo_matrix((length / length.mean(), (pairs[:, 0], pairs[:, 1])), shape=(len(x), len(x)))
    return dijkstra(g.tocsr(), directed=False, indices=s) * length.mean()


@pytest.mark.parametrize("h", [1e-6, 1e-9, 3e-10, 1e-10, 3e-11])
@pytest.mark.parametrize("kw", [dict(ref_compat=True), dict(ref_compat=True, fim_ctas_per_sm=7),
                                dict(ref_compat=True, fim_ctas_per_sm=3), dict(ref_compat=True, block=4),
                                dict(ref_compat=True, flags=lsgb300.PERSISTENT), dict(length_scale=1.0),
                                dict(length_scale=1.0, fim_ctas_per_sm=6), dict(fp64_flagged=True, length_scale=1.0)])
def test_distances_between_straight_lines_and_edge_paths(h, kw):
    kw = dict(kw)
    w = synth.workload("c2", n=8, scale=8 * h)
    w["npart"], w["nparts"] = synth.structured_partition(3, 9, kw.pop("block", 3))
    ls = lsgb300.from_workload(dict(w, update="none"), smallnum=1e-37, **kw)
    x = w["xyz"].astype(np.float64)
    s = 364
    d = ls.eikonal([s], [0.0]).astype(np.float64)
    line = np.linalg.norm(x - x[s], axis=1)
    path = _edge_paths(x, w["elems"], s)
    assert np.all(d >= (1 - 1e-3) * line)
    assert np.all(d <= (1 + 1e-3) * path)


def test_batch_with_one_fine_mesh():
    # one member's length scale makes its lengths short; the others are as alone
    ws = [dict(synth.workload("c2", n=6), update="none"), dict(synth.workload("c2", n=8), update="none")]
    b = lsgb300.LevelSetBatch()
    members = [lsgb300.from_workload(ws[0], setup=False),
               lsgb300.from_workload(ws[1], setup=False, length_scale=1.0 / 8 / 1e-10, smallnum=1e-5)]
    for m in members:
        b.add(m)
    b.setup()
    b.solve(1)
    alone = lsgb300.from_workload(ws[0])
    alone.step(1)
    assert np.array_equal(b.phi(0).view(np.uint32), alone.phi().view(np.uint32))
