"""GPU: the one-copy FIM kernel counts the work that it runs: a candidate whose
check finds it unconverged goes on to be visited from that same sweep, which
counts once in the slab bytes and in the FP64 repeats.

Two tetrahedra on either side of an equilateral triangle 1, 2, 3 (side 1),
apexes 0 and 4 at unit height; patches A = {0}, B = {1, 2, 3}, C = {4}; a seed
at 0, one sweep per visit, every conditioning check flagged (threshold 1e30).
With d = |01| = |02| = |03|:
  1  A, B visited: the faces of the targets hold one finite value, no edge of
     two: no repeats.  1, 2, 3 become d
  2  B visited: targets 1, 2, 3 of the lower tet (their heights over the faces
     with 0 are below d) and 4 of the upper: 4 repeats; nothing lower
  3  A checked: 1, 2, 3 as ghosts: 3 repeats.  C checked: target 4: 1 repeat;
     it drops to d + 1, so C is visited by this sweep
  4  C visited: 4 again (d + 0.999 is below its value): 1 repeat
  5  B checked: as in 2: 4 repeats
"""
import numpy as np
import pytest

import lsgb300

pytestmark = pytest.mark.gpu


def _two_tets(**kw):
    c = np.sqrt(3) / 6
    xyz = np.array([[0.5, c, -1], [0, 0, 0], [1, 0, 0], [0.5, np.sqrt(3) / 2, 0], [0.5, c, 1]], np.float32)
    ls = lsgb300.LevelSet(False, lsgb300.default_params(update_kind=lsgb300.UPDATE_NONE, fim_sweeps=1, **kw))
    ls.set_mesh(xyz, np.array([[0, 1, 2, 3], [4, 1, 3, 2]], np.int32))
    ls.set_partition([0, 1, 1, 1, 2], 3)
    ls.set_phi(np.ones(5, np.float32))
    ls.setup()
    return ls


@pytest.mark.parametrize("flags", [0, lsgb300.FP64_FLAGGED])
def test_a_check_that_becomes_a_visit_counts_once(flags):
    ls = _two_tets(flags=lsgb300.BITEXACT | flags, fim_ctas_per_sm=3, fp64_threshold=1e30)
    ls.eikonal([0], [0.0])
    st = ls.stats()
    assert st["patch_visits"] == 5 and st["check_visits"] == 3
    # bytes of a patch: 9 per owned vertex, 8 per ghost, 32 per copy, 24; a
    # check that stays one writes no values (4 per owned vertex)
    a, b, c = (9 * v + 8 * g + 32 * e + 24 for v, g, e in ((1, 3, 1), (3, 2, 2), (1, 3, 1)))
    assert st["sweep_slab_bytes"] == a + b + b + (a - 4) + c + c + (b - 12)
    assert st["flagged_copies"] == (4 + 3 + 1 + 1 + 4 if flags else 0)
